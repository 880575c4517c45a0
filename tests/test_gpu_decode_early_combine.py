"""The decode combine is launched while the split grid still runs and waits for its end before it reads
a partial: back-to-back calls on one stream with other inputs and lengths, more batch entries than the
in-kernel tile table holds, and a captured graph give what single calls give."""
import pytest
import torch

from attentionfuse_b200.runtime.flash_decode import run_flash_decode
from oracle import attention_oracle as orc
from tests._util import assert_close, qkv

pytestmark = pytest.mark.gpu
DEV = "cuda"


def decode(q, k, v, lens, out):
    return run_flash_decode(None, q, k, v, q.shape[-1] ** -0.5, 0, k.shape[1], out, kv_lens=lens)


@pytest.mark.parametrize("B,L", [(1, 300), (5, 1000), (600, 260)])
def test_back_to_back_calls(B, L):
    Hq, Hkv, D, dtype = 8, 2, 64, torch.bfloat16
    calls = []
    for i in range(4):
        Q, K, V = qkv(8100 + 10 * i, B, Hq, Hkv, 1, L, D, dtype)
        lens = torch.tensor([(L - 37 * b - i) % L for b in range(B)], dtype=torch.int32)
        calls.append((Q, K, V, lens))
    dev = [tuple(t.to(DEV) for t in c) for c in calls]
    outs = [torch.full_like(d[0], float("nan")) for d in dev]
    for d, o in zip(dev, outs):
        decode(*d, o)
    for (Q, K, V, lens), o in zip(calls, outs):
        assert_close(o, orc.attention(Q, K, V, kv_lens=lens), dtype, what=f"back to back B{B} L{L}")


def test_graph_replay_sees_new_inputs():
    B, Hq, Hkv, L, D, dtype = 3, 16, 4, 2000, 128, torch.float16
    Q, K, V = qkv(8200, B, Hq, Hkv, 1, L, D, dtype)
    lens = torch.tensor([2000, 1, 1111], dtype=torch.int32)
    q, k, v, ln = Q.to(DEV), K.to(DEV), V.to(DEV), lens.to(DEV)
    out = torch.empty_like(q)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        decode(q, k, v, ln, out)
        side.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=side):
            decode(q, k, v, ln, out)
    for n in (2000, 777):
        ln.copy_(torch.tensor([n, 5, n // 2], dtype=torch.int32))
        out.zero_()
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        assert_close(out, orc.attention(Q, K, V, kv_lens=torch.tensor([n, 5, n // 2])), dtype, what="graph replay")
