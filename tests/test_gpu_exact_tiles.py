"""The exact (FFMA) forward kernel at the edges of its tiles: 32 query rows per CTA, 64-key tiles that
two groups of threads take in turn (one group above head_dim 128), 16-byte and element-wise row
access.  Against the CPU oracle in 64 bits: fp32 sums of at most 400 terms of order one stay within
1e-5 (a few hundred ulps of 6e-8 bound the worst case, one hundredth of that is typical)."""
import pytest
import torch

import attentionfuse_b200 as af
from attentionfuse_b200.runtime.dispatch import _alibi_slopes
from oracle import attention_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda"
H = 3


def graph(mask, alibi, rope, relu=False):
    def fn(Q, K, V):
        s = af.rope(Q, K) if rope else af.scaled_dot_product(Q, K)
        s = af.alibi(s, H) if alibi else s
        s = af.causal(s) if mask == "causal" else af.sliding_window(s, 70) if mask == "window" else s
        return (af.relu_attention(s) if relu else af.softmax(s)) @ V
    return af.attention(fn)


@pytest.mark.parametrize("N", [1, 31, 33, 64, 65, 128, 129, 193, 400])
@pytest.mark.parametrize("D", [64, 60, 62, 24, 128, 100, 256, 130])
@pytest.mark.parametrize("variant", ["none", "causal", "window", "causal_alibi_rope"])
def test_tiles(N, D, variant):
    mask = variant.split("_")[0]
    extra = "alibi" in variant
    q, k, v = (orc.randn(7000 + N + D + i, (2, H, N, D), torch.float32) for i in range(3))
    kw, okw = {}, {}
    if extra:
        cos, sin = orc.build_rope_cache(N, D, 10000.0, torch.float32)
        kw, okw = dict(cos=cos.to(DEV), sin=sin.to(DEV)), dict(cos=cos, sin=sin, slopes=_alibi_slopes(H, "cpu", "torch.float32"))
    got = graph(mask, extra, extra)(q.to(DEV), k.to(DEV), v.to(DEV), **kw).cpu()
    want = orc.attention(q, k, v, causal=mask == "causal", window=70 if mask == "window" else None, dtype=torch.float64, **okw)
    assert orc.max_abs(got, want) < 1e-5


@pytest.mark.parametrize("layout", ["rows", "offset", "inner"])
def test_strided_and_unaligned_rows_agree(layout):
    """(B, N, H, D) storage keeps the 16-byte path; a base that is 4 bytes off, or an inner stride of
    two, takes the element-wise one."""
    B, N, D = 2, 100, 64
    ts = [orc.randn(7100 + i, (B, H, N, D), torch.float32) for i in range(3)]
    if layout == "rows":
        dev = [t.to(DEV).transpose(1, 2).contiguous().transpose(1, 2) for t in ts]
    elif layout == "offset":
        dev = [torch.zeros(t.numel() + 1, device=DEV)[1:].view(t.shape).copy_(t) for t in ts]
    else:
        dev = [torch.zeros(*t.shape, 2, device=DEV)[..., 0].copy_(t) for t in ts]
    got = graph("causal", False, False)(*dev).cpu()
    assert orc.max_abs(got, orc.attention(*ts, causal=True, dtype=torch.float64)) < 1e-5


def test_relu_merges_both_groups_without_a_maximum():
    ts = [orc.randn(7200 + i, (1, H, 200, 64), torch.float32) for i in range(3)]
    got = graph("none", False, False, relu=True)(*(t.to(DEV) for t in ts)).cpu()
    assert orc.max_abs(got, orc.attention(*ts, relu=True, dtype=torch.float64)) < 1e-5
