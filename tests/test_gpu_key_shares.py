"""Forward problems with fewer query tiles than SMs against a long key axis deal the keys of a tile out
to several items and merge their partials (head_dim 128, calls that keep no log-sum-exp).  Against
the CPU oracle, and against the same call kept whole (one head per CTA, no workspace)."""
import ctypes as C

import pytest
import torch

import attentionfuse_b200 as af
from attentionfuse_b200.runtime import _lib
from attentionfuse_b200.runtime.dispatch import _alibi_slopes, fill_problem
from oracle import attention_oracle as orc
from tests._util import assert_close, qkv

pytestmark = pytest.mark.gpu
DEV, D = "cuda", 128
MASKS = {"none": 0, "causal": 1, "window": 2}


def call(q, k, v, mask, off, slopes, workspace, window=700):
    """af_fwd with or without the workspace it asks for; returns (output, launches, bytes asked for)."""
    lib, params, out = _lib.load(), _lib.AfFwdParams(), torch.full_like(q, float("nan"))
    fill_problem(params.p, q, k, v, sm_scale=D ** -0.5, mask_kind=MASKS[mask], window=window, bias_kind=1 if slopes is not None else 0,
                 slopes=slopes, q_offset=off)
    params.o, params.o_stride = out.data_ptr(), _lib.strides(out)
    need = int(lib.af_fwd_workspace_bytes(C.byref(params)))
    ws = torch.full((max(need, 1),), 0xff, dtype=torch.uint8, device=DEV)      # NaN in every word
    if workspace:
        params.workspace, params.workspace_bytes = ws.data_ptr(), need
    before = _lib.launch_count()
    _lib.check(lib.af_fwd(C.byref(params), _lib.current_stream(q.device)), "af_fwd")
    return out, _lib.launch_count() - before, need


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("mask,alibi", [("none", False), ("causal", False), ("causal", True), ("window", False)])
@pytest.mark.parametrize("shape", [(1, 8, 2, 1, 4097), (1, 4, 1, 64, 5000), (2, 6, 3, 130, 3000), (1, 8, 2, 250, 4011)],
                         ids=lambda s: "x".join(map(str, s)))
def test_shares_match_oracle_and_whole_rows(shape, mask, alibi, dtype):
    B, Hq, Hkv, N_q, N_kv = shape
    off = N_kv - N_q - 5
    Q, K, V = qkv(7300 + N_q, B, Hq, Hkv, N_q, N_kv, D, dtype)
    q, k, v = Q.transpose(1, 2).contiguous().to(DEV).transpose(1, 2), K.to(DEV), V.to(DEV)    # (B, N, H, D) storage
    slopes = _alibi_slopes(Hq, DEV, str(dtype)) if alibi else None
    got, launches, need = call(q, k, v, mask, off, slopes, True)
    whole, one, _ = call(q, k, v, mask, off, slopes, False)
    assert one == 1
    if mask != "window":                       # this one leaves too few tiles to share: see below
        assert launches == 2 and need > 0
    want = orc.attention(Q, K, V, causal=mask == "causal", window=700 if mask == "window" else None, q_offset=off,
                         slopes=None if slopes is None else slopes.cpu(),
                         **(dict(q_positions=torch.full((B,), off)) if N_q == 1 else {}))
    assert_close(got, want, dtype, what=f"key shares {mask} {shape}")
    assert_close(whole, want, dtype, what=f"whole rows {mask} {shape}")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("mask,alibi,shape,off,window", [
    ("window", False, (1, 8, 2, 200, 9000), 4000, 1500), ("window", True, (1, 8, 2, 200, 9000), 4000, 1500),
    ("window", False, (1, 4, 2, 130, 3000), 0, 2500), ("none", True, (1, 8, 2, 250, 4011), 3000, 0),
    ("causal", False, (1, 2, 1, 4096, 4096), 0, 0), ("causal", True, (1, 2, 1, 4096, 4096), 0, 0),
    ("causal", False, (1, 8, 2, 300, 8000), 100, 0)],
    ids=lambda x: "x".join(map(str, x)) if isinstance(x, tuple) else str(x))
def test_shares_of_every_mask(mask, alibi, shape, off, window, dtype):
    """Calls that must share: windows whose first key tile is not tile 0, ALiBi on a dense score, and causal rows
    from the first key on, whose first query tiles have fewer key tiles than shares (partials of
    nothing) -- or, 100 rows in, so few that no call of the length would share."""
    B, Hq, Hkv, N_q, N_kv = shape
    Q, K, V = qkv(7450 + N_q, B, Hq, Hkv, N_q, N_kv, D, dtype)
    q, k, v = Q.to(DEV), K.to(DEV), V.to(DEV)
    slopes = _alibi_slopes(Hq, DEV, str(dtype)) if alibi else None
    got, launches, need = call(q, k, v, mask, off, slopes, True, window or 1)
    if off == 100:
        assert launches == 1 and need == 0     # 4 key tiles at most, of 63
    else:
        assert launches == 2 and need > 0
    want = orc.attention(Q, K, V, causal=mask == "causal", window=window or None, q_offset=off,
                         slopes=None if slopes is None else slopes.cpu())
    assert_close(got, want, dtype, what=f"must share {mask} {shape}")


def test_rotated_chunk_and_training_call():
    """A RoPE chunk puts the partials behind the rotated operands; a call that keeps the log-sum-exp
    (training) is not shared."""
    B, Hq, Hkv, N_q, N_kv, dtype = 1, 8, 2, 200, 4000, torch.bfloat16
    Q, K, V = qkv(7400, B, Hq, Hkv, N_q, N_kv, D, dtype)
    cos, sin = orc.build_rope_cache(N_kv, D, 500000.0, dtype)
    fn = af.attention(lambda q, k, v: af.softmax(af.causal(af.rope(q, k))) @ v)
    before = _lib.launch_count()
    got = fn(Q.to(DEV), K.to(DEV), V.to(DEV), cos=cos.to(DEV), sin=sin.to(DEV), q_offset=N_kv - N_q)
    assert _lib.launch_count() - before == 3   # rotation, shares, merge
    assert_close(got, orc.attention(Q, K, V, causal=True, cos=cos, sin=sin, q_offset=N_kv - N_q), dtype, what="rotated shares")
    dense = af.attention(lambda q, k, v: af.softmax(af.scaled_dot_product(q, k)) @ v)
    before = _lib.launch_count()
    q = Q.to(DEV).requires_grad_(True)
    out = dense(q, K.to(DEV), V.to(DEV))
    assert _lib.launch_count() - before == 1
    assert_close(out, orc.attention(Q, K, V), dtype, what="training call")
