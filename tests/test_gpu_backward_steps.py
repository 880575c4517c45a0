"""The tensor-core backward at the edges of its steps (128 stationary rows; 128 streamed rows a step at
head_dim 64, 64 at 128) and over the range of the row statistics: -L / scale and -delta enter the
products of the key-stationary passes as three bf16 terms each."""
import pytest
import torch

import attentionfuse_b200 as af
from attentionfuse_b200.runtime import _lib
from attentionfuse_b200.runtime.backward import launch_backward
from attentionfuse_b200.runtime.dispatch import launch_forward
from oracle import attention_oracle as orc
from tests._util import assert_close, qkv

pytestmark = pytest.mark.gpu
DEV = "cuda"


def grads(Q, K, V, dO, scale, mask_kind, window=0):
    q, k, v, do = (t.to(DEV) for t in (Q, K, V, dO))
    L = torch.empty(q.shape[:3], dtype=torch.float32, device=DEV)
    out = torch.empty_like(q)
    launch_forward(q, k, v, out, sm_scale=scale, mask_kind=mask_kind, window=window, save_lse=L, family=_lib.AF_FAMILY_TCGEN05)
    return launch_backward(q, k, v, out, L, do, sm_scale=scale, mask_kind=mask_kind, window=window, family=_lib.AF_FAMILY_TCGEN05)


@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("mask,window", [("none", 0), ("causal", 0), ("window", 90)])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("N", [1, 63, 65, 127, 128, 129, 257, 450])
def test_step_edges(N, D, mask, window, deterministic, monkeypatch):
    monkeypatch.setenv("ATTNFUSE_BWD_DETERMINISTIC", "1" if deterministic else "0")
    dtype = torch.float16
    Q, K, V = qkv(7500 + N, 2, 4, 2, N, N, D, dtype)
    dO = orc.randn(7600 + N, Q.shape, dtype)
    got = grads(Q, K, V, dO, D ** -0.5, {"none": 0, "causal": 1, "window": 2}[mask], window)
    _, *want = orc.attention_grads(Q, K, V, dO, causal=mask == "causal", window=window or None)
    for name, g, w in zip(("dQ", "dK", "dV"), got, want):
        if N == 1 and name != "dV":            # one key: P = 1, dQ = dK = 0 up to the rounding of O in delta
            assert g.float().abs().max().item() < 2e-2
        else:
            assert_close(g, w, dtype, grad=True, what=f"steps {mask} N{N} D{D} {name}")


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("scale", [1e-40, 1e-38, 1e-33, 1e-8, 1e-3, 1.0, 4.0])
def test_scale_range(scale, D, dtype):
    """L / scale from beyond fp32 (scales whose reciprocal overflows) and 1e9 (flat rows) down to a few
    (one-hot rows), where a term that was dropped would show as a factor on every probability."""
    N = 200
    Q, K, V = qkv(7700, 1, 2, 1, N, N, D, dtype)
    if scale >= 1.0:
        Q = (Q.float() * 0.25).to(dtype)
    dO = orc.randn(7800, Q.shape, dtype)
    got = grads(Q, K, V, dO, scale, 1)
    _, *want = orc.attention_grads(Q, K, V, dO, causal=True, scale=scale)
    for name, g, w in zip(("dQ", "dK", "dV"), got, want):
        if scale < 1e-4 and name != "dV":      # dQ, dK carry the factor `scale`: below f16's range
            continue
        assert_close(g, w, dtype, grad=True, what=f"scale {scale} D{D} {name}")


def test_rows_without_a_visible_key():
    """Query blocks without any key block: L = -inf, the rows contribute nothing to dK and dV."""
    N, D, H, dtype = 512, 64, 2, torch.bfloat16
    grid = torch.zeros(4, 4, dtype=torch.bool)
    grid[0, 0] = grid[2, 0] = grid[2, 3] = True
    bm = af.BlockMask.from_dense(grid, 128, 128, device=DEV)
    fn = af.attention(lambda q, k, v: af.softmax(af.block_sparse(af.scaled_dot_product(q, k))) @ v)
    Q, K, V = qkv(7900, 1, H, H, N, N, D, dtype)
    dO = orc.randn(7950, Q.shape, dtype)
    q, k, v = (t.to(DEV).requires_grad_(True) for t in (Q, K, V))
    fn(q, k, v, block_mask=bm).backward(dO.to(DEV))
    rows = torch.cat([torch.arange(0, 128), torch.arange(256, 384)])
    mask = orc.block_elem_mask(grid, 128, 128, N, N)
    _, dq, dk, dv = orc.attention_grads(Q[:, :, rows], K, V, dO[:, :, rows], elem_mask=mask[rows])
    assert_close(q.grad[:, :, rows], dq, dtype, grad=True, what="seen rows dQ")
    assert (q.grad[:, :, 128:256] == 0).all() and (q.grad[:, :, 384:] == 0).all()
    assert_close(k.grad, dk, dtype, grad=True, what="dK with unseen rows")
    assert_close(v.grad, dv, dtype, grad=True, what="dV with unseen rows")


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("dtype,logit", [(torch.float16, -26.0), (torch.bfloat16, -126.0)])
@pytest.mark.parametrize("mask,window", [("none", 0), ("window", 90), ("blocks", 0), ("causal", 0)])
@pytest.mark.parametrize("N", [1, 130, 200, 257])
def test_negative_logits_at_a_ragged_key_axis(N, mask, window, dtype, logit, D):
    """Every logit is clearly negative, so that exp(-L) leaves the type: the lanes of the last key tile past
    N_kv have S = 0 and must not reach dQ.  The mean of the logits sits in one column of Q and K, whose
    gradients are sums of dS that cancel: rounding only, compared on the other columns."""
    Q, K, V = qkv(8300 + N, 1, 4, 2, N, N, D, dtype)
    side = (-logit * D ** 0.5) ** 0.5
    Q[..., 0], K[..., 0] = side, -side
    dO = orc.randn(8400 + N, Q.shape, dtype)
    kw = dict(causal=mask == "causal", window=window or None)
    if mask == "blocks":
        nb = (N + 127) // 128
        bm = af.BlockMask.from_dense(torch.ones(nb, nb, dtype=torch.bool), 128, 128, device=DEV)
        fn = af.attention(lambda q, k, v: af.softmax(af.block_sparse(af.scaled_dot_product(q, k))) @ v)
        q, k, v = (t.to(DEV).requires_grad_(True) for t in (Q, K, V))
        fn(q, k, v, block_mask=bm).backward(dO.to(DEV))
        got = q.grad, k.grad, v.grad
    else:
        got = grads(Q, K, V, dO, D ** -0.5, {"none": 0, "causal": 1, "window": 2}[mask], window)
    _, *want = orc.attention_grads(Q, K, V, dO, **kw)
    for name, g, w in zip(("dQ", "dK", "dV"), got, want):
        assert torch.isfinite(g.float()).all(), name
        if N == 1 and name != "dV":            # one key: P = 1, dQ = dK = 0 up to the rounding of O in delta
            assert g[..., 1:].float().abs().max().item() < 2e-2
        elif name == "dV":
            assert_close(g, w, dtype, grad=True, what=f"negative logits {mask} N{N} D{D} dV")
        else:
            assert_close(g[..., 1:], w[..., 1:], dtype, grad=True, what=f"negative logits {mask} N{N} D{D} {name}")
