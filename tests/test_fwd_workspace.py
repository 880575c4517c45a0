"""Nobody else writes the workspace of a forward call (rotated Q and K, partials of shared keys) before its
kernels have run: calls of two threads whose launches interleave on one stream, a captured graph and
later calls do not meet in it."""
import threading

import pytest
import torch

import attentionfuse_b200 as af
from attentionfuse_b200.runtime import _lib, dispatch
from oracle import attention_oracle as orc
from tests._util import assert_close, qkv

causal_rope = af.attention(lambda q, k, v: af.softmax(af.causal(af.rope(q, k))) @ v)


class FakeLibrary:
    """af_fwd notes the workspace it was given and waits there until told to go on."""

    def __init__(self):
        self.seen, self.inside, self.go_on = [], threading.Event(), threading.Event()

    need = 4096

    def af_fwd_workspace_bytes(self, params):
        return self.need

    def af_fwd(self, params, stream):
        p = params._obj
        self.seen.append((p.workspace, p.workspace_bytes))
        if len(self.seen) == 1:
            self.inside.set()
            assert self.go_on.wait(30)
        return 0


@pytest.fixture
def lib(monkeypatch):
    lib = FakeLibrary()
    monkeypatch.setattr(_lib, "load", lambda: lib)
    monkeypatch.setattr(_lib, "current_stream", lambda device: lib.stream)
    monkeypatch.setattr(_lib, "on_device", lambda device: _lib._NO_SWITCH)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: lib.capturing)
    monkeypatch.setattr(dispatch, "_KEPT", dispatch._KeptWorkspaces())
    monkeypatch.setattr(dispatch, "_FWD_TEMPLATES", {})
    lib.stream, lib.capturing = 7, False
    return lib


def rope_call(n=640):
    Q, K, V = (torch.zeros(1, h, n, 64, dtype=torch.bfloat16) for h in (2, 1, 1))
    cos, sin = orc.build_rope_cache(n, 64, 10000.0, torch.bfloat16)
    dispatch.launch_forward(Q, K, V, torch.empty_like(Q), sm_scale=0.125, mask_kind=1, cos=cos, sin=sin)


def test_two_threads_on_one_stream_have_a_workspace_each(lib):
    first = threading.Thread(target=rope_call)
    first.start()
    assert lib.inside.wait(30)
    rope_call()                                        # while the first call is between its launches
    lib.go_on.set()
    first.join()
    (ws_a, n_a), (ws_b, n_b) = lib.seen
    assert n_a == n_b == 4096
    assert abs(ws_a - ws_b) >= 4096


def test_what_is_kept_is_bounded_and_never_a_graphs(lib):
    lib.go_on.set()
    rope_call()
    rope_call()
    assert lib.seen[0] == lib.seen[1]                  # a stream's calls follow one another
    lib.capturing = True
    rope_call()
    lib.capturing = False
    kept = dispatch._KEPT.by_stream
    assert lib.seen[2][0] != lib.seen[0][0] and len(kept) == 1 and kept[None, 7].data_ptr() == lib.seen[0][0]
    for lib.stream in range(1, 20):
        rope_call()
        assert len(kept) <= 4
    lib.need, lib.stream = dispatch._KEPT_MAX_BYTES + 1, 100
    rope_call(700)
    assert all(t.numel() <= dispatch._KEPT_MAX_BYTES for t in kept.values()) and (None, 100) not in kept
    others = []
    thread = threading.Thread(target=lambda: others.append(len(dispatch._KEPT.by_stream)))
    thread.start()
    thread.join()
    assert others == [0]


@pytest.mark.gpu
@pytest.mark.parametrize("N_q,N_kv", [(700, 700), (100, 4000)], ids=["square", "shares"])
def test_a_captured_rope_call_owns_its_workspace(N_q, N_kv):
    """Warm up and capture on a side stream, run a larger call there, fill what it leaves free, replay."""
    Hq, Hkv, D, dtype = 8, 2, 128, torch.bfloat16
    Q, K, V = qkv(8600, 1, Hq, Hkv, N_q, N_kv, D, dtype)
    cos, sin = orc.build_rope_cache(N_kv, D, 500000.0, dtype)
    q, k, v, c, s = (t.cuda() for t in (Q, K, V, cos, sin))
    big = [torch.randn(2, h, 4096, D, device="cuda", dtype=dtype) for h in (Hq, Hkv, Hkv)]
    cb, sb = (t.cuda() for t in orc.build_rope_cache(4096, D, 500000.0, dtype))
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        causal_rope(q, k, v, cos=c, sin=s, q_offset=N_kv - N_q)
        side.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            out = causal_rope(q, k, v, cos=c, sin=s, q_offset=N_kv - N_q)
        causal_rope(*big, cos=cb, sin=sb)
        side.synchronize()
        filled = [torch.full((n,), 3, dtype=torch.uint8, device="cuda") for n in (1 << 20, 4 << 20, 16 << 20, 32 << 20)]
        graph.replay()
    torch.cuda.synchronize()
    assert_close(out, orc.attention(Q, K, V, causal=True, cos=cos, sin=sin, q_offset=N_kv - N_q), dtype, what="replayed")
    assert all(bool((f == 3).all()) for f in filled)


@pytest.mark.gpu
def test_the_workspace_follows_the_environment_and_the_rotation_switch(monkeypatch):
    """A call that could share its keys, first with the layout fixed by the environment, then free; and with
    rotation kept in the kernel, which is no concern of a call without RoPE."""
    q, k, v = (t.cuda() for t in qkv(8700, 1, 8, 2, 64, 4096, 128, torch.bfloat16))
    out = torch.empty_like(q)

    def launches():
        before = _lib.launch_count()
        dispatch.launch_forward(q, k, v, out, sm_scale=0.088, mask_kind=0)
        return _lib.launch_count() - before

    monkeypatch.setenv("ATTNFUSE_FWD_PAIR", "1")
    assert launches() == 1
    monkeypatch.delenv("ATTNFUSE_FWD_PAIR")
    assert launches() == 2                             # shares and their merge
    monkeypatch.setenv("ATTNFUSE_ROPE_IN_KERNEL", "1")
    assert launches() == 2
