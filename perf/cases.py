"""The attention work that a user of this package has it do, as measurable cases.

`listed()` names the cases, `draw(rng)` gives more of the same ranges, `prepare(case, seed)`
makes what a program holds before the call (tensors, rotation tables, block masks, the traced
function), `run(state)` is one call through the public entry points, `work(case)` counts the bytes
and floating-point operations that call cannot do without, and `tolerance(case)` bounds the
difference between two correct implementations at the same precision, and `exact(case, seed)` is the
result in 64 bits.

Kinds: "prefill" (square forward), "chunk" (rows of a prompt against a cache), "train" (forward and
backward of one layer), "blocks" (block-sparse forward and backward) and "decode" (one query row per
sequence against a cache).
"""
from __future__ import annotations

import functools

import numpy as np
import torch

import attentionfuse_b200 as af
from attentionfuse_b200.rope_utils import build_rope_cache

DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}


def _square(name, kind, B, H_q, H_kv, N, D, dtype, mask="causal", window=0, alibi=False, rope=False, base=10000.0):
    return dict(name=name, kind=kind, B=B, H_q=H_q, H_kv=H_kv, N=N, D=D, dtype=dtype, mask=mask, window=window,
                alibi=alibi, rope=rope, base=base)


def _chunk(name, B, H_q, H_kv, N_q, N_kv, D, dtype):
    return dict(name=name, kind="chunk", B=B, H_q=H_q, H_kv=H_kv, N_q=N_q, N=N_kv, D=D, dtype=dtype, mask="causal",
                window=0, alibi=False, rope=False)


def _blocks(name, B, H, N, D, dtype, block):
    return dict(name=name, kind="blocks", B=B, H_q=H, H_kv=H, N=N, D=D, dtype=dtype, block=block)


def _decode(name, B, H_q, H_kv, N, D, dtype, ragged, rotated=False):
    return dict(name=name, kind="decode", B=B, H_q=H_q, H_kv=H_kv, N=N, D=D, dtype=dtype, ragged=ragged,
                rotated=rotated)


def listed():
    return [
        # one token of a single user's chat, Llama-3-8B heads, short cache: pure latency
        _decode("decode_b1_l1024", 1, 32, 8, 1024, 128, "bf16", ragged=False),
        # a serving batch of a RoPE model (70B heads): every row at the end of its own sequence, the
        # cache holds keys that were rotated when they were written
        _decode("decode_rope_b16_l4096", 16, 64, 8, 4096, 128, "bf16", ragged=True, rotated=True),
        # the long-cache decode of the benchmark: lengths spread over [L/2, L]
        _decode("decode_b16_l32768", 16, 32, 8, 32768, 128, "bf16", ragged=True),
        # the golden fp32 problem: the exact path
        _square("fp32_rope_alibi_n512", "prefill", 2, 12, 12, 512, 64, "f32", alibi=True, rope=True),
        # GPT-2 / BERT geometry, the shortest sequence of the forward sweep
        _square("prefill_gpt2_n512", "prefill", 4, 12, 12, 512, 64, "bf16", rope=True),
        # the same geometry at the longest sequence, everything on the score
        _square("prefill_gpt2_rope_alibi_n4096", "prefill", 4, 12, 12, 4096, 64, "f16", alibi=True, rope=True),
        # bidirectional window of an encoder on a ragged sequence length
        _square("window256_n3001", "prefill", 4, 12, 12, 3001, 64, "bf16", mask="window", window=256),
        # Llama-3-8B layer prefill: the headline of bench.py
        _square("prefill_llama_n4096", "prefill", 4, 32, 8, 4096, 128, "bf16", rope=True, base=500000.0),
        # a chunk of a long prompt against its cache, as the transformers hook calls it
        _chunk("chunk_500_of_8011", 1, 32, 8, 500, 8011, 128, "bf16"),
        # a training step of the GPT-2 layer
        _square("train_gpt2_n4096", "train", 4, 12, 12, 4096, 64, "f16"),
        # a training step of the Llama-3-8B layer, rotation included
        _square("train_llama_n4096", "train", 4, 32, 8, 4096, 128, "bf16", rope=True, base=500000.0),
        # BigBird training step, one mask per head
        _blocks("bigbird_n8192", 2, 16, 8192, 64, "f16", 128),
    ]


def _size(rng, lo, hi):
    """Spread over the logarithm of [lo, hi]; every other one is whatever it is, odd ones among them,
    the rest multiples of 64 as padded batches have them."""
    n = int(round(lo * (hi / lo) ** rng.random()))
    return n if rng.random() < 0.5 else max(lo, n // 64 * 64)


def draw(rng):
    half = rng.choice(["bf16", "f16"])
    kind = rng.choice(["decode", "decode", "prefill64", "prefill128", "chunk", "train64", "train128", "blocks", "fp32"])
    if kind == "decode":
        H_q, H_kv = rng.choice([(32, 8), (64, 8), (64, 1)])
        rotated = rng.random() < 0.4 and H_q // H_kv <= 16
        B = rng.choice([1, 2, 3, 5, 8, 12, 16])
        case = _decode("", B, H_q, H_kv, _size(rng, 1024, 32768), 128, half, rng.random() < 0.7, rotated)
    elif kind == "chunk":
        n = _size(rng, 1024, 16384)
        case = _chunk("", rng.choice([1, 2]), 32, 8, min(_size(rng, 64, 1024), n - 1), n, 128, half)
    elif kind == "blocks":
        case = _blocks("", rng.choice([1, 2]), rng.choice([8, 12, 16]), _size(rng, 1024, 8192), 64, half,
                       rng.choice([64, 128]))
    else:
        mask, window = rng.choice([("none", 0), ("causal", 0), ("causal", 0), ("window", 256)])
        extra = dict(mask=mask, window=window)
        if mask == "causal":
            extra.update(alibi=rng.random() < 0.3, rope=rng.random() < 0.6)
        if kind == "fp32":
            case = _square("", "prefill", rng.choice([1, 2]), 12, 12, _size(rng, 128, 1024), 64, "f32", **extra)
        elif kind.endswith("64"):
            case = _square("", kind[:-2], rng.choice([1, 2, 4]), rng.choice([12, 16]), 0, _size(rng, 128, 4096), 64,
                           half, **extra)
            case["H_kv"] = case["H_q"]
        else:
            B = rng.choice([1, 2, 4])
            if kind == "train128" and mask == "none":       # no dearer than the listed step
                B = min(B, 2)
            case = _square("", kind[:-3], B, 32, 8, _size(rng, 512, 4096), 128, half, base=500000.0, **extra)
    del case["name"]
    return case


@functools.lru_cache(maxsize=None)
def _function(mask, window, alibi_heads, rope):
    """The decorated function a user's module defines once."""
    @af.attention
    def fn(Q, K, V):
        s = af.rope(Q, K) if rope else af.scaled_dot_product(Q, K)
        if alibi_heads:
            s = af.alibi(s, alibi_heads)
        if mask == "causal":
            s = af.causal(s)
        elif mask == "window":
            s = af.sliding_window(s, window)
        elif mask == "blocks":
            s = af.block_sparse(s)
        return af.softmax(s) @ V
    return fn


def _bigbird(case, seed):
    """BigBird grid per head: 2 global key blocks and query rows, a band of one block to each side,
    3 random further blocks per row: [H, n, n] of truth values, the count the same for every seed."""
    n = (case["N"] + case["block"] - 1) // case["block"]
    rng = np.random.default_rng(seed)
    grids = np.zeros((case["H_q"], n, n), dtype=bool)
    grids[:, :, :2] = True
    grids[:, :2, :] = True
    for i in range(n):
        grids[:, i, max(0, i - 1):i + 2] = True
    for g in grids:
        for i in range(2, n):
            free = np.flatnonzero(~g[i])
            g[i, rng.choice(free, size=min(3, len(free)), replace=False)] = True
    return grids


def _lengths(case):
    """Valid cache lengths, evenly spread over [L/2, L] (their sum is part of `work`)."""
    B, L = case["B"], case["N"]
    if not case["ragged"]:
        return [L] * B
    return [L - (L // 2) * i // max(1, B - 1) for i in range(B)]


def prepare(case, seed):
    dev, dt = torch.device("cuda"), DTYPES[case["dtype"]]
    gen = torch.Generator(device=dev).manual_seed(seed)
    B, H_q, H_kv, N, D, kind = (case[k] for k in ("B", "H_q", "H_kv", "N", "D", "kind"))

    def rnd(*shape):
        return torch.randn(*shape, generator=gen, device=dev, dtype=dt)

    state = {"kind": kind, "kw": {}}
    if kind == "decode":
        state["q"], state["k"], state["v"] = rnd(B, H_q, 1, D), rnd(B, H_kv, N, D), rnd(B, H_kv, N, D)
        lens = torch.tensor(_lengths(case), dtype=torch.int32)
        lens = lens[torch.from_numpy(np.random.default_rng(seed).permutation(B))].to(dev)
        if case["rotated"]:
            # a position cannot see past itself: the causal rule and the length are the same bound
            state["fn"] = _function("causal", 0, 0, True)
            cos, sin = build_rope_cache(N, D, 500000.0, device=dev, dtype=dt)
            state["kw"] = dict(cos=cos, sin=sin, kv_lens=lens, q_offset=lens - 1, kv_rotated=True)
        else:
            state["fn"] = _function("none", 0, 0, False)
            state["kw"] = dict(kv_lens=lens) if case["ragged"] else {}
        return state
    if kind == "chunk":
        # queries as a projection leaves them: (B, N, H, D) storage seen as (B, H, N, D)
        state["q"] = rnd(B, case["N_q"], H_q, D).transpose(1, 2)
        state["kw"] = dict(q_offset=N - case["N_q"])
    else:
        state["q"] = rnd(B, H_q, N, D)
    state["k"], state["v"] = rnd(B, H_kv, N, D), rnd(B, H_kv, N, D)
    if kind == "blocks":
        state["fn"] = _function("blocks", 0, 0, False)
        grids = torch.from_numpy(_bigbird(case, seed))
        state["kw"] = dict(block_mask=af.create_block_mask_per_head(grids, case["block"], case["block"], device=str(dev)))
    else:
        state["fn"] = _function(case["mask"], case["window"], H_q if case["alibi"] else 0, case["rope"])
        if case["rope"]:
            cos, sin = build_rope_cache(N, D, case["base"], device=dev, dtype=dt)
            state["kw"].update(cos=cos, sin=sin)
    if kind in ("train", "blocks"):
        state["do"] = rnd(B, H_q, N, D)
        for t in ("q", "k", "v"):
            state[t].requires_grad_(True)
    return state


def run(state):
    q, k, v = state["q"], state["k"], state["v"]
    out = state["fn"](q, k, v, **state["kw"])
    if state["kind"] in ("train", "blocks"):
        return (out.detach(), *torch.autograd.grad(out, (q, k, v), state["do"]))
    return out


def _pairs(case):
    """Visible (query, key) pairs of one head."""
    N, w = case["N"], case.get("window", 0)
    if case["kind"] == "chunk":
        n_q = case["N_q"]
        return n_q * (N - n_q) + n_q * (n_q + 1) // 2
    if case["kind"] == "blocks":
        grid, b = _bigbird(dict(case, H_q=1), 0)[0], case["block"]
        side = np.minimum(b, N - b * np.arange(len(grid)))       # the last block may be cut short
        return int(side @ (grid * side).sum(1))
    if case["mask"] == "causal":
        return N * (N + 1) // 2
    if case["mask"] == "window":
        w = min(w, N)
        return N * (2 * w - 1) - w * (w - 1)
    return N * N


def work(case):
    size = 4 if case["dtype"] == "f32" else 2
    B, H_q, H_kv, N, D = (case[k] for k in ("B", "H_q", "H_kv", "N", "D"))
    if case["kind"] == "decode":
        keys = sum(_lengths(case))
        return {"bytes": size * D * (2 * H_kv * keys + 2 * B * H_q), "flops": 4 * H_q * D * keys}
    rows_q, rows_k = B * H_q * case.get("N_q", N), B * H_kv * N
    tables = 2 * N * D * size if case.get("rope") else 0
    if case["kind"] in ("train", "blocks"):
        # forward 2 products, backward 5 (scores again, dP, dQ, dK, dV)
        nbytes = size * D * (4 * rows_q + 4 * rows_k)      # q, dO in; o, dq out; k, v in; dk, dv out
        return {"bytes": nbytes + tables, "flops": 14 * B * H_q * D * _pairs(case)}
    return {"bytes": size * D * (2 * rows_q + 2 * rows_k) + tables, "flops": 4 * B * H_q * D * _pairs(case)}


def tolerance(case):
    # About four times the error of the outputs against a float64 evaluation (2-norm, worst over the
    # kinds): fp32 2.0e-7; bf16 2.9e-3 forward and 3.8e-3 gradients, f16 3.7e-4 and 4.9e-4 (rotated
    # operands, probabilities and results are rounded to the type).
    if case["dtype"] == "f32":
        return {"rel": 1e-6}
    grad = case["kind"] in ("train", "blocks")
    if case["dtype"] == "f16":
        return {"rel": 2e-3 if grad else 1.5e-3}
    return {"rel": 1.5e-2 if grad else 1.2e-2}


def _slopes(n):
    """ALiBi slopes of n heads (Press et al.): geometric for a power of two, else the closest lower
    power of two followed by every other slope of the doubled sequence."""
    def geometric(m):
        return [2.0 ** (-8.0 * (i + 1) / m) for i in range(m)]
    if n & (n - 1) == 0:
        return geometric(n)
    low = 1 << (n.bit_length() - 1)
    return geometric(low) + geometric(2 * low)[0::2][:n - low]


def _rotated(x, cos, sin):
    half = x.shape[-1] // 2
    return x * cos + torch.cat([-x[..., half:], x[..., :half]], dim=-1) * sin


def exact(case, seed):
    """What `run` returns, in 64 bits, one (batch, KV head) group after the other; gradients are
    written out: P and dP of one head, then the four products."""
    state = prepare(case, seed)
    q, k, v = (state[t].detach() for t in ("q", "k", "v"))
    dev, kw, kind = q.device, state["kw"], state["kind"]
    B, H_q, n_q, D = q.shape
    H_kv, n_kv = k.shape[1], k.shape[2]
    group, scale, train = H_q // H_kv, D ** -0.5, kind in ("train", "blocks")
    first = kw.get("q_offset", 0)
    first = first.tolist() if torch.is_tensor(first) else [first] * B
    lens = kw["kv_lens"].tolist() if "kv_lens" in kw else [n_kv] * B
    cols = torch.arange(n_kv, device=dev)
    rope = "cos" in kw
    if rope:
        cos, sin = (kw[t].double().reshape(-1, D) for t in ("cos", "sin"))
    # the slope table is created in the type of the operands
    slopes = torch.tensor(_slopes(H_q), dtype=DTYPES[case["dtype"]]).double().tolist() if case.get("alibi") else None
    grids = torch.from_numpy(_bigbird(case, seed)).to(dev) if kind == "blocks" else None
    out = torch.empty(q.shape, dtype=torch.float64, device=dev)
    if train:
        dq, dk, dv = (torch.zeros(t.shape, dtype=torch.float64, device=dev) for t in (q, k, v))
    for b in range(B):
        rows = torch.arange(n_q, device=dev) + first[b]
        rel = rows[:, None] - cols[None, :]
        keep = None
        if kind == "chunk" or (kind != "decode" and case.get("mask") == "causal"):
            keep = rel >= 0
        elif case.get("mask") == "window":
            keep = rel.abs() < case["window"]
        elif kind == "decode":
            keep = (cols < lens[b])[None, :]
        for h in range(H_q):
            g = h // group
            qh, kh, vh = q[b, h].double(), k[b, g].double(), v[b, g].double()
            if rope:
                qh = _rotated(qh, cos[rows], sin[rows])
                if not case.get("rotated"):
                    kh = _rotated(kh, cos[:n_kv], sin[:n_kv])
            s = (qh @ kh.T).mul_(scale)
            if slopes:
                s -= slopes[h] * rel.abs()
            if kind == "blocks":
                keep = grids[h].repeat_interleave(case["block"], 0).repeat_interleave(case["block"], 1)[:n_q, :n_kv]
            if keep is not None:
                s.masked_fill_(~keep, float("-inf"))
            p = torch.softmax(s, dim=-1)
            del s
            out[b, h] = p @ vh
            if train:
                do = state["do"][b, h].double()
                dv[b, g] += p.T @ do
                ds = do @ vh.T
                ds.sub_((do * out[b, h]).sum(-1, keepdim=True)).mul_(p).mul_(scale)
                gq, gk = ds @ kh, ds.T @ qh
                if rope:          # the transpose of the rotation is the one with -sin
                    gq, gk = _rotated(gq, cos[rows], -sin[rows]), _rotated(gk, cos[:n_kv], -sin[:n_kv])
                dq[b, h] += gq
                dk[b, g] += gk
                del ds
            del p
    return (out, dq, dk, dv) if train else out
