"""Cases that stand for the work a host program has this library do, for timing one build of it against another.

The model behind the sizes is the 27B hybrid of the library's headers: 64 layers, width 5120, feed-forward width 17408,
48 delta-net layers (48 value heads, [128][128] state each) and 16 attention layers (24 query heads over 4 kv heads of
256), weights in PQ2_0.  What such a program calls, token by token and prompt by prompt:

  linear     one decode projection by itself: rotate + quantise + mat-vec, plain or repacked weights
  list       the decode projections of whole layers as one prepared list, independent or waiting for each other
  matmul     a projection of a batch of tokens: norm or SwiGLU, rotation + quantiser, mat-mul
  attention  causal attention of a prompt
  kv_decode  one decoded token in the attention layers: append K and V, attend over the cache
  kv_append  the K and V rows of a prompt into the cache
  delta      one decoded token in the delta-net layers
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "p40-kernel_b200"))
import bonsai_b200 as bb  # noqa: E402

DIM, FFN, HEAD_ROWS = 5120, 17408, 248320
N_HEAD, N_HEAD_KV, HEAD_DIM, KV_LAYERS = 24, 4, 256, 16
GDN_LAYERS, GDN_K_HEADS, GDN_V_HEADS, GDN_DIM = 48, 16, 48, 128
EPS = 1e-6


def listed():
    return [
        # the smallest projection (K or V of an attention layer): a latency, two launches and a call
        {"name": "linear k/v projection", "op": "linear", "n_in": DIM, "n_out": 1024, "repacked": False},
        # the longest rows, from the aligned layout a program repacks its weights into when it loads them
        {"name": "linear down, repacked", "op": "linear", "n_in": FFN, "n_out": DIM, "repacked": True},
        # the four projection shapes of a layer, eight sets, vectors already quantised: weight streaming alone
        {"name": "list layer sweep", "op": "list", "kind": "sweep", "layers": 8},
        # all projections of one decoded token with their RMSNorm and SwiGLU, 6.8 GB of weights
        {"name": "list decode step", "op": "list", "kind": "step", "layers": 64},
        # a batch of eight sequences decoding together, or eight drafted tokens
        {"name": "matmul 8 tokens", "op": "matmul", "n_in": DIM, "n_out": FFN, "n_tok": 8},
        # the ragged end of a prompt on the long rows
        {"name": "matmul 37 tokens", "op": "matmul", "n_in": FFN, "n_out": DIM, "n_tok": 37},
        # one chunk of a prompt
        {"name": "matmul 512 tokens", "op": "matmul", "n_in": DIM, "n_out": FFN, "n_tok": 512},
        {"name": "attention 2048 tokens", "op": "attention", "n_tok": 2048},
        # a decoded token late in a long context, and early in a chat
        {"name": "kv decode at 32767", "op": "kv_decode", "pos": 32767},
        {"name": "kv decode at 700", "op": "kv_decode", "pos": 700},
        {"name": "kv append 512 tokens", "op": "kv_append", "n_tok": 512},
        {"name": "delta-net step", "op": "delta", "layers": GDN_LAYERS},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["linear", "list", "matmul", "attention", "kv_decode", "kv_append", "delta"])
    if op == "linear":
        return {"op": op, "n_in": 1024 * rng.choice([1, 2, 4, 5, 5, 6, 9, 12, 17]), "n_out": _log_int(rng, 64, HEAD_ROWS),
                "repacked": rng.random() < 0.5}
    if op == "list":
        kind = rng.choice(["sweep", "step"])
        return {"op": op, "kind": kind, "layers": _log_int(rng, 1, 24 if kind == "sweep" else 63)}
    if op == "matmul":
        n_in, n_out, n_tok = 1024 * rng.choice([1, 3, 5, 5, 6, 17]), _log_int(rng, 256, 40000), _log_int(rng, 2, 2048)
        return {"op": op, "n_in": n_in, "n_out": max(64, min(n_out, DIM * FFN * 1024 // (n_in * n_tok))), "n_tok": n_tok}
    if op == "attention":
        return {"op": op, "n_tok": _log_int(rng, 16, 2047)}
    if op == "kv_decode":
        return {"op": op, "pos": _log_int(rng, 8, 32766)}
    if op == "kv_append":
        return {"op": op, "n_tok": _log_int(rng, 1, 4096)}
    return {"op": op, "layers": rng.randint(1, GDN_LAYERS - 1)}


# ---- inputs ------------------------------------------------------------------------------------------
def _ok(rc):
    if rc != 0:
        raise RuntimeError("the library returned %d" % rc)


class _Inputs:
    """Tensors made from one seed, on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(seed)
        self.seed, self.blocks = seed, 0

    def normal(self, *shape):
        return torch.randn(*shape, generator=self.g, device="cuda")

    def signs(self, n):
        return torch.randint(0, 2, (n,), generator=self.g, device="cuda").float() * 2 - 1

    def weights(self, n_out, n_in):
        """PQ2_0 rows with the checkpoint's code and scale distribution."""
        n = n_out * (n_in // 128)
        W = torch.empty(n * bb.W_BLOCK_BYTES, dtype=torch.uint8, device="cuda")
        _ok(bb.synth_pq2_0(W, self.blocks, n, self.seed))
        self.blocks += n
        return W


def _blocks(n):
    return torch.empty(n // 32 * bb.A_BLOCK_BYTES, dtype=torch.uint8, device="cuda")


def _floats(*shape):
    return torch.empty(*shape, dtype=torch.float32, device="cuda")


def _step_shapes(layers):
    """(n_in, n_out, role) of the projections of `layers` layers, every fourth of them an attention layer, and of the output head."""
    out = []
    for layer in range(layers):
        if layer % 4 == 3:
            out += [(DIM, 12288, "norm"), (DIM, 1024, "same"), (DIM, 1024, "same"), (6144, DIM, "mix")]
        else:
            out += [(DIM, 10240, "norm"), (DIM, 6144, "same"), (6144, DIM, "mix")]
        out += [(DIM, FFN, "norm"), (DIM, FFN, "same"), (FFN, DIM, "down")]
    return out + [(DIM, HEAD_ROWS, "norm")]


def _sweep_shapes(layers):
    return [(DIM, DIM), (DIM, 1024), (DIM, FFN), (FFN, DIM)] * layers


def _prepare_list(case, inp):
    ops = []
    if case["kind"] == "sweep":      # inputs quantised beforehand, nothing waits
        shapes = _sweep_shapes(case["layers"])
        y = _floats(sum(n_out for _, n_out in shapes))
        xq, at = {}, 0
        for n_in in (DIM, FFN):
            xq[n_in] = _blocks(n_in)
            _ok(bb.fwht_quant(inp.normal(n_in), inp.signs(n_in), xq[n_in], None, n_in))
        for n_in, n_out in shapes:
            ops.append((inp.weights(n_out, n_in), xq[n_in], None, y[at:at + n_out], n_out, n_in, 0))
            at += n_out
        return bb.Chain(ops), y
    # one decoded token.  The residual stream and what attention and delta-net leave behind are vectors of the host
    # program, so the projections that read them wait for what came before; the feed-forward's own values flow.
    shapes = _step_shapes(case["layers"])
    y = _floats(sum(n_out for _, n_out, _ in shapes))
    signs = {n: inp.signs(n) for n in (DIM, 6144, FFN)}
    at, x, w = 0, None, None
    for n_in, n_out, role in shapes:
        out, W = y[at:at + n_out], inp.weights(n_out, n_in)
        wait = bb.OP_DEPENDS if ops else 0
        if role == "norm":
            x, w = inp.normal(DIM), 1 + 0.1 * inp.normal(DIM)
            ops.append((W, x, signs[n_in], out, n_out, n_in, bb.OP_ROTATE | bb.OP_RMSNORM | wait, w, EPS))
        elif role == "same":
            ops.append((W, x, signs[n_in], out, n_out, n_in, bb.OP_ROTATE | bb.OP_RMSNORM | bb.OP_SAME_INPUT, w, EPS))
        elif role == "mix":
            ops.append((W, inp.normal(n_in), signs[n_in], out, n_out, n_in, bb.OP_ROTATE | wait))
        else:
            ops.append((W, y[at - 2 * FFN:at - FFN], signs[n_in], out, n_out, n_in, bb.OP_ROTATE | bb.OP_SWIGLU | bb.OP_DEPENDS, y[at - FFN:at]))
        at += n_out
    return bb.Chain(ops), y


class _Bytes:
    """One array of a cache.  A tensor made from it keeps it, and with it the cache whose memory it is."""

    def __init__(self, kv, ptr, n):
        self.kv = kv
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "|u1", "data": (ptr, False), "version": 3}


def _cache_bytes(kv):
    k, v, n = kv.arrays()
    return [torch.as_tensor(_Bytes(kv, p, n), device="cuda") for p in (k, v)]


def prepare(case, seed):
    inp, op = _Inputs(seed), case["op"]
    s = dict(case)
    if op == "linear":
        n_in, n_out = case["n_in"], case["n_out"]
        W = inp.weights(n_out, n_in)
        if case["repacked"]:
            plain, W = W, torch.empty_like(W)
            _ok(bb.repack(plain, W, n_out, n_in))
        s.update(W=W, x=inp.normal(n_in), signs=inp.signs(n_in), y=_floats(n_out), xq=_blocks(n_in), x_rot=_floats(n_in))
    elif op == "list":
        s["chain"], s["y"] = _prepare_list(case, inp)
    elif op == "matmul":
        n_in, n_out, n_tok = case["n_in"], case["n_out"], case["n_tok"]
        s.update(W=inp.weights(n_out, n_in), signs=inp.signs(n_in), X=_floats(n_tok, n_in), Xq=_blocks(n_in * n_tok), Y=_floats(n_out, n_tok))
        if n_in == FFN:
            s.update(gate=inp.normal(n_tok, n_in), up=inp.normal(n_tok, n_in))
        else:
            s.update(H=inp.normal(n_tok, n_in), norm=1 + 0.1 * inp.normal(n_in))
    elif op == "attention":
        n = case["n_tok"]
        s.update(q=inp.normal(n, N_HEAD, HEAD_DIM), k=inp.normal(n, N_HEAD_KV, HEAD_DIM), v=inp.normal(n, N_HEAD_KV, HEAD_DIM), out=_floats(n, N_HEAD, HEAD_DIM))
    elif op == "kv_decode":
        pos = case["pos"]
        kv = bb.KVCache(pos + 1)
        for layer in range(KV_LAYERS):
            _ok(kv.append_batch(layer, 0, pos, inp.normal(pos, N_HEAD_KV, HEAD_DIM), inp.normal(pos, N_HEAD_KV, HEAD_DIM)))
        q, k, v = inp.normal(KV_LAYERS, N_HEAD, HEAD_DIM), inp.normal(KV_LAYERS, N_HEAD_KV, HEAD_DIM), inp.normal(KV_LAYERS, N_HEAD_KV, HEAD_DIM)
        out = _floats(KV_LAYERS, N_HEAD, HEAD_DIM)
        s.update(kv=kv, cache=_cache_bytes(kv), out=out, rows=[(i, k[i], v[i], q[i], out[i]) for i in range(KV_LAYERS)])
    elif op == "kv_append":
        n = case["n_tok"]
        kv = bb.KVCache(n)
        s.update(kv=kv, cache=_cache_bytes(kv), rows=[(i, inp.normal(n, N_HEAD_KV, HEAD_DIM), inp.normal(n, N_HEAD_KV, HEAD_DIM)) for i in range(KV_LAYERS)])
    else:
        n, unit = case["layers"], GDN_DIM ** -0.5      # q and k of unit length, as the model normalises them
        state = inp.normal(n, GDN_V_HEADS, GDN_DIM, GDN_DIM) * 0.1
        q, k = inp.normal(n, GDN_K_HEADS, GDN_DIM) * unit, inp.normal(n, GDN_K_HEADS, GDN_DIM) * unit
        v, g = inp.normal(n, GDN_V_HEADS, GDN_DIM), -inp.normal(n, GDN_V_HEADS).abs() * 0.1
        beta, out = torch.sigmoid(inp.normal(n, GDN_V_HEADS)), _floats(n, GDN_V_HEADS, GDN_DIM)
        s.update(state=state, out=out, rows=[(state[i], q[i], k[i], v[i], g[i], beta[i], out[i]) for i in range(n)])
    return s


# ---- one pass ----------------------------------------------------------------------------------------
def run(s):
    op = s["op"]
    if op == "linear":
        n_in, n_out = s["n_in"], s["n_out"]
        if s["repacked"]:
            _ok(bb.fwht_quant(s["x"], s["signs"], s["xq"], s["x_rot"], n_in))
            _ok(bb.gemv_repack(s["W"], s["x_rot"], s["y"], n_out, n_in))
        else:
            _ok(bb.linear(s["W"], s["x"], s["signs"], s["y"], s["xq"], n_out, n_in))
        return s["y"]
    if op == "list":
        _ok(s["chain"].run())
        return s["y"]
    if op == "matmul":
        n_in, n_out, n_tok = s["n_in"], s["n_out"], s["n_tok"]
        if n_in == FFN:
            _ok(bb.swiglu(s["gate"], s["up"], s["X"], n_tok * n_in))
        else:
            _ok(bb.rmsnorm(s["H"], s["norm"], s["X"], n_tok, n_in, EPS))
        _ok(bb.quant_batch(s["X"], s["signs"], s["Xq"], n_in, n_tok, True))
        _ok(bb.gemm(s["W"], s["Xq"], s["Y"], n_out, n_in, n_tok))
        return s["Y"]
    if op == "attention":
        _ok(bb.attn(s["q"], s["k"], s["v"], s["out"], s["n_tok"], N_HEAD, N_HEAD_KV, HEAD_DIM, HEAD_DIM ** -0.5))
        return s["out"]
    if op == "kv_decode":
        kv, pos = s["kv"], s["pos"]
        for layer, k, v, q, out in s["rows"]:
            _ok(kv.append(layer, pos, k, v))
            _ok(kv.attn_decode(layer, pos, q, out))
        return [s["out"], s["cache"]]
    if op == "kv_append":
        for layer, k, v in s["rows"]:
            _ok(s["kv"].append_batch(layer, 0, s["n_tok"], k, v))
        return s["cache"]
    for state, q, k, v, g, beta, out in s["rows"]:
        _ok(bb.gdn_step(state, q, k, v, g, beta, out, GDN_K_HEADS, GDN_V_HEADS, GDN_DIM, GDN_DIM))
    return [s["out"], s["state"]]


# ---- what a pass cannot do without -------------------------------------------------------------------
def _weight_bytes(n_out, n_in):
    return n_out * (n_in // 128) * bb.W_BLOCK_BYTES


def work(case):
    """Every input read once (weights, vectors, cache, state), every output written once; two operations per product."""
    op = case["op"]
    if op == "linear":
        n_in, n_out = case["n_in"], case["n_out"]
        return {"bytes": _weight_bytes(n_out, n_in) + 4 * (2 * n_in + n_out), "flops": 2 * n_in * n_out}
    if op == "list":
        shapes = _sweep_shapes(case["layers"]) if case["kind"] == "sweep" else [p[:2] for p in _step_shapes(case["layers"])]
        return {"bytes": sum(_weight_bytes(n_out, n_in) + 4 * (n_in + n_out) for n_in, n_out in shapes), "flops": sum(2 * a * b for a, b in shapes)}
    if op == "matmul":
        n_in, n_out, n_tok = case["n_in"], case["n_out"], case["n_tok"]
        return {"bytes": _weight_bytes(n_out, n_in) + 4 * n_tok * (n_in * (2 if n_in == FFN else 1) + n_out), "flops": 2 * n_in * n_out * n_tok}
    if op == "attention":
        n = case["n_tok"]
        return {"bytes": 4 * n * HEAD_DIM * (2 * N_HEAD + 2 * N_HEAD_KV), "flops": 2 * n * (n + 1) * N_HEAD * HEAD_DIM}
    if op == "kv_decode":
        n, row = case["pos"] + 1, HEAD_DIM // 32 * 34
        return {"bytes": KV_LAYERS * (2 * n * N_HEAD_KV * row + 4 * HEAD_DIM * (2 * N_HEAD + 2 * N_HEAD_KV)), "flops": KV_LAYERS * 4 * n * N_HEAD * HEAD_DIM}
    if op == "kv_append":
        return {"bytes": KV_LAYERS * 2 * case["n_tok"] * N_HEAD_KV * (4 * HEAD_DIM + HEAD_DIM // 32 * 34), "flops": 0}
    n = case["layers"] * GDN_V_HEADS
    return {"bytes": n * 4 * (2 * GDN_DIM * GDN_DIM + 3 * GDN_DIM), "flops": n * 7 * GDN_DIM * GDN_DIM}


def tolerance(case):
    """Sums are fp32 (1e-5).  Where an fp32 value is computed and then quantised to 8 bits inside the pass, its last bits
    decide some roundings: a norm's shift few values by one step of 1 / 127, a SwiGLU of computed projections more.
    Cache bytes are exact: the quantiser's arithmetic is given operation by operation."""
    if case["op"] == "kv_append":
        return "exact"
    if case["op"] == "matmul":
        return {"rel": 3e-4}
    if case["op"] == "list" and case["kind"] == "step":
        return {"rel": 1e-3}
    return {"rel": 1e-5}
