"""Prompt attention on the tensor cores (csrc/attn_tc.cuh) against softmax attention in float64, at the sizes where its
tiles of 128 queries and 64 keys begin, end and are left half empty, and next to the token count from which it is used.

Bound: 2e-6 of the largest output.  The operands carry 22 - 24 bits and the sums are fp32 (at most 2^-23 lost in each of 24
additions per score and 12 per tile of outputs); the largest error seen on the CUDA cores over these sizes is 1.1e-6."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

D = 256
SCALE = D ** -0.5
REL_TOL = 2e-6


def inputs(n, heads, kv_heads, seed, spread=0.0):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    q, k, v = (torch.randn(n, h, D, generator=g, device="cuda") for h in (heads, kv_heads, kv_heads))
    if spread:          # rows of very different size: the planes are scaled row by row
        k = k * torch.exp(spread * torch.randn(n, kv_heads, 1, generator=g, device="cuda")) * 0.2
        v = v * torch.exp(2 * spread * torch.randn(n, kv_heads, 1, generator=g, device="cuda"))
    return q, k, v


def exact(q, k, v):
    import torch
    n, heads, _ = q.shape
    later = torch.ones(n, n, dtype=torch.bool, device="cuda").triu(1)
    out = torch.empty(n, heads, D, dtype=torch.float64, device="cuda")
    for h in range(heads):
        kv = h // (heads // k.shape[1])
        s = (q[:, h].double() @ k[:, kv].double().T) * SCALE
        out[:, h] = torch.softmax(s.masked_fill(later, -float("inf")), -1) @ v[:, kv].double()
    return out


def close(got, want):
    err, top = float((got.double() - want).abs().max()), float(want.abs().max())
    assert err <= REL_TOL * top, (err, top)


@pytest.mark.parametrize("n,heads,kv_heads,spread", [
    (511, 6, 1, 0.0), (512, 24, 4, 0.0), (513, 4, 4, 1.0), (575, 6, 2, 0.0), (577, 6, 2, 0.0), (639, 6, 2, 0.0), (641, 6, 2, 0.0), (831, 6, 2, 0.0), (832, 3, 1, 0.0), (833, 2, 1, 0.0),
    (895, 6, 1, 0.0), (896, 1, 1, 0.0), (897, 6, 1, 1.0), (1601, 24, 4, 0.0)])
def test_against_float64(gpu, n, heads, kv_heads, spread):
    import torch
    q, k, v = inputs(n, heads, kv_heads, n, spread)
    out = torch.full((n, heads, D), float("nan"), device="cuda")
    assert gpu.attn(q, k, v, out, n, heads, kv_heads, D, SCALE) == 0
    close(out, exact(q, k, v))
    # q and out at an odd float offset: same bits
    qo, oo = (torch.zeros(q.numel() + 1, device="cuda") for _ in range(2))
    qo[1:].copy_(q.view(-1))
    assert gpu.attn(qo[1:], k, v, oo[1:], n, heads, kv_heads, D, SCALE) == 0
    assert torch.equal(oo[1:].view_as(out), out)
    assert gpu.device_status() == 0


def test_values_that_do_not_survive_the_split(gpu):
    """Infinities, NaN and huge values give what the CUDA-core kernel gives: rows in front of them are untouched, rows behind
    see them where their weight is not zero."""
    import torch
    n, heads, kv_heads = 1000, 6, 2
    q, k, v = inputs(n, heads, kv_heads, 5)
    v[700, 0, 3], v[901, 1, 7], q[750, 5, 0] = float("inf"), float("nan"), 1e25
    k[903, 0, 9] = 1e30
    out = torch.empty(n, heads, D, device="cuda")
    assert gpu.attn(q, k, v, out, n, heads, kv_heads, D, SCALE) == 0
    clean_v, clean_k, clean_q = v.clone(), k.clone(), q.clone()
    clean_v[700, 0, 3], clean_v[901, 1, 7], clean_k[903, 0, 9], clean_q[750, 5, 0] = 0, 0, 0, 0
    want = exact(clean_q, clean_k, clean_v)
    close(out[:700], want[:700])
    assert bool(torch.isinf(out[700:900, :3, 3]).all())          # kv head 0: the infinity has a weight in every row behind it
    other = [d for d in range(D) if d != 3]
    close(out[700:900, :3][:, :, other], want[700:900, :3][:, :, other])
    # kv head 1: dims other than the NaN's are as without it (a CUDA-core warp takes four queries: 900 .. 903 share a row)
    ok = [d for d in range(D) if d != 7]
    close(out[904:, 3:5][:, :, ok], want[904:, 3:5][:, :, ok])
    assert bool(torch.isnan(out[904:, 3:, 7]).all())


def test_streams_release_and_capture(gpu):
    """More streams than the library keeps buffers for, a release in between, and a captured call: all give the same bits
    (a stream under capture is served by the CUDA-core kernel: same values within the bound)."""
    import torch
    n, heads, kv_heads = 800, 6, 1
    cases = [inputs(n, heads, kv_heads, 40 + i) for i in range(3)]
    want = []
    for q, k, v in cases:
        out = torch.empty(n, heads, D, device="cuda")
        assert gpu.attn(q, k, v, out, n, heads, kv_heads, D, SCALE) == 0
        want.append(out)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(20)]
    outs = []
    for i, st in enumerate(streams):
        q, k, v = cases[i % 3]
        with torch.cuda.stream(st):
            out = torch.empty(n, heads, D, device="cuda")
            assert gpu.attn(q, k, v, out, n, heads, kv_heads, D, SCALE) == 0
            outs.append(out)
        if i == 11:
            torch.cuda.synchronize()
            assert gpu.lib().bonsai_b200_gemm_release() == 0
    torch.cuda.synchronize()
    for i, out in enumerate(outs):
        assert torch.equal(out, want[i % 3]), i
    q, k, v = cases[0]
    out = torch.empty(n, heads, D, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        assert gpu.attn(q, k, v, out, n, heads, kv_heads, D, SCALE) == 0
    graph.replay()
    torch.cuda.synchronize()
    close(out, want[0].double())
    assert gpu.device_status() == 0
