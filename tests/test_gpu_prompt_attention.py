"""Prompt attention on the tensor cores (csrc/attn_tc.cuh) against softmax attention in float64, at the sizes where its
tiles of 128 queries and 64 keys begin, end and are left half empty, and next to the token count from which it is used.

Bound: 2e-6 of the largest output.  The operands carry 22 - 24 bits and the sums are fp32 (at most 2^-23 lost in each of 24
additions per score and 12 per tile of outputs); the largest error seen on the CUDA cores over these sizes is 1.1e-6."""
import numpy as np
import pytest

from captured import launches

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


@pytest.mark.parametrize("n,heads,kv_heads,spread", [
    (1, 3, 3, 0.0), (7, 24, 4, 0.0), (9, 6, 1, 0.0), (17, 2, 2, 0.0), (31, 24, 4, 0.0), (33, 24, 4, 1.0), (49, 24, 4, 0.0), (65, 40, 8, 0.0), (145, 24, 4, 0.0), (161, 24, 4, 1.0),
    (130, 64, 8, 0.0), (191, 24, 4, 0.0), (192, 24, 4, 0.0), (193, 1, 1, 0.0), (255, 6, 2, 0.0), (256, 6, 2, 1.0), (257, 3, 1, 0.0), (319, 4, 4, 0.0), (321, 24, 4, 1.0), (448, 2, 2, 0.0)])
def test_short_prompts(gpu, n, heads, kv_heads, spread):
    """Few queries, by CTAs of 8 and of 16, the lengths next to where the tensor cores begin to serve, and between there and 512 (the same oracle and
    bound)."""
    test_against_float64(gpu, n, heads, kv_heads, spread)


@pytest.mark.parametrize("n,kernels", [(191, 1), (192, 1), (223, 1), (224, 1), (511, 1), (512, 2), (513, 2)])
def test_where_the_tensor_cores_begin(gpu, n, kernels):
    """One launch on the CUDA cores, which up to here are the more exact ones for some inputs; then two, and scratch."""
    import torch
    q, k, v = inputs(n, 24, 4, n)
    out = torch.empty(n, 24, D, device="cuda")
    assert len(launches(lambda: gpu.attn(q, k, v, out, n, 24, 4, D, SCALE))) == kernels
    close(out, exact(q, k, v))


@pytest.mark.parametrize("n", [200, 300])
def test_short_prompts_of_positive_values(gpu, n):
    """Queries four times as large, so that a row's weights fall off steeply, and values of one sign: short prompts keep the exactness of fp32 sums
    (relative error seen on the CUDA cores at most 2.1e-7 and 2.6e-7; of a tensor core, which cuts each of the small terms off, 3.2e-7 and 3.3e-7)."""
    import torch
    q, k, v = inputs(n, 24, 4, 7)
    q, v = 4 * q, v.abs()
    out = torch.empty(n, 24, D, device="cuda")
    assert gpu.attn(q, k, v, out, n, 24, 4, D, SCALE) == 0
    want = exact(q, k, v)
    assert float((out.double() - want).norm() / want.norm()) < 2.9e-7


def signed_error(got, want):
    """Mean error in the direction of the result, relative to it."""
    want = want.double()
    return float(((got.double() - want) * want).sum() / (want * want).sum())


@pytest.mark.parametrize("n", [256, 2048])
def test_what_the_sums_lose(gpu, n):
    """The tensor core cuts sums off, which is put back in the mean and only where something was cut: rows of one key and rows whose softmax sits
    on one key are v to what a plane pair keeps of it (22 bits at least, 2^-23 at most lost, in the mean nothing: a tenth of 2^-22 is allowed), ones
    stay ones in the first row, and the rows of a prompt are right in the mean to 0.6e-7 (1.0e-7 - 1.6e-7 was cut off)."""
    import torch
    heads, kv_heads = 24, 4
    q, k, v = inputs(n, heads, kv_heads, 3)
    own = v.repeat_interleave(heads // kv_heads, 1)

    def run(q, k, v):
        out = torch.full((n, heads, D), float("nan"), device="cuda")
        assert gpu.attn(q, k, v, out, n, heads, kv_heads, D, SCALE) == 0
        return out
    out = run(q, k, v)
    assert float((out[0] - own[0]).abs().max()) <= 2 ** -23 * float(v.abs().max()) and abs(signed_error(out[0], own[0])) < 0.25e-7
    want = exact(q, k, v)
    for rows in (slice(16, 64), slice(64, n)):
        assert abs(signed_error(out[rows], want[rows])) < 0.6e-7, rows
    assert bool((run(q, k, torch.ones_like(v))[0] == 1).all())
    # a query that is ten times its own key: 160 against at most some 50 for any other
    one = run(10 * k.repeat_interleave(heads // kv_heads, 1), k, v)
    assert float((one - own).abs().max()) <= 2 ** -23 * float(v.abs().max()) and abs(signed_error(one, own)) < 0.25e-7


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


ROW_TOL = 3e-6      # of the row's OWN largest output: fp32 sums over up to 600 keys; the CUDA cores' worst row of these cases is 1.9e-6


def rows_close(got, want):
    err = (got.double() - want).abs().amax(-1) / want.abs().amax(-1)
    assert float(err.max()) <= ROW_TOL, (float(err.max()), int(err.max(-1).values.argmax()))


@pytest.mark.parametrize("weight", [True, False])
@pytest.mark.parametrize("at", [320, 351, 383])         # first, middle and last key of a tile
@pytest.mark.parametrize("x", [1e3, 1e5, 1e6, 1e8, 1e10, 1e12, 1e15])
def test_rows_do_not_depend_on_keys_they_do_not_see(gpu, x, at, weight):
    """One key whose v is x, in every dim or in one: the rows in front of it (they do not see it), behind it without a weight for it
    (its score is -100) and with one."""
    import torch
    n, heads, kv_heads = 600, 6, 2
    for dims in (slice(None), slice(200, 201)):
        q, k, v = inputs(n, heads, kv_heads, 9)
        v[at, :, dims] *= x
        if not weight:
            q[:, :, 0], k[:, :, 0] = 16.0, 0.0
            k[at, :, 0] = -100.0
        out = torch.empty(n, heads, D, device="cuda")
        assert gpu.attn(q, k, v, out, n, heads, kv_heads, D, SCALE) == 0
        rows_close(out, exact(q, k, v))
    assert gpu.device_status() == 0


@pytest.mark.parametrize("x", [1e3, 1e4, 1e5, 1e6, 1e9, 1e12])
@pytest.mark.parametrize("large", ["q", "k"])
def test_channels_that_the_other_side_does_not_use(gpu, x, large):
    import torch
    n, heads, kv_heads = 600, 6, 2
    q, k, v = inputs(n, heads, kv_heads, 10)
    a, b = (q, k) if large == "q" else (k, q)
    a[:, :, 7], b[:, :, 7] = x, 0.0
    out = torch.empty(n, heads, D, device="cuda")
    assert gpu.attn(q, k, v, out, n, heads, kv_heads, D, SCALE) == 0
    rows_close(out, exact(q, k, v))


@pytest.mark.parametrize("size", [1e-38, 1e-33, 1e-28, 1e17])
def test_values_of_any_size(gpu, size):
    """All of v very small or large, one dim of it, and tiles of large v whose small weights make them count as much as the rest."""
    import torch
    n, heads, kv_heads = 600, 6, 2
    for dims in (slice(None), slice(9, 10)):
        q, k, v = inputs(n, heads, kv_heads, 11)
        v[:, :, dims] *= size
        out = torch.empty(n, heads, D, device="cuda")
        assert gpu.attn(q, k, v, out, n, heads, kv_heads, D, SCALE) == 0
        want = exact(q, k, v)
        err = (out.double() - want)[:, :, dims].abs().amax(-1) / want[:, :, dims].abs().amax(-1).clamp_min(float(v[:, :, dims].abs().max()) * 0.02)
        assert float(err.max()) <= max(ROW_TOL, 2 ** -149 / size * 600), float(err.max())
    q, k, v = inputs(n, heads, kv_heads, 12)
    q[:, :, 0], k[:, :, 0] = 16.0, 0.0
    k[300:, :, 0] = -28.0
    v[300:] *= 1e12
    out = torch.empty(n, heads, D, device="cuda")
    assert gpu.attn(q, k, v, out, n, heads, kv_heads, D, SCALE) == 0
    rows_close(out, exact(q, k, v))


@pytest.mark.parametrize("how", ["reserve", "plain call"])
def test_captured_with_a_buffer(gpu, how):
    """A captured call on a stream that has a buffer gives the bits of a plain one, also when the stream's buffer has grown since: the
    graph keeps its own."""
    import torch
    n, heads, kv_heads = 800, 6, 1
    q, k, v = inputs(n, heads, kv_heads, 50)
    big = inputs(1700, heads, kv_heads, 51)
    want, out, out_big = (torch.empty(m, heads, D, device="cuda") for m in (n, n, 1700))
    assert gpu.attn(q, k, v, want, n, heads, kv_heads, D, SCALE) == 0
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        if how == "reserve":
            assert gpu.attn_reserve(n, kv_heads) == 0
        else:
            assert gpu.attn(q, k, v, out, n, heads, kv_heads, D, SCALE) == 0
        with torch.cuda.graph(graph, stream=side):
            assert gpu.attn(q, k, v, out, n, heads, kv_heads, D, SCALE) == 0
        assert gpu.attn(*big, out_big, 1700, heads, kv_heads, D, SCALE) == 0
    torch.cuda.current_stream().wait_stream(side)
    for _ in range(3):
        out.fill_(7.0)
        graph.replay()
        assert torch.equal(out, want)
    close(out_big, exact(*big))
    assert gpu.attn_reserve(0, 1) == 1 and gpu.attn_reserve(600, 0) == 1 and gpu.attn_reserve(100, 4) == 0
    del graph
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    assert gpu.gemm_release() == 0
    assert torch.cuda.mem_get_info()[0] > free0
    assert gpu.device_status() == 0


def test_buffers_are_bounded(gpu):
    """200 streams one after the other, destroyed each: never more than 16 buffers, and new streams get one again.  (Buffers of 25 MB,
    seen as device memory.)"""
    import ctypes
    import torch
    n, heads, kv_heads = 1536, 8, 8
    q, k, v = inputs(n, heads, kv_heads, 60)
    want = exact(q, k, v)
    rt = ctypes.CDLL("libcudart.so.12")
    out = torch.empty(n, heads, D, device="cuda")
    torch.cuda.synchronize()
    assert gpu.gemm_release() == 0
    free0, got = torch.cuda.mem_get_info()[0], set()
    for i in range(200):
        st = ctypes.c_void_p()
        assert rt.cudaStreamCreate(ctypes.byref(st)) == 0
        rc = gpu.lib().bonsai_p40_attn(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), n, heads, kv_heads, D, SCALE, st)
        torch.cuda.synchronize()
        assert rc == 0 and rt.cudaStreamDestroy(st) == 0
        if i % 20 == 0:
            close(out, want)
        got.add(free0 - torch.cuda.mem_get_info()[0])
    assert max(got) <= 16 * 32 << 20 and max(got) >= 16 * 24 << 20
    assert gpu.gemm_release() == 0
