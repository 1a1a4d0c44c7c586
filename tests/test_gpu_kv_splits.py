"""Decode attention over the K/V cache at the positions where its splits change: the first and last position of a tile, of a
warp's share of one, one cluster against several, more clusters than are resident; and what the launches share.

Against float64 on the cache's own bytes (quantised query x cache, softmax, value sum).  Bound: 2e-6 of the largest output:
scores are exact integers with fp32 scales, weights carry 22 bits, sums are fp32."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N_LAYERS, N_KV, N_HEADS, D = 16, 4, 24, 256
REL_TOL = 2e-6


def cache_tensors(kv):
    import torch

    class Raw:
        def __init__(self, ptr, n):
            self.__cuda_array_interface__ = {"shape": (n,), "typestr": "|u1", "data": (int(ptr), False), "version": 3}
    kp, vp, n = kv.arrays()
    return [torch.as_tensor(Raw(p, n), device="cuda") for p in (kp, vp)]


def dequantise(raw, cap, layer, kvh, n):
    import torch
    at = (layer * N_KV + kvh) * cap * 272
    b = raw[at:at + n * 272].view(n, 8, 34)
    d = b[:, :, :2].contiguous().view(torch.float16).double()
    return (d * b[:, :, 2:].contiguous().view(torch.int8).double()).view(n, D)


def exact(port, kv, cap, layer, n, q):
    import torch
    K, V = cache_tensors(kv)
    qd = np.stack([port.kv_dequantize_row(port.kv_quantize_row(row)) for row in q.cpu().numpy()])
    qd = torch.from_numpy(qd).cuda().double()
    out = torch.empty(N_HEADS, D, dtype=torch.float64, device="cuda")
    for h in range(N_HEADS):
        s = dequantise(K, cap, layer, h // 6, n) @ qd[h] * 0.0625
        out[h] = torch.softmax(s, 0) @ dequantise(V, cap, layer, h // 6, n)
    return out


def fill(kv, layer, n, seed, spread):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    k, v = torch.randn(n, N_KV, D, generator=g, device="cuda"), torch.randn(n, N_KV, D, generator=g, device="cuda")
    if spread:                      # rows of V of very different size
        v = v * torch.exp(2 * torch.randn(n, N_KV, 1, generator=g, device="cuda"))
    assert kv.append_batch(layer, 0, n, k, v) == 0
    return torch.randn(N_HEADS, D, generator=g, device="cuda")


@pytest.mark.parametrize("n", [1, 15, 16, 17, 63, 64, 65, 127, 128, 129, 1023, 1024, 1025, 2047, 2048, 2049, 4100, 13311, 13312, 14337, 40001])
@pytest.mark.parametrize("spread", [0, 1])
def test_against_float64(gpu, port, n, spread):
    import torch
    cap, layer = n + 3, 5
    kv = gpu.KVCache(cap)
    q = fill(kv, layer, n, n, spread)
    out = torch.full((N_HEADS, D), float("nan"), device="cuda")
    for _ in range(2):              # the second call finds the counters as the first one left them
        assert kv.attn_decode(layer, n - 1, q, out) == 0
    want = exact(port, kv, cap, layer, n, q)
    err, top = float((out.double() - want).abs().max()), float(want.abs().max())
    assert err <= REL_TOL * top, (err, top)
    assert gpu.device_status() == 0
    kv.close()


@pytest.mark.parametrize("n", [70, 1000, 5000])
@pytest.mark.parametrize("size", [1e-4, 1e1, 1e2, 1e3, 1e5, 1e6])
def test_scales_far_apart(gpu, port, n, size):
    """One position with a very large (or small) V: in one dim or all, without weight (its score is -225) or with.  Each head to 2e-6
    of its own largest output in the blocks that the large values leave alone, and in all of them."""
    import torch
    layer, at = 5, n // 3
    for dims in (slice(None), slice(40, 41)):
        for weight in (False, True):
            kv = gpu.KVCache(n)
            g = torch.Generator(device="cuda").manual_seed(n)
            k, v = torch.randn(n, N_KV, D, generator=g, device="cuda"), torch.randn(n, N_KV, D, generator=g, device="cuda") * 0.06
            q = torch.randn(N_HEADS, D, generator=g, device="cuda")
            v[at, :, dims] = size
            if not weight:
                q[:, 0], k[:, :, 0], k[at, :, 0] = 60.0, 0.0, -60.0
            assert kv.append_batch(layer, 0, n, k, v) == 0
            out = torch.full((N_HEADS, D), float("nan"), device="cuda")
            assert kv.attn_decode(layer, n - 1, q, out) == 0
            err, want = out.double(), exact(port, kv, n, layer, n, q)
            err = (err - want).abs()
            for block in (slice(None), slice(64, None)):
                assert float((err[:, block].amax(1) / want[:, block].abs().amax(1)).max()) <= REL_TOL
            kv.close()
    assert gpu.device_status() == 0


def test_infinite_scale(gpu, port):
    """A V block past fp16's range: infinities with their signs where its values are not 0, NaN where they are, nothing else touched."""
    import torch
    n, layer = 1500, 2
    kv = gpu.KVCache(n)
    q = fill(kv, layer, n, 3, 0)
    row = torch.randn(2, 1, N_KV, D, generator=torch.Generator(device="cuda").manual_seed(4), device="cuda")
    row[1, 0, 1, 3], row[1, 0, 1, 4], row[1, 0, 1, 40] = 1e7, -1e7, 1e6
    assert kv.append(layer, 700, row[0], row[1]) == 0
    out = torch.full((N_HEADS, D), float("nan"), device="cuda")
    assert kv.attn_decode(layer, n - 1, q, out) == 0
    want = exact(port, kv, n, layer, n, q)
    hit = out[6:12]
    assert bool((hit[:, 3] == float("inf")).all()) and bool((hit[:, 4] == -float("inf")).all())
    assert bool(torch.isnan(hit[:, [d for d in range(32) if d not in (3, 4)]]).all())
    assert float((hit[:, 32:].double() - want[6:12, 32:]).abs().max()) <= REL_TOL * float(want[6:12, 32:].abs().max())
    rest = [h for h in range(N_HEADS) if not 6 <= h < 12]
    assert float((out[rest].double() - want[rest]).abs().max()) <= REL_TOL * float(want[rest].abs().max())
    kv.close()


def test_layers_on_streams_of_their_own(gpu):
    """Layers have their own records and counters: decoded at the same time on different streams they give the bits that
    they give one after the other."""
    import torch
    n = 9000
    kv = gpu.KVCache(n)
    qs = [fill(kv, layer, n, layer, 0) for layer in range(4)]
    want = [torch.empty(N_HEADS, D, device="cuda") for _ in range(4)]
    for layer in range(4):
        assert kv.attn_decode(layer, n - 1, qs[layer], want[layer]) == 0
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(4)]
    got = [torch.empty(N_HEADS, D, device="cuda") for _ in range(4)]
    torch.cuda.synchronize()
    for _ in range(20):
        for layer, st in enumerate(streams):
            with torch.cuda.stream(st):
                assert kv.attn_decode(layer, n - 1, qs[layer], got[layer]) == 0
    torch.cuda.synchronize()
    for layer in range(4):
        assert torch.equal(got[layer], want[layer]), layer
    kv.close()


def test_append_at_odd_offsets(gpu):
    """Rows at any float address store the bytes of rows at an aligned one."""
    import torch
    kv, cap = gpu.KVCache(40), 40
    g = torch.Generator(device="cuda").manual_seed(1)
    k, v = torch.randn(37, N_KV, D, generator=g, device="cuda"), torch.randn(37, N_KV, D, generator=g, device="cuda")
    odd = [torch.empty(t.numel() + 1, device="cuda") for t in (k, v)]
    for o, t in zip(odd, (k, v)):
        o[1:].copy_(t.view(-1))
    assert kv.append_batch(2, 3, 37, k, v) == 0 and kv.append_batch(3, 3, 37, odd[0][1:], odd[1][1:]) == 0
    for raw in cache_tensors(kv):
        for h in range(N_KV):
            a, b = ((layer * N_KV + h) * cap * 272 + 3 * 272 for layer in (2, 3))
            assert torch.equal(raw[a:a + 37 * 272], raw[b:b + 37 * 272]), h
    kv.close()


@pytest.mark.parametrize("n", [16, 65, 512, 513, 1024, 1025, 3071, 3072])
def test_query_and_output_at_odd_offsets(gpu, n):
    """A query that is not 16-byte aligned is read by words, outputs are stored by words: the bits of aligned ones."""
    import torch
    kv = gpu.KVCache(n)
    q = fill(kv, 3, n, n, 1)
    odd = torch.empty(q.numel() + 1, device="cuda")
    odd[1:].copy_(q.view(-1))
    out, at = torch.full((N_HEADS * D,), float("nan"), device="cuda"), torch.full((N_HEADS * D + 2,), float("nan"), device="cuda")
    assert kv.attn_decode(3, n - 1, q, out) == 0 and kv.attn_decode(3, n - 1, odd[1:], at[1:-1]) == 0
    assert torch.equal(out, at[1:-1]) and bool(torch.isnan(at[[0, -1]]).all())
    kv.close()


def test_create_does_not_wait_for_the_stream(gpu):
    """A cache is made while the caller's stream is busy (a kernel of a tenth of a second); decoding on another stream at once finds its
    counters zero."""
    import torch
    gpu.KVCache(16).close()
    busy, other, done = torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.Event()
    torch.cuda.synchronize()
    with torch.cuda.stream(busy):
        torch.cuda._sleep(200_000_000)
        done.record()
        kv = gpu.KVCache(3000)
        waited = done.query()
    with torch.cuda.stream(other):
        q, out = fill(kv, 1, 3000, 7, 0), torch.full((2, N_HEADS, D), float("nan"), device="cuda")
        assert kv.attn_decode(1, 2999, q, out[0]) == 0 and kv.attn_decode(1, 2999, q, out[1]) == 0
    torch.cuda.synchronize()
    assert not waited
    assert bool(torch.isfinite(out).all()) and torch.equal(out[0], out[1])
    kv.close()
