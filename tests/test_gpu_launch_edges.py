"""Launches that start before their predecessor ends, and work cut into parts: what a call reads must be what the call in
front of it wrote (weights included), and the parts of a tile must add up wherever the cuts fall."""
import numpy as np
import pytest

from bonsai_b200 import synth

pytestmark = pytest.mark.gpu

REL_TOL = 1e-5      # the mat-vec's and mat-mul's bound: max |got - want| <= REL_TOL * max |want|


def dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("n_out,n_in", [(64, 1024), (1024, 5120), (5120, 17408)])
def test_calls_read_what_the_call_before_wrote(gpu, n_out, n_in):
    """Weights, inputs and scratch are written again between the calls, by a copy, by the library's own kernels and by the
    call in front; every result has the bits of the same call made alone."""
    import torch
    Ws = [dev(synth.pq2_0_weights(n_out, n_in, seed=s)) for s in range(2)]
    xs = [dev(synth.activations(n_in, seed=s)) for s in range(3)]
    sg = dev(synth.signs(n_in, seed=1))
    xq = torch.empty(n_in // 32 * 36, dtype=torch.uint8, device="cuda")
    rot = torch.empty(n_in, device="cuda")
    W, R, y = torch.empty_like(Ws[0]), torch.empty_like(Ws[0]), torch.empty(n_out, device="cuda")

    def step(i, sync):
        wait = torch.cuda.synchronize if sync else (lambda: None)
        out = []
        W.copy_(Ws[i % 2]); wait()
        assert gpu.linear(W, xs[i % 3], sg, y, xq, n_out, n_in) == 0; wait()
        out.append(y.clone()); wait()
        assert gpu.repack(W, R, n_out, n_in) == 0; wait()
        assert gpu.gemv_repack(R, rot, y, n_out, n_in) == 0; wait()     # rot: of the step before
        out.append(y.clone()); wait()
        assert gpu.fwht_quant(xs[(i + 1) % 3], sg, xq, rot, n_in) == 0; wait()
        assert gpu.gemv(W, xq, y, n_out, n_in) == 0; wait()
        out.append(y.clone()); wait()
        assert gpu.gemv_repack(R, rot, y, n_out, n_in) == 0; wait()
        out.append(y.clone()); wait()
        assert gpu.synth_pq2_0(W, 0, n_out * (n_in // 128), 7 + i) == 0; wait()
        assert gpu.gemv(W, xq, y, n_out, n_in) == 0; wait()
        out.append(y.clone()); wait()
        assert gpu.quant_activations(rot, xq, n_in) == 0; wait()
        assert gpu.gemv(W, xq, y, n_out, n_in) == 0; wait()
        out.append(y.clone()); wait()
        return out

    rot.copy_(xs[0])
    want = [step(i, True) for i in range(6)]
    rot.copy_(xs[0])
    got = [step(i, False) for i in range(6)]
    torch.cuda.synchronize()
    for i in range(6):
        for a, b in zip(want[i], got[i]):
            assert torch.equal(a, b), i
    assert gpu.device_status() == 0


@pytest.mark.parametrize("n_tok", [2, 5, 8, 9, 16])
@pytest.mark.parametrize("offset", [0, 4])      # of Xq in bytes: bulk copies or plain loads
def test_token_batches_read_what_the_call_before_wrote(gpu, n_tok, offset):
    """Weights, inputs and quantised blocks change between the mat-muls of 2 - 16 tokens: bits of the same calls made one by one."""
    import torch
    n_out, n_in = 1030, 5120
    Ws = [dev(synth.pq2_0_weights(n_out, n_in, seed=s)) for s in range(2)]
    Xs = [dev(synth.activations(n_in, seed=s, batch=n_tok)) for s in range(3)]
    sg, W = dev(synth.signs(n_in, seed=1)), torch.empty_like(Ws[0])
    Xq = torch.empty(n_in // 32 * 36 * n_tok + 16, dtype=torch.uint8, device="cuda")[offset:offset + n_in // 32 * 36 * n_tok]
    Y = torch.empty(n_out, n_tok, device="cuda")

    def step(i, sync):
        wait = torch.cuda.synchronize if sync else (lambda: None)
        out = []
        for rotate in (True, False):
            W.copy_(Ws[(i + rotate) % 2]); wait()
            assert gpu.quant_batch(Xs[i % 3], sg, Xq, n_in, n_tok, rotate) == 0; wait()
            assert gpu.gemm(W, Xq, Y, n_out, n_in, n_tok) == 0; wait()
            out.append(Y.clone()); wait()
        return out

    want = [step(i, True) for i in range(6)]
    got = [step(i, False) for i in range(6)]
    for i in range(6):
        for a, b in zip(want[i], got[i]):
            assert torch.equal(a, b), i
    assert gpu.device_status() == 0


@pytest.mark.parametrize("n_out,n_in,n_tok", [
    (128, 17408, 17), (129, 17408, 64), (5120, 17408, 37), (1000, 5120, 33), (2000, 17408, 95), (300, 17408, 96), (1030, 9216, 130), (6000, 5120, 257)])
@pytest.mark.parametrize("tile", [0, 64, 128])
def test_parts_of_a_tile_add_up(gpu, port, tile, n_out, n_in, n_tok):
    """Tiles of the many-token mat-mul in one to five parts: as the call divides them, and on each tile width."""
    import torch
    W = synth.pq2_0_weights(n_out, n_in, seed=n_tok)
    Xq = port.quantize_batch_chunk_major(synth.activations(n_in, seed=n_out, batch=n_tok))
    Wd, Xd = dev(W), dev(Xq)
    Y = [torch.full((n_out, n_tok), float("nan"), device="cuda") for _ in range(2)]
    try:
        assert gpu.set_option("gemm_tile", tile) == 0
        for y in Y:
            assert gpu.gemm(Wd, Xd, y, n_out, n_in, n_tok) == 0
    finally:
        gpu.set_option("gemm_tile", 0)
    assert torch.equal(Y[0], Y[1])
    rows = np.unique(np.concatenate([np.arange(min(n_out, 64)), np.arange(max(0, n_out - 64), n_out), np.linspace(0, n_out - 1, 64).astype(np.int64)]))
    row_bytes = n_in // 128 * 34
    want = port.gemm(np.concatenate([W[r * row_bytes:(r + 1) * row_bytes] for r in rows]), Xq, len(rows), n_in, n_tok, threads=8)
    err = np.abs(Y[0].cpu().numpy()[rows] - want).max()
    assert err <= REL_TOL * np.abs(want).max(), (err, np.abs(want).max())
    assert gpu.device_status() == 0


@pytest.mark.parametrize("n", [124, 128, 8188, 8189, 8192, 8193, 8196, 65537])
def test_rmsnorm_rows_held_and_not(gpu, port, n):
    """Rows on both sides of what a CTA keeps in registers (8192), in place and not, with 16-byte accesses and without."""
    import torch
    rng = np.random.default_rng(n)
    x, w = rng.uniform(-2, 2, size=(3, n)).astype(np.float32), rng.uniform(0.5, 1.5, size=n).astype(np.float32)
    want = port.rmsnorm(x, w, 1e-6)
    y, xd, wd = torch.empty(3, n, device="cuda"), dev(x), dev(w)
    assert gpu.rmsnorm(xd, wd, y, 3, n, 1e-6) == 0
    assert np.abs(y.cpu().numpy() - want).max() <= REL_TOL * np.abs(want).max()
    odd = torch.empty(3 * n + 1, device="cuda")[1:]
    assert gpu.rmsnorm(xd, wd, odd, 3, n, 1e-6) == 0
    assert torch.equal(odd.view(3, n), y)
    assert gpu.rmsnorm(xd, wd, xd, 3, n, 1e-6) == 0
    assert torch.equal(xd, y)


def test_threads_on_their_per_thread_streams(gpu):
    """Mat-muls cut into parts, from three host threads at once on cudaStreamPerThread (one handle, a stream per thread), with sizes that
    make the scratch grow in between: every result has the bits of the same call made alone."""
    import ctypes
    import threading
    import torch
    per_thread = ctypes.c_void_p(2)
    n_in, cases = 17408, [(128, 17), (640, 37), (300, 64)]
    data = []
    for i, (n_out, n_tok) in enumerate(cases):
        W, Xq = dev(synth.pq2_0_weights(n_out, n_in, seed=i)), torch.empty(n_in // 32 * 36 * 130, dtype=torch.uint8, device="cuda")
        assert gpu.quant_batch(dev(synth.activations(n_in, seed=i, batch=130)), None, Xq, n_in, 130, True) == 0
        toks = [n_tok, n_tok + 3, 2 * n_tok]
        data.append((W, Xq, n_out, toks, [[torch.zeros(n_out, t, device="cuda") for t in toks] for _ in range(21)]))
    torch.cuda.synchronize()
    fn = gpu.lib().bonsai_p40_gemm

    def calls(i, rounds):
        W, Xq, n_out, toks, Y = data[i]
        for r in rounds:
            for t, y in zip(toks, Y[r]):
                failed.append(fn(W.data_ptr(), Xq.data_ptr(), y.data_ptr(), n_out, n_in, t, per_thread))

    failed = []
    for i in range(len(cases)):          # alone
        calls(i, [0])
        torch.cuda.synchronize()
    threads = [threading.Thread(target=calls, args=(i, range(1, 21))) for i in range(len(cases))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not any(failed)
    for _, _, _, toks, Y in data:
        for r in range(1, 21):
            for a, b in zip(Y[0], Y[r]):
                assert torch.equal(a, b), r
    assert gpu.device_status() == 0


def test_plain_launches(gpu):
    """Option "overlap" = 0: the bits of the default, also with "pdl" = 1 beside it."""
    import torch
    n_out, n_in, n = 640, 5120, 300
    W, x, sg = dev(synth.pq2_0_weights(n_out, n_in, seed=3)), dev(synth.activations(n_in, seed=3)), dev(synth.signs(n_in, seed=3))
    kv = gpu.KVCache(n)
    k, q = torch.randn(n, 4, 256, device="cuda"), torch.randn(24, 256, device="cuda")

    def step():
        xq, y, out = torch.empty(n_in // 32 * 36, dtype=torch.uint8, device="cuda"), torch.empty(n_out, device="cuda"), torch.empty(24, 256, device="cuda")
        assert gpu.linear(W, x, sg, y, xq, n_out, n_in) == 0
        assert kv.append_batch(3, 0, n, k, k) == 0 and kv.attn_decode(3, n - 1, q, out) == 0
        return y, out

    want = step()
    try:
        for pdl in (0, 1):
            assert gpu.set_option("overlap", 0) == 0 and gpu.set_option("pdl", pdl) == 0
            assert all(torch.equal(a, b) for a, b in zip(want, step()))
    finally:
        gpu.set_option("overlap", 1), gpu.set_option("pdl", 0)
    kv.close()


@pytest.mark.parametrize("odd", [0, 1])
@pytest.mark.parametrize("n", [60, 128, 1000, 1024, 1028, 2048, 3072, 3076, 5120, 5124, 8192, 8196])
def test_rmsnorm_rows_and_forms(gpu, port, n, odd):
    """Row counts on both sides of the forms' lines (two, three, four and eight rows per SM), in place too: every row has the bits of the
    same row alone, and the first is the host's within the bound."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(n)
    w = torch.randn(n, generator=g, device="cuda")
    for rows in (1, 296, 297, 444, 445, 592, 593, 1185):
        x = torch.empty(rows * n + 1, device="cuda")[odd:rows * n + odd]
        x.copy_(torch.randn(rows * n, generator=g, device="cuda"))
        y = torch.full((rows, n), float("nan"), device="cuda")
        assert gpu.rmsnorm(x, w, y, rows, n, 1e-6) == 0
        for r in (0, rows // 2, rows - 1):
            one = torch.empty(n, device="cuda")
            assert gpu.rmsnorm(x[r * n:(r + 1) * n].clone(), w, one, 1, n, 1e-6) == 0
            assert torch.equal(y[r], one), (rows, r)
        want = port.rmsnorm(x[:n].cpu().numpy().reshape(1, n), w.cpu().numpy(), 1e-6)
        assert np.abs(y[0].cpu().numpy() - want).max() <= REL_TOL * np.abs(want).max()
        assert gpu.rmsnorm(x, w, x, rows, n, 1e-6) == 0
        assert torch.equal(x.view(rows, n), y), rows


@pytest.mark.parametrize("odd", [0, 1])
@pytest.mark.parametrize("blocks", [1, 5, 296, 297, 298, 592, 593, 888, 889, 1480, 1481, 2664, 2665, 4737, 9473])
def test_rotation_and_quantiser_forms(gpu, blocks, odd):
    """Block counts on both sides of the forms' lines and of the overlap's: every block's bytes and rotated values are those of the block
    alone, in one vector and in a batch of tokens."""
    import torch
    N, Q = 1024, 1152
    g = torch.Generator(device="cuda").manual_seed(blocks)
    x = torch.empty(blocks * N + 1, device="cuda")[odd:blocks * N + odd]
    x.copy_(torch.randn(blocks * N, generator=g, device="cuda"))
    sg = torch.randn(blocks * N, generator=g, device="cuda").sign()
    ones = torch.randn(N, generator=g, device="cuda").sign()
    new = lambda n, t=torch.float32: torch.zeros(n, dtype=t, device="cuda")
    xq, both, xb, xn, rot, inplace = new(blocks * Q, torch.uint8), new(blocks * Q, torch.uint8), new(blocks * Q, torch.uint8), new(blocks * Q, torch.uint8), new(blocks * N), x.clone()
    assert gpu.fwht_quant(x, sg, xq, None, blocks * N) == 0 and gpu.fwht_quant(x, sg, both, rot, blocks * N) == 0
    assert gpu.fwht(inplace, sg, blocks * N) == 0
    assert gpu.quant_batch(x, ones, xb, N, blocks, True) == 0 and gpu.quant_batch(x, None, xn, N, blocks, False) == 0
    assert torch.equal(both, xq) and torch.equal(inplace, rot)
    xb, xn = xb.view(32, blocks, 36), xn.view(32, blocks, 36)
    for b in {0, 1 % blocks, blocks // 2, blocks - 1}:
        one, q1, r1, part = x[b * N:(b + 1) * N].clone(), new(Q, torch.uint8), new(N), sg[b * N:(b + 1) * N].clone()
        assert gpu.fwht_quant(one, part, q1, r1, N) == 0
        assert torch.equal(xq[b * Q:(b + 1) * Q], q1) and torch.equal(rot[b * N:(b + 1) * N], r1), b
        assert gpu.fwht_quant(one, ones, q1, None, N) == 0
        assert torch.equal(xb[:, b].reshape(-1), q1), b
        assert gpu.quant_activations(one, q1, N) == 0
        assert torch.equal(xn[:, b].reshape(-1), q1), b


@pytest.mark.parametrize("n_in,n_tok", [(1024, 148), (1024, 149), (3072, 98), (3072, 99), (5120, 61)])
def test_rotation_of_a_batch_on_both_sides_of_a_warp_per_block(gpu, port, n_in, n_tok):
    """Blocks of several per token through both forms of the rotation: the host's bytes, and of a block with an infinity or a NaN (which the
    rotation spreads over it) those of the block alone; rotated in place as one vector."""
    import torch
    X = synth.activations(n_in, seed=n_tok, batch=n_tok) * 1.7
    sg = synth.signs(n_in, seed=n_in)
    want = port.quantize_batch_chunk_major(np.stack([port.fwht_blocks(X[t], sg) for t in range(n_tok)]))
    x, s, xq = torch.from_numpy(X).cuda(), torch.from_numpy(sg).cuda(), torch.zeros(want.size, dtype=torch.uint8, device="cuda")
    assert gpu.quant_batch(x, s, xq, n_in, n_tok, True) == 0
    assert np.array_equal(xq.cpu().numpy(), want)
    flat, signs = x.reshape(-1).clone(), s.repeat(n_tok)
    assert gpu.fwht(flat, signs, n_in * n_tok) == 0
    assert np.array_equal(flat.cpu().numpy(), np.concatenate([port.fwht_blocks(X[t], sg) for t in range(n_tok)]))
    x[5, 7], x[n_tok - 1, n_in - 1] = float("nan"), float("inf")
    assert gpu.quant_batch(x, s, xq, n_in, n_tok, True) == 0
    one = torch.zeros(n_in // 32 * 36, dtype=torch.uint8, device="cuda")
    for t in (4, 5, n_tok - 1):
        assert gpu.quant_batch(x[t:t + 1].clone(), s, one, n_in, 1, True) == 0
        assert torch.equal(xq.view(n_in // 32, n_tok, 36)[:, t].reshape(-1), one), t


@pytest.mark.parametrize("n_rows,n", [(1, 1024), (1, 5120), (1, 8192), (1, 17408), (2, 1024), (2, 5120), (37, 1028), (148, 1000), (149, 1024), (8, 17408), (9, 17408), (148, 1024)])
def test_small_operators_in_front_of_their_projection(gpu, n_rows, n):
    """RMSNorm and SwiGLU on both sides of what lets the next launch in at once, over and over into the same buffers in front of a projection (of
    rows: of a quantiser): the bits of plain launches."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(n_rows * n)
    xs = [torch.randn(n_rows * n, generator=g, device="cuda") for _ in range(3)]
    w, n_out = torch.randn(n, generator=g, device="cuda"), 64
    W = torch.empty(n_out * (n // 128) * 34, dtype=torch.uint8, device="cuda")
    assert n_rows > 1 or gpu.synth_pq2_0(W, 0, n_out * (n // 128), n) == 0
    h, y, xq = torch.empty(n_rows * n, device="cuda"), torch.empty(n_out, device="cuda"), torch.empty(n // 32 * 36 * n_rows, dtype=torch.uint8, device="cuda")

    def steps():
        out = []
        for i in range(6):
            call = (lambda: gpu.rmsnorm(xs[i % 3], w, h, n_rows, n, 1e-6)) if i < 3 else (lambda: gpu.swiglu(xs[i % 3], xs[(i + 1) % 3], h, n_rows * n))
            assert call() == 0
            if n_rows == 1:
                assert gpu.linear(W, h, None, y, xq, n_out, n) == 0
            elif n % 32 == 0:
                assert gpu.quant_batch(h, None, xq, n, n_rows, False) == 0
            out += [h.clone(), y.clone() if n_rows == 1 else xq.clone()]
        return out
    y.zero_(), xq.zero_()
    got = steps()
    try:
        assert gpu.set_option("overlap", 0) == 0
        want = steps()
    finally:
        gpu.set_option("overlap", 1)
    assert all(torch.equal(a.view(torch.int32), b.view(torch.int32)) if a.dtype == torch.float32 else torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("n_out,n_in,n_tok", [(1000, 1024, 17), (5120, 5120, 37), (5120, 17408, 37), (17408, 5120, 130)])
def test_mat_mul_reads_the_weights_written_in_front_of_it(gpu, n_out, n_in, n_tok):
    """The many-token mat-mul fetches its weights while its activations are split: they are written again in front of each call, as are the activations,
    and results have the bits of calls made alone."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(n_out + n_tok)
    xs = [torch.randn(n_tok * n_in, generator=g, device="cuda") for _ in range(2)]
    n = n_out * (n_in // 128)
    W = torch.empty(n * 34, dtype=torch.uint8, device="cuda")
    xq = torch.empty(n_in // 32 * 36 * n_tok, dtype=torch.uint8, device="cuda")
    y = torch.empty(n_tok * n_out, device="cuda")

    def steps(wait):
        out = []
        for i in range(6):
            for call in (lambda: gpu.quant_batch(xs[i % 2], None, xq, n_in, n_tok, True), lambda: gpu.synth_pq2_0(W, 0, n, i), lambda: gpu.gemm(W, xq, y, n_out, n_in, n_tok)):
                assert call() == 0
                wait()
            out.append(y.clone())
            wait()
        return out
    want = steps(torch.cuda.synchronize)
    got = steps(lambda: None)
    assert all(torch.equal(a, b) for a, b in zip(want, got)) and not torch.equal(want[0], want[2])
    assert gpu.device_status() == 0
