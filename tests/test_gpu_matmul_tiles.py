"""The fp16 tensor-core mat-mul at the edges of its tiles: every width that a tile of up to 64 tokens (one CTA, steps of 16) or 128 (a pair
of CTAs, steps of 32) can have, one token beside each, rows that leave a tile or a pair's second CTA empty, tiles whose blocks several
CTAs share, more tiles than CTAs; in the form that the call picks by itself, and in each.  Per token within 1e-5 of its largest |y| in the host's loop: a row's sum of 2 n_in products in fp32 differs by
less than 1e-6 of that from any other order."""
import numpy as np
import pytest

from bonsai_b200 import synth
from captured import capture, launches, pointer_argument, scratch_given_back  # noqa: F401

pytestmark = pytest.mark.gpu


def check(gpu, port, n_out, n_in, n_tok, tile):
    import torch
    W = synth.pq2_0_weights(n_out, n_in, seed=n_tok)
    X = synth.activations(n_in, seed=n_out, batch=n_tok)
    X[::5] *= 300.0
    Xq = port.quantize_batch_chunk_major(X)
    Wd, Xqd = torch.from_numpy(W).cuda(), torch.from_numpy(Xq).cuda()
    flat = torch.full((n_out * n_tok + 64,), 5.0, device="cuda")        # nothing is written behind Y
    Y, again = flat[:n_out * n_tok].view(n_out, n_tok), torch.full((n_out, n_tok), 6.0, device="cuda")
    try:
        assert gpu.set_option("gemm_path", 1) == 0 and gpu.set_option("gemm_tile", tile) == 0
        assert gpu.gemm(Wd, Xqd, Y, n_out, n_in, n_tok) == 0
        assert gpu.gemm(Wd, Xqd, again, n_out, n_in, n_tok) == 0
        torch.cuda.synchronize()
    finally:
        gpu.set_option("gemm_path", -1)
        gpu.set_option("gemm_tile", 0)
    assert gpu.device_status() == 0
    assert torch.equal(Y, again) and (flat[n_out * n_tok:] == 5.0).all()
    rows = np.unique(np.concatenate([np.arange(min(n_out, 200)), np.linspace(0, n_out - 1, 120).astype(np.int64)]))
    row_bytes = n_in // 128 * 34
    want = port.gemm(np.concatenate([W[r * row_bytes:(r + 1) * row_bytes] for r in rows]), Xq, len(rows), n_in, n_tok, threads=8)
    err = np.abs(Y.cpu().numpy()[rows] - want).max(axis=0)
    assert (err <= 1e-5 * np.maximum(np.abs(want).max(axis=0), 1e-30)).all(), err


@pytest.mark.parametrize("n_out,n_in,n_tok", [(128, 1024, t) for t in (17, 32, 33, 48, 49, 63, 64, 65, 81, 95, 96, 97, 127, 128, 129, 161, 193, 257)] +
                         [(1, 2048, 40), (129, 3072, 40), (127, 1024, 100), (128, 2048, 100), (129, 1024, 100), (257, 2048, 130), (385, 6144, 97),
                          (300, 17408, 37), (520, 17408, 160), (19000, 1024, 70), (9700, 1024, 300), (5120, 5120, 33)])
def test_tile_edges(gpu, port, n_out, n_in, n_tok):
    check(gpu, port, n_out, n_in, n_tok, 0)


@pytest.mark.parametrize("tile", [64, 128])
@pytest.mark.parametrize("n_out,n_in,n_tok", [(128, 1024, t) for t in (1, 16, 17, 31, 32, 33, 64, 65, 95, 96, 97, 128, 129, 192, 193, 257)] +
                         [(1, 2048, 40), (127, 1024, 100), (129, 1024, 100), (255, 1024, 96), (257, 2048, 130), (300, 17408, 96), (1030, 9216, 130),
                          (385, 6144, 97), (19000, 1024, 70)])
def test_edges_of_each_tile(gpu, port, n_out, n_in, n_tok, tile):
    check(gpu, port, n_out, n_in, n_tok, tile)


# (4000 x 17408 at 65 tokens: four parts per tile; 5120 x 17408 at 128: five; 2048 x 5120 at 577: three; the others whole tiles in turn)
@pytest.mark.parametrize("n_out,n_in,n_tok", [(4000, 17408, 65), (5120, 17408, 128), (2048, 5120, 577), (6000, 5120, 257), (12288, 1024, 300)])
def test_calls_that_take_pairs_by_themselves(gpu, port, scratch_given_back, n_out, n_in, n_tok):
    import torch
    W, Xq = torch.zeros(n_out * n_in // 128 * 34, dtype=torch.uint8, device="cuda"), torch.zeros(n_in // 32 * 36 * n_tok, dtype=torch.uint8, device="cuda")
    Y = torch.empty(n_out, n_tok, device="cuda")
    assert launches(lambda: gpu.gemm(W, Xq, Y, n_out, n_in, n_tok)) == [1, 2]
    check(gpu, port, n_out, n_in, n_tok, 0)

@pytest.mark.parametrize("n_out,n_in,n_tok,tile", [(300, 17408, 40, 64), (300, 17408, 96, 128), (5120, 17408, 37, 0)])
def test_flags_that_an_earlier_launch_left_raised(gpu, port, scratch_given_back, n_out, n_in, n_tok, tile):
    """A launch whose wait for a part ran out may leave that part's flag raised (all of them here, by a memset): the next calls on the same
    scratch, and replays of a captured one, wait for parts of their own."""
    import torch
    from cuda.bindings import runtime as rt
    X = [torch.from_numpy(port.quantize_batch_chunk_major(synth.activations(n_in, seed=s, batch=n_tok))).cuda() for s in range(2)]
    W, Xq = torch.from_numpy(synth.pq2_0_weights(n_out, n_in, seed=n_tok)).cuda(), X[0].clone()
    Y, want = torch.zeros(n_out, n_tok, device="cuda"), []
    call = lambda: gpu.gemm(W, Xq, Y, n_out, n_in, n_tok)
    try:
        assert gpu.set_option("gemm_path", 1) == 0 and gpu.set_option("gemm_tile", tile) == 0
        graph, kernels, st = capture(call)
        flags = pointer_argument(kernels[1], 4)
        with torch.cuda.stream(st):
            for x in X:
                Xq.copy_(x)
                assert call() == 0
                want.append(Y.clone())
            for again in (call, lambda: graph.replay() or 0):
                for i in range(4):
                    assert int(rt.cudaMemsetAsync(flags, 1, 148 * 16 * 4, st.cuda_stream)[0]) == 0
                    Xq.copy_(X[i % 2])
                    assert again() == 0
                    assert torch.equal(Y, want[i % 2]), i
        torch.cuda.synchronize()
    finally:
        gpu.set_option("gemm_path", -1)
        gpu.set_option("gemm_tile", 0)
    assert gpu.device_status() == 0
