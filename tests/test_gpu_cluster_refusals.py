"""Calls that launch clusters of CTAs where a device lets them, when a launch of clusters is refused: the call runs in the form that needs none
with what it has enqueued so far, and later calls do not try again.  The kernels of a call are read from a capture of it."""
import numpy as np
import pytest

from bonsai_b200 import synth
from captured import launches, scratch_given_back  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.fixture
def refuse(gpu):
    assert gpu.set_option("refuse_clusters", 0) == 0
    yield lambda n: gpu.set_option("refuse_clusters", n)
    gpu.set_option("refuse_clusters", 0)


def test_matmul(gpu, port, scratch_given_back, refuse):
    """Two launches, the activations split once: refused in the capture, refused in the call in front of it and remembered, and not refused."""
    import torch
    n_out, n_in, n_tok = 300, 2048, 200
    W, X = synth.pq2_0_weights(n_out, n_in, seed=1), synth.activations(n_in, seed=2, batch=n_tok)
    Xq = port.quantize_batch_chunk_major(X)
    Wd, Xqd, Y = torch.from_numpy(W).cuda(), torch.from_numpy(Xq).cuda(), torch.zeros(n_out, n_tok, device="cuda")
    want = port.gemm(W, Xq, n_out, n_in, n_tok, threads=8)
    call = lambda: gpu.gemm(Wd, Xqd, Y, n_out, n_in, n_tok)

    def right():
        ok = np.abs(Y.cpu().numpy() - want).max() <= 1e-5 * np.abs(want).max()
        Y.fill_(float("nan"))
        return ok

    try:
        assert gpu.set_option("gemm_tile", 128) == 0
        assert launches(call) == [1, 2] and right()
        assert launches(call, lambda: refuse(1)) == [1, 1] and right()
        assert refuse(0) == 0
        assert launches(call) == [1, 2] and right()
        assert refuse(1) == 0
        assert launches(call) == [1, 1] and right()
        assert call() == 0 and right()
    finally:
        gpu.set_option("gemm_tile", 0)
    assert gpu.device_status() == 0


# (how many fours find an SM for each CTA is the device's: 33 on the one that was looked at)
@pytest.mark.parametrize("n_out,n_in,forms", [(400, 17408, [4]), (400, 5120, [4]), (1024, 5120, [4, 1]), (1060, 5120, [4, 1]), (5120, 17408, [2]), (4160, 9216, [1]),
                                              (4160, 10240, [4, 1]), (4150, 12288, [4, 2]), (5120, 11264, [1]), (700, 4096, [1])])
def test_repacked_matvec(gpu, refuse, n_out, n_in, forms):
    """Fours as far as they find an SM for each CTA, pairs, single CTAs; one launch, and the same bits, refused or not."""
    import torch
    W = torch.from_numpy(synth.pq2_0_weights(n_out, n_in, seed=3)).cuda()
    Wr, xq, x = torch.zeros_like(W), torch.zeros(n_in // 32 * 36, dtype=torch.uint8, device="cuda"), torch.from_numpy(synth.activations(n_in, seed=4)).cuda()
    y, want = torch.zeros(n_out, device="cuda"), torch.zeros(n_out, device="cuda")
    assert gpu.repack(W, Wr, n_out, n_in) == 0 and gpu.quant_activations(x, xq, n_in) == 0 and gpu.gemv(W, xq, want, n_out, n_in) == 0
    call = lambda: gpu.gemv_repack(Wr, x, y, n_out, n_in)

    def right():
        ok = torch.equal(y, want)
        y.fill_(float("nan"))
        return ok

    (ctas,) = launches(call)
    assert ctas in forms and right()
    if ctas > 1:
        assert launches(call, lambda: refuse(1)) == [1] and right()
        assert launches(call) == [1] and right()
        assert refuse(0) == 0
        assert launches(call) == [ctas] and right()
    assert gpu.device_status() == 0
