"""fp32 inputs of a list's ops at every number of units a warp rotates side by side (widths 1024 to 9216 and the longest of the model), by
every CTA for itself and once for the grid: the bits of the per-matrix calls."""
import numpy as np
import pytest

from bonsai_b200 import synth

pytestmark = pytest.mark.gpu


def dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("n_in", [1024 * k for k in (1, 2, 3, 4, 5, 6, 7, 8, 9, 17)])
@pytest.mark.parametrize("signed", [False, True])
def test_rotated_inputs(gpu, n_in, signed):
    import torch
    first, rows, eps = 5120, 37, 1e-6
    x = dev(synth.activations(first, seed=1))
    norm = 1 + 0.1 * dev(synth.activations(n_in, seed=2))
    sg = dev(synth.signs(n_in, seed=3)) if signed else None
    W0, W1 = dev(synth.pq2_0_weights(n_in, first, seed=4)), dev(synth.pq2_0_weights(rows, n_in, seed=5))
    mid, plain, normed = torch.zeros(n_in, device="cuda"), torch.zeros(rows, device="cuda"), torch.zeros(rows, device="cuda")
    ops = [(W0, x, None, mid, n_in, first, gpu.OP_ROTATE), (W1, mid, sg, plain, rows, n_in, gpu.OP_ROTATE | gpu.OP_DEPENDS)]
    if n_in <= 7168:
        ops.append((W1, mid, sg, normed, rows, n_in, gpu.OP_ROTATE | gpu.OP_RMSNORM | gpu.OP_DEPENDS, norm, eps))
    chain = gpu.Chain(ops)
    for _ in range(2):
        assert chain.run() == 0
    torch.cuda.synchronize()
    scratch = torch.empty(17408 // 32 * 36, dtype=torch.uint8, device="cuda")
    h, want, t = torch.empty(n_in, device="cuda"), torch.empty(rows, device="cuda"), torch.empty(n_in, device="cuda")
    assert gpu.linear(W0, x, None, h, scratch, n_in, first) == 0
    assert torch.equal(mid, h)
    assert gpu.linear(W1, h, sg, want, scratch, rows, n_in) == 0
    assert torch.equal(plain, want)
    if n_in <= 7168:
        assert gpu.rmsnorm(h, norm, t, 1, n_in, eps) == 0
        assert gpu.linear(W1, t, sg, want, scratch, rows, n_in) == 0
        assert torch.equal(normed, want)
    chain.close()
    assert gpu.device_status() == 0
