"""fp32 inputs of a list's ops at every number of units that a warp rotates, two at a time or one by one (widths 1024 to 9216 and the longest of the model), by
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


@pytest.mark.parametrize("at", [0, 1024, 6144, 10240, 15356, 15360])
@pytest.mark.parametrize("written", ["norm", "signs"])
def test_factors_that_the_list_writes(gpu, at, written):
    """Norm weights or signs that are an output of an earlier op (all of the first op's, the end of it and the start of the next one's, parts
    of the second's, its last four values and what lies behind them): the values of this run, whatever the buffer held before.  At 15360
    they are a neighbour of the outputs."""
    import torch
    n_in, rows, eps = 5120, 37, 1e-6
    x0 = dev(synth.activations(n_in, seed=1))
    W0, W1, W2 = (dev(synth.pq2_0_weights(n, n_in, seed=k)) for k, n in ((4, n_in), (5, 2 * n_in), (6, rows)))
    buf = torch.zeros(5 * n_in, device="cuda")
    mid, wide, after = buf[:n_in], buf[n_in:3 * n_in], buf[3 * n_in:]
    fac = buf[at:at + n_in]
    ones = torch.ones(n_in, device="cuda")
    norm, sg = (fac, None) if written == "norm" else (ones, fac)
    ops = [(W0, x0, None, mid, n_in, n_in, gpu.OP_ROTATE), (W1, x0, None, wide, 2 * n_in, n_in, gpu.OP_ROTATE),
           (W2, mid, sg, torch.zeros(rows, device="cuda"), rows, n_in, gpu.OP_ROTATE | gpu.OP_RMSNORM | gpu.OP_DEPENDS, norm, eps)]
    chain = gpu.Chain(ops)
    scratch = torch.empty(n_in // 32 * 36, dtype=torch.uint8, device="cuda")
    want_mid, want_wide, want, t = (torch.empty(n, device="cuda") for n in (n_in, 2 * n_in, rows, n_in))
    assert gpu.linear(W0, x0, None, want_mid, scratch, n_in, n_in) == 0
    assert gpu.linear(W1, x0, None, want_wide, scratch, 2 * n_in, n_in) == 0
    for run in range(3):
        buf.fill_(7.0 + run)
        after.copy_(dev(synth.activations(2 * n_in, seed=run)))
        fresh = torch.cat([want_mid, want_wide, after])
        f = fresh[at:at + n_in].clone()
        assert gpu.rmsnorm(want_mid, f if written == "norm" else ones, t, 1, n_in, eps) == 0
        assert gpu.linear(W2, t, None if written == "norm" else f, want, scratch, rows, n_in) == 0
        assert chain.run() == 0
        torch.cuda.synchronize()
        assert torch.equal(mid, want_mid) and torch.equal(wide, want_wide)
        assert torch.equal(ops[2][3], want), run
    chain.close()
    assert gpu.device_status() == 0
