"""The repacked mat-vec's own quantiser at every number of 128-element slices a warp takes side by side (one, two, three, four or five, a
second round of one to five): the bits of quantiser and plain mat-vec in two steps."""
import numpy as np
import pytest

from bonsai_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_in", [1024 * k for k in (1, 2, 3, 4, 5, 6, 7, 9, 10, 12, 14, 17, 19)])
def test_slices(gpu, n_in):
    import torch
    n_out = 37
    x = synth.activations(n_in, seed=n_in) * 1.7
    x[:32] = 0                                          # a chunk without a value
    x[n_in - 32:] *= 1e-7                               # one whose scale is below the 16-bit range
    W, xd = torch.from_numpy(synth.pq2_0_weights(n_out, n_in, seed=7)).cuda(), torch.from_numpy(np.ascontiguousarray(x)).cuda()
    Wr, xq = torch.zeros_like(W), torch.zeros(n_in // 32 * 36, dtype=torch.uint8, device="cuda")
    got, want = torch.zeros(n_out, device="cuda"), torch.ones(n_out, device="cuda")
    assert gpu.repack(W, Wr, n_out, n_in) == 0
    assert gpu.gemv_repack(Wr, xd, got, n_out, n_in) == 0
    assert gpu.quant_activations(xd, xq, n_in) == 0
    assert gpu.gemv(W, xq, want, n_out, n_in) == 0
    torch.cuda.synchronize()
    assert torch.equal(got, want)
    assert gpu.device_status() == 0
