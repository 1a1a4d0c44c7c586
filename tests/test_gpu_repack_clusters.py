"""The repacked mat-vec whose CTAs share the quantiser in fours (up to 128 CTAs, 40 blocks per row and more) and in pairs (96 blocks), the last
cluster with CTAs that have no rows, beside shapes that share nothing: the bits of quantiser and plain mat-vec in two steps, call after call."""
import numpy as np
import pytest

from bonsai_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_out,n_in", [(1, 5120), (13, 17408), (511, 9216), (512, 5120), (1030, 6144), (4644, 12288), (4100, 17408), (5120, 17408),
                                        (9000, 11264), (700, 4096)])
def test_shared_quantiser(gpu, n_out, n_in):
    import torch
    W = torch.from_numpy(synth.pq2_0_weights(n_out, n_in, seed=n_out)).cuda()
    Wr, xq = torch.zeros_like(W), torch.zeros(n_in // 32 * 36, dtype=torch.uint8, device="cuda")
    assert gpu.repack(W, Wr, n_out, n_in) == 0
    got, want = [torch.zeros(n_out, device="cuda") for _ in range(3)], torch.ones(n_out, device="cuda")
    for seed in range(2):
        x = torch.from_numpy(np.ascontiguousarray(synth.activations(n_in, seed=seed) * 1.7)).cuda()
        for y in got:                                   # launches that start while the one in front still runs
            assert gpu.gemv_repack(Wr, x, y, n_out, n_in) == 0
        assert gpu.quant_activations(x, xq, n_in) == 0
        assert gpu.gemv(W, xq, want, n_out, n_in) == 0
        torch.cuda.synchronize()
        assert all(torch.equal(y, want) for y in got)
        assert gpu.device_status() == 0
