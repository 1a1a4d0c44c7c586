"""Decode attention at the lengths between which one cluster of sixteen CTAs serves a kv head: the first and last of them, the first
with a second tile in a split, splits that are empty.  Oracle and bound as in test_gpu_kv_splits."""
import pytest

from test_gpu_kv_splits import D, N_HEADS, REL_TOL, exact, fill

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [512, 513, 528, 529, 769, 1040, 1041, 3071, 3072])
@pytest.mark.parametrize("spread", [0, 1])
def test_against_float64(gpu, port, n, spread):
    import torch
    kv, layer = gpu.KVCache(n), 9
    q = fill(kv, layer, n, n, spread)
    out = torch.full((N_HEADS, D), float("nan"), device="cuda")
    for _ in range(2):
        assert kv.attn_decode(layer, n - 1, q, out) == 0
    want = exact(port, kv, n, layer, n, q)
    err, top = float((out.double() - want).abs().max()), float(want.abs().max())
    assert err <= REL_TOL * top, (err, top)
    assert gpu.device_status() == 0
    kv.close()
