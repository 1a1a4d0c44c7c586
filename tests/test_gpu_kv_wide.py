"""Decode attention at the lengths between which one cluster of sixteen CTAs serves a kv head: the first and last of them, the first
with a second tile in a split, splits that are empty; and with the clusters of eight that serve there where sixteen cannot be placed,
also in the form that reads the others' parts, which serves one cluster where the form that sends them cannot be placed.
Oracle and bound as in test_gpu_kv_splits."""
import ctypes as C

import pytest

from test_gpu_kv_splits import D, N_HEADS, REL_TOL, exact, fill

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [512, 513, 528, 529, 769, 1025, 1040, 1041, 2047, 2048, 3071, 3072])
@pytest.mark.parametrize("spread", [0, 1])
@pytest.mark.parametrize("wide", [1, 0])
def test_against_float64(gpu, port, n, spread, wide):
    import torch
    kv, layer, splits = gpu.KVCache(n), 9, (C.c_int64 * 3)()
    q = fill(kv, layer, n, n, spread)
    out = torch.full((N_HEADS, D), float("nan"), device="cuda")
    try:
        assert gpu.set_option("kv_wide", wide) == 0
        assert gpu.lib().bonsai_b200_kv_splits(n, -1, -1, splits) == 0
        assert splits[0] == (16 if wide and 513 <= n <= 3071 else 8)
        for _ in range(2):
            assert kv.attn_decode(layer, n - 1, q, out) == 0
    finally:
        gpu.set_option("kv_wide", 1)
    want = exact(port, kv, n, layer, n, q)
    err, top = float((out.double() - want).abs().max()), float(want.abs().max())
    assert err <= REL_TOL * top, (err, top)
    assert gpu.device_status() == 0
    kv.close()


@pytest.mark.parametrize("n", [1, 9, 64, 65, 129, 511, 512, 513, 1025, 2047])
@pytest.mark.parametrize("spread", [0, 1])
def test_one_cluster_that_reads(gpu, port, n, spread):
    import torch
    kv, layer = gpu.KVCache(n), 5
    q = fill(kv, layer, n, n, spread)
    sent, read = (torch.full((N_HEADS, D), float("nan"), device="cuda") for _ in range(2))
    try:
        assert gpu.set_option("kv_wide", 0) == 0
        assert kv.attn_decode(layer, n - 1, q, sent) == 0
        assert gpu.set_option("kv_push", 0) == 0
        for _ in range(2):
            assert kv.attn_decode(layer, n - 1, q, read) == 0
    finally:
        gpu.set_option("kv_wide", 1), gpu.set_option("kv_push", 1)
    want = exact(port, kv, n, layer, n, q)
    top = float(want.abs().max())
    for out in (sent, read):
        err = float((out.double() - want).abs().max())
        assert err <= REL_TOL * top, (err, top)
    assert n < 64 or not torch.equal(sent, read)        # scores added in another order: the other kernel did run
    assert gpu.device_status() == 0
    kv.close()
