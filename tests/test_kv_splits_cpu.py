"""How decode attention divides the positions of a cache over clusters of CTAs, on devices of every size (host arithmetic)."""
import ctypes as C

import pytest


def splits(n_pos, resident8, resident16):
    import bonsai_b200
    out = (C.c_int64 * 3)()
    assert bonsai_b200.lib().bonsai_b200_kv_splits(n_pos, resident8, resident16, out) == 0
    cluster, clusters, chunk = out
    assert chunk % 16 == 0 and cluster * clusters * chunk >= n_pos
    return cluster, clusters


@pytest.mark.parametrize("n_pos,want", [(1, (8, 1)), (512, (8, 1)), (513, (16, 1)), (2048, (16, 1)), (3071, (16, 1)), (3072, (8, 3)), (13312, (8, 13)), (262144, (8, 13))])
def test_whole_device(n_pos, want):
    assert splits(n_pos, 52, 20) == want


@pytest.mark.parametrize("resident8", [1, 4, 8, 11, 52])
def test_clusters_of_sixteen_serve_only_where_measured(resident8):
    """Not above 3071 positions however few clusters of eight there are, and not where those of the four kv heads would run in waves."""
    few = max(1, resident8 // 4)
    for n_pos in (3072, 4096, 40000, 262144):
        assert splits(n_pos, resident8, 20) == (8, min(few, n_pos // 1024))
    for n_pos in (513, 1500, 3071):
        assert splits(n_pos, resident8, 4) == (16, 1)
        for resident16 in (0, 1, 2, 3):
            assert splits(n_pos, resident8, resident16) == (8, min(few, max(1, n_pos // 1024)))


def test_rejections():
    import bonsai_b200
    out = (C.c_int64 * 3)()
    f = bonsai_b200.lib().bonsai_b200_kv_splits
    assert f(0, 52, 20, out) == 1 and f(262145, 52, 20, out) == 1 and f(700, 0, 20, out) == 1 and f(700, 52, 20, None) == 1
