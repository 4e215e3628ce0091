"""CPU tests of the MSM's device workspace (planned on the host): the affine tree's lists are bounded."""
import ctypes

import pytest

import zkutil as Z


def workspace(zk, curve, n):
    info = (ctypes.c_size_t * 2)()
    assert zk.lib().zkg_msm_workspace(curve, n, info) == 0, zk.lib().zkg_last_error()
    return list(info)


@pytest.mark.parametrize("curve", Z.CURVES)
def test_tree_lists_are_bounded(zk, curve):
    """Beside the rest of the workspace the tree holds, for a slab of at most 2^27 entries or one window, a
    point for every second entry and for every fourth and a field element for every second: a point an
    entry in all; a quarter more for the padding, the threads' products and the alignment."""
    point = 2 * 8 * Z.NLP[curve]
    for n in [int(2 ** (lg / 3)) for lg in range(54, 81)] + [1 << 26, 1 << 27, 165000000]:
        with_tree, without = workspace(zk, curve, n)
        assert without <= with_tree <= without + 1.25 * max(1 << 27, n) * point, n


@pytest.mark.parametrize("curve", Z.CURVES)
def test_large_msms_windows(zk, curve):
    """long segments for the tree up to the sizes where it pays (16-bit windows), wide windows beyond, and
    never more (window, point) entries than a launch has"""
    L = zk.lib()
    for n in (1 << 22, 6000000, 1 << 23, 1 << 24, 20000000):
        assert L.zkg_msm_window_for(curve, n) == 16, n
    for n in (25000000, 1 << 25, 1 << 27, 165000000):
        c = L.zkg_msm_window_for(curve, n)
        assert c == 20 if curve == Z.BN254 else c >= 16, n
        assert -(-256 // c) * n < 1 << 31, n
        if curve == Z.BN254:
            with_tree, without = workspace(zk, curve, n)
            assert with_tree == without, n
