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
    for n in [int(2 ** (lg / 3)) for lg in range(54, 81)] + [1 << 26, 1 << 27]:
        with_tree, without = workspace(zk, curve, n)
        assert without <= with_tree <= without + 1.25 * max(1 << 27, n) * point, n
