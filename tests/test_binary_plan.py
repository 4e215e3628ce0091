"""CPU tests of the binary MSMs' launch plans (no kernels run): every launch of a call, the last rows and
the last columns included, fits in the workspace the call sets aside for one launch."""
import ctypes
import random

import pytest

import zkutil as Z


def plan(zk, curve, host, nrows, npts):
    info = (ctypes.c_size_t * 3)()
    assert zk.lib().zkg_msm_binary_plan(curve, host, nrows, npts, info) == 0, zk.lib().zkg_last_error()
    return list(info)


RAGGED = [(Z.BN254, 1, 1, 1035752), (Z.BN254, 1, 14, 1035752), (Z.BN254, 1, 64, 1035752), (Z.BN254, 1, 1, 1024000),
          (Z.BLS12_381, 1, 1, 690502), (Z.BLS12_381, 1, 14, 690502), (Z.BN254, 0, 65528, 300000),
          (Z.BN254, 0, 1, (1 << 26) + 1), (Z.BN254, 1, 1, 1), (Z.BLS12_381, 0, 40000, 3)]


@pytest.mark.parametrize("curve,host,nrows,npts", RAGGED)
def test_every_launch_fits_its_workspace(zk, curve, host, nrows, npts):
    given, needed, _ = plan(zk, curve, host, nrows, npts)
    assert needed <= given


def test_every_launch_fits_its_workspace_over_the_range(zk):
    rng = random.Random(5)
    for _ in range(400):
        curve, host = rng.randrange(2), rng.randrange(2)
        nrows = int(2 ** rng.uniform(0, 14))
        npts = int(2 ** rng.uniform(10, 21.5))
        given, needed, _ = plan(zk, curve, host, nrows, npts)
        assert needed <= given, (curve, host, nrows, npts)
