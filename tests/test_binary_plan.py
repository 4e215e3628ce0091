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


@pytest.mark.parametrize("host,nrows,npts", [(0, 16384, 1 << 21), (0, 28000, 1 << 19), (1, 32768, 1 << 20),
                                             (1, 1 << 20, 4096), (0, 1 << 17, 1 << 16), (1, 2048, 1 << 20)])
@pytest.mark.parametrize("curve", Z.CURVES)
def test_many_rows_are_planned_in_bounded_memory(zk, curve, host, nrows, npts):
    """no size is refused, and the workspace is one point a row and one launch: at most 2^26 entries of 12
    bytes, their chunks' partial sums and the buckets, below 2 GiB; not a point a row and column chunk"""
    given, needed, total = plan(zk, curve, host, nrows, npts)
    assert needed <= given <= 2 << 30
    assert total <= given + nrows * 4 * Z.NLP[curve] * 8 + 512
