"""The affine tree in bounded memory: slabs of windows, calls and servers in memory it does not fit."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

import test_knobs_gpu as K
import zkutil as Z
from test_msm_workspace import workspace

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slab,levels", [(1, 1), (7000, 2), (9000, 3), (30000, 2)])
def test_tree_in_slabs_of_windows_changes_no_result(zk, slab, levels, tmp_path):
    """3000 points: slabs of one window, of two or three and of ten, of narrow and wide windows"""
    path = str(tmp_path / "slabs.npz")
    env = dict(os.environ, ZKB_MSM_TREE=str(levels), ZKB_MSM_TREE_SLAB=str(slab), ZKB_DEVICE_CHECKS="1",
               ZKB_MSM_PARTS="2" if slab == 9000 else "1")
    code = "import sys; sys.path.insert(0, %r); import test_knobs_gpu as T; T._dump(%r)" % (K.HERE, path)
    r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    got = np.load(path)
    for k, v in K.compute_all().items():
        assert np.array_equal(got[k], v), k


def test_device_checks_on_the_small_sort_and_binary_rows(zk):
    """with the bounds checks on, valid inputs set no bit and give the same points"""
    code = ("import sys; sys.path.insert(0, %r); import numpy as np, zkutil as Z; zk = Z.load_package()\n"
            "for c in Z.CURVES:\n"
            "    b = Z.gen_bases_cpu(c, Z.rand_fr(c, 900, 1)); s = Z.rand_fr(c, 900, 2)\n"
            "    co = (Z.splitmix64(3, 30 * 900) & np.uint64(1)).astype(np.uint8).reshape(30, 900)\n"
            "    for mont in (True, False):\n"
            "        assert np.array_equal(zk.msm_affine(c, s, b, mont=mont), Z.oracle_msm_affine(c, s, 4, mont, b))\n"
            "    r = zk.binary_multi_msm(c, co, b, affine=True)\n"
            "    z = np.zeros((900, 4), np.uint64); z[:, 0] = co[29]\n"
            "    assert np.array_equal(r[29], Z.oracle_msm_affine(c, z, 4, False, b))\n" % K.HERE)
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, ZKB_DEVICE_CHECKS="1"), capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]


def _bases(zk, curve, n):
    import torch
    b = torch.empty((n, 2 * Z.NLP[curve]), dtype=torch.int64, device="cuda")
    zk.g1_gen_mul_device(curve, n, torch.from_numpy(Z.rand_fr(curve, n, 71000).view(np.int64)).cuda(), b)
    torch.cuda.synchronize()
    return b


@pytest.mark.parametrize("curve", Z.CURVES)
def test_msm_without_room_for_the_tree(zk, curve):
    """device memory for the workspace without the tree's lists but not with them: same point, on device and
    on host buffers"""
    import torch
    n = 1 << 20
    bases = _bases(zk, curve, n)
    s = torch.from_numpy(Z.rand_fr(curve, n, 71001).view(np.int64)).cuda()
    want = zk.msm_device(curve, n, s, bases, mont=True)
    with_tree, without = workspace(zk, curve, n)
    hs, hb = s.cpu().numpy().view(np.uint64), bases.cpu().numpy().view(np.uint64)
    assert zk.lib().zkg_release_cache() == 0
    # room for the host form, whose inputs lie beside the workspaces of its parts, without the tree
    room = 2 * without + hs.nbytes + hb.nbytes + (64 << 20)
    assert room < with_tree
    free, _ = torch.cuda.mem_get_info()
    hold = torch.empty(free - room, dtype=torch.uint8, device="cuda")
    try:
        for _ in range(2):
            assert np.array_equal(zk.msm_device(curve, n, s, bases, mont=True), want)
        assert np.array_equal(zk.msm_affine(curve, hs, hb, mont=True), want)
    finally:
        del hold
        torch.cuda.empty_cache()
    assert np.array_equal(zk.msm_device(curve, n, s, bases, mont=True), want)


@pytest.mark.parametrize("curve", Z.CURVES)
def test_server_budget_without_room_for_the_tree(zk, curve):
    """a budget of one request without the tree's lists is accepted, and its commitment is right"""
    import torch
    k = 20
    bases = _bases(zk, curve, 1 << k)
    with_tree, without = workspace(zk, curve, 1 << k)
    assert with_tree > 1.5 * without
    srv = zk.Server(curve, bases, 1 << k, k, k, 3 * (32 << k) + without + (1 << 16), 2)
    v = torch.from_numpy(Z.rand_fr(curve, 1 << k, 71002).view(np.int64)).pin_memory()
    got = [srv.wait(t)[0] for t in [srv.submit(k, v), srv.submit(k, v)]]
    srv.close()
    coef = zk.inverse_ntt(curve, k, v.numpy().view(np.uint64).reshape(-1, 4))
    want = zk.msm_device(curve, 1 << k, torch.from_numpy(coef.view(np.int64)).cuda(), bases, mont=True)
    assert np.array_equal(got[0], want) and np.array_equal(got[1], want)
