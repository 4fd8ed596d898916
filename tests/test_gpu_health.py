"""Failure detection on the GPU without faulting it.

Kernels never trap: bounded waits and capacity or finiteness checks raise bits
in a device health word, which sph_synchronize turns into an error status.
Each case below makes one such failure happen on purpose from the host (a
withheld predecessor with a short spin limit, a non-finite input) and checks
that the error comes back and that the context stays usable afterwards.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SPH_ERR_DEVICE_HEALTH = 5
SPH_ERR_TIMEOUT = 6


def test_lookback_timeout_is_reported_and_context_recovers(cuda, pkg):
    lib = pkg._lib.load()
    ic = pkg.ic.make_impact(2048, 512, seed=4)
    with pkg.Compute(ic, max_children_in_leaf=16) as c:
        c.step()
        c.synchronize()
        assert lib.sph_selftest_lookback_timeout(c._h, 1000, None) == 0
        rc = lib.sph_synchronize(c._h, None)
        assert rc == SPH_ERR_TIMEOUT, rc
        assert c.health() & pkg._lib.HEALTH["sort_timeout"]
        c.clear_health()
        c.step()
        c.synchronize()  # raises on any error
        assert np.all(np.isfinite(c.download("pos")))


# what is built on a sort whose waits gave up -- the tree, and the cell ranges
# with all that walks them -- stays within its buffers, in both gravity forms
@pytest.mark.parametrize("n,leaf,depth,theta", [(2560, 16, 7, None), (20481, 1, 7, None), (20481, 4, 10, 0.6),
                                                (300000, 32, 7, 0.6)])
def test_passes_after_a_sort_timeout_and_recovery(cuda, pkg, n, leaf, depth, theta):
    lib = pkg._lib.load()
    ic = pkg.ic.make_impact(n - n // 5, n // 5, seed=4)
    gn = np.full(n, 0.1, np.float32)
    got = []
    for disturbed in (True, False):
        with pkg.Compute(ic, max_children_in_leaf=leaf, max_tree_depth=depth) as c:
            if theta:
                c.set_form(gravity="theta", theta=theta)
            for _ in range(2 if disturbed else 0):
                assert lib.sph_selftest_sort_timeout(c._h, 200, None) == 0
                tree = c.get_tree()
                # a whole tree: every particle place in one leaf, every node reached once
                assert tree["n_nodes"] == sum(np.diff(tree["level_offsets"]))
                start = c.download("cell_start")
                assert np.all(start == 0xFFFFFFFF)
                c.gravitationalPass()
                c.densityPass()
                c.accelerationPass()
                assert lib.sph_synchronize(c._h, None) == SPH_ERR_TIMEOUT
                assert c.health() & pkg._lib.HEALTH["sort_timeout"]
                c.clear_health()
            for f in ("h", "rho"):
                c.upload(f, ic[f])
            c.upload("grav_norm", gn)
            c.updateOctreeBuffer()
            c.sort()
            c.gravitationalPass()
            c.densityPass()
            c.accelerationPass()
            c.synchronize()
            got.append([c.get_tree()["tree"]] + [c.download(f) for f in ("cell_start", "cell_end", "h", "rho", "acc")])
    for a, b in zip(*got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("thread", [0, 1, 77, 127])
def test_a_tensor_core_wait_that_gives_up_is_reported_by_any_thread(cuda, pkg, thread):
    lib = pkg._lib.load()
    ic = pkg.ic.make_impact(2048, 512, seed=4)
    with pkg.Compute(ic, max_children_in_leaf=16) as c:
        assert lib.sph_selftest_mlp_timeout(c._h, 128, 16, None) == 1  # no such thread
        assert lib.sph_selftest_mlp_timeout(c._h, thread, 16, None) == 0
        assert lib.sph_synchronize(c._h, None) == SPH_ERR_TIMEOUT
        assert c.health() == pkg._lib.HEALTH["mlp_timeout"]
        c.clear_health()
        c.step()
        c.synchronize()


def test_non_finite_density_is_reported(cuda, pkg):
    lib = pkg._lib.load()
    ic = pkg.ic.make_impact(2048, 512, seed=4)
    with pkg.Compute(ic, max_children_in_leaf=16) as c:
        u = ic["u"].copy()
        u[17] = np.float32("nan")
        c.upload("u", u)
        c.updateOctreeBuffer()
        c.sort()
        c.gravitationalPass()
        c.densityPass()
        rc = lib.sph_synchronize(c._h, None)
        assert rc == SPH_ERR_DEVICE_HEALTH, rc
        assert c.health() & pkg._lib.HEALTH["nan_density"]
        c.clear_health()
        c.upload("u", ic["u"])
        c.step()
        c.synchronize()


def test_tree_capacity_is_reported_and_context_recovers(cuda, pkg):
    lib = pkg._lib.load()
    ic = pkg.ic.make_impact(2048, 512, seed=4)
    with pkg.Compute(ic, max_children_in_leaf=16) as c:
        c.step()
        c.synchronize()
        want_ok = c.download("pos")
        assert lib.sph_selftest_tree_capacity(c._h, None) == 0
        rc = lib.sph_synchronize(c._h, None)
        assert rc == SPH_ERR_DEVICE_HEALTH, rc
        assert c.health() & pkg._lib.HEALTH["tree_capacity"]
        c.clear_health()
        c.step()  # rebuilds a whole tree
        c.synchronize()
        assert np.all(np.isfinite(c.download("pos")))
        assert not np.array_equal(c.download("pos"), want_ok)  # it stepped


def test_async_transfers_round_trip_on_a_stream(cuda, pkg):
    import torch

    ic = pkg.ic.make_impact(2048, 512, seed=6)
    n = int(ic["n"])
    with pkg.Compute(ic, max_children_in_leaf=16) as c:
        s = torch.cuda.Stream()
        pos = torch.from_numpy(ic["pos"].reshape(-1).copy()).pin_memory().numpy()
        u = torch.from_numpy(ic["u"].copy()).pin_memory().numpy()
        out_pos = torch.empty(3 * n, dtype=torch.float32).pin_memory().numpy()
        out_u = torch.empty(n, dtype=torch.float32).pin_memory().numpy()
        pos2 = pos + np.float32(0.25)
        c.upload_async("pos", pos2, s)
        c.upload_async("u", u * np.float32(2.0), s)
        c.download_async("pos", out_pos, s)
        c.download_async("u", out_u, s)
        s.synchronize()
        assert np.array_equal(out_pos, pos2)
        assert np.array_equal(out_u, u * np.float32(2.0))
        # the mass rides in the position records and must survive the upload
        assert np.array_equal(c.download("mass"), ic["mass"])
