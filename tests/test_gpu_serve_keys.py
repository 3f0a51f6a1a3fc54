"""Device memory of finite-depth requests in the server: the keys a slot keeps
stay inside what its request reserved."""
import numpy as np
import pytest
import torch

import __graft_entry__ as g

pytestmark = pytest.mark.gpu


def _hull(pkg):
    rng = np.random.default_rng(3)
    b = pkg.meshgen.cylinder(5.0, 6.0, 33, 13, 6)
    b.nodes = np.where(b.nodes[:, 2:3] < 0, b.nodes * (1 + rng.uniform(-0.02, 0.02, b.nodes.shape)), b.nodes)
    return pkg.meshgen.combine([b])


@pytest.mark.parametrize("form", [0, 1])
def test_slots_hold_no_more_than_the_budget(form):
    pkg = g.load_package()
    hg, mesh, h, nslots = pkg.hamsgpu, _hull(pkg), 25.0, 2
    props = [hg.wave_properties(3, w, h) for w in (0.7, 1.0, 1.4, 1.9)]
    v, wk, w1, wvn = (np.array([p[k] for p in props]) for k in range(4))
    betas = np.array([0.0, 0.5])
    alone, keys = [], 0
    for limit in (0, -1):  # also loads every kernel before memory is read
        s = hg.Solver(precision=form)
        s.set_key_limit(limit)
        s.set_mesh(mesh.nodes, mesh.ncon, mesh.ncn, mesh.xyz_p, mesh.ds, mesh.pnsz, mesh.dxyz_p, mesh.body_ranges)
        alone = [s.solve_frequency(v[i], wk[i], w1[i], h, wvn[i], betas, want_potentials=False)[:3] for i in range(4)]
        keys = s.key_info()["bytes"]
        s.close()
    one = hg.solve_footprint(form, mesh.n, 0, 1, 2)
    assert keys > 4 * one  # what a slot must not hold on top here
    for budget in (1.3 * nslots * one, 40e9):
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        srv = hg.Server(nslots=nslots, budget_bytes=budget, precision=form)
        got = srv.wait(srv.submit(mesh, h, v, wk, w1, wvn, betas))
        held, st = free - torch.cuda.mem_get_info()[0], srv.stats()
        srv.close()
        for i, ref in enumerate(alone):
            for a, b in zip(got[:3], ref):
                np.testing.assert_array_equal(a[i], b)
        # small allocations share pages of 2 MB, some tens of them in each slot
        assert held <= st["peak_reserved_bytes"] + nslots * 64e6 and st["peak_reserved_bytes"] <= budget
        if budget == 40e9:
            assert st["peak_reserved_bytes"] > nslots * (one + keys)


def test_near_pairs_fit_what_is_reserved():
    """With tables only the near pairs are keyed: the reservation covers them, at far less than all pairs would take."""
    pkg = g.load_package()
    hg, mg, h = pkg.hamsgpu, pkg.meshgen, 45.0
    mesh = mg.combine([mg.cylinder(4.0, 6.0, 31, 12, 6, cx=25.0 * k, cy=3.0 * k) for k in range(2)])
    props = [hg.wave_properties(3, w, h) for w in (0.8, 1.3)]
    v, wk, w1, wvn = (np.array([p[k] for p in props]) for k in range(4))
    betas = np.array([0.3])
    s = hg.Solver(precision=hg.HG_PREC_MIXED)
    s.set_mesh(mesh.nodes, mesh.ncon, mesh.ncn, mesh.xyz_p, mesh.ds, mesh.pnsz, mesh.dxyz_p, mesh.body_ranges)
    alone = [s.solve_frequency(v[i], wk[i], w1[i], h, wvn[i], betas, want_potentials=False)[:3] for i in range(2)]
    keys = s.key_info()
    s.close()
    pairs = mesh.n ** 2
    assert pairs >= 1000000 and 0 < keys["pairs"] < pairs // 4
    srv = hg.Server(nslots=2, budget_bytes=40e9)
    got = srv.wait(srv.submit(mesh, h, v, wk, w1, wvn, betas))
    reserved = srv.stats()["peak_reserved_bytes"] / 2
    srv.close()
    for i, ref in enumerate(alone):
        for a, b in zip(got[:3], ref):
            np.testing.assert_array_equal(a[i], b)
    one = hg.solve_footprint(hg.HG_PREC_MIXED, mesh.n, 0, 2, 1)  # 28 bytes a pair of it for the near pairs
    assert reserved >= one - 28 * pairs + keys["peak"]
    assert reserved < one + 100 * pairs + 2 ** 28  # the tables may take 256 MB by themselves
