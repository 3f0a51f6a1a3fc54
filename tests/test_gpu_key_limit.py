"""The memory the finite-depth keys may hold (hg_set_key_limit): less of it
means more passes over smaller tables, none the pair-by-pair kernels, and the
matrices stay the same bits; keys that do not fit are not tried again."""
import numpy as np
import pytest

import __graft_entry__ as g

pytestmark = pytest.mark.gpu


def _mesh(pkg, kind):
    mg = pkg.meshgen
    if kind == "bodies":   # repeated R and depths, lids
        return mg.combine([mg.cylinder(3.0, 6.0, 16, 6, 4, lid_rings=2), mg.cylinder(3.0, 6.0, 16, 6, 4, cx=15.0, lid_rings=2)])
    rng = np.random.default_rng(4)  # no two panels at one depth
    b = mg.cylinder(4.0, 5.0, 21, 9, 5)
    b.nodes = np.where(b.nodes[:, 2:3] < 0, b.nodes * (1 + rng.uniform(-0.03, 0.03, b.nodes.shape)), b.nodes)
    return mg.combine([b])


def _solver(pkg, mesh, form, table, limit=None):
    s = pkg.hamsgpu.Solver(precision=form, fin_table=table)
    s.keep_matrices(True)
    if limit is not None:
        s.set_key_limit(limit)
    s.set_mesh(mesh.nodes, mesh.ncon, mesh.ncn, mesh.xyz_p, mesh.ds, mesh.pnsz, mesh.dxyz_p, mesh.body_ranges,
               mesh.lid_xyz_p if len(mesh.lid_xyz_p) else None)
    return s


def _fill(pkg, s, mesh, w, h):
    lid = len(mesh.lid_xyz_p)
    v, wk, w1, wvn = pkg.hamsgpu.wave_properties(3, w, h)
    s.set_frequency(v, wk, w1, h, wvn)
    s.fill_factor(1 if lid else 0)
    return s.get_matrix(0, mesh.n + lid), s.get_matrix(1, mesh.n + lid)


# plain; mixed with every pair keyed (the contracted build); mixed with tables and the near pairs keyed.  Depths that
# put pairs in all bands, and nearly all of them in the nearest two.
@pytest.mark.parametrize("form,table", [(0, -1), (1, 0), (1, 1)])
@pytest.mark.parametrize("kind,h,w", [("bodies", 20.0, 1.3), ("bodies", 300.0, 0.7), ("irregular", 9.0, 1.7),
                                      ("irregular", 120.0, 1.1)])
def test_same_bits_within_any_limit(form, table, kind, h, w):
    pkg = g.load_package()
    mesh = _mesh(pkg, kind)
    s = _solver(pkg, mesh, form, table)
    want = _fill(pkg, s, mesh, w, h)
    free = s.key_info()
    s.close()
    assert free["pairs"] > 0 and free["keys"] > 0 and 0 < free["bytes"] <= free["peak"]
    for share in (0.8, 0.55, 0.0):
        s = _solver(pkg, mesh, form, table, share * free["peak"])
        got = _fill(pkg, s, mesh, w, h)
        info = s.key_info()
        s.close()
        assert info["peak"] <= share * free["peak"]
        if share == 0.0:
            assert info["pairs"] == 0 and info["bytes"] == 0
        for a, b in zip(got, want):
            assert np.array_equal(a, b), (share, info, np.abs(a - b).max())


def test_tables_in_several_passes():
    """Half the memory of all tables and then little more than the least: bands cut into groups, the same bits."""
    pkg = g.load_package()
    mesh = _mesh(pkg, "irregular")
    s = _solver(pkg, mesh, 0, -1)
    want = _fill(pkg, s, mesh, 1.4, 30.0)
    free = s.key_info()
    assert free["bytes"] == free["peak"]  # the tables, not the build's scratch
    passes = []
    for share in (0.6, 0.45):
        s.set_key_limit(share * free["peak"])
        for turn in range(2):
            got = _fill(pkg, s, mesh, 1.4, 30.0)
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
        info = s.key_info()
        assert info["pairs"] == free["pairs"] and info["keys"] == free["keys"] and info["peak"] <= share * free["peak"]
        passes.append(info["passes"])
    s.close()
    assert free["passes"] < passes[0] < passes[1]


def test_keys_that_do_not_fit_are_not_tried_again():
    pkg = g.load_package()
    mesh = _mesh(pkg, "irregular")
    s = _solver(pkg, mesh, 0, -1, 3e6)
    for w in (0.8, 1.0, 1.2):
        _fill(pkg, s, mesh, w, 20.0)
        assert s.key_info()["builds"] == 1
    _fill(pkg, s, mesh, 0.8, 25.0)      # another depth is tried
    assert s.key_info()["builds"] == 2 and s.key_info()["pairs"] == 0
    s.set_key_limit(-1)                 # and another limit
    _fill(pkg, s, mesh, 0.8, 25.0)
    assert s.key_info()["builds"] == 3 and s.key_info()["pairs"] == mesh.n ** 2
    s.set_key_limit(0)                  # given back at once
    assert s.key_info()["bytes"] == 0
    s.close()


def test_sweep_without_keys():
    pkg = g.load_package()
    hg, mesh = pkg.hamsgpu, _mesh(pkg, "irregular")
    props = [hg.wave_properties(3, w, 20.0) for w in (0.8, 1.0, 1.3)]
    v, wk, w1, wvn = (np.array([p[k] for p in props]) for k in range(4))
    out = []
    for limit in (-1, 0):
        s = _solver(pkg, mesh, hg.HG_PREC_FP64, -1, limit)
        out.append(s.solve_sweep(v, wk, w1, 20.0, wvn, np.array([0.0]), nslots=2)[:3])
        s.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def test_a_failing_allocation_takes_the_keys_back():
    """A call for more memory than any device has fails, but only after every context's keys went; they are not built
    again for their mesh and depth, and the fill gives the same bits without them."""
    pkg = g.load_package()
    mesh = _mesh(pkg, "irregular")
    a, b = (_solver(pkg, mesh, form, -1) for form in (0, 1))
    want = [_fill(pkg, s, mesh, 1.2, 20.0) for s in (a, b)]
    assert a.key_info()["bytes"] > 0 and b.key_info()["bytes"] > 0
    other = pkg.hamsgpu.Solver()
    n = 200000  # 640 GB of matrix: refused before anything is read
    one, piv = np.zeros(2), np.zeros(1, dtype=np.int32)
    rc = other.L.hg_gesv(other.h, 0, n, 0, one.ctypes.data, n, piv.ctypes.data, None, n, None, None)
    assert rc < 0 and b"out of memory" in other.L.hg_last_error(other.h)
    other.close()
    for s, x in zip((a, b), want):
        builds = s.key_info()["builds"]
        assert s.key_info()["bytes"] == 0
        y = _fill(pkg, s, mesh, 1.2, 20.0)
        assert np.array_equal(x[0], y[0]) and np.array_equal(x[1], y[1])
        assert s.key_info()["bytes"] == 0 and s.key_info()["builds"] == builds
        s.close()
