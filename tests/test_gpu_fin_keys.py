"""The keyed finite-depth fill (region methods once per distinct (R, zq, zp))
against the per-pair evaluation of the same points (hg_green_points): the same
operations in the same order, so the matrices agree bit for bit."""
import numpy as np
import pytest

import __graft_entry__ as g

pytestmark = pytest.mark.gpu


def _mesh(kind, pkg):
    mg = pkg.meshgen
    if kind == "symmetric":        # repeated R and depths; a second equal body
        return mg.combine([mg.cylinder(3.0, 6.0, 12, 5, 3), mg.cylinder(3.0, 6.0, 12, 5, 3, cx=15.0)])
    if kind == "lids":             # field rows beyond the sources
        return mg.combine([mg.cylinder(4.0, 5.0, 13, 4, 2, lid_rings=2)])
    if kind == "four":             # fewer pairs than a warp
        return mg.combine([mg.box(2.0, 2.0, 1.0, 2.0)])
    rng = np.random.default_rng(11)  # no two panels at one depth
    b = mg.cylinder(3.0, 4.0, 11, 6, 3)
    b.nodes = np.where(b.nodes[:, 2:3] < 0, b.nodes * (1 + rng.uniform(-0.03, 0.03, b.nodes.shape)), b.nodes)
    return mg.combine([b])


# depths that put pairs in every band: R/h below 0.0005, 0.05, 0.5 and above
@pytest.mark.parametrize("kind,h,w,nk", [("symmetric", 20.0, 1.3, 200), ("symmetric", 150.0, 0.5, 200),
                                         ("lids", 12.0, 0.9, 200), ("irregular", 9.0, 1.7, 200),
                                         ("irregular", 90.0, 1.1, 60), ("four", 8.0, 1.0, 20)])
def test_keyed_fill_equals_per_pair(kind, h, w, nk):
    pkg = g.load_package()
    mesh = _mesh(kind, pkg)
    lid = len(mesh.lid_xyz_p) > 0
    s = pkg.hamsgpu.Solver()
    s.keep_matrices(True)
    s.set_mesh(mesh.nodes, mesh.ncon, mesh.ncn, mesh.xyz_p, mesh.ds, mesh.pnsz, mesh.dxyz_p, mesh.body_ranges,
               mesh.lid_xyz_p if lid else None)
    v, wk, w1, wvn = pkg.hamsgpu.wave_properties(3, w, h)
    for turn in range(2):  # the first fill builds the keys, the second uses them
        s.set_frequency(v, wk, w1, h, wvn[:nk])
        s.fill_factor(1 if lid else 0)
    rows = np.vstack([mesh.xyz_p, mesh.lid_xyz_p]) if lid else mesh.xyz_p
    n, tn = mesh.n, len(rows)
    a, sm = s.get_matrix(0, tn), s.get_matrix(1, tn)
    q = np.broadcast_to(mesh.xyz_p[None], (tn, n, 3))
    p = np.broadcast_to(rows[:, None], (tn, n, 3))
    dist = np.sqrt(((p[..., 0] - q[..., 0]) ** 2 + (p[..., 1] - q[..., 1]) ** 2) + (p[..., 2] - q[..., 2]) ** 2)
    near = dist <= 50.0 * mesh.pnsz
    grn = s.green_points(np.concatenate([q, p], axis=2).reshape(-1, 6), near.ravel().astype(np.int32)).reshape(tn, n, 4)
    s.close()
    ds, nr = mesh.ds, mesh.dxyz_p
    near_ai = ((grn[..., 1].imag * ds) * nr[:, 0] + (grn[..., 2].imag * ds) * nr[:, 1]) + (grn[..., 3].imag * ds) * nr[:, 2]
    far_a = [((c(grn[..., 1]) * nr[:, 0] + c(grn[..., 2]) * nr[:, 1]) + c(grn[..., 3]) * nr[:, 2]) * ds
             for c in (np.real, np.imag)]
    assert np.array_equal(sm.imag, grn[..., 0].imag * ds)
    assert np.array_equal(a.imag, np.where(near, near_ai, far_a[1]))
    far = ~near
    assert np.array_equal(sm.real[far], (grn[..., 0].real * ds)[far])
    assert np.array_equal(a.real[far], far_a[0][far])
