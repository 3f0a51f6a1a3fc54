"""The on-body test of field points near its tolerance, with panel normals of
unit length and not (the single-precision filter holds for unit normals and
leaves the others to the test itself): potentials against the oracle, which
halves where a point counts as on the body."""
import copy

import numpy as np
import pytest

from helpers import case_from_mesh, gpu_frequency, gpu_solver, max_norm_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length", [1.0, 100.0, 0.01])
@pytest.mark.parametrize("shift", [0.0, 3000.0])  # far from the origin single precision rounds a plane's offset
def test_points_at_the_tolerance(pkg, oracle, length, shift):
    base = case_from_mesh(oracle, pkg.meshgen.single_cylinder(), h=-1.0, headings_deg=(0.0,))
    case = copy.deepcopy(base)
    case.dxyz_p = base.dxyz_p * length
    case.xyz_p = base.xyz_p + [shift, -shift, 0.0]
    case.nodes = base.nodes + [shift, -shift, 0.0]
    s = gpu_solver(pkg, case, 0)
    w = 0.9
    mx = gpu_frequency(pkg, s, case, w)[3]
    some = np.arange(0, case.n, 13)
    tolp = np.maximum(1e-6, 1e-3 * case.pnsz[some])[:, None]
    pts = np.vstack([case.xyz_p[some] + f * tolp / length * base.dxyz_p[some, :3] for f in (0.0, 0.9, -0.9, 1.1, -1.1)])
    got = s.field_points(pts, kind=0, isol=2)
    s.close()
    v, wk, w1, wvn = oracle.wave_properties(case.ctl, w)
    ref = oracle.field_potential(case, pts, v, wk, w1, wvn, np.radians(case.ctl.headings), mx, isol=2)
    # a decision the other way is a factor of two in every column
    rel = np.abs(got - ref).max(axis=1) / np.abs(ref).max(axis=1)
    assert rel.max() < 1e-6, (int(rel.argmax()), rel.max())
