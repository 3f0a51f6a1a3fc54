"""GRN_KIND = 4: Green values and panel integrals rounded to single precision
before assembly.  Both forms round the same values, so the mixed form's stored
matrices are the plain form's rounded once more."""
import numpy as np
import pytest

import __graft_entry__ as g

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w", [(-1.0, 1.1), (-1.0, 2.3)])
def test_plain_matrices_round_to_the_mixed_ones(h, w):
    pkg = g.load_package()
    hg, mesh = pkg.hamsgpu, pkg.meshgen.three_cylinders(with_lid=False)
    got = []
    for form in (hg.HG_PREC_FP64, hg.HG_PREC_MIXED):
        s = hg.Solver(precision=form, grn_kind=4)
        s.keep_matrices(True)
        s.set_mesh(mesh.nodes, mesh.ncon, mesh.ncn, mesh.xyz_p, mesh.ds, mesh.pnsz, mesh.dxyz_p, mesh.body_ranges)
        v, wk, w1, wvn = hg.wave_properties(3, w, h)
        s.set_frequency(v, wk, w1, h, wvn)
        s.fill_factor(0)
        got.append([s.get_matrix(k, mesh.n).astype(np.complex64) for k in (0, 1)])
        s.close()
    for plain, mixed in zip(*got):
        assert np.array_equal(plain, mixed)
