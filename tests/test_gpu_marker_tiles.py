"""Interpolation and spreading over marker lattices that the patches of markers
do not divide (1e-12 max-norm relative, as on the regular ones): a last patch
of one column, of one row, fewer rows or columns than a patch, many markers a
cell, and markers so far apart that a patch's box of grid points is not kept
on chip."""
import numpy as np
import pytest

from oracle import channel_oracle as co
from test_gpu_ib import build, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nxb,nzb", [(17, 5), (33, 9), (5, 4), (40, 3), (65, 1), (96, 24), (8, 4), (3, 13)])
def test_interpolation_and_spreading(nxb, nzb):
    p, g, st, ib, ch = build("wall_standing_wave", extra=dict(nxb=nxb, nzb=nzb))
    with ch:
        rng = np.random.default_rng(nxb + nzb)
        U, V, W = (rng.standard_normal(a.shape) for a in (st.U, st.V, st.W))
        co.apply_boundary_conditions(g, U, V, W)
        for name, A in (("U", U), ("V", V), ("W", W)):
            ch.upload(name, A[1:, 1:, 1:])
        assert rel(ch.regT(), ib.ops.E(U, V, W)) < 1e-12
        assert rel(ch.regT_1n(), ib.ops.E1n(U, V, W)) < 1e-12
        Pr = g.rhs_p_array()
        Pr[2:, 2:, 2:] = rng.standard_normal(Pr[2:, 2:, 2:].shape)
        ch.upload("P_INTERIM", Pr[2:, 2:, 2:])
        assert rel(ch.regTc_1n("P_INTERIM"), ib.ops.E1n_c(Pr)) < 1e-12
        f = rng.standard_normal(ib.body.nb)
        for comp, (name, shape) in enumerate((("U_REG", st.U.shape), ("V_REG", st.V.shape), ("W_REG", st.W.shape))):
            ch.reg(comp + 1, f)
            assert rel(ch.download(name), ib.ops.R(comp, f, shape)[1:, 1:, 1:]) < 1e-12, name
