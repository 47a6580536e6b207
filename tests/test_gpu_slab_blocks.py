"""The y-z solve by blocks of rows (slabs with more than 256 columns, or that
need a 16-CTA cluster) against the oracle's Poisson solve, 1e-11 relative
max-norm: one block, a last block of one and of seven rows, more blocks than
the chain takes at once; FP64, and the FP32 form inside one mixed step."""
import numpy as np
import pytest

from oracle import channel_oracle as co

pytestmark = pytest.mark.gpu


def make(nx, ny, nz, mode=None):
    import channel3d_parallel_b200 as c3d
    p = co.channel_params(nx, ny, nz, 0.06 * nx, 0.03 * nz, 1.0 / 5600.0)
    g = co.Grid(p)
    st = co.seeded_initial_state(g, p["dpdx"])
    ch = c3d.Channel(nx_global=nx, ny_global=ny, nz_global=nz, Lxp=p["lxp"], Lzp=p["lzp"], nu=p["nu"], CFL=-1e-3,
                     x_mass_cte=1, grid_type=1, alpha_stretch=2.0, dPdx=p["dpdx"])
    ch.set_grid(g.x[1:], g.y[1:], g.z[1:])
    if mode is not None:
        ch.set_mode(poisson=mode)
    for n in ("U", "V", "W"):
        ch.upload(n, getattr(st, n)[1:, 1:, 1:])
    ch.set_scalars(dPdx=st.dPdx, t=0.0, Qflow_x_0=st.Qflow_x_0)
    ch.compute_dt()
    return g, st, ch


@pytest.mark.parametrize("grid", [(8, 9, 290), (6, 10, 326), (8, 16, 386), (6, 76, 434), (6, 260, 194)])
def test_poisson_solve(grid):
    g, st, ch = make(*grid)
    with ch:
        rng = np.random.default_rng(3)
        rhs = g.rhs_p_array()
        inner = (slice(2, g.nxg - 1), slice(2, g.nyg), slice(2, g.nzg - 1))
        rhs[inner] = rng.standard_normal(rhs[inner].shape)
        rhs[g.nxg - 1, :, :] = rhs[2, :, :]
        rhs[:, :, g.nzg - 1] = rhs[:, :, 2]
        ch.upload("RHS_P", rhs[2:, 2:, 2:])
        ch.solve_poisson_equation()
        ref = co.solve_poisson_equation(g, rhs)[2:, 2:, 2:]
        got = ch.download("RHS_P")
        assert np.abs(got - ref)[:, :, :-1].max() < 1e-11 * np.abs(ref).max()


def test_mixed_step():
    from channel3d_parallel_b200 import lib as L
    g, st, ch = make(8, 19, 290, L.POISSON_MIXED)
    with ch:
        ch.compute_time_step_RK3(1)
        co.compute_time_step_RK3(g, st, 1e-3)
        for n in ("U", "V", "W"):
            ref = getattr(st, n)[1:, 1:, 1:]
            assert np.abs(ch.download(n) - ref).max() < 1e-10 * np.abs(ref).max(), n
        assert ch.check_divergence() < 1e-12
