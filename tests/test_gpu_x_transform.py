"""The x transforms at every kind of stage plan (two stages at least: the
lengths up to 8 are split for it) and at line counts that leave a CTA part
empty: Poisson solve of a random right-hand side (1e-11 relative max-norm) and
one FP64 and one mixed step (1e-10) against the oracle."""
import numpy as np
import pytest

from oracle import channel_oracle as co

pytestmark = pytest.mark.gpu

LENGTHS = [4, 6, 8, 12, 16, 18, 36, 54, 64, 162, 256, 384, 486, 512]


def make(nx, ny, nz, mode):
    import channel3d_parallel_b200 as c3d
    p = co.channel_params(nx, ny, nz, 0.06 * nx, 0.05 * nz, 1.0 / 5600.0)
    g = co.Grid(p)
    st = co.seeded_initial_state(g, p["dpdx"])
    ch = c3d.Channel(nx_global=nx, ny_global=ny, nz_global=nz, Lxp=p["lxp"], Lzp=p["lzp"], nu=p["nu"], CFL=-1e-3,
                     x_mass_cte=1, grid_type=1, alpha_stretch=2.0, dPdx=p["dpdx"])
    ch.set_grid(g.x[1:], g.y[1:], g.z[1:])
    ch.set_mode(poisson=mode)
    for n in ("U", "V", "W"):
        ch.upload(n, getattr(st, n)[1:, 1:, 1:])
    ch.set_scalars(dPdx=st.dPdx, t=0.0, Qflow_x_0=st.Qflow_x_0)
    ch.compute_dt()
    return g, st, ch


@pytest.mark.parametrize("Nx", LENGTHS)
def test_poisson_solve(Nx):
    g, st, ch = make(Nx + 2, 8, 8, 0)
    with ch:
        rng = np.random.default_rng(Nx)
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


@pytest.mark.parametrize("Nx", LENGTHS)
@pytest.mark.parametrize("mode", [0, 1])
def test_step(Nx, mode):
    g, st, ch = make(Nx + 2, 10, 14, mode)
    with ch:
        ch.compute_time_step_RK3(1)
        co.compute_time_step_RK3(g, st, 1e-3)
        for n in ("U", "V", "W"):
            ref = getattr(st, n)[1:, 1:, 1:]
            assert np.abs(ch.download(n) - ref).max() < 1e-10 * np.abs(ref).max(), n
        assert ch.check_divergence() < 1e-12
