"""The fused stage update (projection of one stage formed inside the next
stage's right-hand side) at the edges of its tiles and chunks.

Several steps in one call, whose projected fields are never stored between
stages, against the same steps one call each (bit for bit: both forms round
the same operations) and against the oracle's steps (1e-10 relative
max-norm, as for the other step tests).  Grids: the smallest one, one column
or row past a 32 x 8 tile, an exact multiple, and more planes than one chunk.
"""
import numpy as np
import pytest

from oracle import channel_oracle as co

pytestmark = pytest.mark.gpu

GRIDS = [(6, 5, 6), (8, 9, 8), (34, 9, 14), (38, 10, 20), (66, 18, 26), (20, 35, 258)]


def rel(a, b):
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


def channel(g, st, p, grid, mass):
    import channel3d_parallel_b200 as c3d
    nx, ny, nz = grid
    ch = c3d.Channel(nx_global=nx, ny_global=ny, nz_global=nz, Lxp=p["lxp"], Lzp=p["lzp"], nu=p["nu"], CFL=-1e-3,
                     x_mass_cte=mass, grid_type=1, alpha_stretch=2.0, dPdx=p["dpdx"])
    ch.set_grid(g.x[1:], g.y[1:], g.z[1:])
    for n in ("U", "V", "W"):
        ch.upload(n, getattr(st, n)[1:, 1:, 1:])
    ch.set_scalars(dPdx=st.dPdx, t=0.0, Qflow_x_0=st.Qflow_x_0)
    return ch


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("nsteps,mass", [(2, 1), (3, 0), (5, 1)])
def test_steps_in_one_call(grid, nsteps, mass):
    nx, ny, nz = grid
    p = co.channel_params(nx, ny, nz, 0.06 * nx, 0.05 * nz, 1.0 / 5600.0, x_mass_cte=mass)
    g = co.Grid(p)
    st = co.seeded_initial_state(g, p["dpdx"])
    with channel(g, st, p, grid, mass) as one, channel(g, st, p, grid, mass) as many:
        one.compute_time_step_RK3(nsteps)
        for _ in range(nsteps):
            many.compute_time_step_RK3(1)
            co.compute_time_step_RK3(g, st, 1e-3)
        for n in ("U", "V", "W", "P"):
            got = one.download(n)
            assert np.array_equal(got, many.download(n)), n
            assert rel(got, getattr(st, n)[1:, 1:, 1:]) < 1e-10, n
        assert one.stats()["dPdx"] == many.stats()["dPdx"]
        assert one.check_divergence() < 1e-12
