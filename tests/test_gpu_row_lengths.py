"""Kernels with the row length compiled in, at every such length, 1e-11 relative
max-norm: the y-z solves against the oracle's Poisson solve, in clusters (few
rows of j and many: columns per thread differ) and by blocks, with a
part-filled last block; the x transforms against the oracle's time step (its
divergence with and without the bulk flux), with a part-filled last group of
lines."""
import numpy as np
import pytest

from oracle import channel_oracle as co

pytestmark = pytest.mark.gpu

CLUSTER = (64, 72, 96, 108, 128, 144, 162, 192, 216, 256)
BLOCKS = (192, 216, 256, 288, 324, 384, 432, 486, 512)
CASES = [(n, 17) for n in CLUSTER] + [(n, 127) for n in CLUSTER] + [(n, 259 if n <= 256 else 19) for n in BLOCKS]


@pytest.mark.parametrize("nz,rows", CASES)
def test_poisson_solve(nz, rows):
    import channel3d_parallel_b200 as c3d
    p = co.channel_params(6, rows + 1, nz + 2, 0.36, 0.03 * nz, 1.0 / 5600.0)
    g = co.Grid(p)
    rhs = g.rhs_p_array()
    inner = (slice(2, g.nxg - 1), slice(2, g.nyg), slice(2, g.nzg - 1))
    rhs[inner] = np.random.default_rng(nz + rows).standard_normal(rhs[inner].shape)
    rhs[g.nxg - 1, :, :] = rhs[2, :, :]
    rhs[:, :, g.nzg - 1] = rhs[:, :, 2]
    with c3d.Channel(nx_global=6, ny_global=rows + 1, nz_global=nz + 2, Lxp=p["lxp"], Lzp=p["lzp"], nu=p["nu"],
                     CFL=-1e-3, grid_type=1, alpha_stretch=2.0) as ch:
        ch.set_grid(g.x[1:], g.y[1:], g.z[1:])
        ch.upload("RHS_P", rhs[2:, 2:, 2:])
        ch.solve_poisson_equation()
        got = ch.download("RHS_P")
    ref = co.solve_poisson_equation(g, rhs)[2:, 2:, 2:]
    assert np.abs(got - ref)[:, :, :-1].max() < 1e-11 * np.abs(ref).max()


@pytest.mark.parametrize("nx", (32, 48, 64, 72, 96, 108, 128, 144, 162, 192, 216, 256, 288, 324, 384, 432, 486, 512))
def test_time_step(nx):
    import channel3d_parallel_b200 as c3d
    p = co.channel_params(nx + 2, 8, 8, 0.06 * nx, 0.3, 1.0 / 5600.0)
    g = co.Grid(p)
    st = co.seeded_initial_state(g, p["dpdx"])
    with c3d.Channel(nx_global=nx + 2, ny_global=8, nz_global=8, Lxp=p["lxp"], Lzp=p["lzp"], nu=p["nu"], CFL=-1e-3,
                     x_mass_cte=1, grid_type=1, alpha_stretch=2.0, dPdx=p["dpdx"]) as ch:
        ch.set_grid(g.x[1:], g.y[1:], g.z[1:])
        for n in ("U", "V", "W"):
            ch.upload(n, getattr(st, n)[1:, 1:, 1:])
        ch.set_scalars(dPdx=st.dPdx, t=0.0, Qflow_x_0=st.Qflow_x_0)
        ch.compute_dt()
        ch.compute_time_step_RK3(2)
        for _ in range(2):
            co.compute_time_step_RK3(g, st, 1e-3)
        for n in ("U", "V", "W"):
            ref = getattr(st, n)[1:, 1:, 1:]
            assert np.abs(ch.download(n) - ref).max() < 1e-11 * np.abs(ref).max(), n
