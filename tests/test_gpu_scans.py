"""The one-pass scans over U, V, W at the edges of their runs, rows and warps:
the time step from the fields (exact: a maximum of quotients and scalar
arithmetic in the reference's order), the monitor values and the statistics
profiles against the oracle's restatements, with zero and non-finite entries.
"""
import numpy as np
import pytest

from oracle import channel_oracle as co
from oracle import snapshot as sn

pytestmark = pytest.mark.gpu

GRIDS = [(6, 5, 6), (34, 26, 26), (38, 27, 26), (66, 9, 50)]


def make(grid, seed):
    import channel3d_parallel_b200 as c3d
    nx, ny, nz = grid
    # a viscosity small enough that the convective bound decides
    p = co.channel_params(nx, ny, nz, 0.06 * nx, 0.05 * nz, 1e-6, cfl=1e-4)
    g = co.Grid(p)
    st = co.seeded_initial_state(g, p["dpdx"], project=False)
    rng = np.random.default_rng(seed)
    # velocities kept away from zero, V's walls too, so every component bounds dt
    for a in (st.U, st.V, st.W):
        a[1:, 1:, 1:] = rng.choice((-1.0, 1.0), a[1:, 1:, 1:].shape) * rng.uniform(0.05, 1.0, a[1:, 1:, 1:].shape)
    ch = c3d.Channel(nx_global=nx, ny_global=ny, nz_global=nz, Lxp=p["lxp"], Lzp=p["lzp"], nu=p["nu"], CFL=1e-4,
                     x_mass_cte=0, grid_type=1, alpha_stretch=2.0, dPdx=p["dpdx"])
    ch.set_grid(g.x[1:], g.y[1:], g.z[1:])
    return g, st, ch


def upload(ch, st):
    for n in ("U", "V", "W"):
        ch.upload(n, getattr(st, n)[1:, 1:, 1:])


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("comp", ["U", "V", "W"])
def test_compute_dt_finds_the_slowest_point(grid, comp):
    g, st, ch = make(grid, 1)
    with ch:
        f = getattr(st, comp)
        upper = {"U": (g.nxg - 1, g.nyg - 1, g.nzg - 1), "V": (g.nxg - 1, g.nyg - 1, g.nzg - 1),
                 "W": (g.nxg - 1, g.nyg - 1, g.nzg - 1)}[comp]
        # the smallest velocity of every component at the first and last points
        # of the scan, one component at a time the largest bound
        for at in ((2, 2, 2), upper):
            old = {n: getattr(st, n)[at] for n in ("U", "V", "W")}
            for n in ("U", "V", "W"):
                getattr(st, n)[at] = -1e-3 if n != comp else 2e-3
            upload(ch, st)
            assert ch.compute_dt() == co.compute_dt(g, st)
            for n in ("U", "V", "W"):
                getattr(st, n)[at] = old[n]
        f[3, 3, 3] = 0.0
        upload(ch, st)
        assert ch.compute_dt() == co.compute_dt(g, st)


@pytest.mark.parametrize("grid", GRIDS)
def test_monitor_and_statistics(grid):
    g, st, ch = make(grid, 2)
    with ch:
        upload(ch, st)
        m, r = ch.output_monitor(), sn.monitor_values(g, st)
        for k in ("maxU", "maxV", "maxW"):
            assert m[k] == r[k], k
        for k in ("meanU", "meanV", "meanW"):
            assert abs(m[k] - r[k]) <= 1e-14, k            # values of at most 1
        assert abs(m["max_divergence"] - r["max_divergence"]) <= 1e-12 * r["max_divergence"]
        got, ref = ch.compute_statistics(), sn.compute_statistics(g, st)
        for k in ch.STAT_NAMES:
            assert np.abs(got[k] - ref[k]).max() <= 1e-14, k
        for k in ("Qflow_x", "Qflow_y", "Qflow_z"):
            assert abs(got[k] - ref[k]) <= 1e-14, k
        assert got["nonfinite"] is False
        for n in ("U", "V", "W"):
            a = getattr(st, n)
            keep = a[2, 2, 3]
            a[2, 2, 3] = np.inf
            upload(ch, st)
            assert ch.compute_statistics()["nonfinite"] is True
            a[2, 2, 3] = keep
