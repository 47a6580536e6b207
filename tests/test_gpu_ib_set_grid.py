"""A new grid on a handle whose immersed body has been solved for: the Schur
operator, the preconditioners and whole steps equal, bit for bit, those of a
handle that had that grid from the start (the same kernels on the same tables)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASE = dict(nx_global=34, ny_global=49, nz_global=14, nu=3e-4, CFL=-1e-3, x_mass_cte=1, grid_type=2,
            alpha_stretch=2.0, min_buffer_width=0.45, body_type="wall_standing_wave", nxb=32, nzb=12,
            body_param_1=0.02, body_param_2=1.2, body_param_3=1.0, body_param_4=0.2, cg_tol=1e-12, cg_max_iter=400,
            dPdx=9e-4)


def channel(lx, lz, alpha):
    import channel3d_parallel_b200 as c3d
    return c3d.Channel(**dict(CASE, Lxp=lx, Lzp=lz, alpha_stretch=alpha))


def start(ch, grid):
    import channel3d_parallel_b200 as c3d
    if grid is not None:
        ch.set_grid(grid["x"], grid["y"], grid["z"])
    ch.set_scalars(dPdx=CASE["dPdx"])            # time 0
    ch.setup_IB_geometry()
    ch.setup_IB_operators()
    ch.compute_dt()
    ch.compute_heaviside()
    c3d.seeded_initial_state(ch, CASE["dPdx"], CASE["nu"], amplitude=0.05)
    ch.upload("FB", np.zeros(4 * ch.dims["nb"]))


@pytest.mark.parametrize("mode", ["none", "jacobi", "band"])
def test_new_grid_equals_a_fresh_handle(mode):
    from channel3d_parallel_b200 import lib as L
    code = {"none": L.PRECOND_NONE, "jacobi": L.PRECOND_JACOBI, "band": L.PRECOND_BAND}[mode]
    with channel(2.0, 0.6, 2.0) as old, channel(2.5, 0.7, 2.2) as other:
        grid = other.grid()
        old.set_mode(precond=code)
        start(old, None)
        old.compute_time_step_RK3(1)             # operators, loop and preconditioner of the first grid
        out = []
        with channel(2.0, 0.6, 2.0) as new:
            new.set_mode(precond=code)
            for ch in (old, new):
                start(ch, grid)
                f = np.random.default_rng(1).standard_normal(4 * ch.dims["nb"])
                res = [ch.schur(f), ch.precond_apply(f)]
                ch.compute_time_step_RK3(2)
                out.append(res + [ch.download(n) for n in ("U", "V", "W", "FB")])
        for name, a, b in zip(("schur", "precond", "U", "V", "W", "FB"), *out):
            assert np.array_equal(a, b), (name, np.abs(a - b).max() / np.abs(b).max())


def test_grid_that_changes_the_marker_count_is_refused_whole():
    """double_cylinders_z takes its marker count from the spacings; the device
    arrays keep the first one, so another count is refused without a change: the
    body works on, and with the first grid set again as before."""
    import channel3d_parallel_b200 as c3d
    kw = dict(nx_global=34, ny_global=33, nz_global=14, Lzp=1.0, nu=3e-4, CFL=-0.01, grid_type=0, alpha_stretch=0.0,
              body_type="double_cylinders_z", nxb=0, nzb=6, body_param_1=0.15, body_param_2=0.3, body_param_3=0.015)
    with c3d.Channel(**dict(kw, Lxp=2.0)) as ch, c3d.Channel(**dict(kw, Lxp=1.0)) as wide:
        first, second, nb = ch.grid(), wide.grid(), ch.dims["nb"]
        assert wide.dims["nb"] > nb
        ch.compute_dt()
        ch.compute_heaviside()
        f = np.random.default_rng(2).standard_normal(4 * nb)
        before = ch.schur(f)
        with pytest.raises(c3d.C3DError, match="marker count"):
            ch.set_grid(second["x"], second["y"], second["z"])
        assert len(ch.download("XB")) == nb and np.isfinite(ch.schur(f)).all()
        ch.set_grid(first["x"], first["y"], first["z"])
        ch.compute_heaviside()
        assert np.array_equal(ch.schur(f), before)
