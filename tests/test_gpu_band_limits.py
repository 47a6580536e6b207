"""Marker lattices the banded preconditioner does not take: a row too long for the
block solve (1,100 markers; 1,088 go).  It is refused each time it is asked for,
and the body steps on without it."""
import pytest

pytestmark = pytest.mark.gpu

CASE = dict(nx_global=34, ny_global=49, nz_global=14, Lxp=2.0, Lzp=0.6, nu=3e-4, CFL=-1e-3, grid_type=2,
            alpha_stretch=2.0, min_buffer_width=0.45, body_type="wall_standing_wave", body_param_1=0.02,
            body_param_2=1.2, body_param_3=1.0, body_param_4=0.2, nzb=3, cg_max_iter=3)


@pytest.mark.parametrize("nxb,taken", [(1088, True), (1100, False)])
def test_longest_marker_rows(nxb, taken):
    import channel3d_parallel_b200 as c3d
    with c3d.Channel(nxb=nxb, **CASE) as ch:
        c3d.seeded_initial_state(ch, 9e-4, 3e-4)
        ch.compute_heaviside()
        for mode in (c3d.lib.PRECOND_BAND, c3d.lib.PRECOND_LEARNED, c3d.lib.PRECOND_BAND):
            if taken:
                ch.set_mode(precond=mode)
            else:
                with pytest.raises(c3d.C3DError, match="-6"):
                    ch.set_mode(precond=mode)
        if not taken:
            with pytest.raises(c3d.C3DError):
                ch.precond_probe()
            assert ch.compute_time_step_RK3(1) == c3d.lib.WARN_NOT_CONVERGED
