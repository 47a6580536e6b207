"""Banded preconditioners of two live handles whose marker lattices need different
amounts of shared memory: what the first computes does not change when the
second is set up.  Lattices: many block rows, then few; 250 marker rows (the
direct DFTs, above the default 48 KB), then 10."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASE = dict(nx_global=34, ny_global=49, nz_global=14, Lxp=2.0, Lzp=0.6, nu=3e-4, CFL=-1e-3, grid_type=2,
            alpha_stretch=2.0, min_buffer_width=0.45, body_type="wall_standing_wave", body_param_1=0.02,
            body_param_2=1.2, body_param_3=1.0, body_param_4=0.2)


@pytest.mark.parametrize("first,second", [(dict(nxb=96, nzb=3), dict(nxb=5, nzb=3)),
                                          (dict(nxb=5, nzb=250), dict(nxb=5, nzb=10))])
def test_second_handle_leaves_the_first_alone(first, second):
    import channel3d_parallel_b200 as c3d

    def handle(lat):
        ch = c3d.Channel(**CASE, **lat)
        ch.compute_dt()
        ch.compute_heaviside()
        ch.set_mode(precond=c3d.lib.PRECOND_BAND)
        return ch

    with handle(first) as a:
        v = np.random.default_rng(3).standard_normal(4 * a.dims["nb"])
        before = a.precond_apply(v)
        with handle(second) as b:
            b.precond_apply(np.ones(4 * b.dims["nb"]))
            assert np.array_equal(a.precond_apply(v), before)
