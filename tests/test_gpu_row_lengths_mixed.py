"""The FP32 kernels with the row length compiled in, at every such length: one
mixed step (FP32 solve and one refinement) against the oracle's FP64 step,
1e-10 relative max-norm."""
import numpy as np
import pytest

from oracle import channel_oracle as co

pytestmark = pytest.mark.gpu

X = (32, 48, 64, 72, 96, 108, 128, 144, 162, 192, 216, 256, 288, 324, 384, 432, 486, 512)
Z = (64, 72, 96, 108, 128, 144, 162, 192, 216, 256, 288, 324, 384, 432, 486, 512)


@pytest.mark.parametrize("nx,rows,nz", [(n, 7, 6) for n in X] + [(4, 17, n) for n in Z] +
                         [(4, 127, n) for n in (64, 128, 192, 256)])
def test_mixed_step(nx, rows, nz):
    import channel3d_parallel_b200 as c3d
    from channel3d_parallel_b200 import lib as L
    p = co.channel_params(nx + 2, rows + 1, nz + 2, 0.06 * nx, 0.03 * nz, 1.0 / 5600.0)
    g = co.Grid(p)
    st = co.seeded_initial_state(g, p["dpdx"])
    with c3d.Channel(nx_global=nx + 2, ny_global=rows + 1, nz_global=nz + 2, Lxp=p["lxp"], Lzp=p["lzp"], nu=p["nu"],
                     CFL=-1e-3, x_mass_cte=1, grid_type=1, alpha_stretch=2.0, dPdx=p["dpdx"]) as ch:
        ch.set_grid(g.x[1:], g.y[1:], g.z[1:])
        ch.set_mode(poisson=L.POISSON_MIXED)
        for n in ("U", "V", "W"):
            ch.upload(n, getattr(st, n)[1:, 1:, 1:])
        ch.set_scalars(dPdx=st.dPdx, t=0.0, Qflow_x_0=st.Qflow_x_0)
        ch.compute_dt()
        ch.compute_time_step_RK3(1)
        co.compute_time_step_RK3(g, st, 1e-3)
        for n in ("U", "V", "W"):
            ref = getattr(st, n)[1:, 1:, 1:]
            assert np.abs(ch.download(n) - ref).max() < 1e-10 * np.abs(ref).max(), n
