"""Steps of one call with the mixed Poisson solve (stage fields that alternate
between arrays, the last projection alone at the end) against calls of one step:
the same bits, for odd and even numbers, with and without the mass-flow
correction."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cte", [0, 1])
@pytest.mark.parametrize("nsteps", [3, 4, 5])
def test_calls_of_several_steps(nsteps, cte):
    import channel3d_parallel_b200 as c3d
    out = []
    for calls in ([nsteps], [1] * nsteps):
        with c3d.Channel(nx_global=50, ny_global=34, nz_global=38, Lxp=3.0, Lzp=1.5, nu=1 / 5600.0, CFL=-1e-3,
                         x_mass_cte=cte, grid_type=1, alpha_stretch=2.0, dPdx=3 / 5600.0) as ch:
            c3d.seeded_initial_state(ch, 3 / 5600.0, 1 / 5600.0)
            ch.set_mode(poisson=c3d.lib.POISSON_MIXED)
            for n in calls:
                ch.compute_time_step_RK3(n)
            out.append([ch.download(n) for n in ("U", "V", "W", "P")] + [np.array(ch.stats()["dPdx"])])
    for a, b in zip(*out):
        assert np.array_equal(a, b)
