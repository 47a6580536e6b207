"""The y-z solve either side of the line between 16-CTA clusters and blocks of rows
(few slabs of many rows stay in clusters, many go by blocks), against the oracle
at the tolerances of the block tests: clusters half and nearly full, one and two
waves of them, blocks from 256 columns down; the FP32 forms inside one mixed step."""
import numpy as np
import pytest

from oracle import channel_oracle as co
from test_gpu_slab_blocks import make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,cs", [((6, 301, 18), 16), ((26, 251, 20), 16), ((38, 161, 18), 16), ((38, 501, 18), 16),
                                     ((74, 301, 18), 16), ((98, 251, 130), 16), ((26, 251, 258), 16)])
def test_poisson_solve(grid, cs):
    g, st, ch = make(*grid)
    with ch:
        assert ch.stats()["slab_cluster"][0] == cs
        rng = np.random.default_rng(5)
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


@pytest.mark.parametrize("grid", [(14, 301, 20), (50, 301, 38)])
def test_mixed_step(grid):
    from channel3d_parallel_b200 import lib as L
    g, st, ch = make(*grid, L.POISSON_MIXED)
    with ch:
        ch.compute_time_step_RK3(1)
        co.compute_time_step_RK3(g, st, 1e-3)
        for n in ("U", "V", "W"):
            ref = getattr(st, n)[1:, 1:, 1:]
            assert np.abs(ch.download(n) - ref).max() < 1e-10 * np.abs(ref).max(), n
