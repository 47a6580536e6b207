"""The inverse x transform either side of the line where its CTAs no longer share
SMs (148 CTAs of sixteen lines) and takes fewer threads: rows of one and of two
rounds of threads, against the oracle's Poisson solve at the tolerance of the
other solves."""
import numpy as np
import pytest

from oracle import channel_oracle as co
from test_gpu_slab_blocks import make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [(258, 75, 34), (258, 76, 34), (514, 6, 10), (488, 10, 38), (434, 75, 34),
                                  (434, 76, 34), (74, 76, 34)])
def test_poisson_solve(grid):
    g, st, ch = make(*grid)
    with ch:
        rng = np.random.default_rng(7)
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
