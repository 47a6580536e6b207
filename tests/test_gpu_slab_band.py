"""The y-z solve with a right-hand side in a band of rows alone: Schur applications
whose band does not fit the one-CTA solve (200 KB of shared memory).  Blocks of
rows (288 columns) at radii that start and end the band at different places of a
block, with blocks on both sides of it, and a 16-CTA cluster (thin channel);
against the oracle at the tolerance of the operator's other tests."""
import numpy as np
import pytest

from oracle import ib_oracle as ibo
from test_gpu_ib import build, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius,nx,ny,nz,nzb", [(0.30, 34, 161, 290, 144), (0.33, 34, 161, 290, 144),
                                                 (0.36, 34, 156, 290, 144), (0.70, 34, 161, 290, 144),
                                                 (0.30, 26, 261, 194, 96)])
def test_schur_operator(radius, nx, ny, nz, nzb):
    p, g, st, ib, ch = build("double_cylinders_z", extra=dict(nx_global=nx, ny_global=ny, nz_global=nz, nzb=nzb,
                                                              body_param_1=0.5 * radius, body_param_2=radius))
    with ch:
        lo, hi = ch.stats()["ib_rows"]
        assert lo > 10 and hi < ny - 10 and (hi - lo + 3) * (nz - 2) * 16 > 200 * 1024
        f = np.random.default_rng(9).standard_normal(4 * ib.body.nb)
        assert rel(ch.schur(f), ibo.schur(g, ib, f, -p["cfl"])) < 1e-11
