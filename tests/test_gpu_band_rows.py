"""The block solve of the banded preconditioner at few and odd numbers of block
rows (four markers a row; it runs from both ends to the middle one): as the
regular lattices, precond_apply must return B^-1 v with backward error below
1e-12."""
import numpy as np
import pytest

from test_gpu_band import band_matrix, dense_schur, segments

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nxb", [5, 8, 12, 13, 17, 20, 33, 37])
def test_block_rows(nxb):
    import test_gpu_ib as tib
    from channel3d_parallel_b200 import lib as L
    p, g, st, ib, ch = tib.build("wall_standing_wave", extra=dict(nxb=nxb, nzb=3))
    with ch:
        ch.set_mode(precond=L.PRECOND_BAND)
        nb = ib.body.nb
        lat, segs = segments("wall_standing_wave", ib, p)
        B = band_matrix(dense_schur(ch, 4 * nb), lat, nb // lat, segs)
        v = np.random.default_rng(nxb).standard_normal(4 * nb)
        x = ch.precond_apply(v)
        assert np.abs(B @ x - v).max() < 1e-12 * np.abs(B).sum(axis=1).max() * np.abs(x).max()
