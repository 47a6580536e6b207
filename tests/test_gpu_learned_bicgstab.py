"""The Schur solver called by itself (c3d_bicgstab) with the learned preconditioner,
whose warm start adds a product of its own: the solution of a given right-hand
side is that of the unpreconditioned solver.  Both end at a residual of 1e-12,
against |b| of a few tenths: with the operator's condition, about 2e3, solutions
within some 1e-8 of each other; 1e-6 leaves two orders in hand."""
import numpy as np
import pytest

from test_gpu_ib import build, rel

pytestmark = pytest.mark.gpu


def test_learned_solution_of_a_given_right_hand_side():
    from channel3d_parallel_b200 import lib as L
    p, g, st, ib, ch = build("wall_standing_wave", cg_tol=1e-12, cg_max_iter=600)
    with ch:
        n = 4 * ch.dims["nb"]
        b = ch.schur(np.random.default_rng(4).standard_normal(n))
        sol = {}
        for mode in (L.PRECOND_NONE, L.PRECOND_LEARNED):
            ch.set_mode(precond=L.PRECOND_BAND)
            if mode == L.PRECOND_LEARNED:
                ch.precond_probe()
                ch.precond_train(epochs=300, lr=2e-3)
            ch.set_mode(precond=mode)
            ch.upload("FB", np.zeros(n))
            ch.bicgstab(b)
            assert ch.stats()["last_residual"] < 1e-12
            sol[mode] = ch.download("FB")
            assert rel(ch.schur(sol[mode]), b) < 1e-9
        assert rel(sol[L.PRECOND_LEARNED], sol[L.PRECOND_NONE]) < 1e-6
