"""A grid barrier of a cooperative kernel that gave up (k_inner_small, k_mg_coarse).

QCU_BARRIER_GIVE_UP marks the barrier's state on the host, as a wait that ran out leaves it, before each launch: the
kernels return at once, the call ends with an error at the first step whose scalars it reads, and the next call on the
same device, handle and multigrid finds nothing of it."""
import time

import numpy as np
import pytest

import oracle as O
from util import dev, empty_like_dev, host

pytestmark = pytest.mark.gpu

LATT, KAPPA = [8, 8, 8, 8], 0.124


@pytest.fixture(scope="module")
def q():
    import qcu_b200

    return qcu_b200


def _fails_at_once(q, call, monkeypatch, which):
    """`call` raises within half of the launches that it takes otherwise, and afterwards returns the same again."""
    x0, n0 = call()
    monkeypatch.setenv("QCU_BARRIER_GIVE_UP", which)
    before, t = q.kernel_launches(), time.monotonic()
    with pytest.raises(q.QcuError, match="barrier"):
        call()
    assert q.kernel_launches() - before <= n0 / 2
    assert time.monotonic() - t < 1.0  # no wait ran out
    monkeypatch.delenv("QCU_BARRIER_GIVE_UP")
    x1, _ = call()
    assert np.array_equal(x0, x1)


@pytest.mark.parametrize("clover", [False, True])
def test_inner_solve_of_small_lattices(q, monkeypatch, clover):
    U, b = O.gauge_smooth(LATT, 0.25, 31), dev(O.fermion_gauss(O.full_shape(LATT), 32))
    with q.Gauge(dev(U), LATT, t_boundary=-1.0, clover_coeff=KAPPA if clover else 0.0) as G:

        def call():
            x, before = empty_like_dev(O.full_shape(LATT)), q.kernel_launches()
            info = G.invert(x, b, KAPPA, tol=1e-10, maxiter=4000, solver="gcr", precision=16, inner_iters=8,
                            inner_tol=0.2, gcr_k=4, clover=clover)
            assert info["status"] == 1 and info["reliable_updates"] >= 5, info
            return host(x), q.kernel_launches() - before

        _fails_at_once(q, call, monkeypatch, "inner")


def test_coarse_solve(q, monkeypatch):
    U, b = O.gauge_smooth(LATT, 0.25, 33), dev(O.fermion_gauss(O.full_shape(LATT), 34))
    with q.Gauge(dev(U), LATT, t_boundary=-1.0) as G:
        mg = q.Multigrid(G, KAPPA, n_vec=4, setup_maxiter=8, nu_post=2, coarse_tol=0.05, coarse_maxiter=30)

        def multigrid():
            x, before = empty_like_dev(O.full_shape(LATT)), q.kernel_launches()
            info = mg.invert(x, b, tol=1e-10, maxiter=300)
            assert info["status"] == 1 and info["outer"] >= 5, info
            return host(x), q.kernel_launches() - before

        def preconditioner():
            x, before = empty_like_dev(O.full_shape(LATT)), q.kernel_launches()
            info = G.invert(x, b, KAPPA, tol=1e-10, maxiter=4000, solver="gcr", precision=16, inner_iters=8,
                            inner_tol=0.2, gcr_k=4, precond=3, mg=mg)
            assert info["status"] == 1 and info["reliable_updates"] >= 5, info
            return host(x), q.kernel_launches() - before

        _fails_at_once(q, multigrid, monkeypatch, "coarse")
        _fails_at_once(q, preconditioner, monkeypatch, "coarse")
        _fails_at_once(q, preconditioner, monkeypatch, "inner")
        monkeypatch.setenv("QCU_BARRIER_GIVE_UP", "coarse")
        with pytest.raises(q.QcuError, match="barrier"):
            multigrid()
        orth, gal = mg.check()  # reads no coarse solve: an error before it is not its own
        mg.close()
    assert orth <= 1e-5 and gal <= 1e-5
