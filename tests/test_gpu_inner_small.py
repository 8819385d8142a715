"""The GCR's inner solve on small lattices (one cooperative kernel): its residual, and its ways out."""
import numpy as np
import pytest

import oracle as O
from util import dev, empty_like_dev, host

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def q():
    import qcu_b200

    return qcu_b200


@pytest.mark.parametrize("seed", range(8))
def test_residual_after_a_steep_iteration(q, seed):
    """kappa 1e-3: M_pc = 1 - 1e-6 D D, so one inner iteration takes |r|^2 down to the 16-bit rounding of s and t, some
    1e-10 and 1e-11 of what it was each, 1e-21 together: less than asked for (inner_tol^2 = 1e-24).  No outer step may
    count as done after one iteration, as it does when the residual's sums round to zero at 1e-8 |s|^2."""
    latt, kappa = [4, 4, 4, 4], 1e-3
    U = O.gauge_smooth(latt, 0.3, 60 + seed)
    b = O.fermion_gauss(O.full_shape(latt), 70 + seed)
    x = empty_like_dev(O.full_shape(latt))
    with q.Gauge(dev(U), latt, t_boundary=-1.0) as G:
        info = G.invert(x, dev(b), kappa, tol=1e-12, maxiter=400, solver="gcr", precision=16, inner_iters=40,
                        inner_tol=1e-12, gcr_k=4)
    assert info["status"] == 1 and info["fallback"] == 0, info
    assert info["iterations"] >= 2 * info["reliable_updates"], info
    r = b - O.mfull(host(x), U, latt, kappa, -1.0)
    assert np.linalg.norm(r) <= 1.05e-12 * np.linalg.norm(b)


@pytest.mark.parametrize("clover", [False, True])
@pytest.mark.parametrize("scale", [1e40, 1e-42])
def test_inner_solve_without_a_result(q, clover, scale):
    """Sources beyond FP32: the inner solve finds infinities and NaN, or products of zero, and ends without a direction;
    the plain FP64 solver finishes."""
    latt, kappa = [6, 4, 2, 10], 0.12
    U = O.gauge_smooth(latt, 0.3, 81)
    b = O.fermion_gauss(O.full_shape(latt), 82)
    A = [O.clover_build(U, latt, p, kappa) for p in (0, 1)] if clover else [None, None]
    x = empty_like_dev(O.full_shape(latt))
    with q.Gauge(dev(U), latt, t_boundary=-1.0, clover_coeff=kappa if clover else 0.0) as G:
        kw = dict(tol=1e-10, maxiter=400, solver="gcr", precision=16, inner_iters=16, inner_tol=0.1, gcr_k=4, clover=clover)
        info = G.invert(x, dev(b * scale), kappa, **kw)
        assert info["status"] == 1 and info["fallback"] == 1, info
        r = b - O.mfull(host(x) / scale, U, latt, kappa, -1.0, True, A[0], A[1])
        assert np.linalg.norm(r) <= 1.05e-10 * np.linalg.norm(b)
        b[0].flat[7] = np.nan
        info = G.invert(x, dev(b), kappa, **kw)
        assert info["status"] == 4, info
        b[0].flat[7] = 0  # and nothing of it stays
        info = G.invert(x, dev(b), kappa, **kw)
        assert info["status"] == 1 and info["fallback"] == 0, info


@pytest.mark.parametrize("solver,precision", [("gcr", 16), ("gcr", 32), ("bicgstab", 16), ("bicgstab", 64), ("batch", 16)])
@pytest.mark.parametrize("half", [0, 1])
def test_source_with_an_infinity_ends(q, solver, precision, half):
    """|b|^2 and the target are infinite, so no residual is above the target and no cycle counts as stalled."""
    latt, kappa = [4, 4, 4, 4], 0.12
    U = O.gauge_smooth(latt, 0.3, 83)
    b = O.fermion_gauss(O.full_shape(latt), 84)
    b[half].flat[7] = np.inf
    x = empty_like_dev(O.full_shape(latt))
    with q.Gauge(dev(U), latt, t_boundary=-1.0) as G:
        if solver == "batch":
            info = q.invert_batch([(G, x[None], dev(b[None]), kappa, False)], tol=1e-10, maxiter=400, precision=16)[0][0]
        else:
            info = G.invert(x, dev(b), kappa, tol=1e-10, maxiter=400, solver=solver, precision=precision)
    assert info["status"] == 4, info
