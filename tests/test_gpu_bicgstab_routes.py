"""The plain solver's two graphs: a device-side loop to the next reliable update, and unrolled iterations with gated
updates, which solves with a delta above 0.6 take (0.4 from 2^14 sites per parity on)."""
import numpy as np
import pytest

import oracle as O
from util import dev, empty_like_dev, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [64, 32, 16])
@pytest.mark.parametrize("delta", [0.0, 0.1, 0.4, 0.41, 0.6, 0.61, 0.9, 0.99])
@pytest.mark.parametrize("latt,chunk,limit", [([6, 4, 4, 6], 32, 0.6), ([16, 16, 8, 16], 16, 0.4)])
def test_both_graphs_take_the_same_steps(precision, delta, latt, chunk, limit):
    """The same iterations, updates and bits on either route; the default route by the kernels it launches."""
    import qcu_b200 as q

    kappa = 0.122
    U = O.gauge_smooth(latt, 0.3, 91)
    b = O.fermion_gauss(O.full_shape(latt), 92)
    got = {}
    with q.Gauge(dev(U), latt, t_boundary=-1.0) as G:
        for c in (0, chunk):  # chunk: what the unrolled route takes on a lattice of this size
            x, before = empty_like_dev(O.full_shape(latt)), q.kernel_launches()
            info = G.invert(x, dev(b), kappa, tol=1e-10, maxiter=500, precision=precision, delta=delta, chunk=c)
            assert info["status"] == 1, info
            got[c] = host(x), info["iterations"], info["reliable_updates"], q.kernel_launches() - before
    r = b - O.mfull(got[0][0], U, latt, kappa, -1.0)
    assert np.linalg.norm(r) <= 1.05e-10 * np.linalg.norm(b)
    assert got[0][1:3] == got[chunk][1:3]
    assert np.array_equal(got[0][0], got[chunk][0])
    assert (got[0][3] == got[chunk][3]) == (delta > limit)
