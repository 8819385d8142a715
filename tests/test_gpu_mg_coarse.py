"""The coarse solve's launch shapes: how many aggregates a block takes, where A_c lies, how lanes share a row."""
import pytest

import oracle as O
from util import dev, empty_like_dev, host, rel

pytestmark = pytest.mark.gpu

# aggregates of 2 x 2 x 2 x 4 sites, on 148 multiprocessors
SHAPES = [
    # 225 aggregates: two a block, the last block half empty; 24 rows, in shared memory
    ([6, 10, 10, 12], 12),
    # 375: four a block, the last with three; in shared memory, and (32 rows: 74 KB each) read from L2
    ([10, 10, 10, 12], 12),
    ([10, 10, 10, 12], 16),
    # 735: four of 24 rows a block in two turns, the second not full; eight of 4 and of 16 rows in one
    ([10, 14, 14, 12], 12),
    ([10, 14, 14, 12], 2),
    ([10, 14, 14, 12], 8),
    # 1715: sixteen a block on two warps each, the last with three, of 8, 10 and 14 rows (4, 3 and 2 lanes a row);
    # eight of 16 rows in two turns
    ([14, 14, 14, 20], 4),
    ([14, 14, 14, 20], 5),
    ([14, 14, 14, 20], 7),
    ([14, 14, 14, 20], 8),
    # 3969: a warp each, 2 and 6 rows (16 and 5 lanes a row); 16 rows, 73 MB: four blocks an SM, two each, ragged turns
    ([18, 18, 14, 28], 1),
    ([18, 18, 14, 28], 3),
    ([18, 18, 14, 28], 8),
]


@pytest.mark.parametrize("latt,n_vec", SHAPES)
def test_coarse_solve_shapes(latt, n_vec):
    """P^dag P = 1 and the Galerkin identity; and without a smoother the cycle is P A_c^-1 P^dag, which gives a vector
    x = P c back from M x (M the oracle's): in one outer step, to the condition of A_c (below 100 here) times the coarse
    solve's 1e-6 and the FP32 rounding of A_c, so within 1e-3."""
    import qcu_b200 as q

    kappa = 0.122
    U = O.gauge_smooth(latt, 0.25, 61)
    x, y = empty_like_dev(O.full_shape(latt)), empty_like_dev(O.full_shape(latt))
    with q.Gauge(dev(U), latt, t_boundary=-1.0) as G:
        mg = q.Multigrid(G, kappa, geo_block_size=[2, 2, 2, 4], n_vec=n_vec, setup_maxiter=24, nu_pre=0, nu_post=0,
                         coarse_tol=1e-6, coarse_maxiter=400)
        orth, gal = mg.check()
        assert orth <= 1e-5 and gal <= 1e-5
        mg.invert(x, dev(O.fermion_gauss(O.full_shape(latt), 62)), tol=1e-10, maxiter=1)  # a multiple of P c
        info = mg.invert(y, dev(O.mfull(host(x), U, latt, kappa, -1.0)), tol=1e-3, maxiter=3)
        mg.close()
    assert info["status"] == 1 and info["outer"] == 1 and 1 < info["coarse_iters"] < 400, info
    assert rel(host(y), host(x)) <= 1e-3
