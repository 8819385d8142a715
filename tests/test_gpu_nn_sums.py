"""The training step's sums over many tiles a block."""
import numpy as np
import pytest

import oracle as O
from oracle import nn_ref as R
from util import dev, rel

pytestmark = pytest.mark.gpu


def test_gradient_over_many_tiles_a_block():
    """512 copies of one sample (32768 tiles, some 110 for each of the resident blocks) have the gradient and the loss of
    the one.  A block adds its tiles up in FP32: 6e-8 sqrt(110 / 3) = 3.6e-7 for the sums of one block, at most as much
    for all together; the bar is 5e-7."""
    import qcu_b200 as q

    latt, B = [8, 8, 8, 8], 512
    U = O.gauge_smooth(latt, 0.3, 18)
    e = O.fermion_gauss((1,) + O.half_shape(latt), 20)
    r = e + 0.5 * O.fermion_gauss((1,) + O.half_shape(latt), 19)
    net = q.Network()
    w = np.random.default_rng(21).normal(0, 0.1, net.num_params()).astype(np.float32)
    net.set_weights(w)
    with q.Gauge(dev(U), latt, t_boundary=-1.0) as G:
        many = [dev(np.repeat(v, B, axis=0)) for v in (r, e)]
        loss, grad = net.train_step(G, *many, B, 0.0, want_grad=True)
    lat = R.Lattice(U, latt, -1.0)
    gref, lref = R.gradient(lat, w.astype(np.float64), r.reshape(1, lat.Vh, 4, 3), e.reshape(1, lat.Vh, 4, 3))
    assert abs(loss - lref) <= 5e-7 * lref
    assert rel(grad, gref) <= 5e-7
