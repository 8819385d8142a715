"""The multi-rhs layout kernels with all rows of a tile in a block, and with sixteen where the tiles are few."""
import numpy as np
import pytest

import oracle as O
from util import dev, host, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("latt", [[2, 1, 1, 3], [4, 4, 4, 4], [6, 9, 9, 11]])
@pytest.mark.parametrize("nrhs", [1, 16, 17, 64, 65, 113, 128])
def test_rows_of_a_block(latt, nrhs):
    """3, 128 and 2673 sites: 1 to 32 tiles, whose rows go sixteen to a block, and 335 or 669, the last not full.  Rows
    that end in, at and before the sixteens' ends; one site past the output's end stays as it was."""
    import qcu_b200 as q
    import torch

    U = O.gauge_smooth(latt, 0.25, 75)
    psi = np.stack([O.fermion_gauss(O.half_shape(latt), 950 + j) for j in range(nrhs)])
    inp = dev(psi)
    buf = torch.full((inp.numel() + 12,), float("nan"), dtype=inp.dtype, device=inp.device)
    out = buf[:inp.numel()].view(inp.shape)
    with q.Gauge(dev(U), latt) as G:
        G.dslash_multi_tc(out, inp, nrhs, 1)
    got = host(out)
    assert max(rel(got[j], O.dslash(psi[j], U, latt, 1, 1.0)) for j in range(nrhs)) < 2e-3
    assert bool(torch.isnan(buf[inp.numel():].real).all())
