"""The clover build on PyQuda's link records at the sizes its launch splits differently, and what dslashCloverQcu keeps."""
import os
import subprocess
import sys

import numpy as np
import pytest

import oracle as O
from util import dev, empty_like_dev, host, rel

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("latt", [[18, 18, 18, 22], [10, 2, 6, 4], [2, 1, 1, 3]])
def test_three_rounds_a_block_and_partial_warps(latt):
    """64152 sites per parity are 2005 warps of sites, the last of 24 sites, in blocks of three, the last of one; 240 and
    3 sites take one round.  On records (dslashCloverQcu) and, both parities at once, on packed links (a handle)."""
    import qcu_b200 as q

    U = O.gauge_smooth(latt, 0.1, 41)
    psi = O.fermion_gauss(O.full_shape(latt), 42)
    dU, dpsi = dev(U), dev(psi)
    with q.Gauge(dU, latt, clover_coeff=1.0) as G:
        for p in (0, 1):
            A = O.clover_build(U, latt, p, 1.0)
            expect = O.clover_apply(O.clover_invert(A), O.dslash(psi[1 - p], U, latt, p))
            bar = 1e-14 * max(np.linalg.cond(A).max(), 10)
            out = empty_like_dev(O.half_shape(latt))
            q.dslashCloverQcu(out, dpsi[1 - p], dU, q.QcuParam(latt), p)
            assert q.last_error()[0] == 0
            assert rel(host(out), expect) <= bar
            out = empty_like_dev(O.half_shape(latt))
            G.dslash(out, dpsi[1 - p], p, clover=True)
            assert rel(host(out), expect) <= bar


_KEPT = """
import torch, qcu_b200 as q
def call(latt):
    L = q.Layout(tuple(latt))
    u = torch.eye(3, dtype=torch.complex128, device="cuda").expand(L.gauge).contiguous()
    psi = torch.ones(L.half, dtype=torch.complex128, device="cuda")
    out = torch.empty_like(psi)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    q.dslashCloverQcu(out, psi, u, q.QcuParam(latt), 0)
    assert q.last_error()[0] == 0
    return before - torch.cuda.mem_get_info()[0]
call([4, 4, 4, 4])
print(call([20, 20, 20, 32]))
"""


def test_dslashCloverQcu_keeps_the_inverse_only():
    """What one call leaves allocated on the device: the inverse clover term of one parity, 576 bytes a site (73.7 MB),
    and at most two of the memory pool's 32 MiB granules beside it."""
    r = subprocess.run([sys.executable, "-c", _KEPT], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    kept = int(r.stdout.split()[-1])
    assert kept <= 576 * 128000 + 2 * (32 << 20), kept
