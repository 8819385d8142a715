"""The work that programs have this library do, as cases that can be timed and checked.

A case goes through the public entry points of ``qcu_b200`` as a program calls them, on inputs made from a seed.
``listed()`` gives the fixed cases, ``draw(rng)`` one more of the same ranges, ``prepare(case, seed)`` what a program
holds before the call (fields on the GPU, the gauge handle, the network or the multigrid), ``run(state)`` one pass,
``work(case)`` the bytes and operations that one pass cannot do without, and ``exact(case, seed)`` the same outputs in
64 bits from plain torch.

Fields are complex128 in PyQuda's even-odd layout (``qcu_b200.Layout``).  Links are exp(i eps H) with a Gaussian H, as
the library's own generator and its benchmark use them; sources are complex Gaussians or the point sources of a
propagator.
"""
import math

import numpy as np
import torch

import qcu_b200 as q

EPS = 0.25  # of the links
CSW = 1.0

# The solvers' settings are the benchmark's: FP64 flexible GCR(4) around a BiCGSTAB on 16-bit spinors and links.  The
# tolerance is what the repository's own training pairs are solved to: a solution to which 1e-10 in x is a fair demand.
TOL = 1e-12
CHOSEN = dict(tol=TOL, maxiter=20000, precision=16, solver="gcr", inner_iters=96, inner_tol=0.03, gcr_k=4)
BATCHED = dict(tol=TOL, maxiter=20000, precision=16, inner_iters=96, inner_tol=0.03, gcr_k=4)


def _case(name, kind, latt, **more):
    c = {"kind": kind, "lx": latt[0], "ly": latt[1], "lz": latt[2], "lt": latt[3], **more}
    return {"name": name, **c} if name else c


def listed():
    return [
        # one hop through qcu's own ABI on the smallest lattice in use: a program's unit test, or the innermost call of
        # a Python solver on a toy lattice; the call's latency is what it pays for
        _case("hop_8x8x8x8", "hop", [8, 8, 8, 8], parity=0),
        # the same call on the benchmark's lattice: PyQuda's pyqcu users apply the operator to complex128 fields
        _case("hop_32x32x32x64", "hop", [32, 32, 32, 64], parity=1),
        # qcu's clover call, which takes the links alone and therefore makes the clover term each time
        _case("clover_hop_24x24x24x48", "clover_hop", [24, 24, 24, 48], parity=0),
        # a new gauge configuration: load it with its clover term, apply the full FP64 operator, let it go
        _case("configuration_24x24x24x48", "configuration", [24, 24, 24, 48], csw=CSW, kappa=0.125),
        # the clover operator in the storage of the inner solver, on a lattice whose extents are no powers of two
        _case("operator16_22x18x20x36", "operator", [22, 18, 20, 36], parity=1, precision=16, csw=CSW, kappa=0.125),
        # qcu's own solve call (kappa 0.125, its stop, its random start) on qcu's notebook lattice
        _case("legacy_solve_16x16x16x32", "legacy_solve", [16, 16, 16, 32]),
        # one clover solve on a small lattice: launches and host steps, not bytes, are its time
        _case("solve_8x8x8x16", "solve", [8, 8, 8, 16], csw=CSW, kappa=0.125),
        # the benchmark's near-critical Wilson system
        _case("solve_32x32x32x64", "solve", [32, 32, 32, 64], csw=0.0, kappa=0.1303),
        # a clover propagator: the 12 spin-colour point sources in one batched solve
        _case("propagator_16x16x16x32", "propagator", [16, 16, 16, 32], csw=CSW, kappa=0.1291),
        # the hop on 64 right-hand sides of one system at once
        _case("multi_rhs_16x16x16x32", "multi_rhs", [16, 16, 16, 32], nrhs=64, parity=0),
        # one step's loss and gradient of the learned preconditioner, at its training's lattice and batch
        _case("train_16x16x16x16", "train", [16, 16, 16, 16], batch=16),
        # one solve with a multigrid that the program has set up for its configuration
        _case("multigrid_16x16x16x32", "multigrid", [16, 16, 16, 32], kappa=0.1303),
    ]


def _lattice(rng, lo, hi, step=2, lowest=4):
    """Four extents, multiples of `step`, of a volume spread over the logarithm of [lo, hi] sites."""
    target = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    while True:
        v = [rng.randrange(lowest, 33, step) for _ in range(3)] + [rng.randrange(lowest, 65, step)]
        n = v[0] * v[1] * v[2] * v[3]
        if lo <= n <= hi and abs(math.log(n / target)) < 0.25:
            return v


def draw(rng):
    kind = rng.choice(["hop", "clover_hop", "configuration", "operator", "legacy_solve", "solve", "propagator",
                       "multi_rhs", "train", "multigrid"])
    if kind == "hop":
        return _case(None, kind, _lattice(rng, 4 ** 4, 32 ** 3 * 64), parity=rng.randrange(2))
    if kind == "clover_hop":
        return _case(None, kind, _lattice(rng, 4 ** 4, 24 ** 3 * 48), parity=rng.randrange(2))
    if kind == "configuration":
        return _case(None, kind, _lattice(rng, 8 ** 4, 24 ** 3 * 48), csw=rng.choice([0.0, CSW]),
                     kappa=round(rng.uniform(0.11, 0.129), 4))
    if kind == "operator":
        return _case(None, kind, _lattice(rng, 8 ** 4, 32 ** 3 * 64), parity=rng.randrange(2),
                     precision=rng.choice([64, 32, 16, 3216]), csw=rng.choice([0.0, CSW]), kappa=0.125)
    if kind == "legacy_solve":
        return _case(None, kind, _lattice(rng, 8 ** 4, 16 ** 3 * 32))
    if kind == "solve":
        return _case(None, kind, _lattice(rng, 8 ** 3 * 16, 24 ** 3 * 48, lowest=6), csw=rng.choice([0.0, CSW]),
                     kappa=round(rng.uniform(0.11, 0.128), 4))
    if kind == "propagator":
        return _case(None, kind, _lattice(rng, 8 ** 3 * 16, 16 ** 3 * 32, lowest=6), csw=rng.choice([0.0, CSW]),
                     kappa=round(rng.uniform(0.11, 0.128), 4))
    if kind == "multi_rhs":
        return _case(None, kind, _lattice(rng, 8 ** 4, 16 ** 3 * 32), nrhs=rng.choice([1, 12, 24, 47, 64, 65, 96, 128]),
                     parity=rng.randrange(2))
    if kind == "train":
        return _case(None, kind, _lattice(rng, 8 ** 4, 16 ** 4), batch=rng.randint(1, 16))
    return _case(None, kind, _lattice(rng, 8 ** 3 * 16, 16 ** 3 * 32, step=4, lowest=8),
                 kappa=round(rng.uniform(0.12, 0.13), 4))


# ------------------------------------------------------------------ inputs
def _latt(case):
    return [case["lx"], case["ly"], case["lz"], case["lt"]]


def _rng(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _spinor(shape, gen):
    """Complex N(0, 1) per component."""
    z = torch.empty(tuple(shape) + (2,), dtype=torch.float64, device="cuda").normal_(generator=gen)
    return torch.view_as_complex(z)


def _mul(a, b):
    return (a[:, :, :, None] * b[:, None, :, :]).sum(2)


def _links(latt, gen):
    """exp(i EPS H), H = sum_a h_a lambda_a / 2 with h_a from N(0, 1): a Taylor series, then rows 0 and 1 made
    orthonormal and row 2 their conjugate cross product, so that every link is in SU(3) to the last digits."""
    shape = q.Layout(tuple(latt)).gauge
    out = torch.empty((math.prod(shape[:-2]), 3, 3), dtype=torch.complex128, device="cuda")
    eye = torch.eye(3, dtype=torch.complex128, device="cuda")
    for lo in range(0, out.shape[0], 1 << 20):
        n = min(1 << 20, out.shape[0] - lo)
        h = torch.empty((8, n), dtype=torch.float64, device="cuda").normal_(generator=gen) * (0.5 * EPS)
        a = torch.zeros((n, 3, 3), dtype=torch.complex128, device="cuda")
        a[:, 0, 0] = torch.complex(torch.zeros_like(h[0]), h[2] + h[7] / math.sqrt(3))
        a[:, 1, 1] = torch.complex(torch.zeros_like(h[0]), -h[2] + h[7] / math.sqrt(3))
        a[:, 2, 2] = torch.complex(torch.zeros_like(h[0]), -2 * h[7] / math.sqrt(3))
        for (i, j), (u, v) in {(0, 1): (0, 1), (0, 2): (3, 4), (1, 2): (5, 6)}.items():
            a[:, i, j] = torch.complex(h[v], h[u])
            a[:, j, i] = torch.complex(-h[v], h[u])
        u = eye + a / 10
        for k in range(9, 0, -1):
            u = eye + _mul(a, u) / k
        r0 = u[:, 0] / torch.linalg.vector_norm(u[:, 0], dim=1, keepdim=True)
        r1 = u[:, 1] - (r0.conj() * u[:, 1]).sum(1, keepdim=True) * r0
        r1 = r1 / torch.linalg.vector_norm(r1, dim=1, keepdim=True)
        r2 = torch.stack([r0[:, 1] * r1[:, 2] - r0[:, 2] * r1[:, 1], r0[:, 2] * r1[:, 0] - r0[:, 0] * r1[:, 2],
                          r0[:, 0] * r1[:, 1] - r0[:, 1] * r1[:, 0]], dim=1).conj()
        out[lo:lo + n] = torch.stack([r0, r1, r2], dim=1)
    return out.view(shape)


def _inputs(case, seed):
    """The fields of one case, from the seed alone."""
    gen, latt, kind = _rng(seed), _latt(case), case["kind"]
    L = q.Layout(tuple(latt))
    f = {"u": _links(latt, gen)}
    if kind in ("hop", "clover_hop", "operator"):
        f["psi"] = _spinor(L.half, gen)
    elif kind in ("configuration", "legacy_solve", "solve", "multigrid"):
        f["psi"] = _spinor(L.full, gen)
    elif kind == "propagator":
        at = [int(torch.randint(0, n, (1,), generator=gen, device="cuda")) for n in latt]
        f["psi"] = q.point_sources(latt, at)
    elif kind == "multi_rhs":
        f["psi"] = _spinor((case["nrhs"],) + L.half, gen)
    else:  # train: errors and what stands for their residuals, of like size, and a network on its way
        f["e"] = _spinor((case["batch"],) + L.half, gen)
        f["r"] = f["e"] + 0.5 * _spinor((case["batch"],) + L.half, gen)
        f["w"] = np.random.default_rng(seed).normal(0, 0.1, 2 * 2 * 9 * 16 * 4).astype(np.float32)
    return f


def _clover_coeff(case):
    return case.get("kappa", 0.0) * case.get("csw", 0.0)


def prepare(case, seed):
    f = _inputs(case, seed)
    kind, latt = case["kind"], _latt(case)
    s = {"case": case, **f}
    if kind in ("hop", "clover_hop", "legacy_solve"):
        s["param"] = q.QcuParam(latt)
        s["grid"] = q.QcuParam([1, 1, 1, 1])
    elif kind != "configuration":
        s["gauge"] = q.Gauge(s.pop("u"), latt, t_boundary=-1.0, clover_coeff=_clover_coeff(case))
    if "psi" in s:
        s["out"] = torch.empty_like(s["psi"])
    if kind == "train":
        s["net"] = q.Network(seed=1)
        s["net"].set_weights(s["w"])
    elif kind == "multigrid":
        s["mg"] = q.Multigrid(s["gauge"], case["kappa"], n_vec=12, setup_maxiter=200, nu_post=4, coarse_tol=0.05,
                              coarse_maxiter=50)
    return s


# ------------------------------------------------------------------ one pass
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "train":  # lr 0: the gradient for the program's own optimiser; the weights stay
        loss, grad = s["net"].train_step(s["gauge"], s["r"], s["e"], case["batch"], 0.0, want_grad=True)
        return {"loss": loss, "grad": grad}
    psi, out = s["psi"], s["out"]
    clover = case.get("csw", 0.0) != 0.0
    if kind == "hop":
        q.dslashQcu(out, psi, s["u"], s["param"], case["parity"])
    elif kind == "clover_hop":
        q.dslashCloverQcu(out, psi, s["u"], s["param"], case["parity"])
    elif kind == "configuration":
        with q.Gauge(s["u"], _latt(case), t_boundary=-1.0, clover_coeff=_clover_coeff(case)) as gauge:
            gauge.mat(out, psi, case["kappa"], clover)
    elif kind == "operator":
        s["gauge"].dslash(out, psi, case["parity"], clover, case["precision"])
    elif kind == "legacy_solve":
        q.ncclBistabCgQcu(out, psi, s["u"], s["param"], s["grid"])
    elif kind == "solve":
        s["gauge"].invert(out, psi, case["kappa"], clover=clover, **CHOSEN)
    elif kind == "propagator":
        q.invert_batch([(s["gauge"], out, psi, case["kappa"], clover)], **BATCHED)
    elif kind == "multi_rhs":
        s["gauge"].dslash_multi_tc(out, psi, case["nrhs"], case["parity"])
    else:
        s["mg"].invert(out, psi, tol=TOL, maxiter=1000)
    return out


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    """Inputs read once and outputs written once.  A link is two complex128 rows (96 bytes) where the caller's links
    are read, 24 bytes in the 16-bit storage; a solve's iterations are counted with each operator's fields read and
    written once per application, at the number of iterations such a system takes."""
    kind, vh = case["kind"], math.prod(_latt(case)) // 2
    clover = case.get("csw", 0.0) != 0.0
    links64, spinor, hop = 8 * 96 * vh, 192 * vh, 1320 * vh
    leaves = 24 * 3 * 198 * vh  # the plaquette leaves of one parity's clover term
    clov = (504 if clover else 0) * vh
    if kind == "hop":
        return {"bytes": links64 + 2 * spinor, "flops": hop}
    if kind == "clover_hop":
        return {"bytes": links64 + 2 * spinor, "flops": hop + leaves + 504 * vh}
    if kind == "configuration":
        return {"bytes": links64 + 4 * spinor, "flops": 2 * (hop + clov + (leaves if clover else 0))}
    if kind == "operator":
        b = {64: 8 * 96 + 576 * clover, 32: 8 * 48 + 288 * clover}.get(case["precision"], 8 * 24 + 288 * clover)
        return {"bytes": b * vh + 2 * spinor, "flops": hop + clov}
    if kind == "multi_rhs":
        return {"bytes": 8 * 24 * vh + 2 * spinor * case["nrhs"], "flops": hop * case["nrhs"]}
    if kind == "train":
        b = case["batch"]
        # transports of 4 and 16 channels over 8 links on both parities, mixing of 9 hops, forward and twice back
        return {"bytes": 8 * 48 * vh + 2 * spinor * b, "flops": 3 * b * vh * (2 * 8 * 4 * 66 + 3 * 9 * 64 * 8 * 2)}
    its = {"legacy_solve": 60, "solve": 480 if case.get("kappa", 0) > 0.13 else 60, "propagator": 200, "multigrid": 150}[kind]
    rhs = 12 if kind == "propagator" else 1
    per = 4 * (1152 if kind in ("legacy_solve", "multigrid") else (104 * rhs + 192 + (288 if clover else 0))) * vh
    return {"bytes": links64 + 4 * spinor * rhs + its * per, "flops": its * 4 * (hop + clov) * rhs}


# ------------------------------------------------------------------ the same outputs in 64 bits, from torch alone
class _Grid:
    """Site tables of the even-odd lattice: per parity, the coordinates, the neighbours and the t-boundary phases."""

    def __init__(self, latt, u, t_bc):
        self.latt, self.t_bc = latt, t_bc
        lx, ly, lz, lt = latt
        self.vh = lx * ly * lz * lt // 2
        self.u = u.reshape(4, 2, self.vh, 3, 3)
        i = torch.arange(self.vh, device="cuda")
        xh, y, z, t = i % (lx // 2), i // (lx // 2) % ly, i // (lx // 2 * ly) % lz, i // (lx // 2 * ly * lz)
        self.c = [torch.stack([2 * xh + (y + z + t + p) % 2, y, z, t]) for p in (0, 1)]

    def index(self, c):
        lx, ly, lz, _ = self.latt
        return ((c[3] * lz + c[2]) * ly + c[1]) * (lx // 2) + torch.div(c[0], 2, rounding_mode="floor")

    def shift(self, p, steps):
        """Site index (and parity) of the sites of parity p moved by `steps` = {direction: +1 or -1}."""
        c = list(self.c[p])
        for mu, d in steps.items():
            c[mu] = (c[mu] + d) % self.latt[mu]
        return self.index(c), (p + len(steps)) % 2

    def link(self, p, mu, steps):
        n, par = self.shift(p, steps)
        return self.u[mu, par][n]

    def phase(self, p, mu, d):
        edge = self.latt[3] - 1 if d > 0 else 0
        one = torch.ones(self.vh, dtype=torch.float64, device="cuda")
        return torch.where(self.c[p][3] == edge, self.t_bc * one, one) if mu == 3 else one

    def hops(self, p):
        """(direction, step, source sites, the 3x3 matrix of the transport) of the eight hops onto parity p."""
        for mu in range(4):
            for d in (1, -1):
                n, _ = self.shift(p, {mu: d})
                m = self.u[mu, p] if d > 0 else self.u[mu, 1 - p][n].mH
                yield mu, d, n, m * self.phase(p, mu, d)[:, None, None]


def _gammas():
    """The DeGrand-Rossi gamma matrices, directions x, y, z, t."""
    i = 1j
    g = [[[0, 0, 0, i], [0, 0, i, 0], [0, -i, 0, 0], [-i, 0, 0, 0]],
         [[0, 0, 0, -1], [0, 0, 1, 0], [0, 1, 0, 0], [-1, 0, 0, 0]],
         [[0, 0, i, 0], [0, 0, 0, -i], [-i, 0, 0, 0], [0, i, 0, 0]],
         [[0, 0, 1, 0], [0, 0, 0, 1], [1, 0, 0, 0], [0, 1, 0, 0]]]
    return torch.tensor(g, dtype=torch.complex128, device="cuda")


def _hop(grid, p, psi):
    """D_{p <- 1-p} psi on half spinors [..., Vh, 4, 3]."""
    gam, eye = _gammas(), torch.eye(4, dtype=torch.complex128, device="cuda")
    out = torch.zeros_like(psi)
    for mu, d, n, m in grid.hops(p):
        h = psi[..., n, :, :]
        h = torch.einsum("st,...tc->...sc", eye - d * gam[mu], h)
        out += (m[:, None, :, :] * h[..., None, :]).sum(-1)
    return out


def _clover(grid, p, coeff):
    """A = 1 - coeff/8 sum_{mu<nu} gamma_mu gamma_nu (Q - Q^dag) on parity p, [Vh, 12, 12]."""
    gam = _gammas()
    a = torch.zeros((grid.vh, 4, 3, 4, 3), dtype=torch.complex128, device="cuda")
    for mu in range(4):
        for nu in range(mu + 1, 4):
            def at(d, **s):
                return grid.link(p, d, {mu if k == "m" else nu: v for k, v in s.items()})
            leaf = _mul(_mul(_mul(at(mu), at(nu, m=1)), at(mu, n=1).mH), at(nu).mH)
            leaf = leaf + _mul(_mul(_mul(at(nu), at(mu, m=-1, n=1).mH), at(nu, m=-1).mH), at(mu, m=-1))
            leaf = leaf + _mul(_mul(_mul(at(mu, m=-1).mH, at(nu, m=-1, n=-1).mH), at(mu, m=-1, n=-1)), at(nu, n=-1))
            leaf = leaf + _mul(_mul(_mul(at(nu, n=-1).mH, at(mu, n=-1)), at(nu, m=1, n=-1)), at(mu).mH)
            a += torch.einsum("st,xab->xsatb", gam[mu] @ gam[nu], leaf - leaf.mH)
    return torch.eye(12, dtype=torch.complex128, device="cuda") - (coeff / 8) * a.view(grid.vh, 12, 12)


def _site(a, psi):
    return torch.einsum("xij,...xj->...xi", a, psi.reshape(psi.shape[:-2] + (12,))).view(psi.shape)


class _System:
    """M = A - kappa D and its even-odd preconditioned solve."""

    def __init__(self, grid, kappa, coeff):
        self.g, self.k = grid, kappa
        self.a = [_clover(grid, p, coeff) for p in (0, 1)] if coeff else None
        self.ai = [torch.linalg.inv(a) for a in self.a] if coeff else None

    def inv(self, p, v):
        return _site(self.ai[p], v) if self.ai else v

    def mat(self, psi):
        d = [_site(self.a[p], psi[p]) if self.a else psi[p] for p in (0, 1)]
        return torch.stack([d[p] - self.k * _hop(self.g, p, psi[1 - p]) for p in (0, 1)])

    def mpc(self, v):
        return v - self.k ** 2 * self.inv(1, _hop(self.g, 1, self.inv(0, _hop(self.g, 0, v))))

    def solve(self, b):
        """x of M x = b to rounding, or None: BiCGSTAB on the odd sites, started again from the true residual."""
        rhs = self.inv(1, b[1] + self.k * _hop(self.g, 1, self.inv(0, b[0])))
        x, goal = torch.zeros_like(rhs), 1e-14 * torch.linalg.vector_norm(rhs)
        dot = lambda u, v: (u.conj() * v).sum()  # noqa: E731
        for _ in range(6):
            r = rhs - self.mpc(x)
            start = torch.linalg.vector_norm(r)
            if start <= 3 * goal:
                break
            rt, p, v = r.clone(), torch.zeros_like(r), torch.zeros_like(r)
            rho = alpha = omega = torch.ones((), dtype=r.dtype, device="cuda")
            for _ in range(600):
                rho1 = dot(rt, r)
                p = r + (rho1 / rho) * (alpha / omega) * (p - omega * v)
                v = self.mpc(p)
                rho, alpha = rho1, rho1 / dot(rt, v)
                s = r - alpha * v
                t = self.mpc(s)
                omega = dot(t, s) / dot(t, t)
                x = x + alpha * p + omega * s
                r = s - omega * t
                if torch.linalg.vector_norm(r) <= max(float(goal), 1e-7 * float(start)):
                    break
        if not bool(torch.linalg.vector_norm(rhs - self.mpc(x)) <= 30 * goal):
            return None
        return torch.stack([self.inv(0, b[0] + self.k * _hop(self.g, 0, x)), x])


def _train_exact(case, f, grid):
    """Loss and dL/dW* of N(r) = L2(L1(r)), by torch's own differentiation, one sample at a time."""
    w = torch.view_as_complex(torch.from_numpy(f["w"].astype(np.float64)).cuda().view(-1, 2).contiguous())
    w1 = w[:9 * 64].view(9, 16, 4).clone().requires_grad_(True)
    w2 = w[9 * 64:].view(9, 4, 16).clone().requires_grad_(True)
    hops = [list(grid.hops(p)) for p in (0, 1)]
    total, b = 0.0, case["batch"]

    def moved(v, m, n):
        return (m[:, None, :, :] * v[n][:, :, None, :]).sum(-1)

    for k in range(b):
        r, e = (f[x][k].reshape(grid.vh, 4, 3) for x in ("r", "e"))
        even = sum(torch.einsum("ab,xbc->xac", w1[j + 1], moved(r, m, n)) for j, (_, _, n, m) in enumerate(hops[0]))
        odd = torch.einsum("ab,xbc->xac", w1[0], r)  # r has no even sites to hop from
        out = torch.einsum("ab,xbc->xac", w2[0], odd)
        for j, (_, _, n, m) in enumerate(hops[1]):
            out = out + torch.einsum("ab,xbc->xac", w2[j + 1], moved(even, m, n))
        loss = (out - e).abs().square().sum() / e.abs().square().sum() / b
        loss.backward()
        total += float(loss)
    grad = torch.view_as_real(torch.cat([w1.grad.reshape(-1), w2.grad.reshape(-1)])) / 2
    return {"loss": total, "grad": grad.reshape(-1).cpu().numpy()}


def exact(case, seed):
    kind, latt = case["kind"], _latt(case)
    near = case.get("kappa", 0.0) > 0.13 and math.prod(latt) > 16 ** 3 * 32
    if kind == "propagator" or near:
        return None  # hundreds of applications to many or large fields
    f = _inputs(case, seed)
    legacy = kind in ("hop", "clover_hop", "legacy_solve")
    grid = _Grid(latt, f["u"], 1.0 if legacy else -1.0)
    if kind == "train":
        return _train_exact(case, f, grid)
    psi = f["psi"]
    if kind in ("hop", "clover_hop", "operator", "multi_rhs"):
        p = case["parity"]
        flat = psi.reshape(psi.shape[:-6] + (grid.vh, 4, 3))
        if kind == "multi_rhs":
            return torch.stack([_hop(grid, p, v) for v in flat]).view(psi.shape)
        out = _hop(grid, p, flat)
        coeff = 1.0 if kind == "clover_hop" else _clover_coeff(case)
        if coeff:
            out = _site(torch.linalg.inv(_clover(grid, p, coeff)), out)
        return out.view(psi.shape)
    flat = psi.reshape(2, grid.vh, 4, 3)
    system = _System(grid, case.get("kappa", 0.125), _clover_coeff(case))
    out = system.mat(flat) if kind == "configuration" else system.solve(flat)
    return None if out is None else out.view(psi.shape)
