"""Performance cases of the simulation hot path: what a user's program calls, over
the sizes it is called with.

`listed()` names the cases, `draw(rng)` gives another one of the same ranges,
`prepare(case, seed)` makes on the GPU what such a program has in hand before the
call, `run(state)` is one pass through the public API, `work(case)` the bytes and
operations no implementation can do without, and `exact(case, seed)` the same
outputs from plain torch in 64 bits.

Links are drawn with the plaquette average of the stated beta (Gaussian link
angles under a random gauge transformation), sources are complex Gaussian, and
the draws of a trajectory are Philox4x32-10 keyed by the case's seed, as the
library defines them.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dav-qed2d_b200"))

import qed2d  # noqa: E402

TOL = 1e-24          # |r|^2 < TOL |b|^2: a relative residual of 1e-12, the drivers' setting
MAXITER = 10000
ENSEMBLE_SIZES = (32, 48, 64, 96, 128, 256)


# ---------------------------------------------------------------------------
# the cases
def listed():
    return [
        # one apply of the Dirac operator on the smallest lattice of the configurations:
        # what a measurement script pays per call
        {"name": "dirac_64", "kind": "dirac", "L1": 64, "L2": 64, "dtype": "c128"},
        # the same on a lattice far beyond the caches (master-field measurements)
        {"name": "dirac_4096", "kind": "dirac", "L1": 4096, "L2": 4096, "dtype": "c128"},
        # a propagator in the default precision on the RHMC configuration's lattice
        {"name": "cg_f64_128", "kind": "cg", "L1": 128, "L2": 128, "m0": 0.1, "mu": 0.0, "prec": "f64"},
        # a propagator with the mixed solver on the headline lattice
        {"name": "cg_mixed_512", "kind": "cg", "L1": 512, "L2": 512, "m0": 0.1, "mu": 0.0, "prec": "mixed"},
        # the same on a lattice that leaves the caches
        {"name": "cg_mixed_2048", "kind": "cg", "L1": 2048, "L2": 2048, "m0": 0.1, "mu": 0.0, "prec": "mixed"},
        # one pure-gauge trajectory (beta 11.25, OMF4 ns 10, eps 0.15), many small passes
        {"name": "hmc_gauge_128", "kind": "gauge", "L1": 128, "L2": 128, "beta": 11.25, "eps": 0.15, "ns": 10},
        # one Nf=2 trajectory of a small lattice (beta 4, m0 0.1, leapfrog ns 20, eps 0.05)
        {"name": "hmc_nf2_64", "kind": "nf2", "L1": 64, "L2": 64, "beta": 4.0, "m0": 0.1, "eps": 0.05, "ns": 20,
         "prec": "mixed"},
        # one RHMC trajectory, one flavour with 12 Zolotarev poles, default precision
        {"name": "hmc_rhmc_128", "kind": "rhmc", "L1": 128, "L2": 128, "beta": 4.0, "m0": 0.1, "eps": 0.05, "ns": 20,
         "poles": 12, "prec": "f64"},
        # the headline workload: four Nf=2 chains of 512 x 512 advanced together
        {"name": "batch_hmc_512x4", "kind": "batch", "L1": 512, "L2": 512, "nrep": 4, "beta": 4.0, "m0": 0.1,
         "eps": 0.05, "ns": 20},
        # a batch of small equal lattices (volume or parameter scans): a short trajectory of each
        {"name": "batch_hmc_64x32", "kind": "batch", "L1": 64, "L2": 64, "nrep": 32, "beta": 4.0, "m0": 0.15,
         "eps": 0.1, "ns": 5},
        # the force solve of an ensemble of uneven lattices (sizes, couplings and masses of the ensemble configuration)
        {"name": "ensemble_cg_96", "kind": "ensemble", "nrep": 96, "sizes": "standard", "draw": 2024},
        # pure-gauge integration of a master field, bound by memory
        {"name": "master_omf4_4096", "kind": "omf4", "L1": 4096, "L2": 4096, "beta": 11.25, "eps": 0.025, "ns": 2},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dirac", "cg", "cg", "gauge", "nf2", "rhmc", "batch", "ensemble", "omf4"])
    if kind == "dirac":
        return {"kind": kind, "L1": _log(rng, 16, 4096), "L2": _log(rng, 16, 4096),
                "dtype": rng.choice(["c128", "c64"])}
    if kind == "cg":   # lattices from 24^2 to 1024^2, some with a twisted-mass shift
        return {"kind": kind, "L1": _log(rng, 24, 1024), "L2": _log(rng, 24, 1024),
                "m0": round(rng.uniform(0.05, 0.3), 3), "mu": rng.choice([0.0, 0.0, 0.1]),
                "prec": rng.choice(["f64", "mixed"])}
    if kind == "gauge":
        return {"kind": kind, "L1": _log(rng, 16, 1024), "L2": _log(rng, 16, 1024),
                "beta": round(rng.uniform(2.0, 12.0), 2), "eps": 0.1, "ns": rng.randint(4, 12)}
    if kind == "nf2":
        return {"kind": kind, "L1": _log(rng, 16, 256), "L2": _log(rng, 16, 256),
                "beta": round(rng.uniform(2.0, 6.0), 2), "m0": round(rng.uniform(0.05, 0.3), 3), "eps": 0.05,
                "ns": rng.randint(4, 12), "prec": rng.choice(["mixed", "mixed", "f64"])}
    if kind == "rhmc":
        return {"kind": kind, "L1": _log(rng, 12, 160), "L2": _log(rng, 12, 160),
                "beta": round(rng.uniform(2.0, 6.0), 2), "m0": round(rng.uniform(0.05, 0.3), 3), "eps": 0.05,
                "ns": rng.randint(3, 8), "poles": rng.randint(4, 14), "prec": "f64"}
    if kind == "batch":   # at most the headline's sites in all
        n = rng.randint(2, 16)
        top = int(math.sqrt(2 ** 20 / n))
        return {"kind": kind, "L1": _log(rng, 24, top), "L2": _log(rng, 24, top), "nrep": n,
                "beta": round(rng.uniform(2.0, 6.0), 2), "m0": round(rng.uniform(0.05, 0.3), 3), "eps": 0.05,
                "ns": rng.randint(3, 8)}
    if kind == "ensemble":
        return {"kind": kind, "nrep": rng.randint(8, 64), "sizes": rng.choice(["standard", "any"]),
                "draw": rng.randrange(1 << 30)}
    return {"kind": kind, "L1": _log(rng, 64, 4096), "L2": _log(rng, 64, 4096), "beta": round(rng.uniform(2.0, 12.0), 2),
            "eps": 0.025, "ns": rng.randint(1, 3)}


def _ensemble(case):
    """(sizes, betas, masses) of an ensemble: its parameters are the case's, not the seed's."""
    rng = np.random.default_rng(case["draw"])
    n = case["nrep"]
    if case["sizes"] == "standard":
        sizes = [(int(s), int(s)) for s in rng.choice(ENSEMBLE_SIZES, n)]
    else:
        sizes = [(int(round(math.exp(a))), int(round(math.exp(b))))
                 for a, b in rng.uniform(math.log(24), math.log(256), (n, 2))]
    return sizes, rng.uniform(2.0, 6.0, n).tolist(), rng.uniform(0.05, 0.3, n).tolist()


# ---------------------------------------------------------------------------
# inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _links(shape, beta, g):
    """Links (..., 2, L2, L1) with <Re P> = I1(beta)/I0(beta), as an equilibrium field has it."""
    s = sum((beta / 2) ** (2 * k) / math.factorial(k) ** 2 for k in range(60))
    t = sum((beta / 2) ** (2 * k + 1) / (math.factorial(k) * math.factorial(k + 1)) for k in range(60))
    sigma = math.sqrt(-0.5 * math.log(t / s))
    th = sigma * torch.randn(*shape, dtype=torch.float64, device="cuda", generator=g)
    w = 2 * math.pi * torch.rand(*shape[:-3], *shape[-2:], dtype=torch.float64, device="cuda", generator=g)
    th[..., 0, :, :] += w - torch.roll(w, -1, -1)
    th[..., 1, :, :] += w - torch.roll(w, -1, -2)
    return torch.polar(torch.ones_like(th), th)


def _gauss(shape, g, dtype=torch.complex128):
    return torch.randn(*shape, dtype=dtype, device="cuda", generator=g)


_batch = {}   # the one batch handle in use: a program keeps its handle and feeds it new fields


def _batch_of(key, make):
    if key not in _batch:
        _batch.clear()
        _batch[key] = make()
    return _batch[key]


def _rhmc_interval(case):
    return 0.05, math.sqrt((case["m0"] + 4.0) ** 2 * 1.05)


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    st = {"case": case, "seed": int(seed) & 0x7FFFFFFF}
    qed2d.set_precision(case.get("prec", "f64"))
    if kind == "ensemble":
        sizes, betas, am0s = _ensemble(case)
        b = _batch_of(("ragged", tuple(sizes)), lambda: qed2d.Batch.ragged(sizes, betas))
        U, src = b.field(), b.field()
        for r, (l1, l2) in enumerate(sizes):
            b.replica(U, r).copy_(_links((2, l2, l1), betas[r], g))
            b.replica(src, r).copy_(_gauss((2, l2, l1), g))
        return st | {"batch": b, "U": U, "b": src, "x": b.field(), "am0": am0s}
    L1, L2 = case["L1"], case["L2"]
    if kind == "batch":
        n = case["nrep"]
        b = _batch_of(("equal", n, L1, L2, case["beta"]), lambda: qed2d.Batch(n, L1, L2, case["beta"]))
        U0 = _links((n, 2, L2, L1), case["beta"], g)
        return st | {"batch": b, "U0": U0, "U": U0.clone(), "seeds": [st["seed"] + r for r in range(n)]}
    prm = qed2d.LattParm((L1, L2), case.get("beta", 4.0))
    st["prm"] = prm
    U0 = _links((2, L2, L1), case.get("beta", 4.0), g)
    if kind == "dirac":
        dt = torch.complex64 if case["dtype"] == "c64" else torch.complex128
        si = _gauss((2, L2, L1), g, dt)
        return st | {"U": U0.to(dt), "si": si, "so": torch.empty_like(si)}
    if kind == "cg":
        b = _gauss((2, L2, L1), g)
        return st | {"U": U0, "b": b, "x": torch.zeros_like(b)}
    st |= {"U0": U0, "U": U0.clone()}
    if kind == "omf4":
        mom0 = torch.randn(2, L2, L1, dtype=torch.float64, device="cuda", generator=g)
        return st | {"mom0": mom0, "mom": mom0.clone()}
    if kind == "rhmc":
        ra, rb = _rhmc_interval(case)
        st["rprm"] = [qed2d.get_rhmc_params(case["poles"], ra, rb)]
    return st


# ---------------------------------------------------------------------------
# one pass
def _traj(info, U):
    return {"U": U, "hini": info.hini, "hfin": info.hfin, "accepted": int(info.accepted)}


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "dirac":
        qed2d.gamm5Dw(st["so"], st["U"], st["si"], 0.1, st["prm"])
        return st["so"]
    if kind == "cg":
        if case["mu"]:
            qed2d.CG(st["x"], st["U"], st["b"], case["m0"], case["mu"], MAXITER, TOL, qed2d.gamm5Dw_sqr_musq,
                     st["prm"], None)
        else:
            qed2d.CG(st["x"], st["U"], st["b"], case["m0"], MAXITER, TOL, qed2d.gamm5Dw_sqr_msq, st["prm"], None)
        return st["x"]
    if kind == "ensemble":
        st["batch"].cg(st["x"], st["U"], st["b"], st["am0"], MAXITER, TOL)
        return st["x"]
    # every trajectory starts from the configuration in hand
    U = st["U"].copy_(st["U0"])
    if kind == "omf4":
        mom = st["mom"].copy_(st["mom0"])
        qed2d.OMF4_(mom, U, case["eps"], case["ns"], st["prm"], None)
        return {"U": U, "mom": mom}
    if kind == "batch":
        infos = st["batch"].hmc_nf2(U, case["m0"], case["eps"], case["ns"], MAXITER, TOL, st["seeds"], 0)
        return {"U": U, "hini": np.array([i.hini for i in infos]), "hfin": np.array([i.hfin for i in infos]),
                "accepted": np.array([i.accepted for i in infos], dtype=np.int64)}
    qed2d.seed(st["seed"])
    if kind == "gauge":
        return _traj(qed2d.HMC_(U, case["eps"], case["ns"], [], st["prm"], None), U)
    if kind == "nf2":
        return _traj(qed2d.HMC_(U, case["m0"], case["eps"], case["ns"], [], MAXITER, TOL, st["prm"], None), U)
    return _traj(qed2d.HMC_(U, [case["m0"]], case["eps"], case["ns"], [], MAXITER, TOL, st["prm"], None,
                            st["rprm"]), U)


# ---------------------------------------------------------------------------
# what no implementation can do without: every input read and every output
# written once, and the operations of the algorithm.  Per site one apply of the
# Dirac operator is 4 complex products and 32 additions and scalings (88
# operations), a CG iteration two applies and 56 more, a link update and a gauge
# kick 60 and 48, and a solve takes about ITERS iterations at these masses.
ITERS = 300


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        V = sum(a * b for a, b in _ensemble(case)[0])
        return {"bytes": 96 * V, "flops": V * ITERS * 232}
    V = case["L1"] * case["L2"] * case.get("nrep", 1)
    if kind == "dirac":
        return {"bytes": V * (48 if case["dtype"] == "c64" else 96), "flops": 88 * V}
    if kind == "cg":
        return {"bytes": 96 * V, "flops": V * ITERS * 232}
    steps = case["ns"]
    if kind == "omf4":
        return {"bytes": 96 * V, "flops": V * steps * (5 * 60 + 6 * 48)}
    if kind == "gauge":
        return {"bytes": 64 * V, "flops": V * (steps * (5 * 60 + 6 * 48) + 150)}
    solve = ITERS * 232
    if kind == "rhmc":   # the pole systems share one Krylov space: 24 operations more per pole
        solve += ITERS * 24 * case["poles"]
        return {"bytes": 64 * V, "flops": V * ((steps + 2) * solve + case["poles"] * ITERS * 232)}
    return {"bytes": 64 * V, "flops": V * (steps + 1) * solve}


# ---------------------------------------------------------------------------
# the same in plain torch, 64 bits
def _g5dw(U, s, m0):
    s1, s2 = s[..., 0, :, :], s[..., 1, :, :]
    u1, u2 = U[..., 0, :, :], U[..., 1, :, :]
    f1 = u1 * torch.roll(s1 - s2, -1, -1)
    b1 = torch.roll(u1.conj() * (s1 + s2), 1, -1)
    f2 = u2 * torch.roll(s1 + 1j * s2, -1, -2)
    b2 = torch.roll(u2.conj() * (s1 - 1j * s2), 1, -2)
    o1 = (2 + m0) * s1 - 0.5 * (f1 + b1) - 0.5 * (f2 + b2)
    o2 = -(2 + m0) * s2 - 0.5 * (f1 - b1) - 0.5j * (f2 - b2)
    return torch.stack((o1, o2), -3)


def _dot(a):
    return (a.real ** 2 + a.imag ** 2).sum((-3, -2, -1), keepdim=True)


def _solve(U, b, m0, mu2=0.0, tol=1e-28):
    """((g5Dw)^2 + mu2)^-1 b for every leading index, to a relative residual of sqrt(tol)."""
    x, r, p = torch.zeros_like(b), b.clone(), b.clone()
    bb = rr = _dot(b)
    for k in range(20000):
        t = _g5dw(U, p, m0)
        q = _g5dw(U, t, m0) + mu2 * p if mu2 else _g5dw(U, t, m0)
        a = rr / (_dot(t) + mu2 * _dot(p))
        x = x + a * p
        r = r - a * q
        rn = _dot(r)
        p = r + (rn / rr) * p
        rr = rn
        if k % 25 == 24 and bool((rr < tol * bb).all()):
            return x
    raise RuntimeError("reference solve did not converge")


def _multishift(U, b, m0, mu2, tol=1e-28):
    """((g5Dw)^2 + mu2_i)^-1 b for all i in one Krylov space (hep-lat/9612014)."""
    n = len(mu2)
    base = min(range(n), key=lambda i: mu2[i])
    d = torch.tensor([m - mu2[base] for m in mu2], dtype=torch.float64, device=b.device).view(n, 1, 1, 1)
    x = torch.zeros((n,) + tuple(b.shape), dtype=b.dtype, device=b.device)
    ps = b.expand_as(x).clone()
    r, p = b.clone(), b.clone()
    z = torch.ones_like(d)
    zp = torch.ones_like(d)
    bb = rr = _dot(b)
    a_old, beta = torch.ones_like(rr), torch.zeros_like(rr)
    for k in range(20000):
        t = _g5dw(U, p, m0)
        a = rr / (_dot(t) + mu2[base] * _dot(p))
        r = r - a * (_g5dw(U, t, m0) + mu2[base] * p)
        rn = _dot(r)
        zn = z * zp * a_old / (a * beta * (zp - z) + zp * a_old * (1.0 + d * a))
        zn = torch.where(z.abs() < 1e-60, torch.zeros_like(zn), zn)
        ratio = torch.where(z == 0, torch.zeros_like(z), zn / torch.where(z == 0, torch.ones_like(z), z))
        x = x + (a * ratio) * ps
        beta = rn / rr
        ps = zn * r + (beta * ratio * ratio) * ps
        p = r + beta * p
        zp, z, a_old, rr = torch.where(z == 0, zp, z), zn, a, rn
        if k % 25 == 24 and bool((rr < tol * bb).all()):
            return x
    raise RuntimeError("reference multishift solve did not converge")


def _plaq(U):
    u1, u2 = U[..., 0, :, :], U[..., 1, :, :]
    return u1 * torch.roll(u2, -1, -1) * (torch.roll(u1, -1, -2) * u2).conj()


def _gauge_force(U, beta):
    v = beta * _plaq(U).imag
    return torch.stack((torch.roll(v, 1, -2) - v, v - torch.roll(v, 1, -1)), -3)


def _fermion_force(U, X, G):
    x1, x2, g1, g2 = X[..., 0, :, :], X[..., 1, :, :], G[..., 0, :, :], G[..., 1, :, :]
    u1, u2 = U[..., 0, :, :], U[..., 1, :, :]
    z1 = u1.conj() * torch.roll(x1 - x2, -1, -1).conj() * (g1 + g2) - \
        u1 * (x1 + x2).conj() * torch.roll(g1 - g2, -1, -1)
    z2 = u2.conj() * (torch.roll(x1, -1, -2).conj() - 1j * torch.roll(x2, -1, -2).conj()) * (g1 - 1j * g2) - \
        u2 * (x1.conj() + 1j * x2.conj()) * torch.roll(g1 + 1j * g2, -1, -2)
    return torch.stack((-z1.imag, -z2.imag), -3)


def _rotate(U, mom, eps):
    return U * torch.polar(torch.ones_like(mom), eps * mom)


def _leapfrog(U, mom, force, eps, ns):
    mom = mom + 0.5 * eps * force(U)
    for i in range(ns):
        U = _rotate(U, mom, eps)
        mom = mom + (eps if i < ns - 1 else 0.5 * eps) * force(U)
    return U, mom


def _omf4(U, mom, beta, eps, ns):
    r1, r2, r3, r4 = 0.08398315262876693, 0.2539785108410595, 0.6822365335719091, -0.03230286765269967
    r5, r6 = 0.5 - r1 - r3, 1.0 - 2.0 * (r2 + r4)
    for _ in range(ns):
        for k, c in enumerate((r1, r3, r5, r5, r3, r1)):
            mom = mom + c * eps * _gauge_force(U, beta)
            if k < 5:
                U = _rotate(U, mom, eps * (r2, r4, r6, r4, r2)[k])
    return U, mom


def _philox(n, seed, stream, counter):
    """The four 32-bit words of blocks 0..n-1 of Philox4x32-10 (int64 tensors)."""
    M = 0xFFFFFFFF

    def mul(k, a):   # (high, low) words of k * a; a < 2^32 held in int64
        lo, hi = k * (a & 0xFFFF), k * (a >> 16)
        mid = hi + (lo >> 16)
        return mid >> 16, ((mid & 0xFFFF) << 16) | (lo & 0xFFFF)

    j = torch.arange(n, dtype=torch.int64, device="cuda")
    c = [j & M, j >> 32, torch.full_like(j, stream), torch.full_like(j, counter)]
    k0, k1 = seed & M, (seed >> 32) & M
    for _ in range(10):
        h0, l0 = mul(0xD2511F53, c[0])
        h1, l1 = mul(0xCD9E8D57, c[2])
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
        k0, k1 = (k0 + 0x9E3779B9) & M, (k1 + 0xBB67AE85) & M
    return c


def _normal(n, seed, stream, counter):
    c = _philox((n + 1) // 2, seed, stream, counter)
    a = ((c[0] << 21) | (c[1] >> 11)).double()
    b = ((c[2] << 21) | (c[3] >> 11)).double()
    rad = torch.sqrt(-2.0 * torch.log((a + 0.5) * 2.0 ** -53))
    ph = 2 * math.pi * (b * 2.0 ** -53)
    return torch.stack((rad * torch.cos(ph), rad * torch.sin(ph)), 1).reshape(-1)[:n]


def _uniform(seed, stream, counter):
    c = [int(v[0]) for v in _philox(1, seed, stream, counter)]
    return (((c[0] << 21) | (c[1] >> 11)) + 0.5) * 2.0 ** -53


def _noise(L1, L2, seed, stream):
    z = _normal(4 * L1 * L2, seed, stream, 0).view(-1, 2)
    return (torch.complex(z[:, 0], z[:, 1]) / math.sqrt(2.0)).view(2, L2, L1)


def _energy(U, mom, beta):
    V = U.shape[-1] * U.shape[-2]
    return (mom ** 2).sum((-3, -2, -1)) / 2 + beta * (V - _plaq(U).real.sum((-2, -1)))


def _zolotarev(n, ra, rb):
    """mu_j, nu_j, rho_j of the rational approximation of (g5Dw)^-1 on [ra, rb] (Zolotarev)."""
    m = 1.0 - (ra / rb) ** 2   # parameter k^2
    a, g = [1.0], math.sqrt(1.0 - m)
    c = [math.sqrt(m)]
    while abs(c[-1]) > 1e-17 and len(a) < 40:
        a0 = a[-1]
        a.append((a0 + g) / 2)
        c.append((a0 - g) / 2)
        g = math.sqrt(a0 * g)
    K = math.pi / (2 * a[-1])

    def ar(r):   # cn^2 / sn^2 by the descending Landen transformation
        u = r * K / (2 * n + 1)
        ph = 2.0 ** (len(a) - 1) * a[-1] * u
        for i in range(len(a) - 1, 0, -1):
            ph = (ph + math.asin(c[i] * math.sin(ph) / a[i])) / 2
        return (math.cos(ph) / math.sin(ph)) ** 2

    mu = [rb * math.sqrt(ar(2 * j)) for j in range(1, n + 1)]
    nu = [rb * math.sqrt(ar(2 * j - 1)) for j in range(1, n + 1)]
    rho = []
    for j in range(n):
        v = nu[j] ** 2 - mu[j] ** 2
        for k in range(n):
            if k != j:
                v *= (nu[k] ** 2 - mu[j] ** 2) / (mu[k] ** 2 - mu[j] ** 2)
        rho.append(v)
    return mu, nu, rho


def _decide(U0, U, hini, hfin, seed):
    p = math.exp(-(hfin - hini)) if hfin > hini else 1.0
    acc = 1 if p >= 1.0 or p > _uniform(seed, 3, 0) else 0
    return {"U": U if acc else U0, "hini": hini, "hfin": hfin, "accepted": acc}


def _momenta(L1, L2, seed):
    return _normal(2 * L1 * L2, seed, 1, 0).view(2, L2, L1)


def exact(case, seed):
    st = prepare(case, seed)
    kind = case["kind"]
    if kind == "dirac":
        return _g5dw(st["U"].to(torch.complex128), st["si"].to(torch.complex128), 0.1)
    if kind == "cg":
        return _solve(st["U"], st["b"], case["m0"], case["mu"] ** 2)
    if kind == "ensemble":
        sizes, _, am0 = _ensemble(case)
        b, out = st["batch"], torch.zeros_like(st["x"])
        for size in sorted(set(sizes)):   # equal lattices together
            at = [r for r in range(len(sizes)) if sizes[r] == size]
            m = torch.tensor([am0[r] for r in at], dtype=torch.float64, device="cuda").view(-1, 1, 1)
            x = _solve(torch.stack([b.replica(st["U"], r) for r in at]),
                       torch.stack([b.replica(st["b"], r) for r in at]), m)
            for i, r in enumerate(at):
                b.replica(out, r).copy_(x[i])
        return out
    U0, L1, L2 = st["U0"], case["L1"], case["L2"]
    if kind == "omf4":
        U, mom = _omf4(U0, st["mom0"], case["beta"], case["eps"], case["ns"])
        return {"U": U, "mom": mom}
    sd = st["seed"]
    if kind == "gauge":
        mom0 = _momenta(L1, L2, sd)
        U, mom = _omf4(U0, mom0, case["beta"], case["eps"], case["ns"])
        return _decide(U0, U, float(_energy(U0, mom0, case["beta"])), float(_energy(U, mom, case["beta"])), sd)
    m0, beta = case["m0"], case["beta"]
    if kind in ("nf2", "batch"):
        seeds = st["seeds"] if kind == "batch" else [sd]
        Us = U0 if kind == "batch" else U0[None]
        mom0 = torch.stack([_momenta(L1, L2, s) for s in seeds])
        X = torch.stack([_noise(L1, L2, s, 16) for s in seeds])
        F = _g5dw(Us, X, m0)
        last = {}

        def force(U):
            last["X"] = _solve(U, F, m0)
            return _gauge_force(U, beta) + _fermion_force(U, last["X"], _g5dw(U, last["X"], m0))

        hi = _energy(Us, mom0, beta) + _dot(X).view(-1)
        U, mom = _leapfrog(Us, mom0, force, case["eps"], case["ns"])
        hf = _energy(U, mom, beta) + (last["X"].conj() * F).real.sum((-3, -2, -1))
        each = [_decide(Us[r], U[r], float(hi[r]), float(hf[r]), s) for r, s in enumerate(seeds)]
        if kind == "nf2":
            return each[0]
        return {"U": torch.stack([e["U"] for e in each]), "hini": np.array([e["hini"] for e in each]),
                "hfin": np.array([e["hfin"] for e in each]),
                "accepted": np.array([e["accepted"] for e in each], dtype=np.int64)}
    mu, nu, rho = _zolotarev(case["poles"], *_rhmc_interval(case))
    mu2 = [m * m for m in mu]
    w = torch.tensor(rho, dtype=torch.float64, device="cuda").view(-1, 1, 1, 1)
    mom0, X = _momenta(L1, L2, sd), _noise(L1, L2, sd, 16)
    F = X
    for j in range(case["poles"]):
        F = _g5dw(U0, F, m0) + 1j * mu[j] * F
        F = _solve(U0, F, m0, nu[j] ** 2)
        F = _g5dw(U0, F, m0) - 1j * nu[j] * F

    def force(U):
        xs = _multishift(U, F, m0, mu2)
        return _gauge_force(U, beta) + (w * _fermion_force(U, xs, _g5dw(U, xs, m0))).sum(0)

    hi = float(_energy(U0, mom0, beta)) + float(_dot(X))
    U, mom = _leapfrog(U0, mom0, force, case["eps"], case["ns"])
    xs = F + (w * _multishift(U, F, m0, mu2)).sum(0)
    hf = float(_energy(U, mom, beta)) + float((xs.conj() * F).real.sum())
    return _decide(U0, U, hi, hf, sd)
