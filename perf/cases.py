"""What is timed and compared: the calls that a program built on this library makes, over the sizes it makes them at.

Every system is one of the package's synthetic workloads (``configs.system_params``: 33 up / 33 down at seven shells and its relatives from
7/7 to 66/66).  A case names the call (``kind``), the system, the number of walkers and the arithmetic.  Walkers come from a short
Metropolis walk of the trial wavefunction, written in torch below, so that they have the distances, node distances and local energies
that a run meets and depend on the seed alone; their stored wavefunction values come from the same torch code in 64 bits.
"""
import functools
import math
import random

import numpy as np
import torch

from dmcbcs_project_gb300 import capi, configs
from dmcbcs_project_gb300.abi import make_run, make_system

F64 = torch.float64
M48 = (1 << 48) - 1
WALKER_FIELDS = ("x", "dpsi", "dpsig", "psil", "psigl", "d2psi", "d2psig", "v", "vext", "weight", "psil0", "psigl0", "wt0", "is_", "irn")


# ---- cases -------------------------------------------------------------------------------------------------------------------------
def listed():
    s = lambda name, kind, up, dn, norb, walkers, precision, **more: dict(  # noqa: E731
        name=name, kind=kind, up=up, dn=dn, norb=norb, walkers=walkers, precision=precision, **more)
    return [
        # the smallest run: 7/7, 200 walkers, one DMC generation on a population that the host keeps (the drop-in for step1 + branch)
        s("host_generation_7_7", "host", 7, 7, 5, 200, "fp64", idmc=1),
        # the production run: 33/33, 4096 walkers, a block of DMC generations on the device's own stack, mixed arithmetic
        s("block_33_33_mixed", "block", 33, 33, 7, 4096, "mixed", idmc=1, gens=5),
        # the same in plain FP64, the default arithmetic
        s("block_33_33_fp64", "block", 33, 33, 7, 4096, "fp64", idmc=1, gens=2),
        # a polarised, odd-sized variational run in FP64 (all-particle Metropolis moves)
        s("block_33_30_vmc", "block", 33, 30, 7, 1001, "fp64", idmc=0, gens=4),
        # the largest system: wavefunction and local energy of configurations on the device, mixed arithmetic
        s("hpsi_66_66_mixed", "hpsi", 66, 66, 7, 2048, "mixed"),
        # a parameter study: systems of uneven size advanced together
        s("batch_uneven", "batch", 66, 66, 7, 2048, "fp64", idmc=1, gens=1),
        # determinant, drift and stored inverse of a handful of configurations in host arrays (what single-particle moves start from)
        s("bcs_19_19", "bcs", 19, 19, 7, 37, "fp64"),
        # single-particle ratios from that inverse: the smallest call
        s("move1_33_33", "move1", 33, 33, 7, 64, "fp64"),
        # variational gradients of every parameter (shells, beta function, Jastrow knots)
        s("param_grad_33_33", "param_grad", 33, 33, 7, 2048, "fp64"),
        # stochastic reconfiguration: the sums of one optimisation step over a population
        s("sr_33_33", "sr", 33, 33, 7, 2048, "fp64"),
        # particle-by-particle sweeps with Sherman-Morrison updates
        s("sweeps_33_33", "sweeps", 33, 33, 7, 1024, "mixed", sweeps=2),
        # observables of a block's end: g(r), density, S(q), n(k)
        s("operators_33_33", "operators", 33, 33, 7, 512, "fp64"),
    ]


def draw(rng):
    kind = rng.choice(["host", "block", "block", "hpsi", "batch", "bcs", "move1", "param_grad", "sr", "operators"])
    up, dn, norb = rng.choice([(7, 7, 5), (9, 8, 6), (13, 13, 6), (19, 19, 7), (25, 24, 7), (33, 30, 7), (33, 33, 7), (38, 33, 7),
                               (45, 45, 7), (57, 57, 7), (66, 66, 7)])
    cost = ((up + dn) / 66.0) ** 2.5   # of one walker, against 33/33
    top = {"host": 4096, "block": 2400, "hpsi": 7000, "batch": 2048, "bcs": 2048, "move1": 4096, "param_grad": 2048, "sr": 2048,
           "operators": 512}[kind]
    high = max(40, int(top / max(cost, 0.5)))
    walkers = int(round(math.exp(rng.uniform(math.log(16), math.log(high)))))
    case = dict(kind=kind, up=up, dn=dn, norb=norb, walkers=walkers, precision="fp64")
    if kind in ("host", "block", "hpsi", "batch"):
        case["precision"] = rng.choice(["fp64", "mixed"])
    if kind in ("host", "block"):
        case["idmc"] = rng.choice([0, 1, 1, 2])
    if kind == "batch":
        case["idmc"] = 1
    if kind in ("block", "batch"):
        case["gens"] = rng.choice([1, 2, 3]) if kind == "block" else 1
    return case


# ---- the trial wavefunction in torch, 64 bits --------------------------------------------------------------------------------------
def beta_tables(el, n, b, d, bfact):
    """beta(r), its derivative and its Laplacian on n + 1 points of [0, L/2], images summed; b, d, bfact: 0-dim tensors."""
    e1, e2 = torch.exp(b * el * (1.0 + d)), torch.exp(d * b * el)
    db = d * b * el
    c = 0.5 * (2.0 + 2.0 * db + db**2 * e1 + 2.0 * d * b * b * el * el * e1 + 2.0 * b * el - 2.0 * e2 * b * el - 2.0 * e2) / (
        el * el * (e2 - 1.0 - d + d * e1) * (b * b))
    c0 = d
    c1 = -d + c * d - d * d / 2.0
    c2 = d / 2.0 + d**2 / 2.0 + d**3 / 6.0 + c * (-d - d * d / 2.0)
    c3 = -d / 6.0 - d**2 / 4.0 - d**3 / 6.0 - d**4 / 24.0 + c * (d / 2.0 + d**2 / 2.0 + d**3 / 6.0)
    c4 = d / 24.0 + d**2 / 12.0 + d**3 / 12.0 + d**4 / 24.0 + d**5 / 120.0 - c * (d / 6.0 + d**2 / 4.0 + d**3 / 6.0 + d**4 / 24.0)

    def beta0(r):
        small = r * b < 1.0e-3
        x = torch.where(small, torch.ones_like(r), r) * b
        ex, ex10 = torch.exp(-x), torch.exp(-d * x)
        f = (1.0 + c * x) * (1.0 - ex10) * ex / x
        fp = ex * (-1.0 - x * (1.0 + c * x) + ex10 * (1.0 + x * (1.0 + d) * (1.0 + c * x))) / (x * x)
        fpp = ex * (2.0 + x * (2.0 + x * (1.0 + c * x)) - ex10 * (2.0 + x * (1.0 + d) * (2.0 + x * (1.0 + d) * (1.0 + x * c)))) / x**3
        y = r * b
        f = torch.where(small, c0 + y * (c1 + y * (c2 + y * (c3 + y * c4))), f)
        fp = torch.where(small, c1 + y * (2.0 * c2 + y * (3.0 * c3 + 4.0 * c4 * y)), fp)
        fpp = torch.where(small, 2.0 * c2 + y * (6.0 * c3 + 12.0 * c4 * y), fpp)
        return f / d, b * fp / d, b * b * fpp / d

    def beta(r):
        inside = r <= 0.5 * el
        q = torch.where(inside, r, torch.full_like(r, 0.25 * el))
        h = beta0(torch.full_like(r[:1], 0.5 * el))[0]
        f1, p1, q1 = beta0(q)
        f2, p2, q2 = beta0(el - q)
        zero = torch.zeros_like(r)
        return (torch.where(inside, f1 + f2 - 2.0 * h, zero), torch.where(inside & (q >= 1.0e-14), p1 - p2, zero),
                torch.where(inside, q1 + q2, zero))

    r = torch.arange(n + 1, dtype=F64, device=b.device) * (0.5 * el / n)
    f, fp, fpp = beta(r)
    f2, p2, q2 = beta(el - r)   # the nearest image; farther ones are zero
    f, fp, fpp = f + f2, fp - p2, fpp + q2
    f = f - f[n]
    lap = torch.cat([3.0 * fpp[:1], fpp[1:] + 2.0 * fp[1:] / r[1:]])
    return bfact * f, bfact * fp, bfact * lap


def healed_jastrow(v0, amu, hb, djas, el, ntab):
    """log f, (log f)', (log f)'' of the zero-energy pair solution that is flat at the healing distance; the potential on the grid."""
    dr = 0.5 * el / ntab
    n = int(ntab * djas / (0.5 * el))
    pot = lambda r: -2.0 * v0 * amu**2 * hb / math.cosh(amu * r) ** 2  # noqa: E731
    v = [pot(i * dr) for i in range(ntab + 1)]
    vr, vh, ve = v[:n], [pot(i * dr + 0.5 * dr) for i in range(n)], [pot(i * dr + dr) for i in range(n)]

    def solve(ene):
        p, q, crossings, ps, qs = 0.0, 1.0, 0, [0.0], [1.0]
        for i in range(n):
            a1, b1 = -(ene - vr[i]) * p / hb, q
            a2, b2 = -(ene - vh[i]) * (p + 0.5 * dr * b1) / hb, q + 0.5 * dr * a1
            a3, b3 = -(ene - vh[i]) * (p + 0.5 * dr * b2) / hb, q + 0.5 * dr * a2
            a4, b4 = -(ene - ve[i]) * (p + dr * b3) / hb, q + dr * a3
            q += (a1 + 2.0 * a2 + 2.0 * a3 + a4) * dr / 6.0
            new = p + (b1 + 2.0 * b2 + 2.0 * b3 + b4) * dr / 6.0
            crossings += new != math.copysign(abs(new), p)
            p = new
            ps.append(p)
            qs.append(q)
        return crossings, ps, qs

    low, high = min(v[: n + 1]), 0.001
    while solve(high)[0] <= 0:
        high *= 2.0
    ene = 0.5 * (low + high)
    for _ in range(101):
        _, f, df = solve(ene)
        r = dr * n
        der = (df[n] - f[n] / r) / r / f[n]
        if abs(der) < 1.0e-8:
            break
        low, high = (low, ene) if der < 0.0 else (ene, high)
        ene = 0.5 * (low + high)
    u, du, d2u = np.zeros(ntab + 1), np.zeros(ntab + 1), np.zeros(ntab + 1)
    for i in range(n + 1):
        r = i * dr
        g = df[0] if i == 0 else f[i] / r
        gp = 0.0 if i == 0 else (df[i] - g) / r
        gpp = (v[0] - ene) * df[0] / (3.0 * hb) if i == 0 else (v[i] - ene) * g / hb - 2.0 * gp / r
        u[i], du[i], d2u[i] = math.log(g / (f[n] / (dr * n))), gp / g, gpp / g - (gp / g) ** 2
    return u, du, d2u, np.array(v)


def knot_basis(el, ntab):
    """The 16 knots' basis functions with two derivatives on the pair grid, [3][16][ntab + 1]."""
    h = el / 34.0
    t = np.arange(ntab + 1) * (0.5 * el / ntab) / h

    def bspline(t):
        a, s = np.abs(t), np.where(t < 0.0, -1.0, 1.0)
        q = 2.0 - a
        out = [np.where(a < 1.0, 2.0 / 3.0 - a * a + 0.5 * a**3, q**3 / 6.0), s * np.where(a < 1.0, -2.0 * a + 1.5 * a * a, -0.5 * q * q),
               np.where(a < 1.0, -2.0 + 3.0 * a, q)]
        return np.array([np.where(a < 2.0, o, 0.0) for o in out])

    f = np.array([bspline(t - k) + (bspline(t + k) if k else 0.0) for k in range(16)])
    return np.stack([f[:, 0], f[:, 1] / h, f[:, 2] / h**2])


class Trial:
    """The pair wavefunction with its Jastrow factor: |Psi| = exp(U) |det S|, masses 1."""

    def __init__(self, up, dn, norb, dev):
        self.params = configs.system_params(up, dn, norb)
        self.up, self.dn, self.norb, self.dev = up, dn, norb, dev
        p = self.params
        self.n, self.nd, self.ntab, self.hbar = up + dn, up, p["ntab"], p["hbar"]
        self.el = (self.n / p["rho"]) ** (1.0 / 3.0)
        self.kunit2 = (3.0 * math.pi**2 * self.n / self.el**3) ** (2.0 / 3.0)
        self.eunit = 0.6 * self.hbar * self.kunit2   # reduced mass 1/2
        half = {}
        top = 2 * norb
        for a in range(-6, 7):
            for b in range(-6, 7):
                for c in range(-6, 7):
                    n2 = a * a + b * b + c * c
                    if 0 < n2 <= top and (a, b, c) > (0, 0, 0):
                        half.setdefault(n2, []).append((a, b, c))
        shells = sorted(half)[: norb - 1]
        ks = [(k, s + 1) for s, n2 in enumerate(shells) for k in half[n2]]
        T = lambda v: torch.tensor(v, dtype=F64, device=dev)  # noqa: E731
        self.k = T([k for k, _ in ks]) * (2.0 * math.pi / self.el)
        self.k2 = (self.k**2).sum(1)
        self.shell = torch.tensor([s for _, s in ks], device=dev)
        self.theta0 = T(p["vorb"] + [p["bfact"], p["bbeta"], p["dbeta"]])
        u, du, d2u, v = healed_jastrow(p["v0"], p["amu"], 2.0 * self.hbar, p["djas"], self.el, self.ntab)
        self.jas = T(np.stack([u, du, d2u]))
        self.pot = T(v)
        self.knots = T(knot_basis(self.el, self.ntab))
        self.kex = T([list(k) for k in p["ikup"]] or [[0, 0, 0]]) * (2.0 * math.pi / self.el)
        self.sinex = [next((c < 0 for c in reversed(k) if c), False) for k in p["ikup"]]
        self.nex = p["nexup"]
        self.btab = beta_tables(self.el, self.ntab, self.theta0[norb + 1], self.theta0[norb + 2], self.theta0[norb])

    def image(self, d):
        return d - self.el * torch.round(d / self.el)

    def weights(self, r):
        s = r * (self.ntab / (0.5 * self.el))
        i = s.to(torch.int64).clamp(1, self.ntab - 2)
        t = s - i
        a, b, c = t - 1.0, t - 2.0, t + 1.0
        return i, (-t * a * b / 6.0, c * a * b / 2.0, -c * t * b / 2.0, c * t * a / 6.0)

    @staticmethod
    def look(table, iw):
        i, w = iw
        return sum(w[m] * table[i + (m - 1)] for m in range(4))

    def matrix(self, x, vorb, btab):
        """S, the pair vectors (up - down), their lengths and table weights."""
        xu, xd = x[:, : self.up], x[:, self.up:]
        d = self.image(xu[:, :, None] - xd[:, None])
        r = d.norm(dim=3)
        iw, inside = self.weights(r), r <= 0.5 * self.el
        amp = 2.0 * vorb[self.shell]
        au, ad = xu @ self.k.T, xd @ self.k.T
        s = (torch.cos(au) * amp) @ torch.cos(ad).mT + (torch.sin(au) * amp) @ torch.sin(ad).mT + vorb[0]
        s = s + torch.where(inside, self.look(btab[0], iw), 0.0)
        if self.nex:
            arg = xu @ self.kex.T
            s = torch.cat([s, torch.stack([torch.sin(arg[..., j]) if self.sinex[j] else torch.cos(arg[..., j]) for j in range(self.nex)], 2)], 2)
        return s, d, r, iw, inside, au, ad, amp

    def log_psi(self, x):
        s, _, r, iw, inside, *_ = self.matrix(x, self.theta0[: self.norb], self.btab)
        sign, logdet = torch.linalg.slogdet(s)
        return logdet + torch.where(inside, self.look(self.jas[0], iw), 0.0).sum((1, 2)), sign

    def evaluate(self, x, theta=None, knots=None):
        """Every quantity of hpsi, with the determinant's own parts and the inverse."""
        if theta is None:
            theta, btab = self.theta0, self.btab
        else:
            btab = beta_tables(self.el, self.ntab, theta[self.norb + 1], theta[self.norb + 2], theta[self.norb])
        jas = self.jas if knots is None else self.jas + torch.einsum("k,dki->di", knots, self.knots)
        s, d, r, iw, inside, au, ad, amp = self.matrix(x, theta[: self.norb], btab)
        sign, logdet = torch.linalg.slogdet(s)
        inv = torch.linalg.inv(s)
        w = inv[:, : self.dn].mT   # [walker][up][down] = inv(S)[down][up]
        rs = r.clamp(min=1.0e-14)
        cut = lambda t: torch.where(inside, self.look(t, iw), 0.0)  # noqa: E731
        u, v = cut(jas[0]).sum((1, 2)), cut(self.pot).sum((1, 2))
        uf = cut(jas[1]) / rs
        pair = (d * uf[..., None])
        du = torch.cat([pair.sum(2), -pair.sum(1)], 1)
        d2u = 2.0 * (cut(jas[2]) + 2.0 * uf).sum((1, 2)) + (du**2).sum((1, 2))
        # grad and Laplacian of S_ij with respect to the up particle (down: minus the gradient)
        cu, su, cd, sd = torch.cos(au), torch.sin(au), torch.cos(ad), torch.sin(ad)
        gc, gs = w @ cd, w @ sd                       # [walker][up][k]
        hc, hs = w.mT @ cu, w.mT @ su                 # [walker][down][k]
        tu, td = amp * (cu * gs - su * gc), amp * (cd * hs - sd * hc)
        lu = -(amp * self.k2 * (cu * gc + su * gs)).sum(2)
        ld = -(amp * self.k2 * (cd * hc + sd * hs)).sum(2)
        wb = (w * cut(btab[1]) / rs)[..., None] * d
        wl = w * cut(btab[2])
        gup, gdn = tu @ self.k + wb.sum(2), td @ self.k - wb.sum(1)
        lup, ldn = lu + wl.sum(2), ld + wl.sum(1)
        for j in range(self.nex):
            arg = x[:, : self.up] @ self.kex[j]
            col = inv[:, self.dn + j]
            val, der = (torch.sin(arg), torch.cos(arg)) if self.sinex[j] else (torch.cos(arg), -torch.sin(arg))
            gup = gup + (col * der)[..., None] * self.kex[j]
            lup = lup - col * val * (self.kex[j] ** 2).sum()
        dphi, d2phi = torch.cat([gup, gdn], 1), lup.sum(1) + ldn.sum(1)
        psil, d2psi = logdet + u, d2phi + d2u + 2.0 * (du * dphi).sum((1, 2))
        return dict(psil=psil, sign=sign, dpsi=dphi + du, d2psi=d2psi, v=v, logdet=logdet, dphi=dphi, d2phi=d2phi, inv=inv)

    def parts(self, x, **kw):
        """evaluate() in slices of walkers that fit the card."""
        step = max(1, int(4.0e6 / (self.up * self.dn)))
        got = [self.evaluate(x[i: i + step], **kw) for i in range(0, len(x), step)]
        return {k: torch.cat([g[k] for g in got]) for k in got[0]}

    def walk(self, count, seed):
        """count configurations of a short Metropolis walk: pairs at random, then moves of all particles at once."""
        g = torch.Generator(device=self.dev)
        g.manual_seed(seed)
        normal = lambda n: torch.randn(n, self.n, 3, dtype=F64, device=self.dev, generator=g)  # noqa: E731
        few = min(count, 256)
        xu = self.el * (torch.rand(few, self.up, 3, dtype=F64, device=self.dev, generator=g) - 0.5)
        x = torch.cat([xu, xu[:, : self.dn]], 1) + 0.8 * normal(few)
        step = 0.12 * math.sqrt(66.0 / self.n)
        for k in range(90):
            if k == 80 and count > few:
                x = x.repeat(-(-count // few), 1, 1)[:count]
            if k in (0, 80):
                old, _ = self.log_psi(x)
            y = x + step * normal(len(x))
            new, _ = self.log_psi(y)
            take = torch.log(torch.rand(len(x), dtype=F64, device=self.dev, generator=g)) < 2.0 * (new - old)
            x, old = torch.where(take[:, None, None], y, x), torch.where(take, new, old)
        return self.image(x)


@functools.lru_cache(maxsize=16)
def trial(up, dn, norb):
    return Trial(up, dn, norb, torch.device("cuda"))


def systems(case):
    """(up, dn, norb, walkers) of each system of a case."""
    if case["kind"] != "batch":
        return [(case["up"], case["dn"], case["norb"], case["walkers"])]
    n = case["walkers"]
    return [(case["up"], case["dn"], case["norb"], max(1, n // 4)), (33, 33, 7, n), (38, 33, 7, max(1, n // 2)), (7, 7, 5, max(1, (3 * n) // 4))]


def run_values(case, walkers, seed):
    return make_run(configs.run_params(walkers, 0.001, idmc=case.get("idmc", 1), seed=17 + 2 * seed))


def knot_values(seed):
    return np.random.default_rng(seed).uniform(-0.3, 0.3, 16) * np.exp(-0.15 * np.arange(16))


def population(t, walkers, seed):
    """A population as the library exchanges it: positions, their stored evaluation, random number states."""
    x = t.walk(walkers, seed)
    e = t.parts(x)
    a = {k: e[k].cpu().numpy() for k in ("dpsi", "psil", "d2psi", "v")}
    zero = np.zeros(walkers)
    sign = e["sign"].cpu().numpy()
    rng = np.random.default_rng([seed, walkers])
    return dict(x=x.cpu().numpy(), dpsi=a["dpsi"], dpsig=a["dpsi"], psil=a["psil"], psigl=a["psil"], d2psi=a["d2psi"], d2psig=a["d2psi"],
                v=a["v"], vext=zero, weight=np.ones(walkers), psil0=zero, psigl0=zero, wt0=sign.astype(np.float64),
                is_=sign.astype(np.int32), irn=rng.integers(1, 1 << 47, walkers, dtype=np.int64) * 2 + 1)


def pinned(npart, cap, values=None):
    """Population arrays in page-locked memory, as a host program keeps them for the GPU."""
    out = {}
    for k in WALKER_FIELDS:
        shape = (cap, npart, 3) if k in ("x", "dpsi", "dpsig") else (cap,)
        kind = {"is_": torch.int32, "irn": torch.int64}.get(k, F64)
        out[k] = torch.empty(shape, dtype=kind, pin_memory=True).numpy()
        out[k][:] = 0
        if values is not None:
            out[k][: len(values[k])] = values[k]
    out["n"] = 0 if values is None else len(values["irn"])
    out["cap"] = cap
    return out


def room(walkers):
    """Rows of a host's population arrays: population control keeps the count within a tenth of the target, branching adds a little."""
    return walkers + walkers // 4 + 64


def prepare(case, seed):
    kind = case["kind"]
    members = []
    for m, (up, dn, norb, walkers) in enumerate(systems(case)):
        t = trial(up, dn, norb)
        ctx = capi.Context(make_system(t.params), run_values(case, walkers, seed), precision=case["precision"])
        s = dict(ctx=ctx, trial=t)
        if kind in ("host", "block", "batch", "sweeps", "operators", "sr"):
            cap = room(walkers)
            s["in"] = pinned(t.n, walkers, population(t, walkers, seed + m))
            s["out"] = pinned(t.n, cap)
        else:
            s["x"] = t.walk(walkers, seed)
        members.append(s)
    state = dict(case=case, members=members, **members[0])
    ctx, t, n = state["ctx"], state["trial"], case["walkers"]
    if kind == "hpsi":
        dev = lambda *shape: torch.zeros(shape, dtype=F64, device="cuda")  # noqa: E731
        state["o"] = dict(psil=dev(n), is_=torch.zeros(n, dtype=torch.int32, device="cuda"), dpsi=dev(n, t.n, 3), d2psi=dev(n), v=dev(n),
                          vext=dev(n), psigl=dev(n), dpsig=dev(n, t.n, 3), d2psig=dev(n))
        torch.cuda.synchronize()
    if kind in ("bcs", "move1", "param_grad"):
        state["hx"] = state["x"].cpu().numpy()
    if kind == "move1":
        state.update(moves(t, state["x"], seed))
    if kind == "param_grad":
        ctx.set_jastrow_spline(knot_values(seed))
    if kind == "operators":
        ctx.set_operators(200, 8, 20)
    if kind in ("operators", "sr"):
        ctx.put_walkers(state["in"])
    if kind == "batch":
        state["batch"] = capi.Batch([s["ctx"] for s in members])
    return state


def moves(t, x, seed):
    """A single-particle move of each walker and the inverses it starts from."""
    rng = np.random.default_rng([seed, 3])
    n = len(x)
    inv = t.parts(x)["inv"]
    return dict(smati=inv.mT.reshape(n, -1).cpu().numpy().copy(), ipart=rng.integers(1, t.n + 1, n).astype(np.int32),
                shift=rng.normal(0.0, 0.4, (n, 3)))


def whole(arrs):
    """A host's population arrays with every row; the count that comes beside them says how many are walkers."""
    return {k: arrs[k] for k in WALKER_FIELDS}


def run(state):
    case, ctx, kind = state["case"], state["ctx"], state["case"]["kind"]
    if kind == "host":
        ctx.zero_estimators()
        n = ctx.generation_host(state["in"], state["out"], True)
        return dict(walkers=whole(state["out"]), n=n, sums=np.array(ctx.estimators()))
    if kind == "block":
        ctx.put_walkers(state["in"])
        ctx.zero_estimators()
        for g in range(case["gens"]):
            _generation(ctx, g == case["gens"] - 1)
        val, err = ctx.block_update()
        n = ctx.get_walkers_into(state["out"])
        return dict(walkers=whole(state["out"]), n=n, val=val)
    if kind == "batch":
        for s in state["members"]:
            s["ctx"].put_walkers(s["in"])
            s["ctx"].zero_estimators()
        state["batch"].generations(case["gens"], opcomp_last=True)
        n = np.array([s["ctx"].get_walkers_into(s["out"]) for s in state["members"]])
        return dict(walkers=[whole(s["out"]) for s in state["members"]], n=n,
                    val=np.array([s["ctx"].block_update()[0] for s in state["members"]]))
    if kind == "hpsi":
        o = state["o"]
        order = ("psil", "is_", "dpsi", "d2psi", "v", "vext", "psigl", "dpsig", "d2psig")
        ctx._check(capi.load().dmc_hpsi_device(ctx._h, case["walkers"], state["x"].data_ptr(), *[o[k].data_ptr() for k in order],
                                               torch.cuda.current_stream().cuda_stream))
        return o
    if kind == "bcs":
        return ctx.bcs(state["hx"], want_inverse=True)
    if kind == "move1":
        at = np.arange(case["walkers"]), state["ipart"] - 1
        return ctx.move1(state["hx"], state["smati"], state["ipart"], state["hx"][at] + state["shift"])
    if kind == "param_grad":
        return ctx.param_grad(state["hx"])
    if kind == "sr":
        ctx.sr_zero()
        ctx.sr_accumulate()
        return ctx.sr_sums()
    if kind == "sweeps":
        ctx.put_walkers(state["in"])
        accepted, _ = ctx.sm_sweeps(case["sweeps"], 16)
        n = ctx.get_walkers_into(state["out"])
        return dict(accepted=accepted, walkers=whole(state["out"]), n=n)
    ctx.zero_operators()
    ctx.add_operators()
    return [ctx.operators(w, raw=True)[0] for w in range(4)]


def _generation(ctx, last):
    """A generation of a block: the population count is not asked for, so nothing waits for it."""
    ctx._check(capi.load().dmc_generation(ctx._h, int(last), None))


def work(case):
    total = dict(bytes=0.0, flops=0.0)
    for up, dn, norb, n in systems(case):
        t = trial(up, dn, norb)
        cols = 2 * len(t.k) + 1
        p, nd = up + dn, up
        hpsi = 10.0 * up * dn * cols + 2.0 * nd**3 + 8.0 * nd * p + 30.0 * p * (p - 1) + 40.0 * up * dn + 30.0 * p
        state = 8.0 * (9 * p + 13)
        kind = case["kind"]
        if kind in ("host", "block", "batch"):
            flops, byts = hpsi * case.get("gens", 1), 2 * state
        elif kind == "hpsi":
            flops, byts = hpsi, 8.0 * (9 * p + 8)
        elif kind == "bcs":
            flops, byts = hpsi - 30.0 * p * (p - 1), 8.0 * (6 * p + nd * nd + 3)
        elif kind == "move1":
            flops, byts = 4.0 * nd * cols + 60.0 * p, 8.0 * (3 * p + nd * nd + 5)
        elif kind == "param_grad":
            flops, byts = 2.0 * hpsi + 4.0 * nd**3, 8.0 * (3 * p + 2 * (norb + 19))
        elif kind == "sr":
            flops, byts = 2.0 * up * dn * cols + 2.0 * nd**3 + 2.0 * up * dn * (cols - 1), state
        elif kind == "sweeps":
            flops, byts = hpsi + case["sweeps"] * p * (2.0 * nd * cols + 4.0 * nd * nd), 2 * state
        else:
            flops, byts = 2.0 * up * dn * cols + 2.0 * nd**3 + 10.0 * p * (2.0 * nd * cols + 2.0 * nd), state
        total["flops"] += flops * n
        total["bytes"] += byts * n
    return total


# ---- the same in 64 bits with torch and numpy alone ----------------------------------------------------------------------------------
def ran(state, a, c):
    """One step of a 48-bit congruential generator."""
    return (state * np.uint64(a) + np.uint64(c)) & np.uint64(M48)


def ran1(s):
    return ran(s, 44485709377909, 96309754297)


def ran2(s):
    return ran(s, 34522712143931, 55789347517)


def uniform(s):
    return (s | np.uint64(1)).astype(np.float64) * 2.0**-48


def branch(w, factor):
    """Copies of each walker by its weight, top of the stack first."""
    w = {k: v[::-1] for k, v in w.items()}
    s = ran1(w["irn"].astype(np.uint64))
    wt = w["weight"] * factor
    copies = np.maximum(0, (wt + uniform(s)).astype(np.int64))
    at = np.repeat(np.arange(len(s)), copies)
    rank = np.arange(len(at)) - np.repeat(np.cumsum(copies) - copies, copies)
    out = {k: v[at] for k, v in w.items()}
    st = s[at]
    for k in range(int(copies.max(initial=0))):
        st = np.where(rank >= k, ran2(st), st)
    out["irn"], out["weight"] = st.astype(np.int64), np.copysign(np.ones(len(at)), wt[at])
    return out


def generation(t, case, target, w):
    """One generation of the walker loop on a population."""
    r = configs.run_params(target, 0.001, idmc=case["idmc"])
    dt, idmc, n3 = r["dt"], case["idmc"], 3 * t.n
    old = {k: v[::-1] for k, v in w.items()}
    n = len(old["irn"])
    s = old["irn"].astype(np.uint64)
    u = []
    for _ in range(2 * ((n3 + 1) // 2)):
        s = ran1(s)
        u.append(uniform(s))
    u = np.array(u).T
    ang, rad = 2.0 * np.pi * u[:, 0::2], np.sqrt(-2.0 * np.log(u[:, 1::2]))
    g = np.stack([np.sin(ang) * rad, np.cos(ang) * rad], 2).reshape(n, -1)
    if n3 % 2:
        g[:, n3 - 1] = g[:, n3]
    sig = math.sqrt(2.0 * t.hbar * dt)
    img = lambda d: d - t.el * np.rint(d / t.el)  # noqa: E731
    xo = img(old["x"])
    drift = old["dpsig"] * sig**2
    dx = drift + sig * g[:, :n3].reshape(n, t.n, 3)
    x = img(xo + dx)
    e = {k: v.cpu().numpy() for k, v in t.parts(torch.from_numpy(x).to(t.dev)).items() if k != "inv"}
    sign = np.rint(e["sign"]).astype(np.int32)
    new = dict(x=x, dpsi=e["dpsi"], dpsig=e["dpsi"], psil=e["psil"], psigl=e["psil"], d2psi=e["d2psi"], d2psig=e["d2psi"], v=e["v"], is_=sign)
    take = np.ones(n, bool)
    if idmc != 1:
        dn = e["dpsi"] * sig**2
        prob = 2.0 * (e["psil"] - old["psil"]) + ((drift + dn) * (drift - dn - 2.0 * dx)).sum((1, 2)) / (2.0 * sig**2)
        s = ran1(s)
        take = uniform(s) < np.exp(np.minimum(0.0, prob))
    kept = dict(old, x=xo)
    mix = lambda a, b: np.where(take.reshape((-1,) + (1,) * (a.ndim - 1)), a, b)  # noqa: E731
    out = dict(kept, **{k: mix(v, kept[k]) for k, v in new.items()})
    out["irn"] = s.astype(np.int64)
    eo, en = -t.hbar * old["d2psi"] + old["v"], -t.hbar * e["d2psi"] + e["v"]
    et = r["etrial"] * t.eunit * t.n
    if idmc == 0:
        out["wt0"] = np.where(take, sign.astype(np.float64), old["wt0"])
    else:
        move = np.where(sign != old["is_"], 0.0, np.minimum(r["wtcut"], np.exp(-(0.5 * (eo + en) - et) * dt)))
        stay = np.minimum(r["wtcut"], np.exp(-(eo - et) * dt) * old["weight"])
        out["weight"] = np.where(take, move, stay)
        out = branch(out, 1.0)
    n = len(out["irn"])
    if n > r["popup"] * target or n < r["popdn"] * target:
        out = branch(out, target / n)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("sweeps", "operators"):
        return None   # thousands of dependent single-particle decisions, or draws, per walker
    if kind in ("host", "block", "batch"):
        got = []
        for m, (up, dn, norb, walkers) in enumerate(systems(case)):
            t = trial(up, dn, norb)
            w = population(t, walkers, seed + m)
            for _ in range(case.get("gens", 1)):
                w = generation(t, case, walkers, w)
            rows = room(walkers)
            got.append({k: np.concatenate([w[k], np.zeros((rows - len(w[k]),) + w[k].shape[1:], w[k].dtype)]) for k in WALKER_FIELDS})
        return dict(walkers=got if kind == "batch" else got[0], n=None, **{"sums" if kind == "host" else "val": None})
    t = trial(case["up"], case["dn"], case["norb"])
    x = t.walk(case["walkers"], seed)
    if kind == "param_grad":
        knots = torch.tensor(knot_values(seed), dtype=F64, device=t.dev)
        point = torch.cat([t.theta0, knots])
        m = len(t.theta0)

        def values(theta, part):
            e = t.evaluate(part, theta=theta[:m], knots=theta[m:])
            return e["psil"], -t.hbar * e["d2psi"] + e["v"]

        cols = []
        for q in range(len(point)):
            way = torch.zeros_like(point)
            way[q] = 1.0
            step = max(1, int(1.0e6 / (t.up * t.dn)))
            cols.append([torch.cat(c) for c in zip(*[torch.func.jvp(lambda th: values(th, x[i: i + step]), (point,), (way,))[1]  # noqa: B023
                                                     for i in range(0, len(x), step)])])
        return tuple(torch.stack([c[o] for c in cols], 1).cpu().numpy() for o in (0, 1))
    e = t.parts(x)
    if kind == "hpsi":
        return dict(psil=e["psil"], is_=None, dpsi=e["dpsi"], d2psi=e["d2psi"], v=e["v"], vext=torch.zeros_like(e["v"]), psigl=e["psil"],
                    dpsig=e["dpsi"], d2psig=e["d2psi"])
    if kind == "bcs":
        return dict(phil=e["logdet"], is_=None, dphi=e["dphi"], d2phi=e["d2phi"], smati=e["inv"].mT.reshape(len(x), -1))
    if kind == "move1":
        mv = moves(t, x, seed)
        y = x.clone()
        y[torch.arange(len(x)), torch.from_numpy(mv["ipart"]).long() - 1] += torch.from_numpy(mv["shift"]).to(t.dev)
        (a, sa), (b, sb) = t.log_psi(x), t.log_psi(y)
        return sa * sb * torch.exp(b - a)
    # sr: derivatives of log|det| with respect to the shells' amplitudes, with the local energies
    w = e["inv"][:, : t.dn].mT
    au, ad = x[:, : t.up] @ t.k.T, x[:, t.up:] @ t.k.T
    per_k = 2.0 * ((torch.cos(au) * (w @ torch.cos(ad))).sum(1) + (torch.sin(au) * (w @ torch.sin(ad))).sum(1))
    der = torch.zeros(len(x), t.norb, dtype=F64, device=t.dev)
    der.index_add_(1, t.shell, per_k)
    der[:, 0] = w.sum((1, 2))
    ene = (-t.hbar * e["d2psi"] + e["v"]) / t.eunit / t.n
    return dict(ovec=der.sum(0), ovecw=(der * ene[:, None]).sum(0), pmat=der.mT @ der, e=torch.stack([ene.sum(), (ene**2).sum()]), n=None)


if __name__ == "__main__":
    print(listed(), draw(random.Random(0)))
