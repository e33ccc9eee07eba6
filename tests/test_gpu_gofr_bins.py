"""The pair-distance histogram counts what direct FP64 arithmetic counts where
pairs meet the bins' edges exactly: particles on simple cubic lattices, in and out
of the box, half a box apart, on one point, and far outside.  Counts are whole
numbers: no tolerance.
"""
from fractions import Fraction as F

import numpy as np
import pytest

from dmcbcs_project_gb300 import abi, capi, configs

pytestmark = pytest.mark.gpu


def fma(a, b, c):
    return float(F(a) * F(b) + F(c))


def distance(xi, xj, el):
    """Minimum-image distance with the multiply-adds of the device's direct form."""
    r2 = 0.0
    for a, b in zip(xi, xj):
        dx = float(a) - float(b)
        q = abs(dx / el)
        n = np.floor(q)
        n = float(n + (q - n >= 0.5)) * (1.0 if dx >= 0.0 else -1.0)   # nearest, halves away from zero
        dx = fma(-el, n, dx)
        r2 = fma(dx, dx, r2)
    return float(np.sqrt(r2))


@pytest.mark.parametrize("nup,ndn,m,ntabg", [(7, 7, 4, 64), (7, 6, 6, 60), (9, 9, 5, 100), (33, 33, 6, 60), (33, 30, 4, 100)])
def test_pairs_on_the_edges_of_bins(nup, ndn, m, ntabg):
    n, nw = nup + ndn, 6
    rng = np.random.default_rng(n)
    with capi.Context(abi.make_system(configs.system_params(nup, ndn, 2)), abi.make_run(configs.run_params(nw, 0.001))) as ctx:
        el = ctx.info.el
        sites = np.array([[i, j, k] for i in range(m) for j in range(m) for k in range(m)])
        x = np.stack([el * ((sites[rng.choice(len(sites), n, replace=n > len(sites))] + 0.5) / m - 0.5) for _ in range(nw)])
        x[1] += el * rng.integers(-3, 4, (n, 3))     # images
        x[2] += 0.125 * el                           # across the box's faces
        x[3, 1] = x[3, 0]                            # on one point
        x[4, 0] += 1.0e4 * el                        # far outside
        x[5] = el * (rng.random((n, 3)) - 0.5)       # anywhere
        one, vec = np.ones(nw), np.zeros((nw, n, 3))
        ctx.put_walkers(dict(n=nw, x=x, dpsi=vec, dpsig=vec, psil=0 * one, psigl=0 * one, d2psi=one, d2psig=one, v=one, vext=one,
                             weight=one, psil0=one, psigl0=one, wt0=one, is_=np.ones(nw, np.int32), irn=np.arange(1, nw + 1, dtype=np.int64)))
        ctx.set_operators(ntabg, 0, 0)
        ctx.add_operators()
        got = ctx.operators(0, raw=True)[0].reshape(3, ntabg + 1)
    scale = 1.0 / (0.5 * el / ntabg)
    want = np.zeros((3, ntabg + 1))
    for w in range(nw):
        for i in range(n):
            for j in range(i + 1, n):
                r = distance(x[w, i], x[w, j], el)
                want[0 if i < nup <= j else (1 if j < nup else 2), int(scale * r) if r < 0.5 * el else ntabg] += 2.0
    assert np.array_equal(got, want)
