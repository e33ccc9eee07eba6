"""The FP64 path's list of pairs inside the healing distance against the
oracle: pair counts on both sides of the list's limit (512), every pair in the
list, none, one, pairs either side of the healing distance and of a grid point,
coincident particles' neighbours, and a spline that reaches L/2 (no list).
Tolerance: the parity bar of the FP64 path, 1e-10 relative to max(|ref|, 1).
"""
import numpy as np
import pytest

import oracle
from dmcbcs_project_gb300 import abi, capi, configs

TOL = 1e-10
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nup,ndn", [(23, 22), (32, 16), (23, 23), (33, 33), (41, 40), (64, 64)])
@pytest.mark.parametrize("spline", [False, True])
def test_jastrow_terms_with_the_list(nup, ndn, spline):
    sysd = abi.make_system(configs.system_params(nup, ndn, 7))
    rund = abi.make_run(configs.run_params(4, 0.001))
    orc = oracle.Oracle(sysd, rund)
    rng = np.random.default_rng(nup * ndn)
    n = nup + ndn
    with capi.Context(sysd, rund) as ctx:
        if spline:
            knots = rng.uniform(-0.3, 0.3, 16)
            ctx.set_jastrow_spline(knots)
            orc.set_jastrow_spline(knots)
        el = ctx.info.el
        heal, dr = float(sysd.djas), 0.5 * el / int(sysd.ntab)
        x = el * (rng.random((5, n, 3)) - 0.5)
        x[0] *= 0.5 / el                                                   # every pair inside
        x[1, :nup] = 0.1 * rng.random((nup, 3)) - 0.24 * el                # none
        x[1, nup:] = 0.1 * rng.random((ndn, 3)) + 0.24 * el
        x[2] = x[1]
        x[2, n - 1] = x[2, nup - 1] + [0.0, 0.3, 0.0]                      # one, the last pair
        for j in range(ndn):                                               # about the healing distance
            x[3, nup + j] = x[3, j % nup] + [heal + (j - ndn // 2) * 0.5 * dr, 0.0, 0.0]
        x[4, nup:] = x[4, :ndn] + rng.normal(0.0, 0.4, (ndn, 3))           # pairs, as in a run
        got, ref = ctx.getphi(x), [orc.getphi(xw) for xw in x]
    for w in range(5):
        for k in ("u", "du", "d2u", "v"):
            a, b = np.asarray(got[k][w], float), np.asarray(ref[w][k], float)
            assert np.max(np.abs(a - b)) < TOL * max(float(np.max(np.abs(b))), 1.0), (k, w)
