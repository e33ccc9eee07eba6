"""The FP64 path's pair function in 64-bit fixed point against the oracle's
plane-wave sums: every shell count on both sides of the symmetric form's limit
(|n|^2 <= 6, seven shells) up to the octant form's largest vectors, the
smallest systems, odd and polarised ones, particles far outside the box, on a
common coordinate and close together.  Tolerance: the parity bar of the FP64
path, 1e-10 relative to max(|ref|, 1), or where it is larger the forward error
of an FP64 inverse, nd cond(S) 2^-52 (the configurations are random); an
entry's fixed-point error is below 2^-57 of the amplitudes' sum, inside both.
"""
import numpy as np
import pytest

import oracle
from dmcbcs_project_gb300 import abi, capi, configs

TOL = 1e-10
pytestmark = pytest.mark.gpu


def rel(a, b):
    a, b = np.asarray(a, float), np.asarray(b, float)
    return float(np.max(np.abs(a - b)) / max(float(np.max(np.abs(b))), 1.0))


@pytest.mark.parametrize("nup,ndn,norb", [(1, 1, 1), (2, 1, 2), (7, 7, 1), (8, 7, 6), (13, 13, 7), (9, 9, 8), (17, 16, 10),
                                          (7, 7, 17), (5, 5, 32), (41, 40, 7), (60, 52, 9)])
def test_every_shell_count(nup, ndn, norb):
    sysd = abi.make_system(configs.system_params(nup, ndn, norb))
    rund = abi.make_run(configs.run_params(4, 0.001))
    orc = oracle.Oracle(sysd, rund)
    rng = np.random.default_rng(norb)
    with capi.Context(sysd, rund) as ctx:
        el, n = ctx.info.el, nup + ndn
        x = el * (rng.random((4, n, 3)) - 0.5)
        x[1] += el * rng.integers(-4, 5, (n, 3))          # images of any box
        x[2, nup] = x[2, 0] + [0.0, 0.1, 0.0]             # two common coordinates, close together
        x[3, nup] = x[3, 0] + [0.499 * el, 0.0, 1.0e-9]   # near the tables' end
        got, ref = ctx.hpsi(x), orc.hpsi(x)
        bcs, rbcs = ctx.bcs(x, want_inverse=True), orc.bcs(x, want_inverse=True)
        jas, rjas = ctx.getphi(x), [orc.getphi(xw) for xw in x]
    assert np.array_equal(got["is_"], ref["is_"])
    for w in range(4):
        inverse = rbcs["smati"][w].reshape(nup, nup)
        tol = max(TOL, nup * np.linalg.cond(inverse) * 2.0 ** -52)
        for k in ("psil", "d2psi", "v", "dpsi"):
            assert rel(got[k][w], ref[k][w]) < tol, (k, w)
        for k in ("phil", "d2phi", "dphi"):
            assert rel(bcs[k][w], rbcs[k][w]) < tol, (k, w)
        assert rel(bcs["smati"][w], inverse.reshape(-1)) < tol
        for k in ("u", "du", "d2u", "v"):
            assert rel(jas[k][w], rjas[w][k]) < TOL, (k, w)


def test_amplitudes_that_are_not_finite_stay_visible():
    sysd = abi.make_system(configs.system_params(7, 7, 5))
    with capi.Context(sysd, abi.make_run(configs.run_params(4, 0.001))) as ctx:
        x = ctx.info.el * (np.random.default_rng(1).random((2, 14, 3)) - 0.5)
        good = ctx.bcs(x)["phil"]
        v = np.array(list(sysd.vorb)[:5])
        ctx.set_vorb(np.where(np.arange(5) == 2, np.nan, v))
        assert not np.isfinite(ctx.bcs(x)["phil"]).any() and (ctx.walker_status(2) & 2).all()
        ctx.set_vorb(v)
        assert np.array_equal(ctx.bcs(x)["phil"], good)
