"""The walker kernel's inverse on both sides of every change of its panel's warps
and widths (32, 52, 64, 96 rows; 96 with eight warps, and with sixteen for few
shells, mixed), against the oracle.  Tolerance, relative to max(|ref|, 1): the
parity bars of the two precisions (1e-10; 1e-6), or where it is larger the forward
error of an inverse of random configurations, nd cond(S) 2^-52 (2^-44 in
double-float).
"""
import numpy as np
import pytest

import oracle
from dmcbcs_project_gb300 import abi, capi, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("nup,ndn,norb", [(32, 32, 5), (33, 31, 5), (52, 52, 5), (53, 53, 5), (64, 60, 5), (65, 65, 7), (70, 70, 3), (76, 76, 7),
                                          (96, 96, 7), (97, 97, 7)])
def test_inverse_at_every_width(nup, ndn, norb, prec):
    sysd, rund = abi.make_system(configs.system_params(nup, ndn, norb)), abi.make_run(configs.run_params(4, 0.001))
    orc = oracle.Oracle(sysd, rund)
    with capi.Context(sysd, rund, precision=prec) as ctx:
        x = ctx.info.el * (np.random.default_rng(nup).random((2, nup + ndn, 3)) - 0.5)
        got, ref = ctx.bcs(x, want_inverse=True), orc.bcs(x, want_inverse=True)
    assert np.array_equal(got["is_"], ref["is_"])
    for w in range(2):
        inv = ref["smati"][w].reshape(nup, nup)
        bar, eps = (1e-10, 2.0 ** -52) if prec == "fp64" else (1e-6, 2.0 ** -44)
        tol = max(bar, nup * np.linalg.cond(inv) * eps)
        for k in ("phil", "dphi", "d2phi", "smati"):
            a, b = np.asarray(got[k][w], float), np.asarray(ref[k][w], float)
            assert np.max(np.abs(a - b)) < tol * max(1.0, np.max(np.abs(b))), k
