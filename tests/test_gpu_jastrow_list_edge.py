"""Jastrow terms on both sides of the healing distance from which the pair list is
left (a sixth of the box) and where every pair is inside it (half of the box),
against the oracle: the parity bar of the FP64 path, 1e-10 relative to
max(|ref|, 1).
"""
import numpy as np
import pytest

import oracle
from dmcbcs_project_gb300 import abi, capi, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("share", [0.1664, 0.1667, 0.1669, 0.25, 0.4999])
@pytest.mark.parametrize("nup,ndn", [(23, 23), (40, 33)])
def test_healing_distance_about_the_list_s_limit(nup, ndn, share):
    par = configs.system_params(nup, ndn, 7)
    par["djas"] = share * ((nup + ndn) / configs.RHO_KF1) ** (1.0 / 3.0)
    sysd, rund = abi.make_system(par), abi.make_run(configs.run_params(4, 0.001))
    orc = oracle.Oracle(sysd, rund)
    with capi.Context(sysd, rund) as ctx:
        x = ctx.info.el * (np.random.default_rng(nup).random((3, nup + ndn, 3)) - 0.5)
        got, ref = ctx.getphi(x), [orc.getphi(xw) for xw in x]
    for w in range(3):
        for k in ("u", "du", "d2u", "v"):
            a, b = np.asarray(got[k][w], float), np.asarray(ref[w][k], float)
            assert np.max(np.abs(a - b)) < 1e-10 * max(float(np.max(np.abs(b))), 1.0), (k, w)
