"""Parameters changed on a live context (shell amplitudes, beta, Jastrow knots)
give the bits of a context made with them, for the smallest tables and ordinary
ones, in the symmetric and the octant form; and the interval cubics made on the
device reproduce the tables: FP64 values against the oracle at the parity bar
(1e-10 relative to max(|ref|, 1)).
"""
import numpy as np
import pytest

import oracle
from dmcbcs_project_gb300 import abi, capi, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ntab", [8, 9, 60, 10000])
@pytest.mark.parametrize("norb", [4, 9])
def test_changed_parameters_are_a_new_context_s(norb, ntab):
    par, rund = configs.system_params(7, 6, norb, ntab=ntab), abi.make_run(configs.run_params(4, 0.001))
    new = dict(par, vorb=[0.9 * v + 0.01 for v in par["vorb"]], bbeta=1.1, dbeta=4.0, bfact=0.8)
    rng = np.random.default_rng(ntab)
    one, two = rng.uniform(-0.3, 0.3, 16), rng.uniform(-0.3, 0.3, 16)
    with capi.Context(abi.make_system(par), rund) as live, capi.Context(abi.make_system(new), rund) as fresh:
        x = live.info.el * (rng.random((6, 13, 3)) - 0.5)
        for spline in (False, True):
            if spline:
                live.set_jastrow_spline(one)
            live.param_grad(x)   # tables of the old parameters
            live.set_vorb(new["vorb"])
            live.set_beta(1.1, 4.0, 0.8)
            if spline:
                live.set_jastrow_spline(two)
                fresh.set_jastrow_spline(two)
            for a, b in zip(live.param_grad(x), fresh.param_grad(x)):
                assert np.array_equal(a, b)
            for call in ("hpsi", "bcs", "getphi"):
                a, b = getattr(live, call)(x), getattr(fresh, call)(x)
                assert all(np.array_equal(a[k], b[k]) for k in a if a[k] is not None), call
            orc = oracle.Oracle(abi.make_system(new), rund)
            if spline:
                orc.set_jastrow_spline(two)
            got, ref = fresh.hpsi(x), orc.hpsi(x)
            for k in ("psil", "v", "dpsi", "d2psi"):
                assert np.max(np.abs(got[k] - ref[k])) < 1e-10 * max(1.0, np.max(np.abs(ref[k]))), k
            live.set_vorb(par["vorb"])
            live.set_beta(par["bbeta"], par["dbeta"], par["bfact"])
