"""Layout tuning of systems with one shell, whose mixed layout is smaller than
the FP64 kernel's: with the union region in global memory the mixed kernel fits
two CTAs per SM where the FP64 kernel does not.  The tuner keeps a layout for
both, and every evaluation its values (FP64 parity bar, 1e-10 relative to
max(|ref|, 1), mixed 1e-6).
"""
import numpy as np
import pytest

from dmcbcs_project_gb300 import abi, capi, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nup,ndn,nexdn", [(88, 79, 0), (87, 80, 1), (86, 81, 2), (88, 80, 0), (87, 79, 0)])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_tuner_with_one_shell(nup, ndn, nexdn, prec):
    par = configs.system_params(nup, ndn, 1)
    waves = [[0, 0, 0], [1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0], [0, 0, 1], [0, 0, -1], [1, 1, 0], [1, -1, 0], [-1, 1, 0], [-1, -1, 0],
             [1, 0, 1], [1, 0, -1]]
    par.update(nexup=nup - ndn + nexdn, ikup=waves[:nup - ndn + nexdn], nexdn=nexdn, ikdn=waves[:nexdn])
    with capi.Context(abi.make_system(par), abi.make_run(configs.run_params(16, 0.001)), precision=prec) as ctx:
        ctx.init_walkers()
        ctx.initial_eval()
        x = ctx.walkers()["x"]
        ref = ctx.hpsi(x)
        kind, ms = ctx.tune_layout(1)
        got = ctx.hpsi(x)
    assert kind >= 0 and ms > 0.0
    tol = 1e-10 if prec == "fp64" else 1e-6
    for k in ("psil", "d2psi", "v"):
        assert np.max(np.abs(got[k] - ref[k])) <= tol * max(1.0, np.max(np.abs(ref[k]))), k
