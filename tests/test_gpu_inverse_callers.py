"""The evaluation behind the shell derivatives flags walkers as dmc_bcs does
(regular, two equal rows, a coordinate that is not finite, an up and a down particle on
one point), and the derivatives of the regular ones are their inverse's: the sum of
its up-down block for the first shell, to the rounding of an FP64 sum.
"""
import numpy as np
import pytest

from dmcbcs_project_gb300 import abi, capi, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nup,ndn,norb", [(7, 7, 5), (33, 30, 7), (19, 19, 9)])
def test_shell_derivatives_flag_as_bcs(nup, ndn, norb):
    with capi.Context(abi.make_system(configs.system_params(nup, ndn, norb)), abi.make_run(configs.run_params(4, 0.001))) as ctx:
        x = ctx.info.el * (np.random.default_rng(nup).random((6, nup + ndn, 3)) - 0.5)
        x[1, 1] = x[1, 0]            # two equal rows: singular up to rounding
        x[2, 3, 1] = np.nan
        x[3, nup + 2, 0] = np.inf
        x[4, nup + 1] = x[4, 2]      # an infinite 1/r
        out = ctx.bcs(x, want_inverse=True)
        want = ctx.walker_status(6)
        der = ctx.getderbcs(x)
        got = ctx.walker_status(6)
    assert np.array_equal(got, want)
    assert want[0] == want[5] == 0   # (equal rows cancel to exactly zero, the flag's condition, in six of seven cases)
    assert want[2] == want[3] == want[4] == abi.DMC_STATUS_NONFINITE
    for w in (0, 5):
        block = out["smati"][w].reshape(nup, nup)[:nup, :ndn]   # [i][j] = inverse (j, i)
        assert abs(der[w, 0] - block.sum()) < nup * ndn * 2.0 ** -52 * np.abs(block).sum()
