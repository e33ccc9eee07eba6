"""A coordinate that is not finite shows in the Jastrow-only evaluation: the
walker's flag, its Laplacian, and that component of the gradient of the particle
and of every opposite-spin partner, with the pairs taken one by one (7/7, and a
spline that reaches L/2) and from the list (33/33); the sums over distances keep
the reference's clamp (coshpot.f90:170) and stay finite.  The walkers beside it
are the same bits as without it.
"""
import numpy as np
import pytest

from dmcbcs_project_gb300 import abi, capi, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("nup,ndn,spline", [(7, 7, False), (33, 33, False), (33, 33, True)])
def test_a_coordinate_that_is_not_finite_is_seen(nup, ndn, spline, value):
    sysd = abi.make_system(configs.system_params(nup, ndn, 7))
    with capi.Context(sysd, abi.make_run(configs.run_params(4, 0.001))) as ctx:
        if spline:
            ctx.set_jastrow_spline(np.random.default_rng(0).uniform(-0.3, 0.3, 16))
        x = ctx.info.el * (np.random.default_rng(1).random((3, nup + ndn, 3)) - 0.5)
        good = ctx.getphi(x)
        x[1, 2, 1] = value              # an up particle
        x[2, nup + 4, 0] = value        # a down particle
        got, flags = ctx.getphi(x), ctx.walker_status(3)
    assert list(flags) == [0, abi.DMC_STATUS_NONFINITE, abi.DMC_STATUS_NONFINITE]
    for k in ("u", "du", "d2u", "v"):
        assert np.array_equal(got[k][0], good[k][0]), k
    assert np.isfinite(got["u"]).all() and np.isfinite(got["v"]).all() and not np.isfinite(got["d2u"][1:]).any()
    want = np.zeros((3, nup + ndn, 3), bool)
    want[1, 2, 1] = want[1, nup:, 1] = True
    want[2, nup + 4, 0] = want[2, :nup, 0] = True
    assert np.array_equal(~np.isfinite(got["du"]), want)
