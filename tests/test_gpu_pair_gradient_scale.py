"""The drift of a pair function whose k = 0 amplitude is far larger than the others
(the gradient does not contain it), in the symmetric form (seven shells) and the
octant form (nine), against the oracle.  One pair, no beta function: the drift is
grad phi / phi, so its error is theirs.  Tolerance: the kernel's 2^-57 of the
amplitudes' sums (of phi's, and of the gradient's without k = 0) is far inside the
oracle's (nk + 30) 2^-52 of them (FP64 sums of nk terms with arguments k.r below 30);
at these positions phi and the gradient's largest component are above a hundredth
of those sums, so 200 (nk + 30) 2^-52 relative to it.
"""
import numpy as np
import pytest

import oracle
from dmcbcs_project_gb300 import abi, capi, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("small", [1.0, 1.0e-6, 1.0e-12, 1.0e-25])
@pytest.mark.parametrize("norb", [2, 7, 9])
def test_a_large_constant_amplitude(norb, small):
    par = configs.system_params(1, 1, norb)
    par["bfact"] = 0.0
    par["vorb"] = [0.7] + [small * v for v in par["vorb"][1:]]
    sysd, rund = abi.make_system(par), abi.make_run(configs.run_params(4, 0.001))
    orc = oracle.Oracle(sysd, rund)
    with capi.Context(sysd, rund) as ctx:
        x = ctx.info.el * (np.random.default_rng(norb + 25).random((8, 2, 3)) - 0.5)
        got, ref, nk = ctx.bcs(x), orc.bcs(x), ctx.info.nk
    assert np.array_equal(got["is_"], ref["is_"])
    assert np.max(np.abs(got["phil"] - ref["phil"])) < 100 * (nk + 30) * 2.0 ** -52
    for w in range(8):
        assert np.max(np.abs(got["dphi"][w] - ref["dphi"][w])) < 200 * (nk + 30) * 2.0 ** -52 * np.max(np.abs(ref["dphi"][w]))
