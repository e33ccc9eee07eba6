"""Single-particle moves on both sides of the size from which their positions are
copied to the device (512 KB), with the inverse's rows in one and in several parts
(8 MB of page-locked memory), up and down particles, the symmetric and the general
pair function: a walker's ratio does not depend on the others, so the same bits as
in a small call, which is compared with the oracle (the FP64 bar, 1e-10 relative to
max(|ref|, 1)).
"""
import numpy as np
import pytest

import oracle
from dmcbcs_project_gb300 import abi, capi, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nup,ndn,norb,total", [(1, 1, 2, 60000), (7, 7, 5, 150001), (7, 6, 5, 1500), (33, 33, 7, 900), (33, 33, 9, 300), (66, 66, 7, 400)])
def test_ratios_do_not_depend_on_the_call_s_size(nup, ndn, norb, total):
    few, n = 60, nup + ndn
    sysd, rund = abi.make_system(configs.system_params(nup, ndn, norb)), abi.make_run(configs.run_params(4, 0.001))
    orc = oracle.Oracle(sysd, rund)
    rng = np.random.default_rng(total)
    with capi.Context(sysd, rund) as ctx:
        x = ctx.info.el * (rng.random((few, n, 3)) - 0.5)
        inv, d = rng.normal(size=(few, nup * nup)), rng.normal(0.0, 0.3, (few, 3))
        ip = np.concatenate([[1, n, nup, nup + 1], rng.integers(1, n + 1, few - 4)]).astype(np.int32)
        det, jas = ctx.bcsone(x, inv, ip, d), ctx.getphione(x, ip, d)
        pick = np.arange(total) % few
        for k in (total, 1, total - 1):
            sel = pick[:k]
            assert np.array_equal(ctx.bcsone(x[sel], inv[sel], ip[sel], d[sel]), det[sel])
            assert np.array_equal(ctx.getphione(x[sel], ip[sel], d[sel]), jas[sel])
    for w in range(8):
        i = int(ip[w])
        for got, ref in ((det[w], orc.bcsone(x[w], d[w], i, inv[w])), (jas[w], orc.getphione(x[w], d[w], i))):
            assert abs(got - ref) < 1e-10 * max(abs(ref), 1.0)
