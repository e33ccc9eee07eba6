"""The sweeps' launch variants (four or two warps per walker, the cos/sin table
on chip or in global memory) give the same bits: a population of copies of the
same walkers, large enough for another variant, against the walkers alone.  On
152 SMs 7/7 takes two warps from 1217 walkers, 66/66 the global table from 457;
33/33 and 17/16 (entries and pairs that no warp count divides) sit between.
"""
import numpy as np
import pytest

from dmcbcs_project_gb300 import abi, capi, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nup,ndn,norb,copies", [(1, 1, 1, 200), (7, 7, 5, 160), (17, 16, 7, 130), (33, 33, 7, 90), (66, 66, 7, 45)])
def test_variants_give_the_same_bits(nup, ndn, norb, copies):
    few, out = 16, []
    sysd = abi.make_system(configs.system_params(nup, ndn, norb))
    with capi.Context(sysd, abi.make_run(configs.run_params(few, 0.001)), precision="mixed") as ctx:
        ctx.init_walkers()
        ctx.initial_eval()
        start = {k: np.array(v) for k, v in ctx.walkers().items() if np.ndim(v)}
    for n in (few, few * copies):
        many = {k: np.concatenate([v] * (n // few)) for k, v in start.items()}
        with capi.Context(sysd, abi.make_run(configs.run_params(n, 0.001)), precision="mixed") as ctx:
            ctx.put_walkers(dict(many, n=n))
            accepted, moves = ctx.sm_sweeps(3, 2)
            got = ctx.walkers()
            out.append((accepted / moves, {k: got[k] for k in ("x", "irn", "psil", "dpsi", "is_")}, ctx.sm_inverse(n)))
    assert out[0][0] == out[1][0] and 0.0 < out[0][0] < 1.0
    for k, v in out[1][1].items():
        assert np.array_equal(v, np.concatenate([out[0][1][k]] * copies)), k
    assert np.array_equal(out[1][2], np.concatenate([out[0][2]] * copies))
