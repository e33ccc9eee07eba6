"""Populations that take one warp per walker in the sweeps (small systems beyond
one round of the other forms, on 152 SMs) give the bits of a few walkers, which
take four: one particle a species, partly filled and full warps of entries, an
unpaired particle, and a count that leaves a CTA with one walker.
"""
import numpy as np
import pytest

from dmcbcs_project_gb300 import abi, capi, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nup,ndn,norb,n", [(1, 1, 1, 2721), (5, 5, 3, 2721), (19, 18, 5, 4993), (26, 25, 7, 4098), (32, 32, 4, 2451)])
def test_one_warp_gives_the_same_bits(nup, ndn, norb, n):
    few, out = 16, []
    sysd = abi.make_system(configs.system_params(nup, ndn, norb))
    with capi.Context(sysd, abi.make_run(configs.run_params(few, 0.001)), precision="mixed") as ctx:
        ctx.init_walkers()
        ctx.initial_eval()
        start = {k: np.array(v) for k, v in ctx.walkers().items() if np.ndim(v)}
    for k in (few, n):
        pick = np.arange(k) % few
        with capi.Context(sysd, abi.make_run(configs.run_params(k, 0.001)), precision="mixed") as ctx:
            ctx.put_walkers(dict({f: v[pick] for f, v in start.items()}, n=k))
            ctx.sm_sweeps(3, 2)
            got = ctx.walkers()
            out.append(({f: got[f] for f in ("x", "irn", "psil", "dpsi", "is_")}, ctx.sm_inverse(k)))
    pick = np.arange(n) % few
    for f, v in out[1][0].items():
        assert np.array_equal(v, out[0][0][f][pick]), f
    assert np.array_equal(out[1][1], out[0][1][pick])
    assert not np.array_equal(out[0][0]["x"], start["x"])
