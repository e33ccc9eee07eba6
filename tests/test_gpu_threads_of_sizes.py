"""Contexts of different sizes on their own host threads at once: sweeps, operators,
adjoint gradients, shell derivatives and inverses of each give the bits that they
give alone, and no launch is refused (the kernels' shared-memory limits are the
process's).
"""
import threading

import numpy as np
import pytest

from dmcbcs_project_gb300 import abi, capi, configs

pytestmark = pytest.mark.gpu
SIZES = [(5, 5, 3), (33, 33, 7), (60, 60, 9)]


def calls(nup, ndn, norb, passes):
    out, rng = [], np.random.default_rng(nup)
    with capi.Context(abi.make_system(configs.system_params(nup, ndn, norb)), abi.make_run(configs.run_params(8, 0.001))) as ctx:
        ctx.init_walkers()
        ctx.initial_eval()
        ctx.set_operators(50, 4, 4)
        x, a = ctx.walkers()["x"], rng.normal(size=(2, nup + 3, nup + 3))
        for _ in range(passes):
            ctx.zero_operators()
            ctx.add_operators()
            ctx.sm_sweeps(1, 1)
            out.append([ctx.walkers()["x"], ctx.operators(0, raw=True)[0], ctx.operators(3, raw=True)[0], *ctx.param_grad(x),
                        ctx.getderbcs(x), ctx.matinv(a)[0]])
    return out


def test_threads_of_different_sizes():
    alone = [calls(*s, 12) for s in SIZES]
    together, errors = [None] * len(SIZES), []

    def run(k):
        try:
            together[k] = calls(*SIZES[k], 12)
        except Exception as e:   # reported below, on the test's own thread
            errors.append(e)

    threads = [threading.Thread(target=run, args=(k,)) for k in range(len(SIZES))]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert not errors, errors
    for a, b in zip(alone, together):
        assert all(np.array_equal(u, v) for p, q in zip(a, b) for u, v in zip(p, q))
