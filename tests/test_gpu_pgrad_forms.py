"""The two forms of the adjoint gradients' shell derivatives against each other:
an eighth shell of amplitude zero takes a system from the symmetric form (seven
shells, |n|^2 <= 6) to the sums over k vectors without changing the
wavefunction, so every other parameter's gradient has to stay.  Smallest
systems, fewer pairs than a warp, a few more than a CTA's threads, unpaired
columns, particles outside the box, coincident coordinates, a pair at distance
zero.  Tolerance, relative to a walker's largest gradient: 1e-10, or 16 nd
cond(S) 2^-52 where that is larger (two products with the inverse each way).
"""
import numpy as np
import pytest

from dmcbcs_project_gb300 import abi, capi, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nup,ndn,spline", [(1, 1, True), (2, 1, False), (5, 5, True), (16, 16, True), (17, 16, True), (33, 30, False),
                                            (33, 33, True)])
def test_the_shell_forms_agree(nup, ndn, spline):
    params = configs.system_params(nup, ndn, 7)
    rng = np.random.default_rng(nup + ndn)
    n, got = nup + ndn, []
    el = (n / params["rho"]) ** (1.0 / 3.0)
    xu = el * (rng.random((4, nup, 3)) - 0.5)
    x = np.concatenate([xu, xu[:, :ndn] + rng.normal(0.0, 0.8, (4, ndn, 3))], axis=1)
    x[1] += el * rng.integers(-4, 5, (n, 3))
    x[2, nup] = x[2, 0] + [0.0, 0.1, 0.0]
    x[3, nup] = x[3, 0]
    knots = rng.uniform(-0.3, 0.3, 16)
    for norb in (7, 8):
        p = dict(params, norb=norb, vorb=(list(params["vorb"]) + [0.0])[:norb])
        with capi.Context(abi.make_system(p), abi.make_run(configs.run_params(4, 0.001))) as ctx:
            if spline:
                ctx.set_jastrow_spline(knots)
            dl, de = ctx.param_grad(x)
            cond = [np.linalg.cond(s.reshape(nup, nup)) for s in ctx.bcs(x[:3], want_inverse=True)["smati"]]
        got.append([np.delete(g, 7, axis=1) if norb == 8 else g for g in (dl, de)])
    for a, b in zip(*got):
        for w in range(3):
            tol = max(1e-10, 16 * nup * cond[w] * 2.0 ** -52)
            assert np.abs(a[w] - b[w]).max() <= tol * max(np.abs(b[w]).max(), 1.0), w
        # the pair at distance zero: the same parameters stay finite
        assert np.array_equal(np.isfinite(a[3]), np.isfinite(b[3]))
