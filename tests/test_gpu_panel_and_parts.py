"""The inverse at the sizes where the panel's rows, warps and widths change
(32, 64, 96 rows; panels of 6 and 8 columns with remainders), with pivots in
every warp, equal candidates and singular matrices; and single-particle moves
of more walkers than one part holds.

Tolerances.  Inverse: n cond(A) 2^-52 of the largest entry, the forward error
of an FP64 elimination with partial pivoting, times 8 for its growth, for both
the kernel's and numpy's; log|det| likewise, with the sum of the columns'
logarithms on top.  Moves: a part's walkers do not see each other, so
the ratios are the same bits.
"""
import numpy as np
import pytest

from dmcbcs_project_gb300 import abi, capi, configs

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -52


@pytest.fixture(scope="module")
def ctx():
    with capi.Context(abi.make_system(configs.system_params(33, 33, 7)), abi.make_run(configs.run_params(4, 0.001))) as c:
        yield c


@pytest.mark.parametrize("n", [1, 5, 6, 7, 31, 32, 33, 37, 63, 64, 65, 66, 95, 96, 97, 104, 112])
def test_inverse_at_the_panel_edges(ctx, n):
    rng = np.random.default_rng(n)
    a = rng.normal(size=(4, n, n))
    scale = np.ones((4, n))
    scale[1] = 2.0 ** rng.integers(-60, 60, n)   # columns of any size: the same pivots, exactly scaled
    a[2] = np.eye(n)[rng.permutation(n)] * rng.choice([-1.0, 1.0], n)   # one candidate a column
    a[3] = np.where(rng.random((n, n)) < 0.5, -1.0, 1.0) + 2.0 * n * np.eye(n)[rng.permutation(n)]   # equal candidates
    inv, logdet, sign = ctx.matinv(a * scale[:, None, :])
    inv, logdet = inv * scale[:, :, None], logdet - np.log(scale).sum(axis=1)
    for w in range(4):
        s, ld = np.linalg.slogdet(a[w])
        ref, tol = np.linalg.inv(a[w]), 8 * n * np.linalg.cond(a[w]) * EPS
        assert np.max(np.abs(inv[w] - ref)) < 2 * tol * np.abs(ref).max(), w
        assert abs(logdet[w] - ld) < 2 * tol * max(1.0, abs(ld)) + 64 * n * EPS * 60 and sign[w] == s, w


@pytest.mark.parametrize("n,col", [(6, 5), (33, 32), (33, 7), (64, 40), (96, 95), (112, 60)])
def test_a_singular_matrix_is_seen_by_every_panel_warp(ctx, n, col):
    a = np.random.default_rng(n).normal(size=(2, n, n))
    a[0, :, col] = 0.0
    inv, logdet, sign = ctx.matinv(a)
    assert logdet[0] < -1.0e10 and np.isfinite(inv[1]).all()
    assert abs(logdet[1] - np.linalg.slogdet(a[1])[1]) < 8 * n * np.linalg.cond(a[1]) * EPS * max(1.0, abs(logdet[1]))


def test_moves_in_parts_are_the_moves_of_one_part(ctx):
    rng = np.random.default_rng(2)
    few, copies = 450, 21   # 9450 walkers: two parts and a remainder
    x = ctx.info.el * (rng.random((few, 66, 3)) - 0.5)
    inv, d = rng.normal(size=(few, 33 * 33)), rng.normal(0.0, 0.3, (few, 3))
    ip = rng.integers(1, 67, few).astype(np.int32)
    many = [np.concatenate([v] * copies) for v in (x, inv, ip, d)]
    one, whole = ctx.bcsone(x, inv, ip, d), ctx.bcsone(*many)
    assert np.array_equal(whole, np.concatenate([one] * copies))
    one, whole = ctx.getphione(x, ip, d), ctx.getphione(many[0], many[2], many[3])
    assert np.array_equal(whole, np.concatenate([one] * copies))
