"""GPU: the decisions of a trust-region step that csrc/fa_solve.cu takes from parallel sums with an error bound
and, where the bound does not decide, from the ordered sums: at and around every threshold the answers are
those of the ordered sums (the device's own statement, and the oracle's subproblem, bit for bit)."""
import numpy as np
import pytest

import fa_b200 as fa
import oracle_py as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    ok, msg = fa.gpu_support()
    assert ok, msg
    return fa.Context()


def _band(rng, nD, n_dim):
    P = nD * n_dim
    J = np.zeros((4 * P, P))
    for i in range(nD):
        rows = slice(4 * i * n_dim, 4 * (i + 1) * n_dim)
        J[rows, i * n_dim:(i + 1) * n_dim] = rng.normal(size=(4 * n_dim, n_dim))
        if i + 1 < nD:
            J[rows, (i + 1) * n_dim:(i + 2) * n_dim] = rng.normal(size=(4 * n_dim, n_dim))
    H = J.T @ J
    blk = np.arange(P) // n_dim
    H[np.abs(blk[:, None] - blk[None, :]) > 1] = 0.0
    return H


SIZES = [(1, 2), (2, 3), (10, 2), (32, 3), (86, 3), (200, 2)]  # fewer parameters than a warp, than the block, more


@pytest.mark.parametrize("nD,n_dim", SIZES)
def test_ratio_at_its_thresholds(ctx, nD, n_dim):
    rng = np.random.default_rng(nD)
    H, g = _band(rng, nD, n_dim), rng.normal(size=nD * n_dim) * 10
    eps = np.finfo(np.float64).eps
    for p in (-np.linalg.solve(H, g), -g * 1e-3, rng.normal(size=g.size), np.zeros_like(g), g * 1e-160):
        pred, _, _ = fa.test_ratio(ctx, nD, n_dim, H, g, p, [1.0])
        near = 1.0 + np.concatenate([np.arange(-40, 41) * eps, [-1e-6, -1e-9, -1e-11, -1e-13, 1e-13, 1e-11, 1e-9, 1e-6]])
        meas = np.concatenate([k * abs(pred) * near for k in (0.0, 0.25, 0.75, 1.0, 1 / eps, -0.25, -1 / eps)] +
                              [[0.0, -0.0, 5e-324, -5e-324, 1e-250, 1e250, -1e250, np.inf, -np.inf, np.nan]])
        _, taken, ordered = fa.test_ratio(ctx, nD, n_dim, H, g, p, meas)
        assert np.array_equal(taken, ordered)
        if np.isfinite(pred) and abs(pred) > 1e-100:  # every answer is met
            assert {1, 2, 8, 10, 12} <= set(taken.tolist())


@pytest.mark.parametrize("bad", [np.nan, np.inf, 1e300])
def test_ratio_of_sums_that_are_not_finite(ctx, bad):
    rng = np.random.default_rng(1)
    H, g = _band(rng, 9, 3), rng.normal(size=27)
    p = rng.normal(size=27)
    p[13] = bad
    _, taken, ordered = fa.test_ratio(ctx, 9, 3, H, g, p, [0.0, 1.0, -1.0, 1e300, np.nan])
    assert np.array_equal(taken, ordered)


@pytest.mark.parametrize("nD,n_dim", SIZES)
def test_subproblem_at_the_length_of_the_newton_step(ctx, nD, n_dim):
    rng = np.random.default_rng(100 + nD)
    H, g = _band(rng, nD, n_dim), rng.normal(size=nD * n_dim) * 10
    newton, inside = O.tr_subproblem(H, g, 1e6)
    assert not inside
    length = 0.0
    for v in newton:  # the ordered norm
        length += v * v
    length = np.sqrt(length)
    for k in (-3, -2, -1, 0, 1, 2, 3, 1000, -1000):
        radius = length * (1.0 + k * np.finfo(np.float64).eps)
        p_dev, b_dev = fa.test_tr_subproblem(ctx, nD, n_dim, H, g, radius)
        p_cpu, b_cpu = O.tr_subproblem(H, g, radius)
        assert b_dev == b_cpu and np.array_equal(p_dev, p_cpu), k


@pytest.mark.parametrize("nD,n_dim", SIZES)
def test_subproblem_without_a_factor_and_without_a_gradient(ctx, nD, n_dim):
    rng = np.random.default_rng(200 + nD)
    H, g = _band(rng, nD, n_dim), rng.normal(size=nD * n_dim) * 10
    flat = H.copy()
    flat[-1, :] = flat[:, -1] = 0.0  # singular: no factor of H itself
    for M, v in ((flat, g), (-H, g), (H, np.zeros_like(g))):
        for radius in (0.5, 40.0):
            p_dev, b_dev = fa.test_tr_subproblem(ctx, nD, n_dim, M, v, radius)
            p_cpu, b_cpu = O.tr_subproblem(M, v, radius)
            assert b_dev == b_cpu and np.array_equal(p_dev, p_cpu)
