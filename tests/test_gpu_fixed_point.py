"""The FP64 tier's fixed-point kernel (csrc/mw_apply_fx.cu) at every order it is compiled for: the row and
column tiles of K = 4..8 (one row tile, 2K <= 16) and of K = 9, 10 (a remainder of 2 and 4 rows, columns and
contraction indices), odd K (a Z pair that straddles the halves), the root scale (no exclusion) and finer
scales (exclusion), rows of one and of several items.

Tolerance: a pass is within 2^-57 of row 1-norm x column maximum, six to seven bits above the values
themselves, and FP64's own rounding in the oracle is 2^-53 per operation with sums of a few hundred items:
2e-14 relative covers both.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TERMS = [(1.3, 2.0, (0.1, -0.2, 0.3), (1, 0, 0)), (0.7, 5.0, (-0.4, 0.1, 0.0), (0, 2, 1)),
         (0.2, 11.0, (0.5, 0.4, -0.3), (0, 0, 0))]


def rel_l2(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("basis", ["interpolating", "legendre"])
@pytest.mark.parametrize("order", range(3, 10))
def test_apply_and_adjoint_against_the_oracle(engine, oracle, order, basis):
    prec = 1e-3
    mra, omra = engine.MultiResolutionAnalysis(order, basis=basis), oracle.MRA(order, basis=basis)
    of = oracle.project_gauss(prec, oracle.Tree(omra), TERMS)
    k, c, _ = of.export()
    f = engine.FunctionTree(mra).upload(k, c)
    P = engine.PoissonOperator(mra, prec)
    V, oV = engine.FunctionTree(mra), oracle.Tree(omra)
    st = engine.apply(prec, V, P, f)
    oracle.apply(prec, oV, oracle.poisson(omra, prec), of)
    k1, c1, _ = V.download()
    k2, c2, _ = oV.export()
    assert st["items_fp64"] == st["items"] and st["rows_fp64"] < st["items_fp64"]
    assert np.array_equal(k1, k2) and rel_l2(c1, c2) <= 2e-14
    # the adjoint takes the same kernel with the roles of output and input swapped
    A, AT = engine.FunctionTree(mra), engine.FunctionTree(mra)
    engine.copy_grid(A, f)
    engine.apply_fixed(prec, A, P, f, abs_prec=True)
    engine.apply_adjoint(prec, AT, P, f, f)
    lhs, rhs = engine.dot(f, A), engine.dot(AT, f)
    assert abs(lhs - rhs) <= 1e-13 * abs(lhs)


@pytest.mark.parametrize("order,power", [(5, 200), (5, -200), (8, 200), (9, -200)])
def test_scaling_by_a_power_of_two_is_exact(engine, order, power):
    prec = 1e-3
    mra = engine.MultiResolutionAnalysis(order)
    f = engine.project(prec, engine.FunctionTree(mra), TERMS)
    k, c, _ = f.download()
    g = engine.FunctionTree(mra).upload(k, c * 2.0 ** power)
    P = engine.PoissonOperator(mra, prec)
    a, b = engine.FunctionTree(mra), engine.FunctionTree(mra)
    engine.apply(prec, a, P, f, max_iter=0)
    engine.apply(prec, b, P, g, max_iter=0)
    assert np.array_equal(a.download()[1] * 2.0 ** power, b.download()[1])


@pytest.mark.parametrize("order", [4, 9])
@pytest.mark.parametrize("value", [np.nan, np.inf, 1e200])
def test_values_outside_the_kernels_range_take_the_fp64_kernel(engine, order, value):
    prec = 1e-3
    mra = engine.MultiResolutionAnalysis(order)
    f = engine.project(prec, engine.FunctionTree(mra), TERMS)
    k, c, _ = f.download()
    c[0, 0] = value
    g = engine.FunctionTree(mra).upload(k, c)
    V = engine.FunctionTree(mra)
    engine.apply(prec, V, engine.PoissonOperator(mra, prec), g, max_iter=0)
    v = V.download()[1]
    assert not np.isfinite(v).all() if not np.isfinite(value) else np.abs(v).max() > 1e190


@pytest.mark.parametrize("precision", ["fp64", "df"])
def test_batch_of_more_operators_and_trees_than_one_launch_takes(engine, precision):
    # 66 trees and operators over at most four groups: more than the 16 that one launch of the digit kernels
    # takes.  The items of a node are the same as alone, only grouped otherwise: FP64 rounding of sums.
    prec, n = 1e-2, 66
    mra = engine.MultiResolutionAnalysis(3)
    fs = [engine.project(prec, engine.FunctionTree(mra), [(1.0, 2.0 + 0.1 * i, (0.02 * i - 0.5, 0.1, -0.2), (0, 0, 0))])
          for i in range(n)]
    Hs = [engine.HelmholtzOperator(mra, 0.5 + 0.02 * i, prec) for i in range(n)]
    many = [engine.FunctionTree(mra) for _ in range(n)]
    st = engine.apply_batch([prec] * n, many, Hs, fs, precision=precision)
    # "df" leaves the root scale's items, among others, to the FP64 tier
    assert st["items_df"] + st["items_fp64"] == st["items"] and (st["items_df"] > 0) == (precision == "df")
    for f, H, v in zip(fs, Hs, many):
        one = engine.FunctionTree(mra)
        engine.apply(prec, one, H, f, precision=precision)
        (k1, c1, _), (k2, c2, _) = v.download(), one.download()
        assert np.array_equal(k1, k2) and rel_l2(c1, c2) <= 2e-14


def test_transforms_of_more_pairs_than_one_slice(engine):
    # the two-scale transforms after an FP64 apply take 512 parents of a scale at a time: 320 trees over four
    # groups with eight parents at each of several scales.  Against each apply alone, as above.
    prec, n = 1e-2, 320
    mra = engine.MultiResolutionAnalysis(3)
    H = engine.HelmholtzOperator(mra, 1.0, prec)
    fs = [engine.project(prec, engine.FunctionTree(mra), [(1.0, 2.0 + 0.01 * i, (0.005 * i - 0.5, 0.1, -0.2), (0, 0, 0))])
          for i in range(n)]
    many = [engine.FunctionTree(mra) for _ in range(n)]
    engine.apply_batch([prec] * n, many, [H] * n, fs)
    finest = [np.bincount(v.download()[0][:, 0] + 32).max() // 8 for v in many[:n // 4]]
    assert sum(finest) > 512
    for f, v in list(zip(fs, many))[::13]:
        one = engine.FunctionTree(mra)
        engine.apply(prec, one, H, f)
        (k1, c1, l1), (k2, c2, l2) = v.download(), one.download()
        assert np.array_equal(k1, k2) and np.array_equal(l1, l2) and rel_l2(c1, c2) <= 2e-14
        # the norms that come with the blocks
        assert abs(v.norm() - one.norm()) <= 2e-14 * one.norm()
