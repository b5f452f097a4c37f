"""Sums of trees for one and for several outputs in one launch (combine_kernel: 1, 4 or 8 outputs per CTA):
the output counts at the edges of those groups, orders from the smallest block to one that is no multiple of
the CTA, inputs missing under leaves at several depths, an output given twice, and coefficients that are not
finite.  The oracle's add has the same order of summation, so a few roundings (1e-14) separate the two."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def trees(oracle, omra, prec):
    out = []
    for a, x, pw in ((1.0, 0.0, (0, 0, 0)), (40.0, 0.6, (1, 0, 0)), (4.0, -1.3, (0, 1, 1)), (150.0, 0.1, (0, 0, 2)), (0.4, 1.0, (2, 0, 0))):
        out.append(oracle.project_gauss(prec, oracle.Tree(omra), [(1.0, a, (x, 0.3 * x, -x), pw)]))
    return out


@pytest.mark.parametrize("order,nout", [(3, 1), (4, 2), (5, 4), (6, 5), (7, 8), (8, 9), (9, 3)])
def test_rotate_against_the_oracle(engine, oracle, order, nout):
    mra, omra = engine.MultiResolutionAnalysis(order), oracle.MRA(order)
    oin = trees(oracle, omra, 1e-3)
    ins = [engine.FunctionTree(mra).upload(*t.export()[:2]) for t in oin]
    U = np.random.default_rng(order).standard_normal((nout, len(ins)))
    U[0, 1] = 0.0
    outs = [engine.FunctionTree(mra) for _ in range(nout)]
    engine.rotate(outs, ins, U)
    for o, row in zip(outs, U):
        ref = oracle.Tree(omra)
        oracle.add(1e-3, ref, row, oin)
        k1, c1, _ = o.download()
        k2, c2, _ = ref.export()
        assert np.array_equal(k1, k2)
        assert np.linalg.norm(c1 - c2) <= 1e-14 * np.linalg.norm(c2)
        s = engine.FunctionTree(mra)
        engine.add(1e-3, s, list(zip(row, ins)))
        assert np.array_equal(s.download()[1], c1)
        assert abs(o.squared_norm() - s.squared_norm()) <= 1e-14 * s.squared_norm()


def test_an_output_given_twice_holds_its_last_row(engine, oracle):
    mra, omra = engine.MultiResolutionAnalysis(4), oracle.MRA(4)
    ins = [engine.FunctionTree(mra).upload(*t.export()[:2]) for t in trees(oracle, omra, 1e-3)[:2]]
    a, b = engine.FunctionTree(mra), engine.FunctionTree(mra)
    U = np.array([[1.0, 2.0], [0.5, -1.0], [3.0, 0.25]])
    engine.rotate([a, b, a], ins, U)
    s = engine.FunctionTree(mra)
    engine.add(1e-3, s, [(3.0, ins[0]), (0.25, ins[1])])
    assert np.array_equal(a.download()[1], s.download()[1])


@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_coefficients_that_are_not_finite_reach_every_value(engine, oracle, value):
    mra, omra = engine.MultiResolutionAnalysis(4), oracle.MRA(4)
    ins = [engine.FunctionTree(mra).upload(*t.export()[:2]) for t in trees(oracle, omra, 1e-3)[:2]]
    s = engine.FunctionTree(mra)
    engine.add(1e-3, s, [(1.0, ins[0]), (value, ins[1])])
    c = s.download()[1]
    # infinity times a zero coefficient is NaN, times any other infinite
    assert not np.isfinite(c).any()


@pytest.mark.parametrize("other", [4, 6])
def test_rotate_refuses_outputs_of_another_context(engine, oracle, other):
    # one launch writes all outputs: of another context they have a stream, and here an order, of their own
    mra, omra = engine.MultiResolutionAnalysis(6), oracle.MRA(6)
    ins = [engine.FunctionTree(mra).upload(*t.export()[:2]) for t in trees(oracle, omra, 1e-3)[:2]]
    a, b = engine.FunctionTree(mra), engine.FunctionTree(engine.MultiResolutionAnalysis(other))
    for outs in ([a, b], [b, a]):
        with pytest.raises(engine.MWError, match="different contexts"):
            engine.rotate(outs, ins, np.eye(2))


@pytest.mark.parametrize("n,nout", [(16385, 1), (30001, 1), (16384, 2)])
def test_sums_of_more_trees_than_shared_memory_has_coefficients_for(engine, oracle, n, nout):
    # the same few trees many times over; against their sum with the added coefficients, whose rounding differs by
    # at most n roundings of the sum of absolute values
    mra, omra = engine.MultiResolutionAnalysis(3), oracle.MRA(3)
    ins = [engine.FunctionTree(mra).upload(*t.export()[:2]) for t in trees(oracle, omra, 1e-1)[:3]]
    U = np.random.default_rng(n).standard_normal((nout, n))
    outs = [engine.FunctionTree(mra) for _ in range(nout)]
    many = [ins[k % 3] for k in range(n)]
    if nout == 1:
        engine.add(1e-1, outs[0], list(zip(U[0], many)))
    else:
        engine.rotate(outs, many, U)
    for o, row in zip(outs, U):
        s = engine.FunctionTree(mra)
        engine.add(1e-1, s, [(float(np.sum(row[k::3])), ins[k]) for k in range(3)])
        d = o.download()[1] - s.download()[1]
        assert np.linalg.norm(d) <= n * 2.3e-16 * np.abs(row).sum() * max(t.norm() for t in ins)
