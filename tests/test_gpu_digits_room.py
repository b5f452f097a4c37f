"""Applies and adjoints whose digits find no room, or whose inputs are outside the fixed-point kernel's range, run
the kernel that reads the FP64 blocks: for all of the call, for single levels (the inputs' digits fit, an
operator's do not) and for one tree of a batch.

Both kernels round like FP64 or better: 2e-14 relative, as against the oracle.  In the norm-tiered modes the other
tiers stay as they are, and a rounding may move no item across a tier: the same bound."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TERMS = [(1.3, 2.0, (0.1, -0.2, 0.3), (1, 0, 0)), (0.7, 25.0, (-0.4, 0.1, 0.0), (0, 2, 1))]
ROOMS = [0, 1 << 16, 1 << 20, 1 << 22, 1 << 24, 1 << 26]


def mra_with_room(engine, monkeypatch, order, room):
    if room is not None:
        monkeypatch.setenv("MW_DIGITS_ROOM", str(room))
    m = engine.MultiResolutionAnalysis(order)
    monkeypatch.delenv("MW_DIGITS_ROOM", raising=False)
    return m


@pytest.mark.parametrize("screening", ["gpu", "host"])
@pytest.mark.parametrize("precision", ["fp64", "mixed", "mixed-near64", "mixed-fp32", "df"])
@pytest.mark.parametrize("order", [3, 7, 9])
def test_applies_at_every_room(engine, monkeypatch, order, precision, screening):
    prec = 1e-4

    def run(room):
        mra = mra_with_room(engine, monkeypatch, order, room)
        mra.set_screening(screening)
        f = engine.project(prec, engine.FunctionTree(mra), TERMS)
        Hs = [engine.HelmholtzOperator(mra, 1.0 + i, prec) for i in range(2)]
        outs = [engine.FunctionTree(mra) for _ in Hs]
        st = engine.apply_batch([prec] * 2, outs, Hs, [f, f], precision=precision)
        return st, [o.download()[:2] for o in outs]

    st, ref = run(None)
    assert st["items_fp64"] + st["items_df"] > 0
    for room in ROOMS if screening == "gpu" else ROOMS[::2]:
        s, got = run(room)
        assert all(s[k] == st[k] for k in ("items", "items_fp64", "items_df", "items_tf32"))
        for (k1, c1), (k2, c2) in zip(got, ref):
            assert np.array_equal(k1, k2) and np.linalg.norm(c1 - c2) <= 2e-14 * np.linalg.norm(c2), room


@pytest.mark.parametrize("order", [4, 8])
def test_adjoints_at_every_room(engine, monkeypatch, order):
    prec = 1e-4

    def run(room, scale=1.0):
        mra = mra_with_room(engine, monkeypatch, order, room)
        f = engine.project(prec, engine.FunctionTree(mra), TERMS)
        k, c, _ = f.download()
        y = engine.FunctionTree(mra).upload(k, c * scale)
        out = engine.FunctionTree(mra)
        engine.apply_adjoint(prec, out, engine.PoissonOperator(mra, prec), f, y)
        return out.download()[1]

    ref = run(None)
    for room in ROOMS:
        assert np.linalg.norm(run(room) - ref) <= 2e-14 * np.linalg.norm(ref), room
    # a seed too large for the fixed-point kernel; a power of two scales every number exactly
    big = run(None, 2.0 ** 505)
    assert np.linalg.norm(big / 2.0 ** 505 - ref) <= 2e-14 * np.linalg.norm(ref)


@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_adjoint_of_a_seed_that_is_not_finite(engine, value):
    mra = engine.MultiResolutionAnalysis(5)
    f = engine.project(1e-3, engine.FunctionTree(mra), TERMS)
    k, c, _ = f.download()
    c[0, 0] = value
    y, out = engine.FunctionTree(mra).upload(k, c), engine.FunctionTree(mra)
    engine.apply_adjoint(1e-3, out, engine.PoissonOperator(mra, 1e-3), f, y)
    assert not np.isfinite(out.download()[1]).all()


@pytest.mark.parametrize("precision", ["mixed", "mixed-near64", "df"])
@pytest.mark.parametrize("value", [np.nan, np.inf, 1e200])
def test_reduced_modes_with_an_input_outside_the_range(engine, precision, value):
    # the root scale's items of a relative apply are the FP64 tier's in every mode
    prec = 1e-3
    mra = engine.MultiResolutionAnalysis(6)
    f = engine.project(prec, engine.FunctionTree(mra), TERMS)
    k, c, _ = f.download()
    c[0, 0] = value
    bad = engine.FunctionTree(mra).upload(k, c)
    H = engine.HelmholtzOperator(mra, 1.0, prec)
    outs = [engine.FunctionTree(mra) for _ in range(2)]
    engine.apply_batch([prec] * 2, outs, [H, H], [bad, f], max_iter=0, precision=precision)
    v = outs[0].download()[1]
    assert np.abs(v).max() > 1e190 if np.isfinite(value) else not np.isfinite(v).all()
    one = engine.FunctionTree(mra)
    engine.apply(prec, one, H, f, max_iter=0, precision=precision)
    (k1, c1, _), (k2, c2, _) = outs[1].download(), one.download()
    assert np.array_equal(k1, k2) and np.linalg.norm(c1 - c2) <= 2e-14 * np.linalg.norm(c2)
