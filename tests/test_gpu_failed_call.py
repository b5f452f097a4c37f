"""A call that fails half-way leaves nothing running on any stream of its context: what it read and wrote can be
freed and reused, and the context goes on working."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_apply_that_fails_after_its_uploads_started(engine, monkeypatch, precision):
    # generation tables beyond the screening's limit: every apply screened on the GPU ends with an error, here
    # after its inputs' uploads and conversions went out on their streams
    prec, n = 1e-4, 4
    monkeypatch.setenv("MW_SCREEN_GEN_SLOTS", str(1 << 27))
    mra = engine.MultiResolutionAnalysis(7)
    monkeypatch.delenv("MW_SCREEN_GEN_SLOTS")
    srcs = [engine.project(prec, engine.FunctionTree(mra), [(1.0, 3.0 + i, (0.2 * i, 0.1, -0.3), (0, 0, 0))])
            for i in range(n)]
    host = []
    for f in srcs:
        k, c, _ = f.download()
        host.append((k, engine.pin_host(mra, np.ascontiguousarray(c))))
    for _ in range(5):
        Hs = [engine.HelmholtzOperator(mra, 1.0 + 0.1 * i, prec) for i in range(n)]
        outs, inps = [engine.FunctionTree(mra) for _ in srcs], [engine.FunctionTree(mra) for _ in srcs]
        with pytest.raises(engine.MWError, match="generation tables"):
            engine.apply_batch_host([prec] * n, outs, Hs, inps, host, precision=precision)
        del Hs, inps, outs  # freed at once
    mra.set_screening("host")
    Hs = [engine.HelmholtzOperator(mra, 1.0 + 0.1 * i, prec) for i in range(n)]
    a, b = [engine.FunctionTree(mra) for _ in srcs], [engine.FunctionTree(mra) for _ in srcs]
    engine.apply_batch_host([prec] * n, a, Hs, [engine.FunctionTree(mra) for _ in srcs], host, precision=precision)
    engine.apply_batch([prec] * n, b, Hs, srcs, precision=precision)
    for x, y in zip(a, b):
        (k1, c1, _), (k2, c2, _) = x.download(), y.download()
        assert np.array_equal(k1, k2) and np.array_equal(c1, c2)
    for _, c in host:
        engine.unpin_host(mra, c)
