"""Overlaps and norms (csrc/mw_kernels.cu dot_kernel, block_norms) at every order: blocks smaller than one round
of the kernels' threads (K = 4: 448 wavelet coefficients, 64 per component) up to K = 10, remainders of the
unrolled loops, trees that share only part of their nodes.

Tolerance: every partial sum is a sum of at most some 10^5 products, each rounded to 2^-53: 1e-13 of the sum of
the products' magnitudes.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", range(3, 10))
def test_dot_and_norm_of_partly_shared_grids(engine, order):
    mra = engine.MultiResolutionAnalysis(order)
    K3 = (order + 1) ** 3
    f = engine.project(1e-3, engine.FunctionTree(mra), [(1.0, 3.0, (0.4, 0.1, -0.3), (1, 0, 0))])
    g = engine.project(1e-4, engine.FunctionTree(mra), [(0.7, 9.0, (-0.2, 0.3, 0.1), (0, 0, 1)), (1.0, 1.0, (0.1, 0, 0), (0, 0, 0))])
    (kf, cf, _), (kg, cg, _) = f.download(), g.download()
    other = {tuple(k): i for i, k in enumerate(kg)}
    total = size = 0.0
    common = 0
    for k, a in zip(kf, np.asarray(cf).reshape(len(kf), -1)):
        j = other.get(tuple(k))
        if j is None:
            continue
        common += 1
        p = a * np.asarray(cg).reshape(len(kg), -1)[j]
        p = p if k[0] == kf[:, 0].min() else p[K3:]
        total += p.sum()
        size += np.abs(p).sum()
    assert 8 <= common < max(len(kf), len(kg))
    assert abs(engine.dot(f, g) - total) <= 1e-13 * size
    assert engine.dot(f, g) == engine.dot(f, g)
    wavelets = np.asarray(cf).reshape(len(kf), -1).copy()
    wavelets[kf[:, 0] > kf[:, 0].min(), :K3] = 0.0
    n2 = float((wavelets ** 2).sum())
    assert abs(f.norm() ** 2 - n2) <= 1e-13 * n2
