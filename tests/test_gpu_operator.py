"""Operator blocks (csrc/mw_opbuild.cu) against the oracle's at the lowest, a middle and the highest order: the
translations whose blocks the band walk keeps (l < 3) and those computed again, wide kernels (one Legendre table
for all) and narrow ones, moments of negative translations taken from their mirror images.

Tolerance: as for the samples in test_gpu_parity.py, 1e-12 of the (term, scale)'s block NS(0).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [3, 6, 9])
def test_blocks_of_all_kinds_match_the_oracle(engine, oracle, order):
    prec = 1e-4
    mra, omra = engine.MultiResolutionAnalysis(order), oracle.MRA(order)
    P, Q = engine.HelmholtzOperator(mra, 0.8, prec), oracle.helmholtz(omra, 0.8, prec)
    computed_again = 0
    for t in range(0, P.nterms, 4):
        for n in (-5, -3, 0, 5):
            L = P.band(t, n)
            assert L == Q.band(t, n)
            if L < 0:
                continue
            scale = max(np.abs(Q.block(t, n, 0)[0]).max(), 1e-300)
            for l in {0, 1, 2, min(L, 3), min(L, 4), L} if L >= 2 else range(L + 1):
                computed_again += l >= 3
                for sl in {l, -l}:
                    b1, n1 = P.block(t, n, sl)
                    b2, n2 = Q.block(t, n, sl)
                    assert np.abs(b1 - b2).max() <= 1e-12 * scale
                    assert np.allclose(n1, n2, rtol=1e-12, atol=1e-12 * scale)
    assert computed_again > 0
