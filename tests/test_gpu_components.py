"""Component by component: the fixed-point kernel (csrc/mw_apply_fx.cu) must not lose the small components of a block,
the pure wavelet ones of a smooth output above all, which vanish beside the scaling part.

One apply from a single root box to a row of root boxes, near and far, where the output is the plain sum of the items
(the root scale has no excluded path and no screening, a single scale no two-scale transforms).  The reference sums
the same items in double-double arithmetic.  The kernel that reads FP64 blocks runs the same apply on the input
times 2^505 (outside the fixed-point kernel's range; every number is scaled exactly): the fixed-point kernel's error
may be at most twice as large in any component of any node, or two roundings of the component itself.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def two_sum(a, b):
    s = a + b
    t = s - a
    return s, (a - (s - t)) + (b - t)


def split(a):
    c = 134217729.0 * a
    hi = c - (c - a)
    return hi, a - hi


def two_prod(a, b):
    p = a * b
    (ah, al), (bh, bl) = split(a), split(b)
    return p, ((ah * bh - p) + ah * bl + al * bh) + al * bl


def contract(A, hi, lo):
    """sum_k A[r, k] (hi + lo)[k, :] in double-double."""
    s, e = np.zeros((A.shape[0], hi.shape[1])), np.zeros((A.shape[0], hi.shape[1]))
    for k in range(A.shape[1]):
        p, q = two_prod(A[:, k:k + 1], hi[k][None])
        s, d = two_sum(s, p)
        e += d + (q + A[:, k:k + 1] * lo[k][None])
    return two_sum(s, e)


def cube(block, K):
    c = block.reshape(2, 2, 2, K, K, K)  # cz, cy, cx, z, y, x
    return np.ascontiguousarray(c.transpose(0, 3, 1, 4, 2, 5).reshape(2 * K, 2 * K, 2 * K))


def reference(op, key, block, keys, K, scale):
    c, _ = op.terms()
    N = 2 * K
    out = []
    for k in keys:
        s, e = np.zeros((N, N, N)), np.zeros((N, N, N))
        d = [int(k[i]) - int(key[i]) for i in (1, 2, 3)]
        for t in range(op.nterms):
            if op.band(t, scale) < max(abs(v) for v in d):
                continue
            hi, lo = cube(block, K), np.zeros((N, N, N))
            for axis, l in ((2, d[0]), (1, d[1]), (0, d[2])):
                A = op.block(t, scale, l)[0]
                h, g = (np.moveaxis(x, axis, 0).reshape(N, N * N) for x in (hi, lo))
                h, g = contract(A, np.ascontiguousarray(h), np.ascontiguousarray(g))
                hi, lo = (np.moveaxis(x.reshape(N, N, N), 0, axis) for x in (h, g))
            p, q = two_prod(np.full_like(hi, c[t]), hi)
            s, r = two_sum(s, p)
            e += r + (q + c[t] * lo)
        out.append((s, e))
    return out


@pytest.mark.parametrize("order,basis,corner,centre,kind", [
    (3, "interpolating", (0, 0, 0), 0.5, "poisson"), (4, "legendre", (0, 0, 0), 0.4, "helmholtz"),
    (5, "interpolating", (0, 0, 0), 0.5, "poisson"), (6, "interpolating", (0, 0, 0), 0.6, "helmholtz"),
    (7, "interpolating", (0, 0, 0), 0.5, "poisson"), (7, "legendre", (0, 0, 0), 0.3, "poisson"),
    (8, "interpolating", (0, 0, 0), 0.5, "poisson"), (9, "interpolating", (0, 0, 0), 0.5, "poisson"),
    (9, "legendre", (0, 0, 0), 0.4, "helmholtz")])
def test_components_against_double_double(engine, order, basis, corner, centre, kind):
    K, scale, box = order + 1, 0, 1.0
    mra = engine.MultiResolutionAnalysis(order, root_scale=scale, corner=corner, boxes=(2, 1, 3), basis=basis)
    prec = 1e-4
    op = engine.PoissonOperator(mra, prec) if kind == "poisson" else engine.HelmholtzOperator(mra, 2.0, prec)
    f = engine.project(1e3, engine.FunctionTree(mra), [(1.0, 12.0, (centre * box,) * 3, (0, 0, 0))], abs_prec=True)
    keys, coefs, _ = f.download()
    keys, coefs = keys[keys[:, 0] == scale], coefs[keys[:, 0] == scale]  # the roots alone
    assert len(keys) == 6
    src = int(np.argmax(np.linalg.norm(coefs, axis=1)))
    only = np.zeros_like(coefs)
    only[src] = coefs[src]
    got = {}
    for power in (0, 505):
        x, y = engine.FunctionTree(mra).upload(keys, only * 2.0 ** power), engine.FunctionTree(mra)
        engine.apply(prec, y, op, x, max_iter=0)
        k2, c2, _ = y.download()
        assert len(k2) == 6
        got[power] = {tuple(k): cube(c * 2.0 ** -power, K) for k, c in zip(k2, c2)}
    ref = reference(op, keys[src], only[src], keys, K, scale)
    worst = []
    for k, (s, e) in zip(keys, ref):
        for comp in range(8):
            at = tuple(slice(K * b, K * b + K) for b in ((comp >> 2) & 1, (comp >> 1) & 1, comp & 1))
            err = {p: np.linalg.norm((got[p][tuple(k)][at] - s[at]) - e[at]) for p in got}
            size = np.linalg.norm(s[at])
            worst.append((err[0] / (2.0 * err[505] + 2.0 ** -52 * size), tuple(int(v) for v in k), comp, err[0] / size, err[505] / size))
    worst.sort(reverse=True)
    print(order, basis, kind, worst[:3])
    assert worst[0][0] <= 1.0, worst[:4]
