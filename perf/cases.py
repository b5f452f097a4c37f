"""The work that programs on this framework's hot path give it: convolution applies (single and
batched, plain FP64 and norm-tiered, with operators built on the way and with host buffers), the
exchange step, potential and density products, orbital rotations, overlaps and the adjoint apply.

Inputs are orbitals and densities made of Gaussians, projected here in 64 bits (plain torch)
and uploaded, so that they do not depend on the framework's own projection.  Every tree a pass
computes is read back into page-locked host buffers, as a program that keeps its SCF state on the
host does.
"""
import math

import numpy as np
import torch

import mrchem_gb300 as mw

ROOT_SCALE, CORNER, BOXES = -5, -1, 2  # the world [-32, 32]^3 of the reference's test fixture

_MRA = {}  # one context per (order, basis), as in a program


def _mra(case):
    key = (case["order"], case["basis"])
    if key not in _MRA:
        _MRA[key] = mw.MultiResolutionAnalysis(case["order"], basis=case["basis"])
    return _MRA[key]


# ------------------------------------------------------------------ cases

def listed():
    def c(name, kind, order, prec, n, mode="fp64", basis="interpolating"):
        return {"name": name, "kind": kind, "order": order, "prec": prec, "n": n, "mode": mode, "basis": basis}
    return [
        # the size of the reference's Coulomb tests: one charge at order 5, prec 1e-3; the smallest apply
        c("coulomb_k5_fp64", "poisson", 5, 1e-3, 1),
        # one density's Coulomb potential in plain FP64 (4 Gaussians, order 7, prec 1e-5)
        c("poisson_k7_fp64", "poisson", 7, 1e-5, 4),
        # the drop-in precision of the Helmholtz apply: plain FP64 at order 9
        c("helmholtz2_k9_fp64", "helmholtz", 9, 1e-6, 2),
        # the benchmark batch: 16 orbitals, order 9, prec 1e-6, norm-tiered
        c("helmholtz16_k9_mixed", "helmholtz", 9, 1e-6, 16, "mixed"),
        # an odd batch at another order, basis and accuracy
        c("helmholtz5_k6_mixed", "helmholtz", 6, 1e-4, 5, "mixed", "legendre"),
        # one SCF iteration's Helmholtz step from host state: new operators for the new energies, inputs
        # up, apply, outputs down
        c("scf_step8_k9_mixed", "scf", 9, 1e-5, 8, "mixed"),
        # exchange: all pair products of 8 orbitals, then their Poisson applies steered by the orbitals
        c("exchange8_k7_mixed", "exchange", 7, 1e-5, 8, "mixed"),
        # V * phi for 8 orbitals (the local potential of the Fock operator)
        c("vphi8_k7", "vphi", 7, 1e-5, 8),
        # the electron density of 6 orbitals
        c("density6_k7", "density", 7, 1e-5, 6),
        # rotation of 8 orbitals (localisation, Loewdin)
        c("rotate8_k9", "rotate", 9, 1e-5, 8),
        # the overlap matrix of 6 orbitals: many small calls
        c("overlap6_k7", "overlap", 7, 1e-5, 6),
        # the gradient of the Coulomb energy: adjoint apply of a 6-Gaussian density
        c("adjoint_k8_fp64", "adjoint", 8, 1e-5, 6),
    ]


def draw(rng):
    kind = rng.choice(["poisson", "helmholtz", "helmholtz", "helmholtz", "scf", "exchange", "vphi", "density",
                       "rotate", "overlap", "adjoint"])
    order = rng.choice([4, 5, 6, 7, 8, 9])
    # accuracies that the order is used for: from 2e-3 down to 10^-(order - 2), 1e-6 at most
    prec = float("%.3g" % 10 ** rng.uniform(-min(6.0, max(3.0, order - 2.0)), -2.7))
    basis = rng.choice(["interpolating", "interpolating", "legendre"])
    mode = rng.choice(["fp64", "mixed"]) if kind in ("poisson", "helmholtz") else "mixed"
    if kind in ("scf", "exchange"):
        n = rng.randint(2, 8)
    elif kind == "helmholtz" and mode == "fp64":
        n = rng.randint(1, 2)
    elif kind == "helmholtz":
        n = rng.randint(1, 16)
    elif kind in ("poisson", "adjoint"):
        n = rng.randint(1, 6)
        if kind == "adjoint":
            order, mode = min(order, 8), "fp64"
            prec = max(prec, 1e-5)
    else:
        n = rng.randint(2, 8)
    if kind in ("vphi", "density", "rotate", "overlap"):
        mode = "fp64"
    return {"kind": kind, "order": order, "prec": prec, "n": n, "mode": mode, "basis": basis}


# ------------------------------------------------------------------ plain 64-bit multiwavelets

class Basis:
    """Scaling basis of the given order on [0, 1], its quadrature maps and the two-scale filter."""

    def __init__(self, order, kind):
        K = self.K = order + 1
        t, w = np.polynomial.legendre.leggauss(K)
        self.x, w = 0.5 * (t + 1.0), 0.5 * w
        leg = lambda x: np.stack([math.sqrt(2 * j + 1) * np.polynomial.legendre.Legendre.basis(j)(2 * x - 1)
                                  for j in range(K)], axis=-1)
        if kind == "legendre":
            self.phi = leg
        else:
            rows = leg(self.x)
            self.phi = lambda x: np.sqrt(w) * (leg(x) @ rows.T)
        self.c2v = self.phi(self.x)               # values at the nodes from coefficients
        self.v2c = (w[:, None] * self.c2v).T      # coefficients from values
        W = np.zeros((2 * K, 2 * K))
        for b in range(2):
            W[:K, b * K:(b + 1) * K] = math.sqrt(0.5) * (self.phi(0.5 * (self.x + b)) * w[:, None]).T @ self.c2v
        for j in range(K):  # wavelets: (e_j, -e_j) / sqrt 2, orthonormalised against all earlier rows
            v = np.zeros(2 * K)
            v[j], v[K + j] = math.sqrt(0.5), -math.sqrt(0.5)
            for _ in range(2):
                for r in range(K + j):
                    v -= (W[r] @ v) * W[r]
                v /= np.linalg.norm(v)
            W[K + j] = v
        self.W = W


def _t(a, dev):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)


def _cube3(M, x):
    """(M (x) M (x) M) on the cubes x[n, Z, Y, X]."""
    x = torch.matmul(x, M.T)
    x = torch.matmul(M, x)
    n, a, b, c = x.shape
    return torch.matmul(M, x.reshape(n, a, b * c)).reshape(n, M.shape[0], b, c)


def _blocks(cubes, K):
    """cubes[n, Z, Y, X] as node blocks [n, 8 K^3] (component cx | cy << 1 | cz << 2, x fastest)."""
    n = cubes.shape[0]
    return cubes.reshape(n, 2, K, 2, K, 2, K).permute(0, 1, 3, 5, 2, 4, 6).reshape(n, 8 * K ** 3)


class Tree:
    """keys[n, 4], cubes[n, 2K, 2K, 2K]; a complete octree from the root boxes."""

    def __init__(self, basis, keys, cubes):
        self.b, self.keys, self.cubes = basis, keys, cubes
        self.index = {tuple(k): i for i, k in enumerate(keys.tolist())}
        self.made = {}
        self.WT = _t(basis.W.T, cubes.device)

    def is_leaf(self, key):
        return (key[0] + 1, 2 * key[1], 2 * key[2], 2 * key[3]) not in self.index

    def cube(self, key):
        """The block at a node, reconstructed from its leaf ancestor where the tree ends above it."""
        i = self.index.get(key)
        if i is not None:
            return self.cubes[i]
        if key not in self.made:
            up = (key[0] - 1, key[1] >> 1, key[2] >> 1, key[3] >> 1)
            K = self.b.K
            full = _cube3(self.WT, self.cube(up)[None])[0]
            s = torch.zeros_like(full)
            x, y, z = (K * (key[1 + d] & 1) for d in range(3))
            s[:K, :K, :K] = full[z:z + K, y:y + K, x:x + K]
            self.made[key] = s
        return self.made[key]

    def compress(self):
        """Every branch node's block from its children's scaling parts, finest first."""
        K, n = self.b.K, self.keys[:, 0]
        W = self.WT.T.contiguous()
        for s in range(int(n.max()) - 1, ROOT_SCALE - 1, -1):
            par = [i for i in np.nonzero(n == s)[0].tolist() if not self.is_leaf(tuple(self.keys[i].tolist()))]
            if not par:
                continue
            kid = np.array([[self.index[(s + 1,) + tuple(2 * self.keys[p, 1 + d] + ((c >> d) & 1) for d in range(3))]
                             for c in range(8)] for p in par])
            ch = self.cubes[torch.as_tensor(kid.reshape(-1), device=self.cubes.device)][:, :K, :K, :K]
            ch = ch.reshape(len(par), 2, 2, 2, K, K, K).permute(0, 1, 4, 2, 5, 3, 6).reshape(len(par), 2 * K, 2 * K, 2 * K)
            self.cubes[torch.as_tensor(np.array(par), device=self.cubes.device)] = _cube3(W, ch)
        return self

    def wavelet2(self):
        K = self.b.K
        return (self.cubes ** 2).sum((1, 2, 3)) - (self.cubes[:, :K, :K, :K] ** 2).sum((1, 2, 3))

    def arrays(self):
        """(keys, blocks) in canonical order: by scale, then Morton order, z most significant."""
        def morton(k):
            u = [k[1 + d] - CORNER * (1 << (k[0] - ROOT_SCALE)) for d in range(3)]
            return (k[0], sum(((u[d] >> i) & 1) << (3 * i + d) for i in range(k[0] - ROOT_SCALE + 2) for d in range(3)))
        order = sorted(range(len(self.keys)), key=lambda i: morton(self.keys[i].tolist()))
        return self.keys[order], _blocks(self.cubes[torch.as_tensor(order, device=self.cubes.device)], self.b.K)


def _children(keys):
    c = np.array([[c & 1, (c >> 1) & 1, c >> 2] for c in range(8)])
    k = np.concatenate([np.repeat(keys[:, :1] + 1, 8, 0), (2 * keys[:, None, 1:] + c).reshape(-1, 3)], 1)
    return k


def _roots():
    return np.array([[ROOT_SCALE, CORNER + x, CORNER + y, CORNER + z] for z in range(BOXES) for y in range(BOXES)
                     for x in range(BOXES)])


def _orbital_cubes(basis, keys, orb, dev):
    """p(r - R) exp(-a |r - R|^2) on the nodes: coefficients of the children's scaling functions, compressed."""
    poly, alpha, R = orb
    K = basis.K
    h = 2.0 ** -(keys[:, 0] + 1.0)
    f1 = []
    for d in range(3):
        x = h[:, None] * (2 * keys[:, 1 + d, None] + np.repeat([0, 1], K) + np.tile(basis.x, 2)) - R[d]
        g = np.exp(-np.minimum(alpha * x * x, 700.0))
        v = np.stack([g * x ** p for p in range(poly.shape[0])], 1).reshape(len(keys), -1, 2, K)
        f1.append(_t((v @ basis.v2c.T).reshape(len(keys), -1, 2 * K) * np.sqrt(h)[:, None, None], dev))
    c = torch.einsum("abc,nax->nbcx", _t(poly, dev), f1[0])
    c = torch.einsum("nbcx,nby->ncyx", c, f1[1])
    c = torch.einsum("ncyx,ncz->nzyx", c, f1[2])
    return _cube3(_t(basis.W, dev), c)


def _project(basis, orbs, prec, dev, norm=True):
    """sum of orbs on an adaptive grid: a box is split while its wavelet part exceeds prec 2^-(n+1)/2 or a
    Gaussian near it is narrower than the box's quadrature."""
    K, keys, all_keys, all_cubes = basis.K, _roots(), [], []
    while len(keys):
        cubes = sum(_orbital_cubes(basis, keys, o, dev) for o in orbs)
        w = ((cubes ** 2).sum((1, 2, 3)) - (cubes[:, :K, :K, :K] ** 2).sum((1, 2, 3))).clamp(min=0).sqrt().cpu().numpy()
        h = 2.0 ** -keys[:, 0].astype(float)
        split = w > prec * 2.0 ** (-0.5 * (keys[:, 0] + 1))
        for _, alpha, R in orbs:
            gap = np.maximum(np.abs((keys[:, 1:] + 0.5) * h[:, None] - R) - 0.5 * h[:, None], 0.0).max(1)
            split |= (gap * math.sqrt(alpha) < 2.0) & (h * math.sqrt(alpha) > 4.0)
        all_keys.append(keys)
        all_cubes.append(cubes)
        keys = _children(keys[split])
    t = Tree(basis, np.concatenate(all_keys), torch.cat(all_cubes)).compress()
    if norm:
        t.cubes /= torch.sqrt(t.wavelet2().sum() + (t.cubes[:8, :K, :K, :K] ** 2).sum())
    return t


def _inputs(case, seed):
    """(basis, input trees, random generator) of a case: cubic-polynomial Gaussian orbitals (exponents
    log-uniform in [0.3, 20], [0.5, 10] for order below 9; centres in [-2, 2]^3), or one density."""
    rng = np.random.default_rng(seed)
    basis = Basis(case["order"], case["basis"])
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    n, kind = case["n"], case["kind"]
    lo, hi = (0.3, 20.0) if case["order"] == 9 else (0.5, 10.0)

    def gaussians(m, a_lo, a_hi):
        out = []
        for _ in range(m):
            a = math.exp(rng.uniform(math.log(a_lo), math.log(a_hi)))
            out.append((np.full((1, 1, 1), (a / math.pi) ** 1.5), a, rng.uniform(-2.0, 2.0, 3)))
        return out

    def orbital():
        p = np.zeros((4, 4, 4))
        for a in range(4):
            for b in range(4 - a):
                for c in range(4 - a - b):
                    p[a, b, c] = rng.standard_normal()
        return (p, math.exp(rng.uniform(math.log(lo), math.log(hi))), rng.uniform(-2.0, 2.0, 3))

    if kind == "poisson":
        return basis, [_project(basis, gaussians(n, 0.5, 50.0), case["prec"], dev, False)], rng
    if kind == "adjoint":
        return basis, [_project(basis, gaussians(n, 1.0, 30.0), case["prec"], dev, False)], rng
    trees = [_project(basis, [orbital()], case["prec"], dev) for _ in range(n)]
    if kind == "vphi":  # a smooth screened potential of four sites
        trees.append(_project(basis, gaussians(4, 0.5, 4.0), case["prec"], dev, False))
    return basis, trees, rng


# ------------------------------------------------------------------ host buffers

def _room(case):
    """Nodes that a program sets room aside for, of all output trees together."""
    kind, n = case["kind"], case["n"]
    if kind in ("poisson", "adjoint"):
        return 1200
    if kind == "exchange":
        return 24 * n * (n + 1) + 200
    if kind == "density":
        return 4000
    if kind == "rotate":
        return 1300 * n
    return int(400 * n + 400 * math.sqrt(n))


SCF_ROOM = 640  # nodes per orbital in the host-buffer step


class Readback:
    """Page-locked buffers that a program reads its trees into, one after the other (grown when they do not fit);
    the rows that no tree fills stay zero."""

    def __init__(self, bs, rows):
        self.bs, self.rows = bs, 0
        self.grow(rows)

    def grow(self, rows):
        if rows > self.rows:
            self.rows = rows
            self.coefs = torch.zeros((rows, self.bs), dtype=torch.float64).pin_memory().numpy()
            self.keys = np.zeros((rows, 4), dtype=np.int32)
            self.leaf = np.zeros(rows, dtype=np.uint8)

    def read(self, trees):
        at = np.cumsum([0] + [t.nnodes for t in trees])
        self.grow(int(at[-1]))
        mw.download_batch(trees, [(self.keys[a:b], self.coefs[a:b], self.leaf[a:b]) for a, b in zip(at[:-1], at[1:])])
        return {"first": at, "keys": self.keys, "coefs": self.coefs}


# ------------------------------------------------------------------ preparing and running

def prepare(case, seed):
    mra, kind, prec, n = _mra(case), case["kind"], case["prec"], case["n"]
    bs = 8 * mra.K ** 3
    _, trees, rng = _inputs(case, seed)
    arrays = [(np.ascontiguousarray(k, dtype=np.int32), c.cpu()) for k, c in (t.arrays() for t in trees)]
    s = {"case": case, "mra": mra}
    if kind == "scf":  # the orbitals and the room for the new ones live on the host
        s["host"] = [(k, c.pin_memory().numpy()) for k, c in arrays]
        s["room"] = []
        for _ in arrays:
            r = Readback(bs, SCF_ROOM)
            s["room"].append((r.keys, r.coefs, r.leaf))
        s["in"] = [mw.FunctionTree(mra) for _ in arrays]
    else:
        s["in"] = mw.upload_batch([mw.FunctionTree(mra) for _ in arrays], [(k, c.numpy()) for k, c in arrays])
    mus = np.sqrt(-2.0 * rng.uniform(-2.0, -0.1, n))
    outs = n
    if kind in ("poisson", "exchange", "adjoint"):
        s["op"] = mw.PoissonOperator(mra, prec)
    if kind == "helmholtz":
        s["ops"] = mw.HelmholtzOperator.batch(mra, mus, prec)
    if kind == "scf":
        s["mus"] = mus
    if kind == "exchange":
        s["pairs"] = [(i, j) for i in range(n) for j in range(i, n)]
        s["rho"] = [mw.FunctionTree(mra) for _ in s["pairs"]]
        outs = len(s["pairs"])
    if kind in ("poisson", "density", "adjoint"):
        outs = 1
    if kind == "rotate":
        s["U"] = np.linalg.qr(rng.standard_normal((n, n)))[0]
    if kind == "density":
        s["occ"] = np.full(n, 2.0)
    if kind == "overlap":
        return s
    s["out"] = [mw.FunctionTree(mra) for _ in range(outs)]
    if kind != "scf":
        s["back"] = Readback(bs, _room(case))
    return s


def run(s):
    case, mra, inp = s["case"], s["mra"], s["in"]
    kind, prec, mode, n = case["kind"], case["prec"], case["mode"], case["n"]
    if kind == "overlap":
        return np.array([mw.dot(inp[i], inp[j]) for i in range(n) for j in range(i, n)])
    out = s["out"]
    if kind != "rotate":
        for t in out:
            t.clear()
    if kind == "poisson":  # relative precision, as the Coulomb potential's apply
        s["stats"] = mw.apply(prec, out[0], s["op"], inp[0], precision=mode)
    elif kind == "helmholtz":
        s["stats"] = mw.apply_batch([prec] * n, out, s["ops"], inp, abs_prec=True, precision=mode)
    elif kind == "scf":
        ops = mw.HelmholtzOperator.batch(mra, s["mus"], prec)
        st = mw.apply_batch_host([prec] * n, out, ops, inp, s["host"], abs_prec=True, precision=mode, outputs=s["room"])
        s["stats"] = st
        got = []
        for t, room, full in zip(out, s["room"], st["outputs_filled"]):
            k, c, _ = room if full else t.download()
            got.append((k, c))
        for o in ops:
            o.close()
        return got
    elif kind == "exchange":  # the accuracies of the reference's exchange: prec / 10 for products, 10 prec for potentials
        for t in s["rho"]:
            t.clear()
        pairs = s["pairs"]
        mw.multiply_batch(prec / 10, s["rho"], 1.0, [inp[i] for i, _ in pairs], [inp[j] for _, j in pairs], abs_prec=True,
                          use_max_norms=True)
        s["stats"] = mw.apply_batch(prec * 10, out, [s["op"]] * len(pairs), s["rho"],
                                    prec_trees=[[inp[i], inp[j]] if i != j else [inp[i]] for i, j in pairs],
                                    abs_prec=True, precision=mode)
    elif kind == "vphi":
        mw.multiply_batch(prec, out, 1.0, [inp[n]] * n, inp[:n], abs_prec=True)
    elif kind == "density":
        mw.density(prec, out[0], inp, s["occ"])
    elif kind == "rotate":
        mw.rotate(out, inp, s["U"])
    elif kind == "adjoint":
        s["stats"] = mw.apply_adjoint(prec, out[0], s["op"], inp[0], inp[0])
    return s["back"].read(out)


# ------------------------------------------------------------------ what the results are, in 64 bits

def exact(case, seed):
    """Overlaps, rotations, products and densities from their definitions.  An adaptive apply has no such
    value here: its result is defined by the operator's fit, bands and screening."""
    kind, n = case["kind"], case["n"]
    if kind not in ("overlap", "rotate", "vphi", "density"):
        return None
    b, trees, rng = _inputs(case, seed)
    if kind == "overlap":
        return np.array([_dot(trees[i], trees[j]) for i in range(n) for j in range(i, n)])
    if kind == "vphi":
        return _result(case, [_product(trees[n], t, case["prec"], _roots(), True) for t in trees[:n]])
    if kind == "density":
        sq = [_product(t, t, case["prec"], t.keys, False) for t in trees]
        return _result(case, [_crop(_combine(sq, [2.0] * n), case["prec"] / (2.0 * n))])
    rng.uniform(-2.0, -0.1, n)
    U = np.linalg.qr(rng.standard_normal((n, n)))[0]
    return _result(case, [_combine(trees, row) for row in U])


def _result(case, trees):
    got = [t.arrays() for t in trees]
    at = np.cumsum([0] + [len(k) for k, _ in got])
    rows = max(_room(case), int(at[-1]))
    keys, coefs = np.zeros((rows, 4), dtype=np.int32), np.zeros((rows, got[0][1].shape[1]))
    for a, (k, c) in zip(at, got):
        keys[a:a + len(k)], coefs[a:a + len(k)] = k, c.cpu().numpy()
    return {"first": at, "keys": keys, "coefs": coefs}


def _dot(a, b):
    K = a.b.K
    common = [k for k in a.index if k in b.index]
    x = a.cubes[torch.as_tensor([a.index[k] for k in common], device=a.cubes.device)]
    y = b.cubes[torch.as_tensor([b.index[k] for k in common], device=a.cubes.device)]
    p = x * y
    inner = torch.as_tensor([k[0] != ROOT_SCALE for k in common], device=p.device)
    return float(p.sum()) - float(p[inner][:, :K, :K, :K].sum())


def _combine(trees, coefs):
    """sum_k coefs[k] trees[k] on the union grid."""
    keys = sorted(set().union(*(t.index for t in trees)))
    cubes = torch.stack([sum(float(c) * t.cube(k) for c, t in zip(coefs, trees)) for k in keys])
    return Tree(trees[0].b, np.array(keys), cubes)


def _product(f, g, prec, keys, absolute):
    """f g: values at the children's quadrature points, refined from the given grid's leaves while the product's
    wavelet part exceeds prec R 2^-(n+1)/2 (R: 1, or the norm over the leaves so far)."""
    basis, K, dev = f.b, f.b.K, f.cubes.device
    c2v, v2c = (_t(np.kron(np.eye(2), m), dev) for m in (basis.c2v, basis.v2c))
    up, down = c2v @ _t(basis.W.T, dev), _t(basis.W, dev) @ v2c
    have = {}
    start = set(map(tuple, keys.tolist()))
    work = sorted(k for k in start if (k[0] + 1, 2 * k[1], 2 * k[2], 2 * k[3]) not in start)
    leaves = {}
    while work:
        a, b = (_cube3(up, torch.stack([t.cube(k) for k in work])) for t in (f, g))
        scale = _t(np.array([2.0 ** (1.5 * (k[0] + 1)) for k in work]), dev)
        p = _cube3(down, a * b * scale[:, None, None, None])
        full = (p ** 2).sum((1, 2, 3))
        w = (full - (p[:, :K, :K, :K] ** 2).sum((1, 2, 3))).clamp(min=0).sqrt().cpu().numpy()
        full = full.cpu().numpy()
        for i, k in enumerate(work):
            have[k], leaves[k] = p[i], full[i]
        R = 1.0 if absolute else math.sqrt(sum(leaves.values()))
        nxt = []
        for i, k in enumerate(work):
            if w[i] > prec * R * 2.0 ** (-0.5 * (k[0] + 1)):
                del leaves[k]
                nxt += [tuple(c) for c in _children(np.array([k])).tolist()]
        work = nxt
    every = sorted(set(have) | start)
    zero = torch.zeros((2 * K,) * 3, dtype=torch.float64, device=dev)
    return Tree(basis, np.array(every), torch.stack([have.get(k, zero) for k in every])).compress()


def _crop(t, prec):
    """Leaves go, finest first, where eight siblings' wavelet parts together stay below prec 2^-(n+1)/2."""
    w = dict(zip(map(tuple, t.keys.tolist()), t.wavelet2().cpu().tolist()))
    alive = set(w)
    for k in sorted(w, reverse=True):
        kids = [tuple(c) for c in _children(np.array([k])).tolist()]
        if kids[0] not in alive or any((c[0] + 1, 2 * c[1], 2 * c[2], 2 * c[3]) in alive for c in kids):
            continue
        if math.sqrt(sum(max(0.0, w[c]) for c in kids)) < prec * 2.0 ** (-0.5 * (k[0] + 2)):
            alive -= set(kids)
    keep = sorted(alive)
    return Tree(t.b, np.array(keep), torch.stack([t.cube(k) for k in keep]))


# ------------------------------------------------------------------ the work a pass cannot do without

def work(case):
    """Input and output blocks once each; 2 (2K)^4 flops per cube pass (one per contraction along x, two more
    per run of contractions that share y and z), per product node six, per rotation two flops a value."""
    s = prepare(case, 0)
    K, kind, n = case["order"] + 1, case["kind"], case["n"]
    run(s)
    nin = sum(t.nnodes for t in s["in"])
    if kind == "overlap":
        vals = sum(8 * K ** 3 * min(s["in"][i].nnodes, s["in"][j].nnodes) for i in range(n) for j in range(i, n))
        return {"bytes": 8 * 8 * K ** 3 * nin, "flops": 2 * vals}
    nout = sum(t.nnodes for t in s["out"])
    w = {"bytes": 8 * 8 * K ** 3 * (nin + nout), "flops": 0}
    cube = 2 * (2 * K) ** 4
    st = s.get("stats")
    if st:
        rows = sum(st["rows_" + t] for t in ("fp64", "fp32", "tf32", "df")) or st["items"]
        w["flops"] += cube * (st["items"] + 2 * rows)
    if kind == "exchange":
        w["flops"] += cube * 3 * sum(t.nnodes for t in s["rho"])
    if kind in ("vphi", "density"):
        w["flops"] += 6 * cube * nout
    if kind == "rotate":
        w["flops"] += 2 * n * 8 * K ** 3 * nout
    return w
