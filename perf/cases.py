"""The work that users of this framework have it do, as cases to be timed.

A case is one call (or one short chain of calls, as a program makes it) of the
public entry points: batched evaluation, eager and as a captured plan; the
training step and the vector-Jacobian product of evaluation; integration;
operator application with truncation, alone and batched; the linear solver.

Networks have one digit per vertex, base 2, on the three graphs that the
framework's configurations use (a path of one variable, a comb with one tooth
per variable, a heap-ordered binary tree whose vertices carry the variables'
digits in turn).  Tensors are Gaussian, or the block-diagonal tensors of sums
of damped waves as the elementary constructors write them.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "itensornumericalanalysis.jl_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import itensornumericalanalysis as ina  # noqa: E402
from itensornumericalanalysis import _lib  # noqa: E402
from itensornumericalanalysis.network import topology_struct  # noqa: E402

_NET = {"f64": _lib.F64, "f32": _lib.F32, "c128": _lib.C128, "mixed": _lib.F32}
_TORCH = {"f64": torch.float64, "f32": torch.float32, "c128": torch.complex128, "mixed": torch.float32}
_OUT = {"f64": torch.float64, "f32": torch.float32, "c128": torch.complex128, "mixed": torch.float64}
_KIND = {"f64": _lib.OUT_F64, "f32": _lib.OUT_F32, "c128": _lib.OUT_C128, "mixed": _lib.OUT_F64}
_PREC = {"f64": _lib.PREC_F64, "f32": _lib.PREC_F32, "c128": _lib.PREC_F64, "mixed": _lib.PREC_MIXED}


# ------------------------------------------------------------------- cases ----
def listed():
    return [
        # the smallest call: a latency-bound loop (an optimiser, a sampler) that
        # evaluates a low-rank function on a fixed buffer through a captured plan
        {"name": "plan path20 chi2", "kind": "plan", "graph": "path", "nvar": 1, "L": 20, "chi": 2, "init": "waves",
         "type": "f64", "points": 4096},
        # the ordinary interactive call: a sum of elementary functions at a few
        # thousand points held in a numpy array
        {"name": "host path20 chi6", "kind": "host", "graph": "path", "nvar": 1, "L": 20, "chi": 6, "init": "waves",
         "type": "f64", "points": 4096},
        # plotting or sampling the same kind of function densely
        {"name": "eval path20 chi2 1e7", "kind": "eval", "graph": "path", "nvar": 1, "L": 20, "chi": 2,
         "init": "waves", "type": "f64", "points": 10_000_000},
        # the forward pass of a fit: two variables of 12 bits, bond 32, FP32
        {"name": "eval comb2x12 chi32 f32", "kind": "eval", "graph": "comb", "nvar": 2, "L": 12, "chi": 32,
         "init": "gauss", "type": "f32", "points": 1 << 20},
        # the heaviest evaluation: three variables of 20 bits on a binary tree,
        # bond 128, FP32 tensors, mixed precision
        {"name": "eval binary60 chi128 mixed", "kind": "eval", "graph": "binary", "nvar": 3, "L": 20, "chi": 128,
         "init": "unit", "type": "mixed", "points": 500_000},
        # plain FP64 at a medium bond and an odd number of points
        {"name": "eval binary33 chi48 f64", "kind": "eval", "graph": "binary", "nvar": 3, "L": 11, "chi": 48,
         "init": "gauss", "type": "f64", "points": 20_011},
        # one training step (forward, loss, backward) of the fit above
        {"name": "train comb2x12 chi32 f32", "kind": "train", "graph": "comb", "nvar": 2, "L": 12, "chi": 32,
         "init": "gauss", "type": "f32", "points": 1 << 20},
        # a gradient from numpy arrays, small bond, odd sizes (the rrule called from a host program)
        {"name": "vjp comb3x8 chi11 f64", "kind": "vjp", "graph": "comb", "nvar": 3, "L": 8, "chi": 11,
         "init": "gauss", "type": "f64", "points": 4097},
        # integral of the heaviest network
        {"name": "integrate binary60 chi128", "kind": "integrate", "graph": "binary", "nvar": 3, "L": 20, "chi": 128,
         "init": "gauss", "type": "f32"},
        # derivative of one function, compressed, then looked at
        {"name": "operate path24 chi40", "kind": "operate", "graph": "path", "nvar": 1, "L": 24, "chi": 40,
         "init": "gauss", "type": "f64", "points": 4096, "n": 1, "precision": "f64"},
        # derivatives of many functions of uneven length and bond in one pass
        {"name": "operate batched 96 mixed", "kind": "operate", "graph": "path", "nvar": 1, "L": 30, "chi": 128,
         "init": "gauss", "type": "f64", "points": 64, "n": 96, "precision": "mixed"},
        # the Laplace solve with Dirichlet boundaries on a two-variable comb
        {"name": "linsolve comb2x12", "kind": "linsolve", "nvar": 2, "L": 12, "points": 4096},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plan", "host", "eval", "eval", "eval", "eval", "train", "vjp", "integrate", "operate",
                       "operate", "linsolve"])
    if kind in ("plan", "host"):
        c = {"kind": kind, "graph": "path", "nvar": 1, "L": rng.randint(12, 30), "chi": rng.randint(2, 8),
             "init": "waves", "type": rng.choice(["f64", "f64", "f32", "c128"]), "points": _log(rng, 700, 20000)}
        if kind == "host" and c["type"] == "f32":
            c["type"] = "f64"
        return c
    if kind == "eval":
        how = rng.choice(["path", "comb", "tree", "mixed"])
        if how == "path":
            c = {"kind": kind, "graph": "path", "nvar": 1, "L": rng.randint(14, 30), "chi": _log(rng, 2, 32),
                 "init": "waves", "type": rng.choice(["f64", "f64", "f32", "c128"])}
            top = 2e11
        elif how == "comb":
            nvar = rng.randint(2, 3)
            c = {"kind": kind, "graph": "comb", "nvar": nvar, "L": rng.randint(6, 14), "chi": _log(rng, 4, 48),
                 "init": "gauss", "type": rng.choice(["f64", "f32", "f32", "c128"])}
            top = 2e11
        elif how == "tree":
            c = {"kind": kind, "graph": "binary", "nvar": 3, "L": rng.randint(5, 20), "chi": _log(rng, 8, 64),
                 "init": "gauss", "type": rng.choice(["f64", "f64", "f32"])}
            top = 2e11
        else:
            c = {"kind": kind, "graph": "binary", "nvar": 3, "L": rng.randint(5, 20), "chi": rng.choice([64, 128]),
                 "init": "unit", "type": "mixed"}
            top = 1e13
        per = _direct_flops(c) * (4 if c["type"] == "c128" else 1)
        c["points"] = _log(rng, 2000, max(4000, min(10_000_000, top / per)))
        return c
    if kind == "train":
        c = {"kind": kind, "graph": "comb", "nvar": 2, "L": rng.randint(8, 14), "chi": _log(rng, 8, 32),
             "init": "gauss", "type": "f32"}
        c["points"] = _log(rng, 10_000, 1 << 20)
        return c
    if kind == "vjp":
        nvar = rng.randint(2, 3)
        return {"kind": kind, "graph": "comb", "nvar": nvar, "L": rng.randint(5, 12), "chi": _log(rng, 3, 20),
                "init": "gauss", "type": "f64", "points": _log(rng, 500, 30_000)}
    if kind == "integrate":
        return {"kind": kind, "graph": "binary", "nvar": 3, "L": rng.randint(8, 20), "chi": _log(rng, 24, 128),
                "init": "gauss", "type": rng.choice(["f32", "f64"])}
    if kind == "operate":
        n = rng.choice([1, _log(rng, 16, 96)])
        return {"kind": kind, "graph": "path", "nvar": 1, "L": rng.randint(14, 30),
                "chi": _log(rng, 12, 48) if n == 1 else _log(rng, 24, 128), "init": "gauss", "type": "f64",
                "points": 1000 if n == 1 else 64, "n": n, "precision": rng.choice(["f64", "mixed"]) if n > 1 else "f64"}
    return {"kind": kind, "nvar": 2, "L": rng.randint(8, 12), "points": _log(rng, 500, 5000)}


# ------------------------------------------------------------------- trees ----
def _tree(case):
    """(parent of every vertex, numbered breadth first; (variable, digit) of every vertex)."""
    nvar, L = case["nvar"], case["L"]
    if case["graph"] == "path":
        return [-1] + list(range(L - 1)), [(1, v + 1) for v in range(L)]
    if case["graph"] == "binary":
        V = nvar * L
        return [(v - 1) // 2 if v else -1 for v in range(V)], [(v % nvar + 1, v // nvar + 1) for v in range(V)]
    order, up, todo = [], [], [(1, 1, -1)]
    while todo:  # breadth first; a spine vertex has its tooth before the next spine vertex
        j, k, p = todo.pop(0)
        me = len(order)
        order.append((j, k))
        up.append(p)
        if k < L:
            todo.append((j, k + 1, me))
        if k == 1 and j < nvar:
            todo.append((j + 1, 1, me))
    return up, order


def _children(parent):
    kids = [[] for _ in parent]
    for v, p in enumerate(parent):
        if p >= 0:
            kids[p].append(v)
    return kids


def _below(parent):
    """Vertices in the subtree of every vertex."""
    n = [1] * len(parent)
    for v in range(len(parent) - 1, 0, -1):
        n[parent[v]] += n[v]
    return n


def _links(case, parent):
    """Bond to the parent of every vertex: chi, and no more than the digits on either side allow."""
    below, V = _below(parent), len(parent)
    cap = case["init"] != "waves" and case["kind"] == "operate"
    return [1 if p < 0 else min(case["chi"], 2 ** min(below[v], V - below[v], 30)) if cap else case["chi"]
            for v, p in enumerate(parent)]


def _shapes(parent, link):
    kids = _children(parent)
    return [(2, link[v]) + tuple(link[c] for c in kids[v]) for v in range(len(parent))]


def _map(case, parent, digits):
    g = ina.NamedGraph(range(len(parent)), [(p, v) for v, p in enumerate(parent) if p >= 0])
    where = [[v for _, v in sorted((d[1], v) for v, d in enumerate(digits) if d[0] == j + 1)]
             for j in range(case["nvar"])]
    s = ina.continuous_siteinds(g, where)
    if s.layout.order != list(range(len(parent))):
        raise RuntimeError("the layout numbers the vertices otherwise")
    return s


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 11)


def _tensors(case, seed, parent, link):
    """The vertex tensors, on the GPU, in the case's type."""
    g, out = _gen(seed), []
    dt = _TORCH[case["type"]]
    if case["init"] == "waves":  # sum over blocks of amp * exp(-k x) * cos(w x + phi), one 2x2 block each
        r = np.random.default_rng([int(seed), 5])
        V, chi = len(parent), case["chi"]
        nb = (chi + 1) // 2
        k, w, phi, amp = r.uniform(0, 2, nb), r.uniform(1, 20, nb), r.uniform(0, 6, nb), r.uniform(0.5, 1.5, nb)
        for v in range(V):
            t = np.zeros((2, chi, chi))
            for s in range(2):
                x = s * 2.0 ** -(v + 1)
                for b in range(nb):
                    e, c, sn = math.exp(-k[b] * x), math.cos(w[b] * x), math.sin(w[b] * x)
                    i = 2 * b
                    t[s, i, i] = e * c
                    if i + 1 < chi:
                        t[s, i, i + 1], t[s, i + 1, i], t[s, i + 1, i + 1] = -e * sn, e * sn, e * c
            left, right = np.zeros(chi), np.zeros(chi)
            left[0::2], right[0::2] = 1.0, amp * np.cos(phi)
            right[1::2] = (amp * np.sin(phi))[: chi // 2]
            if v == 0:
                t = np.einsum("a,sab->sb", left, t)[:, None, :]
            if v == V - 1:
                t = t @ right
            t = torch.from_numpy(np.ascontiguousarray(t)).cuda()
            out.append((t * (0.8 + 0.6j) if v == 0 else t).to(dt) if dt.is_complex else t.to(dt))
        return out
    for shape in _shapes(parent, link):
        t = torch.randn(shape, generator=g, device="cuda", dtype=dt)
        if case["init"] == "unit":
            t /= torch.linalg.vector_norm(t)
        else:
            t /= math.sqrt(math.prod(shape[2:]))
        out.append(t)
    return out


def _network(case, seed):
    parent, digits = _tree(case)
    link = _links(case, parent)
    s = _map(case, parent, digits)
    flat = torch.cat([t.reshape(-1) for t in _tensors(case, seed, parent, link)])
    topo, keep = topology_struct(s, link)
    h, ctx = ctypes.c_void_p(), _lib.default_context()
    torch.cuda.synchronize()
    ctx.call("tnfa_net_create", ctypes.byref(topo), _NET[case["type"]], ctypes.c_void_p(flat.data_ptr()),
             _lib.MEM_DEVICE, ctypes.byref(h))
    return ina.ITensorNetworkFunction(s, h, ctx), flat


def _points(case, seed):
    return torch.rand((case["points"], case["nvar"]), generator=_gen(seed + 1000), device="cuda", dtype=torch.float64)


def _ops(case, seed):
    """The (length, bond) of every function of an operator case: one, or many of uneven length and bond."""
    if case["n"] == 1:
        return [(case["L"], case["chi"])]
    r = np.random.default_rng([int(seed), 3])
    return [(int(r.integers(max(8, case["L"] // 3), case["L"] + 1)),
             int(round(math.exp(r.uniform(math.log(8), math.log(case["chi"]))))) ) for _ in range(case["n"])]


# --------------------------------------------------------------- preparing ----
def prepare(case, seed):
    kind = case["kind"]
    if kind == "linsolve":
        L = case["L"]
        s = ina.continuous_siteinds(ina.named_comb_tree((2, L)), [[(1, j) for j in range(L, 0, -1)],
                                                                  [(2, j) for j in range(1, L + 1)]])
        b = _source(seed) * (ina.sin_itn(s, k=np.pi, dim=1) * ina.sin_itn(s, k=np.pi, dim=2))
        return {"case": case, "A": ina.laplacian_operator(s), "b": b, "X": _points(case, seed).cpu().numpy()}
    if kind == "operate":
        fs, ops, X, made = [], [], [], {}
        for i, (L, chi) in enumerate(_ops(case, seed)):
            one = dict(case, L=L, chi=chi)
            f, _ = _network(one, seed + 100 * i)
            if L not in made:
                made[L] = ina.first_derivative_operator(f.s)
            fs.append(f)
            ops.append(made[L])
            X.append(_points(case, seed + 100 * i).cpu().numpy())
        return {"case": case, "fs": fs, "ops": ops, "X": X}
    f, flat = _network(case, seed)
    st = {"case": case, "f": f}
    if kind == "integrate":
        return st
    X = _points(case, seed)
    dims = list(range(1, case["nvar"] + 1))
    if kind == "host":
        st["X"] = X.cpu().numpy()
    elif kind == "plan":
        st["X"], st["out"] = X, torch.empty(len(X), dtype=_OUT[case["type"]], device="cuda")
        torch.cuda.synchronize()
        names = {"f64": "f64", "f32": "f32", "c128": "c128"}
        st["plan"] = f.evaluation_plan(X, st["out"], dims, out_kind=names[case["type"]])
    elif kind == "eval":
        st["X"], st["dims"] = X, (ctypes.c_int32 * len(dims))(*dims)
    elif kind == "train":
        st["X"], st["params"], st["dims"] = X, flat.requires_grad_(True), dims
        st["y"] = _target(X).to(flat.dtype)
    elif kind == "vjp":
        st["X"] = X.cpu().numpy()
        st["dout"] = _weights(case, seed).cpu().numpy()
        st["dims"] = dims
    return st


def _source(seed):
    return float(np.random.default_rng([int(seed), 9]).uniform(0.5, 2.0))


def _target(X):
    return torch.sin(3 * X[:, 0]) * torch.cos(5 * X[:, 1]) * torch.exp(-(X ** 2).sum(1))


def _weights(case, seed):
    return torch.randn(case["points"], generator=_gen(seed + 2000), device="cuda", dtype=torch.float64)


# ----------------------------------------------------------------- running ----
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "plan":
        st["plan"].launch()
        return st["out"]
    if kind == "host":
        return st["f"].evaluate_batch(st["X"])
    if kind == "eval":
        f, X, t = st["f"], st["X"], case["type"]
        out = torch.empty(len(X), dtype=_OUT[t], device="cuda")
        f.ctx.call("tnfa_evaluate", f.handle, X.data_ptr(), len(X), case["nvar"], st["dims"], _lib.MEM_DEVICE,
                   out.data_ptr(), _KIND[t], _lib.MEM_DEVICE, _PREC[t])
        return out
    if kind == "train":
        p = st["params"]
        p.grad = None
        out = ina.TTNEvaluate.apply(p, st["X"], st["f"], st["dims"])
        ((out - st["y"]) ** 2).mean().backward()
        return [out.detach(), p.grad]
    if kind == "vjp":
        return ina.evaluate_vjp(st["f"], st["X"], st["dout"], st["dims"])
    if kind == "integrate":
        return ina.integrate(st["f"])
    if kind == "operate":
        if case["n"] == 1:
            g = ina.operate(st["ops"][0], st["fs"][0], cutoff=1e-10)
            return g.evaluate_batch(st["X"][0])
        gs = ina.operate_batched(st["ops"], st["fs"], cutoff=1e-10, precision=case["precision"])
        return np.stack([g.evaluate_batch(x) for g, x in zip(gs, st["X"])])
    x = ina.linsolve(st["A"], st["b"], nsweeps=2, maxdim=16, cutoff=1e-20, tol=1e-8)
    return x.evaluate_batch(st["X"], [1, 2])


# ------------------------------------------------------------ in 64 bits ----
def _bits(X, digits):
    """The digit of every vertex at every point (x in [0, 1), base 2)."""
    cols = []
    for var, d in digits:
        cols.append(torch.floor(X[:, var - 1] * 2.0 ** d).to(torch.int64) & 1)
    return cols


def _tree_value(tensors, parent, digits, X):
    """f at the rows of X: messages up the tree, one for every combination of digits below that occurs."""
    kids, S = _children(parent), _bits(X, digits)
    rows, where = {}, {}
    for v in reversed(range(len(parent))):
        key, sizes = S[v], []
        for c in kids[v]:
            key = key * rows[c].shape[0] + where[c]
            sizes.append(rows[c].shape[0])
        key, where[v] = torch.unique(key, return_inverse=True)
        idx = []
        for n in reversed(sizes):
            idx.insert(0, key % n)
            key = torch.div(key, n, rounding_mode="floor")
        parts = []
        for s in range(2):
            t = tensors[v][s]
            mine = torch.nonzero(key == s).reshape(-1)
            if len(sizes) == 0:
                parts.append(t.reshape(1, -1).expand(len(mine), -1))
                continue
            step = max(1, (1 << 27) // max(1, t.numel() // t.shape[-1]))
            for q in range(0, len(mine), step):
                m = mine[q:q + step]
                last = rows[kids[v][-1]][idx[-1][m]]
                y = last @ t.reshape(-1, t.shape[-1]).T
                if len(sizes) == 2:
                    y = torch.einsum("pab,pb->pa", y.reshape(len(m), t.shape[0], t.shape[1]),
                                     rows[kids[v][0]][idx[0][m]])
                parts.append(y)
        rows[v] = torch.cat(parts)  # the keys are sorted, the digit of v first
    return rows[0][where[0], 0]


def _wide(case):
    return torch.complex128 if case["type"] == "c128" else torch.float64


def exact(case, seed):
    kind = case["kind"]
    if kind == "linsolve":
        N = 2 ** case["L"]
        x = np.arange(N) / N
        lam = -(2 - 2 * np.cos(np.pi * np.arange(1, N + 1) / (N + 1))) * float(N) ** 2
        Q = np.sqrt(2 / (N + 1)) * np.sin(np.pi * np.outer(np.arange(1, N + 1), np.arange(1, N + 1)) / (N + 1))
        B = _source(seed) * np.outer(np.sin(np.pi * x), np.sin(np.pi * x))
        U = Q @ ((Q @ B @ Q) / (lam[:, None] + lam[None, :])) @ Q
        at = np.floor(_points(case, seed).cpu().numpy() * N).astype(np.int64)
        return U[at[:, 0], at[:, 1]]
    if kind == "operate":
        got = []
        for i, (L, chi) in enumerate(_ops(case, seed)):
            one = dict(case, L=L, chi=chi)
            parent, digits = _tree(one)
            T = _tensors(one, seed + 100 * i, parent, _links(one, parent))
            X, h = _points(case, seed + 100 * i), 2.0 ** -L
            X = torch.floor(X / h) * h
            y = 0
            for w, Z in ((0.5, X + h), (-0.5, X - h)):
                inside = ((Z >= 0) & (Z < 1)).reshape(-1)
                y = y + w / h * torch.where(inside, _tree_value(T, parent, digits, torch.where(inside[:, None], Z, X)), 0.0)
            got.append(y.cpu().numpy())
        return got[0] if case["n"] == 1 else np.stack(got)
    parent, digits = _tree(case)
    T = [t.to(_wide(case)) for t in _tensors(case, seed, parent, _links(case, parent))]
    if kind == "integrate":
        kids, m = _children(parent), {}
        for v in reversed(range(len(parent))):
            t = T[v].mean(0)
            for c in reversed(kids[v]):
                t = t @ m[c]
            m[v] = t
        return float(m[0])
    X = _points(case, seed)
    if kind in ("train", "vjp"):
        T = [t.requires_grad_(True) for t in T]
        f = _tree_value(T, parent, digits, X)
        if kind == "train":
            ((f - _target(X).to(torch.float32).to(f.dtype)) ** 2).mean().backward()
            return [f.detach(), torch.cat([t.grad.reshape(-1) for t in T])]
        (f * _weights(case, seed)).sum().backward()
        return {v: t.grad.cpu().numpy() for v, t in enumerate(T)}
    f = _tree_value(T, parent, digits, X)
    return f.cpu().numpy() if kind == "host" else f


# -------------------------------------------------------------------- work ----
def _direct_flops(case):
    parent, _ = _tree(case)
    return 2.0 * sum(math.prod(s[1:]) for s in _shapes(parent, _links(case, parent)))


def _tree_flops(case, P):
    """Flops of one evaluation at P points when a message is formed once for
    every combination of the digits below it (at most 2^below, at most P), and
    a child with few of them is contracted into the vertex tensor first."""
    parent, _ = _tree(case)
    link, below, kids = _links(case, parent), _below(parent), _children(parent)
    total = 0.0
    for v in range(len(parent)):
        rows = min(P, 2.0 ** below[v])
        full = link[v] * math.prod(link[c] for c in kids[v])
        ways = [rows * full] + [2 * min(P, 2.0 ** below[c]) * full + rows * full / link[c] for c in kids[v]]
        total += 2.0 * min(ways) if kids[v] else 0.0
    return total


def work(case):
    kind = case["kind"]
    if kind == "linsolve":  # the operator, the source and the solution (bonds of about 8) and the points; two sweeps of two-site updates
        return {"bytes": 8.0 * 2 * case["L"] * 3 * 4 * 64 + 24.0 * case["points"],
                "flops": 2 * 3 * 2.0 * case["L"] * (2 / 3) * (4 * 8 * 8) ** 3}
    if kind == "operate":
        flops = nbytes = 0.0
        for L, chi in _ops(case, 1):
            one = dict(case, L=L, chi=chi)
            parent, _ = _tree(one)
            link = _links(one, parent) + [1]
            for v in range(L):  # per vertex: the product with bond 3, one QR and one SVD of the (chi + 2)-wide bond
                l, r = link[v], link[v + 1]
                m, n = 2 * (l + 2), r + 2
                m, n = max(m, n), min(m, n)
                flops += 2.0 * 4 * 9 * l * r + 2 * (2.0 * m * n * n) + 12.0 * n ** 3
                nbytes += 8.0 * (2 * l * r + 2 * (l + 2) * (r + 2))
            nbytes += 16.0 * case["points"]
        return {"bytes": nbytes, "flops": flops}
    parent, _ = _tree(case)
    n = sum(math.prod(s) for s in _shapes(parent, _links(case, parent)))
    size = {"f64": 8, "f32": 4, "c128": 16, "mixed": 4}[case["type"]]
    if kind == "integrate":
        return {"bytes": float(n * size), "flops": 2.0 * n}
    P = case["points"]
    flops = _tree_flops(case, P) * (4 if case["type"] == "c128" else 1)
    nbytes = n * size + P * (8.0 * case["nvar"] + {"f64": 8, "f32": 4, "c128": 16, "mixed": 8}[case["type"]])
    if kind in ("train", "vjp"):
        flops, nbytes = 3 * flops, nbytes + n * size + 8.0 * P
    return {"bytes": nbytes, "flops": flops}
