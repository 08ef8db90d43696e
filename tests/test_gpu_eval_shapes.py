"""Which networks evaluation takes does not depend on its schedule: vertices of
more than 8 children and bonds beyond the per-point kernels' shared memory are
refused, and what the stored order takes is taken in any orientation."""
import ctypes as C

import numpy as np
import pytest

import oracle as O
from _helpers import upload_oracle

pytestmark = pytest.mark.gpu


def _star(ina, n):
    graph = (list(range(n + 1)), [(0, i) for i in range(1, n + 1)])
    net = O.random_net(O.siteinds(graph), 2, np.random.default_rng(n), normalize=True)
    return upload_oracle(ina, graph, net)[0], net


@pytest.mark.parametrize("n", [7, 8, 9, 10])
@pytest.mark.parametrize("precision", ["f64", "f32", "mixed"])
def test_degree(ina, n, precision):
    f, net = _star(ina, n)
    X = np.random.default_rng(1).random((600, 1))
    if n > 8:
        with pytest.raises(ina.TnfaError, match="UNSUPPORTED"):
            f.evaluate_batch(X, precision=precision)
        return
    ref = O.evaluate_batch(net, X)
    tol = 1e-4 if precision == "f32" else 1e-12
    assert np.max(np.abs(f.evaluate_batch(X, precision=precision) - ref)) < tol * np.max(np.abs(ref))


def test_degree_plan(ina):
    import torch

    X = torch.rand((600, 1), dtype=torch.float64, device="cuda")
    out = torch.empty(600, dtype=torch.float64, device="cuda")
    _star(ina, 8)[0].evaluation_plan(X, out).launch()
    f, _ = _star(ina, 9)
    with pytest.raises(ina.TnfaError, match="UNSUPPORTED"):
        f.evaluation_plan(X, out)
    with pytest.raises(ina.TnfaError, match="UNSUPPORTED"):
        f.ctx.call("tnfa_evaluate_noalloc", f.handle, C.c_void_p(X.data_ptr()), 600, 1, (C.c_int32 * 1)(1),
                   C.c_void_p(out.data_ptr()), ina._lib.OUT_F64, ina._lib.PREC_F64)


@pytest.mark.parametrize("dtype,size", [("f64", 8), ("f32", 4)])
def test_bond(ina, dtype, size):
    """8 rows of a child's bond and 64 bytes within 200 KB."""
    top = (200 * 1024 - 64) // (8 * size)
    s = ina.continuous_siteinds(ina.named_path_graph(3))
    a, b, c = s.layout.order
    L, rng = ina._lib, np.random.default_rng(2)
    X = np.array([0.0, 0.3, 0.9])
    d = np.floor(X[:, None] * [2, 4, 8]).astype(int) & 1
    for chi in (top, top + 1):
        ts = {a: rng.random((2, 1, 2)), b: rng.random((2, 2, chi)), c: rng.random((2, chi))}
        f = ina.ITensorNetworkFunction.from_tensors(s, ts, dtype=L.F32 if dtype == "f32" else L.F64)
        if chi > top:
            with pytest.raises(ina.TnfaError, match="UNSUPPORTED"):
                f.evaluate_batch(X, precision=dtype)
            continue
        ref = [ts[a][i, 0] @ ts[b][j] @ ts[c][k] for i, j, k in d]
        got = f.evaluate_batch(X, precision=dtype)
        # positive terms: a sum of chi of them in FP32, chi 2^-24
        assert np.max(np.abs(got / ref - 1)) < (4e-4 if dtype == "f32" else 1e-12)


@pytest.mark.parametrize("n", [5, 40000])
def test_bond_taken_from_above(ina, n):
    """Toward the digits below child a (bond 2) the vertex takes in its parent (bond
    3000) and child b (bond 300), together above the limit, neither above it alone."""
    V = 14
    verts = ["u", "v", "b"] + list(range(V))
    g = ina.NamedGraph(verts, [("u", "v"), ("v", "b"), ("v", 0)] + [(i, i + 1) for i in range(V - 1)])
    legs = {w: [] for w in ("u", "b")}
    legs["v"] = [ina.SiteLeg("v", 1, 1, 2, "real")]
    legs.update({i: [ina.SiteLeg(i, 1, i + 2, 2, "real")] for i in range(V)})
    s = ina.IndsNetworkMap(g, legs, False)
    rng, lay = np.random.default_rng(3), s.layout
    bond = {frozenset(("u", "v")): 3000, frozenset(("v", "b")): 300}
    ts = {}
    for i, w in enumerate(lay.order):
        nb = lay.neighbours_in_layout_order(i)
        shape = [bond.get(frozenset((w, lay.order[j])), 2) for j in nb]
        if lay.parent[i] < 0:
            shape = [1] + shape
        ts[w] = rng.random(([2] if legs[w] else []) + shape)
    assert lay.order[0] == "u"
    f = ina.ITensorNetworkFunction.from_tensors(s, ts)
    X = rng.random(n)
    got = f.evaluate_batch(X)
    d = np.floor(X[:, None] * 2.0 ** np.arange(1, V + 2)).astype(int) & 1
    row = ts[V - 1][d[:, V]]
    for i in range(V - 2, -1, -1):
        row = np.einsum("pab,pb->pa", ts[i][d[:, i + 1]], row)
    kids = [lay.order[c] for c in lay.children[lay.order.index("v")]]
    tv = ts["v"] if kids == ["b", 0] else np.swapaxes(ts["v"], 2, 3)
    mid = np.einsum("u,supq,p->sq", ts["u"].ravel(), tv, ts["b"].ravel())
    ref = np.einsum("pq,pq->p", mid[d[:, 0]], row)
    assert np.max(np.abs(got / ref - 1)) < 1e-12
