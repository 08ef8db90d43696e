"""The table schedule of evaluation's vector-Jacobian product: a batch large
enough for tables on every subtree against the oracle's gradient on a few
points, and against the sum over small batches (whose vertices run point by
point)."""
import numpy as np
import pytest

import oracle as O
from _helpers import oracle_to_tensors, upload_oracle

pytestmark = pytest.mark.gpu

GRAPHS = {
    "path11": O.path_graph(11),
    "comb3x4": O.comb_tree_graph((3, 4)),
    "binary14": O.binary_tree_graph(14),
    # degrees up to 5: vertices that never have a table
    "star": (list(range(1, 14)), [(1, 2), (2, 3), (2, 4), (2, 5), (2, 6), (6, 7), (6, 8), (6, 9), (9, 10),
                                  (10, 11), (10, 12), (12, 13)]),
}


@pytest.mark.parametrize("gname", list(GRAPHS))
@pytest.mark.parametrize("chi,base,nd", [(1, 2, 1), (5, 3, 2), (17, 2, 2), (33, 2, 2)])
@pytest.mark.parametrize("dtype", ["f64", "f32", "c128"])
def test_vjp_tables(ina, gname, chi, base, nd, dtype):
    if gname == "star" and chi > 5:
        chi = 6
    L = ina._lib
    rng = np.random.default_rng(2000 + chi)
    s_or = O.siteinds(GRAPHS[gname], map_dimension=nd, base=base)
    net = O.random_net(s_or, chi, rng, normalize=True)
    f, s = upload_oracle(ina, GRAPHS[gname], net, dtype=L.F32 if dtype == "f32" else L.F64)
    dims = list(range(1, nd + 1))
    n = 1500
    X = rng.random((n, nd))
    dout = rng.standard_normal(n)
    dout[3] = 0.0
    tol = 1e-4 if dtype == "f32" else 1e-11  # sums of 1500 terms
    few = ina.evaluate_vjp(f, X[:6], dout[:6], dims)
    grads = O.gradient(net, X[:6], dims, dout[:6])
    ref = oracle_to_tensors(O.Net(net.s, {v: O.Tensor(grads[v], net.T[v].inds) for v in net.s.verts}, net.link), s)
    scale = max(np.max(np.abs(r)) for r in ref.values())
    for v in s.layout.order:
        assert np.max(np.abs(few[v] - ref[v])) <= tol * scale, v
    if dtype == "c128":
        f = f.astype(L.C128)
        f.scale_vertex(s.layout.order[0], 0.6 - 0.8j)
    whole = ina.evaluate_vjp(f, X, dout, dims)
    parts = [ina.evaluate_vjp(f, X[i:i + 100], dout[i:i + 100], dims) for i in range(0, n, 100)]
    total = {v: sum(p[v] for p in parts) for v in s.layout.order}
    scale = max(np.max(np.abs(r)) for r in total.values())
    for v in s.layout.order:
        assert np.max(np.abs(whole[v] - total[v])) <= tol * scale, v
