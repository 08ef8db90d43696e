"""The table schedule of batched evaluation (messages formed once per digit
combination, any centre edge, absorbed tensors) against the oracle, at point
counts on both sides of every table size and at tile edges."""
import numpy as np
import pytest

import oracle as O
from _helpers import rel_err, upload_oracle

pytestmark = pytest.mark.gpu

GRAPHS = {
    "path11": O.path_graph(11),
    "comb3x4": O.comb_tree_graph((3, 4)),
    "binary14": O.binary_tree_graph(14),
    # degrees up to 5: several kids per vertex on either side of a centre edge
    "star": (list(range(1, 14)), [(1, 2), (2, 3), (2, 4), (2, 5), (2, 6), (6, 7), (6, 8), (6, 9), (9, 10),
                                  (10, 11), (10, 12), (12, 13)]),
}


@pytest.mark.parametrize("gname", list(GRAPHS))
@pytest.mark.parametrize("chi,base,nd", [(1, 2, 1), (5, 3, 2), (17, 2, 2), (33, 2, 3)])
@pytest.mark.parametrize("dtype", ["f64", "f32", "c128"])
def test_tables_match_oracle(ina, monkeypatch, gname, chi, base, nd, dtype):
    if gname == "star" and chi > 5:
        chi = 6  # the largest tensor has chi^5 entries
    monkeypatch.setenv("TNFA_EVAL_FUSED", "0")  # small bonds through the tables too
    L = ina._lib
    rng = np.random.default_rng(1000 + chi)
    s_or = O.siteinds(GRAPHS[gname], map_dimension=nd, base=base)
    net = O.random_net(s_or, chi, rng, normalize=True)
    f, _ = upload_oracle(ina, GRAPHS[gname], net, dtype=L.F32 if dtype == "f32" else L.F64)
    if dtype == "c128":
        f = f.astype(L.C128)
        f.scale_vertex(f.s.layout.order[1], 0.6 - 0.8j)
    dims = list(range(1, nd + 1))
    X = rng.random((2100, nd))
    X[5], X[6], X[7] = 0.0, 1.0, 1.0 - 2.0**-53  # first, saturated and last grid points
    ref = O.evaluate_batch(net, X, dims) * ((0.6 - 0.8j) if dtype == "c128" else 1.0)
    tol = 2e-5 if dtype == "f32" else 1e-12
    scale = np.max(np.abs(ref))
    for n in (1, 2, 9, 33, 129, 2100):
        got = f.evaluate_batch(X[:n], dims, precision="f32" if dtype == "f32" else "f64")
        assert np.max(np.abs(got - ref[:n])) <= tol * scale, n
    assert rel_err(got, ref) < tol


@pytest.mark.parametrize("V,chi", [(9, 8), (12, 5), (17, 7), (24, 8)])
def test_walk_or_tables(ina, V, chi):
    """FP64 paths of bond 5 to 8 on both sides of the point count where tables
    take over from the walk, against the oracle."""
    rng = np.random.default_rng(3000 + V)
    net = O.random_net(O.siteinds(O.path_graph(V)), chi, rng, normalize=True)
    f, _ = upload_oracle(ina, O.path_graph(V), net)
    limit = int((4.6e-6 * V - 39e-6) * 5.4e11 / (64 * V))
    X = rng.random((limit + 40, 1))
    ref = O.evaluate_batch(net, X, [1])
    scale = np.max(np.abs(ref))
    for n in (limit - 33, limit, limit + 1, limit + 40):
        assert np.max(np.abs(f.evaluate_batch(X[:n]) - ref[:n])) <= 1e-12 * scale, n
