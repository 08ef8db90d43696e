"""Tensor slices that no point reads do not reach the gradient, finite or not:
the gradient is the one of the network with those slices at zero."""
import numpy as np
import pytest

import oracle as O
from _helpers import upload_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.inf, np.nan])
@pytest.mark.parametrize("at", range(8))
@pytest.mark.parametrize("gname", ["path8", "comb2x4", "binary8"])
@pytest.mark.parametrize("dtype", ["f64", "f32", "c128"])
def test_unread_slices(ina, dtype, gname, at, value):
    L = ina._lib
    graph = {"path8": O.path_graph(8), "comb2x4": O.comb_tree_graph((2, 4)), "binary8": O.binary_tree_graph(8)}[gname]
    f, s = upload_oracle(ina, graph, O.random_net(O.siteinds(graph), 5, np.random.default_rng(at), normalize=True))
    v = s.layout.order[at]
    digit = s.legs[v][0].digit
    rng = np.random.default_rng(1)
    X = rng.random(4000)
    X = X[(np.floor(X * 2**digit).astype(int) & 1) == 0]  # the first slice of v alone
    dout = rng.standard_normal(len(X))

    def gradient(fill):
        ts = {w: t.copy() for w, t in f.tensors().items()}
        ts[v][1] = fill
        g = ina.ITensorNetworkFunction.from_tensors(s, ts, dtype=L.F32 if dtype == "f32" else L.F64)
        return ina.evaluate_vjp(g.astype(L.C128) if dtype == "c128" else g, X[:, None], dout)

    got, ref = gradient(value), gradient(0.0)
    scale = max(np.max(np.abs(r)) for r in ref.values())
    for w in ref:  # the atomic sums of 2000 terms in another order
        assert np.max(np.abs(got[w] - ref[w])) <= (1e-4 if dtype == "f32" else 1e-11) * scale, w
