"""Small bonds near the point counts where tables take over from the walk: either
against the oracle, and calls whose many small tables cost more than the walk."""
import numpy as np
import pytest

import oracle as O
from _helpers import upload_oracle

pytestmark = pytest.mark.gpu

GRAPHS = {"path20": O.path_graph(20), "comb3x7": O.comb_tree_graph((3, 7)), "binary30": O.binary_tree_graph(30)}


def _case(ina, gname, chi, dtype, n):
    L, rng = ina._lib, np.random.default_rng(4000 + chi)
    so = O.siteinds(GRAPHS[gname], map_dimension=2)
    net = O.random_net(so, chi, rng, normalize=True)
    f, s = upload_oracle(ina, GRAPHS[gname], net, dtype=L.F32 if dtype == "f32" else L.F64)
    if dtype == "c128":
        f = f.astype(L.C128)
        f.scale_vertex(s.layout.order[1], 0.6 - 0.8j)
    return f, net, rng.random((n, 2)), (0.6 - 0.8j) if dtype == "c128" else 1.0


def _check(f, net, X, z, dtype):
    f.ctx.kernel_stats(reset=True)
    got = f.evaluate_batch(X, [1, 2], precision="f32" if dtype == "f32" else "f64")
    launches = sum(v["launches"] for v in f.ctx.kernel_stats(reset=True).values())
    pick = slice(None, None, max(1, len(X) // 1500))
    ref = O.evaluate_batch(net, X[pick], [1, 2]) * z
    assert np.max(np.abs(got[pick] - ref)) <= (2e-5 if dtype == "f32" else 1e-12) * np.max(np.abs(ref))
    return launches


@pytest.mark.parametrize("gname", list(GRAPHS))
@pytest.mark.parametrize("chi", [2, 3, 5, 8])
@pytest.mark.parametrize("dtype", ["f64", "f32", "c128"])
def test_either_side(ina, gname, chi, dtype):
    f, net, X, z = _case(ina, gname, chi, dtype, 64000)
    for n in (500, 2001, 8000, 16001, 32000, 64000):
        _check(f, net, X[:n], z, dtype)


@pytest.mark.parametrize("chi,dtype,n", [(2, "c128", 16000), (3, "f64", 16000), (4, "f64", 8000), (6, "f32", 32000)])
def test_trees_walk(ina, chi, dtype, n):
    assert _check(*_case(ina, "binary30", chi, dtype, n), dtype) == 1
