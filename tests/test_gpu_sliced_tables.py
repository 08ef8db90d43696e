"""Sliced tensor-core tables: levels of up to 16 vertices in launches of 8,
tiles cut along the parent's values (2 and 4 blocks of 32), and batches on
both sides of one wave of tiles, against the FP64 evaluation: a row computed
from a wrong tile, part or vertex is off by its own size, the slices by 1e-9
per point at most."""
import numpy as np
import pytest

import oracle as O
from _helpers import upload_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,chi,points", [(63, 64, 300), (63, 64, 9000), (31, 128, 300), (31, 128, 20000),
                                          (15, 128, 1)])
def test_sliced_tables(ina, n, chi, points):
    rng = np.random.default_rng(7 * n + chi)
    graph = O.binary_tree_graph(n)
    net = O.random_net(O.siteinds(graph, map_dimension=3), chi, rng, normalize=True)
    f, _ = upload_oracle(ina, graph, net)
    X = rng.random((points, 3))
    got = f.evaluate_batch(X, [1, 2, 3], precision="mixed")
    ref = f.evaluate_batch(X, [1, 2, 3], precision="f64")
    err = np.abs(got - ref) / np.abs(ref)
    assert np.max(err) < 1e-9
