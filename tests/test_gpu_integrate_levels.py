"""The integral level by level: row widths around the lane groups, leaves that
are summed by their parent and leaves that are not, vertices of many children,
levels of more vertices than one launch takes, and rows too long for the lanes
or for shared memory.  The tensors are positive, so that a relative error of a
few roundings per entry and vertex is the bound: (rows of a task + the lanes' sum)
x 14 vertices, or 10 x 90, times 2^-24 < 1e-4 in FP32, and 1e-12 in FP64 with its sums of
partial sums."""
import numpy as np
import pytest

import oracle as O
from _helpers import upload_oracle

pytestmark = pytest.mark.gpu

GRAPHS = {
    "path1": O.path_graph(1),
    "path2": O.path_graph(2),
    "path9": O.path_graph(9),
    "binary14": O.binary_tree_graph(14),
    "comb30x3": O.comb_tree_graph((30, 3)),
    "star": (list(range(1, 12)), [(1, 2), (2, 3), (2, 4), (2, 5), (2, 6), (2, 7), (2, 8), (8, 9), (9, 10), (9, 11)]),
}
CASES = [(g, chi, base) for g in ("path9", "binary14") for chi in (1, 2, 4, 7, 31, 32, 33, 40) for base in (2, 10)] + [
    ("path1", 1, 2), ("path1", 1, 10), ("comb30x3", 3, 2), ("comb30x3", 4, 10), ("star", 4, 2), ("star", 3, 10),
    ("path9", 64, 2), ("path9", 130, 2), ("path9", 260, 2), ("path9", 516, 2), ("path9", 1028, 2), ("path2", 6200, 2),
]


@pytest.mark.parametrize("gname,chi,base", CASES)
@pytest.mark.parametrize("dtype", ["f64", "f32", "c128"])
def test_integrate_levels(ina, gname, chi, base, dtype):
    L = ina._lib
    rng = np.random.default_rng(100 * chi + base)
    net = O.random_net(O.siteinds(GRAPHS[gname], base=base), chi, rng)
    for v in net.s.verts:
        t = net.T[v]
        net.T[v] = O.Tensor(rng.random(t.arr.shape) / chi, t.inds)
    f, s = upload_oracle(ina, GRAPHS[gname], net, dtype=L.F32 if dtype == "f32" else L.F64)
    phase = 1.0
    if dtype == "c128":
        f, phase = f.astype(L.C128), 0.6 - 0.8j
        f.scale_vertex(s.layout.order[0], phase)
    ref = O.integrate(net) * phase
    assert abs(f.integrate() - ref) <= (1e-4 if dtype == "f32" else 1e-12) * abs(ref)
