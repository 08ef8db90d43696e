"""The integral where rows are longer than a warp's lanes hold (1024 FP32, 512
FP64, 256 complex entries): lengths around whole passes of the lanes (4096 FP32
entries, half and a quarter of that), several rows to a task, several children,
messages in shared memory with and without an unscaled copy, and beyond it.
Positive tensors, bounds as in test_gpu_integrate_levels: 1e-12, FP32 (a lane
sums 2 vectors of a pass and 8 passes' worth in order) 1e-5."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("last", [260, 516, 1028, 1032, 2044, 2048, 2052, 4092, 4096, 4100, 6300, 12500, 26000])
@pytest.mark.parametrize("kids", [1, 2, 3])
@pytest.mark.parametrize("dtype", ["f32", "f64", "c128"])
def test_integrate_long_rows(ina, dtype, kids, last):
    L = ina._lib
    rng = np.random.default_rng(last + kids)
    dims = {1: [], 2: [37], 3: [3, 5]}[kids] + [last]
    verts = list(range(kids + 2))
    g = ina.NamedGraph(verts, [(0, 1)] + [(1, 2 + i) for i in range(kids)])
    s = ina.continuous_siteinds(g)
    o = s.layout.order
    up = 9
    ts = {o[0]: rng.random((2, 1, up)), o[1]: rng.random([2, up] + dims)}
    for v, d in zip(o[2:], dims):
        ts[v] = rng.random((2, d)) * 2.0 ** rng.integers(-30, 30)
    mid = ts[o[1]].sum(0)
    for v in reversed(o[2:]):
        mid = mid @ ts[v].sum(0)
    ref = ts[o[0]].sum((0, 1)) @ mid / 2.0 ** len(verts)
    f = ina.ITensorNetworkFunction.from_tensors(s, ts, dtype=L.F32 if dtype == "f32" else L.F64)
    if dtype == "c128":
        f = f.astype(L.C128)
        f.scale_vertex(o[0], 0.6 - 0.8j)
        ref = ref * (0.6 - 0.8j)
    assert abs(f.integrate() - ref) <= (1e-5 if dtype == "f32" else 1e-12) * abs(ref)
