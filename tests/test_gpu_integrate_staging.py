"""The integral where the children's messages just fit the shared memory of a
launch, and just do not: 48 KB less 256 bytes is 4074 FP32, 6112 FP64 and 3056
complex entries, of one child or of two.  Positive tensors: a few roundings per
entry and vertex (8192 entries, warps' and tasks' sums: below 64 x 2^-24 in FP32,
1e-12 in FP64)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,chi", [("f32", c) for c in (4073, 4074, 4075, 4090, 4096, 4097)] +
                         [("f64", c) for c in (6111, 6112, 6113, 6144, 6145)] +
                         [("c128", c) for c in (3055, 3056, 3057, 3072, 3073)])
@pytest.mark.parametrize("kids", [1, 2])
def test_integrate_staging(ina, dtype, chi, kids):
    L = ina._lib
    rng = np.random.default_rng(chi)
    if kids == 1:
        s = ina.continuous_siteinds(ina.named_path_graph(2))
        a, b = s.layout.order
        ts = {a: rng.random((2, 1, chi)), b: rng.random((2, chi))}
        ref = ts[a].sum((0, 1)) @ ts[b].sum(0) / 4
    else:
        g = ina.NamedGraph([1, 2, 3], [(1, 2), (1, 3)])
        s = ina.continuous_siteinds(g)
        a, b, c = s.layout.order
        d = chi - 8  # the sum of both bonds is what counts
        ts = {a: rng.random((2, 1, d, 8)), b: rng.random((2, d)), c: rng.random((2, 8))}
        ref = ts[b].sum(0) @ ts[a].sum((0, 1)) @ ts[c].sum(0) / 8
    f = ina.ITensorNetworkFunction.from_tensors(s, ts, dtype=L.F32 if dtype == "f32" else L.F64)
    if dtype == "c128":
        f = f.astype(L.C128)
        f.scale_vertex(a, 0.6 - 0.8j)
        ref = ref * (0.6 - 0.8j)
    assert abs(f.integrate() - ref) <= (4e-6 if dtype == "f32" else 1e-12) * abs(ref)
