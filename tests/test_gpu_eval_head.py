"""The first levels of the tables, one block each: shared memory at the size of
a plain launch, and rows whose entries lie far apart."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_shared_memory_of_a_plain_launch(ina):
    """48 KB of tensors, tables and jobs, beside the kernel's own words (19 digits of
    base 4, these bonds and this many points give 49152 bytes).  FP32, positive
    tensors: 19 vertices x (20 terms + 2) roundings of 2^-24 < 3e-5."""
    V, base, n = 19, 4, 2630267
    link = [1] + [[20, 2, 6, 12][v % 4] for v in range(1, V)] + [1]
    s = ina.continuous_siteinds(ina.named_path_graph(V), base=base)
    rng = np.random.default_rng(0)
    ts = {v: rng.random([base, link[i]] + ([link[i + 1]] if i + 1 < V else [])) / link[i + 1]
          for i, v in enumerate(s.layout.order)}
    f = ina.ITensorNetworkFunction.from_tensors(s, ts, dtype=ina._lib.F32)
    X = rng.random((n, 1))
    got = f.evaluate_batch(X, precision="f32")
    some = np.arange(0, n, 10007)
    digits = (np.floor(X[some, 0][:, None] * float(base) ** np.arange(1, V + 1)) % base).astype(int)
    row = np.ones((len(some), 1))
    for i, v in enumerate(s.layout.order):
        t = ts[v] if i + 1 < V else ts[v][..., None]
        row = np.einsum("pa,pab->pb", row, t[digits[:, i]])
    assert np.max(np.abs(got[some] / row[:, 0] - 1)) < 3e-5


@pytest.mark.parametrize("dtype", ["f64", "f32", "c128"])
@pytest.mark.parametrize("sign", [-1, 1])
def test_entries_far_apart(ina, dtype, sign):
    """Two terms whose sizes differ by 2^96 (FP32) or 2^704 at the centre; the last
    digit leaves the smaller one alone.  The terms of either side of the centre
    carry 2^39 or 2^399, in turn.  16 vertices x 2 roundings and the centre's: 40 eps."""
    V, f32 = 16, dtype == "f32"
    step, side, eps = (2.0**-12, 2.0**39, 2.0**-24) if f32 else (2.0**-88, 2.0**399, 2.0**-53)
    s = ina.continuous_siteinds(ina.named_path_graph(V))
    ts, small = {}, []
    for i, v in enumerate(s.layout.order):
        # FP32 values, so that both networks hold the same ones
        x = np.float32([1.7, 1.3]) * np.float32(1 + 0.01 * i)
        big, low = np.ones(2), x * (step if i < V // 2 else 1.0)
        if i == V - 1:
            big = np.array([1.0, 0.0])
        scale = side**sign if i == 0 else side**-sign if i == V - 1 else 1.0
        small.append(np.float64(x))
        if i == 0:
            ts[v] = np.stack([big, low], -1)[:, None, :] * scale
        elif i < V - 1:
            ts[v] = np.stack([np.diag([big[d], low[d]]) for d in range(2)])
        else:
            ts[v] = np.stack([big, low], -1) * scale
    f = ina.ITensorNetworkFunction.from_tensors(s, ts, dtype=ina._lib.F32 if f32 else ina._lib.F64)
    if dtype == "c128":
        f = f.astype(ina._lib.C128)
    n = 1 << 21
    cells = np.random.default_rng(0).integers(0, 2 ** (V - 1), n) * 2 + 1
    got = f.evaluate_batch((cells / 2.0**V)[:, None], precision="f32" if f32 else "f64")
    ref = np.ones(n)
    for i in range(V):
        ref *= small[i][(cells >> (V - 1 - i)) & 1]
    assert np.max(np.abs(got / (ref * step ** (V // 2)) - 1)) < 40 * eps
