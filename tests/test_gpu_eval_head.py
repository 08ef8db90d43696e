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
