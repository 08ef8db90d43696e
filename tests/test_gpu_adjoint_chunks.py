"""The gradient of more points than the scratch holds at once: the same as the
sum over calls of one chunk each, and the tables' backward pass, which every
chunk repeats, over few chunks.  FP64 sums of 4 x 10^6 terms of either sign: a
few thousand roundings of the largest entry's size at most, 1e-10."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_vjp_chunks(ina):
    f = ina.rand_itn(ina.continuous_siteinds(ina.named_path_graph(48)), link_space=46, rng=3)
    rng = np.random.default_rng(0)
    n, part = 4_000_000, 500_000
    X, dout = rng.random((n, 1)), rng.standard_normal(n)
    f.ctx.kernel_stats(reset=True)
    whole = ina.evaluate_vjp(f, X, dout)
    launches = {k: v["launches"] for k, v in f.ctx.kernel_stats(reset=True).items()}
    # about 20 levels a chunk, and 616000 points of these bonds fit one
    assert 2 <= launches["digitize"] <= 16 and launches["adjoint_rows"] <= 24 * launches["digitize"]
    total = None
    for i in range(0, n, part):
        g = ina.evaluate_vjp(f, X[i:i + part], dout[i:i + part])
        total = g if total is None else {v: total[v] + g[v] for v in g}
    scale = max(np.max(np.abs(g)) for g in total.values())
    for v in total:
        assert np.max(np.abs(whole[v] - total[v])) <= 1e-10 * scale, v
