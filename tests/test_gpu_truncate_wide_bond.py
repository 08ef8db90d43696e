"""Truncation of one path whose bond exceeds the rank-revealing QR's 1024
reflectors: the sweeps run once, without it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chi", [1024, 1040])
def test_wide_bond(ina, chi):
    s = ina.continuous_siteinds(ina.named_path_graph(4), base=40)
    rng = np.random.default_rng(chi)
    dims = [1, 40, chi, 40, 1]
    ts = {v: rng.standard_normal([40, dims[i]] + ([dims[i + 1]] if i < 3 else [])) / np.sqrt(dims[i + 1])
          for i, v in enumerate(s.layout.order)}
    f = ina.ITensorNetworkFunction.from_tensors(s, ts)
    f.ctx.kernel_stats(reset=True)
    g = ina.truncate(f, cutoff=1e-20)
    launches = {k: v["launches"] for k, v in f.ctx.kernel_stats(reset=True).items()}
    # one QR per bond in the first sweep, at most two per bond in front of its SVD
    assert launches["qr_f64"] <= 9, launches
    assert launches["svd_f64"] == 3, launches
    X = rng.random((500, 1))
    ref = f.evaluate_batch(X)
    assert np.max(np.abs(g.evaluate_batch(X) - ref)) < 1e-9 * np.max(np.abs(ref))
