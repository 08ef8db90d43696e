"""The dense kernels behind truncation and linsolve at the sizes where their
tiles, lane groups and storage change: f + f truncated back to f's bonds
(rank-revealing QR, QR, Jacobi, products: bonds 1 to 130, tall and square,
one network and several, real, complex and mixed) and full-rank linsolve
(local systems of 4 to 1024 unknowns, in shared memory up to 165).

Truncating at 1e-24 leaves sqrt(5 bonds x 1e-24) = 2e-12 of the norm; the
factorisations add a few n eps per bond, below 1e-11 for n = 260: 1e-10 of the
rms value.  linsolve: condition number about 65, so 65 n eps < 2e-11 at n = 1024."""
import numpy as np
import pytest

import oracle as O
from _helpers import upload_oracle

pytestmark = pytest.mark.gpu


def _sum(ina, graph, base, chi, seed, dtype):
    net = O.random_net(O.siteinds(graph, base=base), chi, np.random.default_rng(seed), normalize=True)
    f, s = upload_oracle(ina, graph, net)
    if dtype == "c128":
        f = f.astype(ina._lib.C128)
        f.scale_vertex(s.layout.order[0], 0.6 - 0.8j)
    return f


@pytest.mark.parametrize("chi", [1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 48, 63, 64, 65, 127, 128, 130])
@pytest.mark.parametrize("mode", ["f64", "c128", "mixed", "several", "comb"])
def test_truncate_shapes(ina, chi, mode):
    if mode == "comb" and chi > 33:
        chi = 34
    graph, base = (O.comb_tree_graph((2, 3)), 3) if mode == "comb" else (O.path_graph(6), 6)
    fs = [_sum(ina, graph, base, chi, 50 + i, mode) for i in range(5 if mode == "several" else 1)]
    sums = [f + f for f in fs]
    if mode == "several":
        gs = ina.truncate_batched(sums, cutoff=1e-24)
    else:
        gs = [ina.truncate(sums[0], cutoff=1e-24, precision="mixed" if mode == "mixed" else "f64")]
    X = np.random.default_rng(9).random(400)
    for f, g in zip(fs, gs):
        assert g.maxlinkdim() <= chi
        ref = 2 * f.evaluate_batch(X)
        err = np.max(np.abs(g.evaluate_batch(X) - ref)) / np.sqrt(np.mean(np.abs(ref) ** 2))
        assert err < 1e-10, err


@pytest.mark.parametrize("L", [2, 3, 4, 5, 6, 7, 8, 9, 10])
def test_linsolve_shapes(ina, L):
    s = ina.continuous_siteinds(ina.named_path_graph(L))
    b = ina.truncate(ina.rand_itn(s, link_space=2 ** (L // 2), rng=11), cutoff=0.0)
    a1 = -16.0 / 4.0**L
    x = ina.linsolve(ina.second_derivative_operator(s), b, b, a0=1.0, a1=a1, nsweeps=2, cutoff=0.0, tol=0.0)
    n = 2**L
    M = 4.0**L * (np.diag(np.ones(n - 1), 1) + np.diag(np.ones(n - 1), -1) - 2 * np.eye(n))
    xs = np.arange(n) / n
    ref = np.linalg.solve(np.eye(n) + a1 * M, b.evaluate_batch(xs))
    assert np.linalg.norm(x.evaluate_batch(xs) - ref) < 1e-10 * np.linalg.norm(ref)
