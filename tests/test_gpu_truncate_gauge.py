"""Truncation where the tensors behind a bond say nothing about the weight in
the function: sums whose blocks differ by many orders of magnitude at a vertex
(an exponential's amplitude is spread over all vertices), and a summand whose
scale sits on one vertex.

Unless the cutoff is larger, 1e-24 leaves sqrt(20 bonds x 1e-24) < 5e-12 of the
norm and the factorisations a few n eps per bond, below 1e-11: 1e-10.  A first
difference loses 2 |f| / |f(x + d) - f(x - d)| < 2^20 / 10 of that rounding:
20 bonds x 10 eps x 1e5 = 2e-9, 1e-8."""
import numpy as np
import pytest

import oracle as O
from _helpers import upload_oracle

pytestmark = pytest.mark.gpu

L = 20
X = np.linspace(0.0, 1.0, 4001, endpoint=False)


def _cosh(ina, k):
    s = ina.continuous_siteinds(ina.named_path_graph(L))
    f = ina.cosh_itensornetwork(s, k=float(k), a=-k / 2)
    return s, f, np.cosh(k * np.floor(X * 2**L) / 2**L - k / 2)


def _l2(got, ref):
    return np.linalg.norm(got - ref) / np.linalg.norm(ref)


@pytest.mark.parametrize("k", [10, 44, 60, 100])
@pytest.mark.parametrize("cutoff", [0.0, 1e-24])
def test_truncate_cosh(ina, k, cutoff):
    _, f, ref = _cosh(ina, k)
    assert _l2(f.evaluate_batch(X), ref) < 1e-12
    assert _l2(ina.truncate(f, cutoff=cutoff).evaluate_batch(X), ref) < 1e-10


@pytest.mark.parametrize("k", [10, 44, 100])
@pytest.mark.parametrize("op", ["shift", "derivative"])
def test_operate_cosh(ina, k, op):
    s, f, _ = _cosh(ina, k)
    o = ina.forward_shift_op(s) if op == "shift" else ina.first_derivative_operator(s)
    ref = ina.operate_exact(o, f).evaluate_batch(X)
    got = ina.operate(o, f, cutoff=1e-24).evaluate_batch(X)
    assert _l2(got, ref) < (1e-10 if op == "shift" else 1e-8)


def _lopsided(ina, seed, dtype):
    """f + g with f's scale 1e-20 at the last vertex and 1e20 at the root; the values of f + g."""
    graph, rng = O.path_graph(12), np.random.default_rng(seed)
    fs, vals = [], 0
    for i in range(2):
        f, s = upload_oracle(ina, graph, O.random_net(O.siteinds(graph), 3, rng, normalize=True))
        if dtype == "c128":
            f = f.astype(ina._lib.C128)
            f.scale_vertex(s.layout.order[0], 0.6 - 0.8j)
        vals = vals + f.evaluate_batch(X)
        fs.append((f, s))
    f, s = fs[0]
    f.scale_vertex(s.layout.order[-1], 1e-20)
    f.scale_vertex(s.layout.order[0], 1e20)
    return f + fs[1][0], vals


@pytest.mark.parametrize("dtype", ["f64", "c128"])
@pytest.mark.parametrize("cutoff,tol", [(0.0, 1e-10), (1e-24, 1e-10), (1e-12, 1e-5)])
def test_truncate_lopsided(ina, dtype, cutoff, tol):
    h, ref = _lopsided(ina, 5, dtype)
    assert _l2(ina.truncate(h, cutoff=cutoff).evaluate_batch(X), ref) < tol


# the batched sweep may leave 1e-13 sqrt(40 columns) of every column per bond: 20 bonds, 2e-11
@pytest.mark.parametrize("precision", ["f64", "mixed"])
@pytest.mark.parametrize("cutoff", [0.0, 1e-24])
def test_truncate_batched_cosh(ina, precision, cutoff):
    nets = [_cosh(ina, k)[1:] for k in (10, 44, 60, 100)]
    gs = ina.truncate_batched([f for f, _ in nets], cutoff=cutoff, precision=precision)
    for g, (_, ref) in zip(gs, nets):
        assert _l2(g.evaluate_batch(X), ref) < 1e-10


def test_operate_batched_cosh(ina):
    nets = [_cosh(ina, k) for k in (10, 44, 100)]
    ops = [ina.forward_shift_op(s) for s, _, _ in nets]
    for (_, f, _), o, g in zip(nets, ops, ina.operate_batched(ops, [f for _, f, _ in nets], cutoff=1e-24)):
        assert _l2(g.evaluate_batch(X), ina.operate_exact(o, f).evaluate_batch(X)) < 1e-10


@pytest.mark.parametrize("dtype", ["f64", "c128"])
@pytest.mark.parametrize("cutoff,tol", [(0.0, 1e-10), (1e-12, 1e-5)])
def test_truncate_batched_lopsided(ina, dtype, cutoff, tol):
    nets = [_lopsided(ina, 5 + i, dtype) for i in range(3)]
    for g, (_, ref) in zip(ina.truncate_batched([h for h, _ in nets], cutoff=cutoff), nets):
        assert _l2(g.evaluate_batch(X), ref) < tol


@pytest.mark.parametrize("mindim", [3, 5, 8, 20])
@pytest.mark.parametrize("precision,dtype", [("f64", "f64"), ("f64", "c128"), ("mixed", "f64")])
@pytest.mark.parametrize("batched", [False, True])
def test_mindim_of_a_low_rank(ina, mindim, precision, dtype, batched):
    graph = O.path_graph(8)
    f, _ = upload_oracle(ina, graph, O.random_net(O.siteinds(graph), 2, np.random.default_rng(7), normalize=True))
    if dtype == "c128":
        f = f.astype(ina._lib.C128)
    g = f + f
    h = g + g  # rank 2, stored with bonds of 8
    kw = dict(cutoff=1e-20, mindim=mindim, precision=precision)
    for t in ina.truncate_batched([h, h], **kw) if batched else [ina.truncate(h, **kw)]:
        assert [t.linkdims()[e] for e in h.linkdims()] == [min(mindim, 8, 2**i, 2 ** (8 - i)) for i in range(1, 8)]
        assert _l2(t.evaluate_batch(X), 4 * f.evaluate_batch(X)) < 1e-9


@pytest.mark.parametrize("value", [np.inf, np.nan])
@pytest.mark.parametrize("at", [0, 3, 7])
@pytest.mark.parametrize("chi", [4, 40])
def test_not_finite(ina, value, at, chi):
    """A batch refuses entries that are not finite; a single call answers with them."""
    graph = O.path_graph(8)
    f, s = upload_oracle(ina, graph, O.random_net(O.siteinds(graph, base=3), chi, np.random.default_rng(0)))
    ts = {v: t.copy() for v, t in f.tensors().items()}
    ts[s.layout.order[at]].flat[1] = value
    f = ina.ITensorNetworkFunction.from_tensors(s, ts)
    with pytest.raises(ina.TnfaError, match="TNFA_ERR_DOMAIN"):
        ina.truncate_batched([f, f], cutoff=1e-20)
    assert not np.any(np.isfinite(ina.truncate(f, cutoff=1e-20).evaluate_batch(X[::100])))
