"""The error word of a synchronous call: a point outside the domain is reported
by its own call and by no other, past the point where the words are reused."""
import numpy as np
import pytest

import oracle as O
from _helpers import upload_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chi", [2, 20])
def test_error_word(ina, chi):
    net = O.random_net(O.siteinds(O.path_graph(8)), chi, np.random.default_rng(5))
    f, _ = upload_oracle(ina, O.path_graph(8), net)
    X = np.random.default_rng(6).random((300, 1))
    bad = X.copy()
    bad[-1] = -0.5
    ref = f.evaluate_batch(X)
    for i in range(1100):
        if i % 50 == 7:
            with pytest.raises(ina.TnfaError, match="coordinate"):
                f.evaluate_batch(bad)
        elif i % 50 == 33:
            with pytest.raises(ina.TnfaError, match="coordinate"):
                ina.evaluate_vjp(f, bad, np.ones(300), [1])
        else:
            assert np.array_equal(f.evaluate_batch(X), ref)
