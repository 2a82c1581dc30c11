"""Calls of growing sizes in turn on one surrogate: each of its buffers is as large
as the call needs, whichever call sized the others.  Results as from an object
that saw one call only (summation by atomics: 1e-5)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_calls_of_growing_sizes(eng):
    rng = np.random.default_rng(3)
    x = rng.standard_normal((1000, 32)).astype(np.float32)
    y = rng.standard_normal(1000).astype(np.float32)
    with eng.Surrogate(seed=3, cutoff=3.0) as s:
        for m, n in ((128, 300), (300, 1000), (31, 999)):
            s.loss_grad(x[:m], y[:m])
            t, d = s.net(x[:n])
            loss, g = s.loss_grad(x[:n], y[:n])
            with eng.Surrogate(seed=3, cutoff=3.0) as one:
                assert np.array_equal(one.params(), s.params())
                l1, g1 = one.loss_grad(x[:n], y[:n])
            with eng.Surrogate(seed=3, cutoff=3.0) as one:
                t1, d1 = one.net(x[:n])
            assert np.array_equal(t, t1) and np.array_equal(d, d1)
            assert abs(loss - l1) <= 1e-5 * l1
            assert np.abs(g - g1).max() <= 1e-5 * np.abs(g1).max()
