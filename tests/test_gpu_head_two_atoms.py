"""The direct head's forward with two atoms a lane (from 9,729 atoms, widths 32 and
64): full blocks of 64 atoms and last ones of 1, 33 and 63.  The gradient comes from
the activations that the forward keeps, against the CPU restatement (FP32 sums
over the rows in another order: 1e-4 of the largest)."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
from oracle import surrogate_ref as sref  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden", [32, 64])
@pytest.mark.parametrize("n", [9728, 9729, 9761, 9791, 9792])
def test_two_atoms_a_lane(eng, n, hidden):
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, 32)).astype(np.float32)
    v = rng.standard_normal((n, 32)).astype(np.float32)
    with eng.Surrogate(seed=4, cutoff=3.0) as s:
        s.set_model(1, hidden)
        p = s.head_params()
        p = s.head_params(p + rng.standard_normal(len(p)).astype(np.float32) * 0.05)
        g = s.head_grad(x, v)
    gr = sref.head_grad(p, x, v, hidden)
    assert np.abs(g - gr).max() < 1e-4 * np.abs(gr).max()
