"""The surrogate's pair kernels (descriptors, forces, residual transform) from no
neighbour to 56: even and odd counts (the last step of an even one is half a
step), more than a warp's 32, pairs across the periodic faces, against the CPU
restatement.  Bars: FP32 sums of up to 2,016 terms whose powers carry 16 roundings
(2e-6) and whose radial exponents four times that: 5e-5 of a feature's scale;
projections on a random direction 1e-4 of the sum of their terms' sizes."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
from moleculardynamics_gb300 import lattice as lat  # noqa: E402
from oracle import surrogate_ref as sref  # noqa: E402

pytestmark = pytest.mark.gpu


# atoms, spacing, box: up to 0, 1, 2, 6, 18, 23 and 56 neighbours within 3 angstrom
@pytest.mark.parametrize("n,a,L", [(8, 3.3, 20.0), (2, 1.5, 20.0), (3, 1.5, 20.0),
                                   (125, 2.8, 14.0), (125, 2.0, 12.0), (216, 1.75, 10.5),
                                   (125, 1.3, 12.0)])
def test_neighbour_counts(eng, n, a, L):
    rng = np.random.default_rng(n)
    pos = np.zeros((n, 4))
    k = int(np.ceil(n ** (1.0 / 3.0) - 1e-9))
    pos[:, :3] = lat.lattice(k, a, np.zeros((1, 3)), n) + rng.uniform(-0.05, 0.05, (n, 3))
    e3 = rng.standard_normal((n, 3)) * 0.1
    cfg = eng.make_config(n_mb=n, use_lj=0, use_mb=1, mb_rs=3.5, mb_rcut=3.0, dt=0.5, periodic=1,
                          box=L, species=0)
    hidden, istd, scale = 32, 0.1, 0.5
    with eng.Engine(cfg) as e, eng.Surrogate(seed=3, cutoff=3.0) as s:
        e.upload(pos, np.zeros((n, 3)))
        e.begin(0.0)
        s.set_model(1, hidden)
        s.normalisation(np.zeros(32), np.full(32, istd))
        par = s.head_params()
        par = s.head_params(par + rng.standard_normal(len(par)).astype(np.float32) * 0.05)
        s.head_scale(scale)
        p, _ = e.download()
        g = s.descriptors(e)
        q = s.desc_directional(e, e3)
        f, _ = s.forces(e)
    ref = sref.descriptors(p, L)
    assert np.all(np.abs(g - ref) <= 5e-5 * (np.abs(ref).max(0) + 1e-12))
    h = 1e-4
    pp, pm = p.copy(), p.copy()
    pp[:, :3] += h * e3
    pm[:, :3] -= h * e3
    qr = (sref.descriptors(pp, L) - sref.descriptors(pm, L)) / (2 * h)
    coef = sref.head_forward(par, ref * istd, hidden) * scale * istd
    terms = coef * qr
    assert abs((coef * q).sum() - terms.sum()) <= 1e-4 * np.abs(terms).sum() + 1e-12
    assert abs((f * e3).sum() + terms.sum()) <= 1e-4 * np.abs(terms).sum() + 1e-12


@pytest.mark.parametrize("n", [1, 127, 128, 129])
def test_network_row_counts(eng, n):
    # the ends of the tensor-core tiles of 128 rows; odd counts (the gradient rows
    # leave in 16-byte stores); bars as for the whole tiles
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, 32)).astype(np.float32)
    y = rng.standard_normal(n).astype(np.float32)
    v = rng.standard_normal((n, 32)).astype(np.float32) * 0.1
    with eng.Surrogate(cutoff=3.0) as s:
        p = s.params(rng.standard_normal(s.nparams).astype(np.float32) * 0.3)
        t, d = s.net(x)
        loss, g = s.loss_grad(x, y)
        gf = s.force_grad(x, v)
    tr, dr = sref.net(p, x)
    assert np.abs(t - tr).max() <= 2e-3 * np.abs(tr).max()
    assert np.abs(d - dr).max() <= 2e-3 * np.abs(dr).max()
    lr, gr = sref.loss_grad(p, x, y)
    assert abs(loss - lr) <= 1e-4 * lr
    for got, ref in ((g, gr), (gf, sref.force_grad(p, x, v))):
        for a, b in ((0, 2048), (2048, 2112), (2112, 6208), (6208, 6272), (6272, 6336)):
            assert np.abs(got[a:b] - ref[a:b]).max() <= 5e-3 * np.abs(ref[a:b]).max() + 1e-30


@pytest.mark.parametrize("hidden", [32, 64, 128])
@pytest.mark.parametrize("n", [1, 33, 129])
def test_head_row_counts(eng, n, hidden):
    # the direct head's gradient comes from the activations its forward keeps (FP32)
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
