"""The row scheme that a list build chooses by itself: ensembles of one-cell
replicas (minimum images), of larger ones and of both give the same bits as with
either scheme asked for."""
import numpy as np
import pytest

from moleculardynamics_gb300 import lattice as lat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nmin,nmax", [(160, 500), (256, 3000), (2000, 2500)])
def test_ensemble_defaults(eng, nmin, nmax):
    pos, vel, natoms, boxes, _ = lat.make_batch(6, nmin, nmax, seed=nmax)
    out = []
    for loads in (0, 1, 2):
        cfg = eng.make_config(dt=2.0, periodic=1, precision=eng.PREC_MIXED,
                              species=eng.SPECIES_ARGON, cluster_row_loads=loads)
        with eng.Batch(cfg, natoms, boxes) as b:
            b.upload(pos, vel)
            b.begin(0.0)
            b.step(30)
            out.append(b.download())
    for p, v in out[1:]:
        assert np.array_equal(p, out[0][0]) and np.array_equal(v, out[0][1])
