"""The plain FP64 form with a skin too thin to skip a step: the launches walk full
rows and refresh the compact ones, in a periodic box and within walls (where the
forces after a wall hit walk them too), at each number of lanes per atom.  Positions
and velocities equal the oracle's bit for bit, and trips are counted."""
import numpy as np
import pytest

from conftest import run_params
from moleculardynamics_gb300 import lattice as lat

pytestmark = pytest.mark.gpu

RC, RS = 8.0, 8.00005


def _run(eng, oracle, pos, vel, steps, vxcm, **kw):
    n = len(pos)
    cfg = eng.make_config(n_lj=n, dt=2.0, lj_rs=RS, lj_rcut=RC, energy_loss=0.5,
                          species=eng.SPECIES_ARGON, **kw)
    with eng.Engine(cfg) as e:
        e.upload(pos, vel)
        e.begin(vxcm)
        e.step(steps)
        p, v = e.download()
        st = e.stats()
    ref = oracle.run(run_params(n_lj=n, timesteps=steps, dt=2.0, lj_rs=RS, lj_rcut=RC,
                                energy_loss=0.5, vxcm=vxcm, species=eng.SPECIES_ARGON,
                                threads=oracle.max_threads(), **kw), pos, vel)
    assert np.array_equal(p, ref["pos"]) and np.array_equal(v, ref["vel"])
    assert st["wall_hits"] == ref["wall_hits"]
    return st


@pytest.mark.parametrize("n", [864, 2400, 6912, 13500])
def test_periodic(eng, oracle, n):
    cells = int(np.ceil((n / 4.0) ** (1.0 / 3.0)))
    pos, vel, L = lat.make_system("fcc", cells, 94.4, seed=9, natoms=n, noise=0.05)
    st = _run(eng, oracle, pos, vel, 6, 0.0, periodic=1, box=L)
    assert st["list_trips"] >= 5


def walls_system(n):
    # a few atoms fly at the walls, which lie 52.8 n^(1/3) angstrom away
    cells = int(np.ceil((n / 4.0) ** (1.0 / 3.0)))
    pos, vel, _ = lat.make_system("fcc", cells, 94.4, seed=5, natoms=n, a=6.5)
    fast = np.arange(0, n, max(40, n // 12))
    k = np.arange(len(fast))
    vel[fast, k % 3] += np.where(k // 3 % 2, -1.0, 1.0) * 0.45 * n ** (1.0 / 3.0)
    return pos, vel


@pytest.mark.parametrize("n", [32, 864, 2500, 6000])
def test_walls(eng, oracle, n):
    pos, vel = walls_system(n)
    st = _run(eng, oracle, pos, vel, 80, 0.0)
    assert st["list_trips"] > 75 and st["wall_hits"] > 0
