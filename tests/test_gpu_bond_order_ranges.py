"""The FP64 bond-order kernel where its paths change: short lists beyond a tile of
32 and beyond the 64 force slots, distances outside the fixed point's range (below
0.5 angstrom, beyond 8), and a bond without a third body, against the oracle
(1e-10 relative RMS, the bar of the bond-order forces)."""
import numpy as np
import pytest

from conftest import rel_rms
from moleculardynamics_gb300 import lattice as lat

pytestmark = pytest.mark.gpu


def _grid(n, a, noise, seed=5):
    rng = np.random.default_rng(seed)
    k = int(np.ceil(n ** (1.0 / 3.0)))
    pos = np.zeros((n, 4))
    pos[:, :3] = lat.lattice(k, a, np.zeros((1, 3)), n) + rng.uniform(-noise, noise, (n, 3))
    pos[:, 3] = rng.integers(0, 2, n)
    return pos


def _system(name):
    if name == "two tiles":  # up to 57 neighbours within the cutoff
        return _grid(216, 1.3, 0.05), 3.5, 3.0
    if name == "beyond the slots":  # up to 92
        return _grid(216, 1.1, 0.05), 3.5, 3.0
    if name == "close":
        pos = _grid(64, 1.7, 0.05)
        pos[1, :3] = pos[0, :3] + [0.2, 0.1, -0.25]
        return pos, 3.5, 3.0
    if name == "far":  # third bodies beyond 8 angstrom
        return _grid(125, 2.6, 0.1), 10.0, 9.5
    return _grid(int(name), 1.6, 0.05), 3.5, 3.0


@pytest.mark.parametrize("name", ["two tiles", "beyond the slots", "close", "far", "2", "3", "7"])
def test_forces(eng, oracle, name):
    pos, rs, rc = _system(name)
    n = len(pos)
    vel = np.zeros((n, 3))
    cfg = eng.make_config(n_mb=n, use_lj=0, use_mb=1, mb_rs=rs, mb_rcut=rc, dt=0.5, species=0)
    with eng.Engine(cfg) as e:
        e.upload(pos, vel)
        e.begin(0.0)
        p, _ = e.download()
        f, en = e.compute_forces()
    nl = oracle.build_list(p.copy(), rs, oracle.ready_list(p, vel)[1])
    fo, _, eo = oracle.mb_forces(p, nl, n, oracle.settings(rs, rc)[2], energy=True)
    oracle.free_list(nl)
    assert rel_rms(f, fo) < 1e-10
    assert abs(en[3] - eo[0]) <= 1e-10 * abs(eo[0])
