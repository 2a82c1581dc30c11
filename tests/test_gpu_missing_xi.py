"""The count of third bodies whose bond was not evaluated (a neon atom among the
bond-order atoms, BondOrderFuncs.h:339-393) equals the oracle's, for short lists
within a tile of 32, beyond it, and beyond the slots of the forces on third bodies."""
import numpy as np
import pytest

from moleculardynamics_gb300 import lattice as lat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("a", [1.7, 1.3, 1.1])
def test_missing_count(eng, oracle, a):
    rng = np.random.default_rng(5)
    n = 216
    pos = np.zeros((n, 4))
    pos[:, :3] = lat.lattice(6, a, np.zeros((1, 3)), n) + rng.uniform(-0.05, 0.05, (n, 3))
    pos[::9, 3] = lat.SPECIES_NG
    vel = np.zeros((n, 3))
    cfg = eng.make_config(n_mb=n, use_lj=0, use_mb=1, mb_rs=3.5, mb_rcut=3.0, dt=0.5, species=0)
    with eng.Engine(cfg) as e:
        e.upload(pos, vel)
        e.begin(0.0)  # one evaluation
        got = e.stats()["missing_xi"]
        p, _ = e.download()
    nl = oracle.build_list(p.copy(), 3.5, oracle.ready_list(p, vel)[1])
    want = oracle.mb_forces(p, nl, n, oracle.settings(3.5, 3.0)[2])[1]
    oracle.free_list(nl)
    assert want > 0 and got == want
