"""The precision bond order at the block counts where its launches start early or
do not (152 and 1,216 blocks of four atoms): forces against the FP64 form (1e-4), and
a run within walls, where the gated launches start early and the others do not."""
import numpy as np
import pytest

from conftest import rel_rms
from moleculardynamics_gb300 import lattice as lat
from systems import DIAMOND_A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [608, 609, 4864, 4865])
def test_forces_and_steps(eng, n):
    cells = int(np.ceil((n / 8.0) ** (1.0 / 3.0)))
    pos, vel, _ = lat.make_system("diamond", cells, 300.0, seed=n, a=DIAMOND_A, noise=0.02,
                                  species=lat.SPECIES_N, mass_table="neon", natoms=n)
    out = []
    for prec in (eng.PREC_FP64, eng.PREC_MIXED):
        cfg = eng.make_config(n_mb=n, use_lj=0, use_mb=1, mb_rs=3.5, mb_rcut=3.0, dt=0.25,
                              species=0, precision=prec, output_timesteps=2)
        with eng.Engine(cfg) as e:
            e.upload(pos, vel)
            e.begin(0.0)
            f, _ = e.compute_forces()
            e.step(4)
            out.append((f, e.download()[1], e.records()))
    assert rel_rms(out[1][0], out[0][0]) < 1e-4
    assert rel_rms(out[1][1], out[0][1]) < 1e-4
    assert len(out[0][2]) == len(out[1][2]) == 2  # of the start and of step 2
    assert np.allclose(out[1][2][:, 3], out[0][2][:, 3], rtol=1e-4)
