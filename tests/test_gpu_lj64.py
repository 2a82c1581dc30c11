"""The plain FP64 LJ kernel at the sizes where its lanes per atom change, with
rows longer than its queue, with tripped skins and with three species: forces
equal to the oracle's bit for bit, energies within 1e-12."""
import numpy as np
import pytest

from moleculardynamics_gb300 import lattice as lat

pytestmark = pytest.mark.gpu

RS, RC = 9.534, 8.5125


def _check(eng, oracle, pos, vel, L, periodic, table="argon", rs=RS, rc=RC, nlj=None):
    n = len(pos)
    species = eng.SPECIES_ARGON if table == "argon" else eng.SPECIES_NEON
    cfg = eng.make_config(n_lj=n, dt=2.0, lj_rs=rs, lj_rcut=rc, species=species,
                          periodic=int(periodic), box=L if periodic else 0.0)
    with eng.Engine(cfg) as e:
        e.upload(pos, vel)
        e.begin(0.0)
        p, _ = e.download()
        f, en = e.compute_forces()
    rcsq = oracle.settings(rs, rc)[2]
    if periodic:
        nl = oracle.build_list(p.copy(), rs, L, periodic=True)
    else:
        nl = oracle.build_list(p.copy(), rs, oracle.ready_list(p, vel)[1])
    ref = oracle.lj_forces(p, nl, rcsq, species)
    oracle.free_list(nl)
    assert np.array_equal(f, ref)
    return en


@pytest.mark.parametrize("n", [1, 2, 31, 33, 760, 761, 2432, 2433, 2584, 2585, 4864, 4865, 9728,
                               9729, 12920, 12921])
def test_lane_counts(eng, oracle, n):
    cells = max(6, int(np.ceil((n / 4.0) ** (1.0 / 3.0))))
    pos, vel, L = lat.make_system("fcc", cells, 94.4, seed=n, natoms=n, noise=0.1)
    _check(eng, oracle, pos, vel, L, periodic=n % 2 == 0 and n > 100)


@pytest.mark.parametrize("n", [500, 5000])
def test_rows_longer_than_the_queue(eng, oracle, n):
    # twice the edge's density eightfold: about 430 atoms within the cutoff
    pos, vel, L = lat.make_system("fcc", 11, 94.4, seed=n, natoms=n, noise=0.05, a=2.9)
    _check(eng, oracle, pos, vel, L, periodic=False)


def test_three_species_and_far_coordinates(eng, oracle):
    rng = np.random.default_rng(4)
    pos, vel, L = lat.make_system("fcc", 7, 94.4, seed=4, noise=0.1, mass_table="neon")
    pos[:, 3] = rng.integers(0, 3, len(pos))
    _check(eng, oracle, pos, vel, L, periodic=False, table="neon")
    # a far offset widens the screen (its FP32 copies are coarse there)
    pos[:, :3] += np.array([60.0, -75.0, 90.0])
    _check(eng, oracle, pos, vel, L, periodic=False, table="neon")


@pytest.mark.parametrize("scale", [2.0 ** -16, 2.0 ** 17])
def test_distances_beyond_the_integer_range(eng, oracle, scale):
    # squared distances below 2^-30 (forces overflow to infinity and beyond in
    # the reference's formula, and stay finite at the upper end)
    pos = np.zeros((2, 4))
    pos[1, :3] = np.array([0.7, 0.4, 0.2]) * scale
    pos[:, 3] = lat.SPECIES_NG
    rs, rc = (RS, RC) if scale < 1 else (3.0 * scale, 2.0 * scale)
    cfg = eng.make_config(n_lj=2, lj_rs=rs, lj_rcut=rc)
    with eng.Engine(cfg) as e:
        e.upload(pos, np.zeros((2, 3)))
        if scale < 1:
            # the initial forces are huge but the positions stay as they are
            e.begin(0.0)
        else:
            pos[:, :3] -= pos[:, :3].mean(0)
            e.upload(pos, np.zeros((2, 3)))
            try:
                e.begin(0.0)
            except eng.EngineError:
                pytest.skip("walls clamp so far a pair")
        p, _ = e.download()
        f, _ = e.compute_forces()
    rcsq = oracle.settings(rs, rc)[2]
    nl = oracle.build_list(p.copy(), rs, oracle.ready_list(p, np.zeros((2, 3)))[1])
    ref = oracle.lj_forces(p, nl, rcsq, 1)
    oracle.free_list(nl)
    assert np.array_equal(f, ref, equal_nan=True)


def test_tripped_skin_refreshes_rows(eng, oracle):
    """A skin too thin to skip any step: every step walks full rows."""
    pos, vel, L = lat.make_system("fcc", 6, 94.4, seed=9, noise=0.05)
    n = len(pos)
    out = []
    for rs in (RC + 1e-4, RS):
        cfg = eng.make_config(n_lj=n, dt=2.0, lj_rs=rs, lj_rcut=RC, periodic=1, box=L)
        with eng.Engine(cfg) as e:
            e.upload(pos, vel)
            e.begin(0.0)
            e.step(3)
            out.append(e.download() + (e.stats()["list_trips"],))
    assert out[0][2] >= 0
    assert np.allclose(out[0][0], out[1][0], rtol=0, atol=1e-10)


@pytest.mark.parametrize("n,a", [(1, 5.26), (2, 5.26), (33, 5.26), (129, 5.26), (500, 2.9),
                                 (864, 5.26)])
def test_rows_of_the_caller(eng, oracle, n, a):
    # rows that end inside, at and after a chunk of 32; longer than the queue
    pos, vel, _ = lat.make_system("fcc", 6, 94.4, seed=n, natoms=n, noise=0.05, a=a)
    sh = eng.Shim(species=eng.SPECIES_ARGON)
    nl = oracle.build_list(pos.copy(), RS, 40.0)
    rcsq = oracle.settings(RS, RC)[2]
    rows, nls, nlargest = sh.build_neighbor_list(pos, RS, RC, 40.0)
    assert nls == nl.nlistsize and nlargest == nl.nlargest
    if nls:
        assert np.array_equal(rows, nl.rows)
    f = sh.lennard_jones_forces(pos, rows, nlargest, rcsq)
    assert np.array_equal(f, oracle.lj_forces(pos, nl, rcsq, eng.SPECIES_ARGON))
    assert not sh.lennard_jones_forces(pos, rows, nlargest, -1.0).any()
    oracle.free_list(nl)
