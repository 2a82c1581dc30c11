"""Uploads between steps on the cluster path: the rows in place keep the scheme
that they were built with, whatever the next list build will choose.  Forces
against the FP64 form (1e-4 relative RMS, the precision form's bar)."""
import numpy as np
import pytest

from conftest import rel_rms
from systems import argon_fcc

pytestmark = pytest.mark.gpu


def _engine(eng, n, L, **kw):
    kw = dict(dict(precision=eng.PREC_MIXED, lj_kernel=eng.LJ_CLUSTER), **kw)
    return eng.Engine(eng.make_config(n_lj=n, dt=2.0, periodic=1, box=L, **kw))


def _types(pos):
    pos = pos.copy()
    pos[::7, 3] = 0
    pos[3::11, 3] = 1
    return pos


def _fp64_forces(eng, pos, vel, L, **kw):
    with _engine(eng, len(pos), L, **dict(kw, precision=eng.PREC_FP64, lj_kernel=0)) as e:
        e.upload(pos, vel)
        e.begin(0.0)
        return e.compute_forces()[0]


def test_upload_after_a_build_that_fell_back(eng):
    # a list radius of 19.5 angstrom stages more atoms than the register-prefetch
    # rows address: the build takes block tiles, before and after the upload
    pos, vel, L = argon_fcc(14, noise=0.05)
    kw = dict(lj_rs=19.5, lj_rcut=18.5, species=eng.SPECIES_ARGON)
    with _engine(eng, len(pos), L, **kw) as e:
        e.upload(pos, vel)
        e.begin(0.0)
        assert e.stats()["cluster_max_staged"] >= 4095
        p, v = e.download()
        e.upload(p, v)
        f = e.compute_forces()[0]
        e.step(2)
        p2, v2 = e.download()
        f2 = e.compute_forces()[0]
    assert rel_rms(f, _fp64_forces(eng, p, v, L, **kw)) < 1e-4
    assert rel_rms(f2, _fp64_forces(eng, p2, v2, L, **kw)) < 1e-4


@pytest.mark.parametrize("first", ["one", "three"])
def test_upload_changes_the_species(eng, first):
    # rows built for one species, forces for three, and the other way round
    pos, vel, L = argon_fcc(10, noise=0.1)
    order = (pos, _types(pos)) if first == "one" else (_types(pos), pos)
    with _engine(eng, len(pos), L, species=0) as e:
        e.upload(order[0], vel)
        e.begin(0.0)
        e.step(2)
        p, v = e.download()
        p[:, 3] = order[1][:, 3]
        e.upload(p, v)
        f = e.compute_forces()[0]
        e.step(2)
        p2, v2 = e.download()
        f2 = e.compute_forces()[0]
    assert rel_rms(f, _fp64_forces(eng, p, v, L, species=0)) < 1e-4
    assert rel_rms(f2, _fp64_forces(eng, p2, v2, L, species=0)) < 1e-4


def test_species_changed_twice_between_steps(eng):
    # The launches of one species hand out segments by counters that each step's
    # launch clears for the next one; the steps of three species between do not.
    # Blocks of one warp, more segments than can be resident (32 an SM): a counter
    # left behind would leave atoms out.  Every tiling gives the same bits.
    pos, vel, L = argon_fcc(36, noise=0.1)
    out = []
    for kw in (dict(cluster_row_loads=1), dict(cluster_threads=32, cluster_row_loads=2)):
        with _engine(eng, len(pos), L, species=0, **kw) as e:
            e.upload(pos, vel)
            e.begin(0.0)
            for one in (True, False, True, False, True):
                p, v = e.download()
                p[:, 3] = pos[:, 3] if one else _types(pos)[:, 3]
                e.upload(p, v)
                e.step(2)
            st = e.stats()
            out.append(e.download())
    assert st["cluster_segments"] > 32 * 152 and st["list_builds"] == 1
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
