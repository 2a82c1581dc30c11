"""Animation frames around the size from which several threads copy them (8 MiB in
pieces of 4 MiB and the remainder): the float conversion of the state, for both
parts together and for either alone."""
import numpy as np
import pytest

from systems import argon_fcc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [299593, 299594, 449391, 1000003])
def test_large_frames(eng, n):
    pos, vel, L = argon_fcc(64 if n > 320000 else 43, natoms=n)
    cfg = eng.make_config(n_lj=n, periodic=1, box=L, precision=eng.PREC_MIXED)
    with eng.Engine(cfg) as e:
        e.set_animation(10, 1)
        e.upload(pos, vel)
        e.begin(0.0)
        e.step(1)  # the frame of step 0
        assert e.animation_count() == 1
        fp, fv = e.animation_frame(0)
        p1, v1 = np.zeros_like(fp), np.zeros_like(fv)
        assert e.lib.md_get_animation_frame(e.h, 0, p1.ctypes.data, None) == 0
        assert e.lib.md_get_animation_frame(e.h, 0, None, v1.ctypes.data) == 0
    assert np.array_equal(p1, fp) and np.array_equal(v1, fv)
    # unit-scale proof that every piece arrived: the state's own atoms, one step on
    assert np.abs(fp[:, :3] - pos[:, :3]).max() < 0.1 and np.array_equal(fp[:, 3], pos[:, 3])
    assert (fv != 0).any(1).all()
