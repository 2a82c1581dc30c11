"""A frame is the float conversion of the state that it was taken of, for both parts
together and for either alone, below and above the size from which several threads
copy it (8 MiB in pieces of 4 MiB and the remainder)."""
import numpy as np
import pytest

from systems import argon_fcc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1001, 299594, 449391, 1000003])
@pytest.mark.parametrize("fp64", [False, True])
def test_frame_is_the_state(eng, n, fp64):
    if fp64 and n > 300000:
        pytest.skip("the copy does not depend on the form")
    pos, vel, L = argon_fcc(64 if n > 320000 else (43 if n > 1001 else 7), natoms=n)
    cfg = eng.make_config(n_lj=n, periodic=1, box=L,
                          precision=eng.PREC_FP64 if fp64 else eng.PREC_MIXED)
    with eng.Engine(cfg) as e:
        e.set_animation(3, 2)
        e.upload(pos, vel)
        e.begin(0.0)  # the first frame
        states = [e.download()]
        e.step(4)     # steps 0 to 3: the frame of step 3, the last one
        states.append(e.download())
        assert e.animation_count() == 2
        for k, (p, v) in enumerate(states):
            fp, fv = e.animation_frame(k)
            p1, v1 = np.full_like(fp, 7.0), np.full_like(fv, 7.0)
            assert e.lib.md_get_animation_frame(e.h, k, p1.ctypes.data, None) == 0
            assert e.lib.md_get_animation_frame(e.h, k, None, v1.ctypes.data) == 0
            for got in (fp, p1):
                assert np.array_equal(got, p.astype(np.float32)), k
            for got in (fv, v1):
                assert np.array_equal(got, v.astype(np.float32)), k
