"""Animation frames of atom counts that are no multiple of four: a frame's
positions are stored on the device as float4, so both of its slots have to
start on a 16-byte boundary whatever the count.  Every frame is the float
conversion of the state at its step."""
import numpy as np
import pytest

from systems import argon_fcc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [857, 858, 859, 860])
@pytest.mark.parametrize("mixed", [False, True])
def test_frames_of_odd_counts(eng, n, mixed):
    pos, vel, L = argon_fcc(6, natoms=n, noise=0.05)
    cfg = eng.make_config(n_lj=n, periodic=1, box=L,
                          precision=eng.PREC_MIXED if mixed else eng.PREC_FP64)
    with eng.Engine(cfg) as e:
        e.set_animation(3, 4)
        e.upload(pos, vel)
        e.begin(0.0)
        states = [e.download()]
        # a frame holds the state after its step (steps 3, 6 and 9, counted from 0)
        for steps in (4, 3, 3):
            e.step(steps)
            states.append(e.download())
        assert e.animation_count() == 4
        for k, (p, v) in enumerate(states):
            fp, fv = e.animation_frame(k)
            assert np.array_equal(fp, p.astype(np.float32)), k
            assert np.array_equal(fv, v.astype(np.float32)), k
