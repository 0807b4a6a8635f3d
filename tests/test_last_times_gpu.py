"""The times of the last run stay readable when the next events need larger
buffers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("more", [1, 2, 300])
def test_times_after_new_events(more):
    from sdl_gb300 import Chain, build, synth
    build.build()
    det = synth.detector("barrel_flat")
    ev = synth.make_event(det, 998, "barrel_flat")
    ch = Chain(0)
    ch.upload_detector(det)
    ch.set_events([ev])
    ch.run(4)
    want = ch.times()
    assert np.all(want > 0) and want[:6].sum() <= want[6] * 1.05
    ch.set_events([ev] * more)
    assert np.array_equal(ch.times(), want)
    ch.run(4)
    assert np.all(ch.times() > 0)
