"""Layer-pair tracklets, whose candidates are judged by the first window and the
phi cut ahead of their rows: against the exact cuts on every candidate, by
module-map and by layer-pair segments, and on the same event scaled off its
modules; and the objects against the CPU restatement."""
import numpy as np
import pytest

from test_joins_gpu import check

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def world():
    from sdl_gb300 import Chain, build, synth
    build.build()
    det = synth.detector("full")
    ch = Chain(0)
    ch.upload_detector(det)
    return ch, det, synth.make_event(det, 1001, "full", n_pu=1000)


@pytest.mark.parametrize("flags", [2, 3, 2 | 4])
@pytest.mark.parametrize("scale", [(1.0, 1.0), (2.0, 1.0), (0.5, 1.0), (1.0, 3.0), (3.0, 0.5)])
def test_layer_tracklets(scale, flags, world, oracle_lib):
    ch, det, ev = world
    x, y, z = (np.float32(s) * v for s, v in ((scale[0], ev.x), (scale[0], ev.y), (scale[1], ev.z)))
    events = [type(ev)(**{**ev.__dict__, "x": x, "y": y, "z": z})]
    ch.set_events(events)
    ch.run(2, flags)
    r = ch.tl_phase_a_check()
    assert r["mismatches"] == 0 and r["settled"] + r["exact"] == r["candidates"] > 0, r
    if scale == (1.0, 1.0):
        ch.run(4, flags)
        check(ch, oracle_lib, det, events, flags)
