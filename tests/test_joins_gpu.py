"""The triplets and track candidates as joins: geometries whose connection
lists repeat modules (the reference's nested loops then make segments, triplets
and track candidates several times), runs split between any two stages, and
batches on both sides of the size where the prefix sums change their tiles,
against the CPU restatement."""
import copy

import numpy as np
import pytest

from test_gpu_parity import describe

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from sdl_gb300 import Chain, build
    build.build()
    return Chain(0)


def check(gpu, oracle_lib, det, events, flags):
    orc = oracle_lib.Oracle(det)
    for e, ev in enumerate(events):
        ref, cnt, _ = orc.run(ev, mode=flags)
        for s in range(5):
            got = gpu.objects(s, e)
            assert oracle_lib.digest(got) == oracle_lib.digest(ref[s]), describe(oracle_lib, got, ref[s], s)
        assert np.array_equal(gpu.counters(e), cnt)


def repeated(det):
    """`det` with every third connection list ending in its first module again, every fifth twice over"""
    out = copy.copy(det)
    out.conn = {}
    for k, (d, v) in enumerate(sorted(det.conn.items())):
        out.conn[d] = list(v) + (list(v) if k % 5 == 0 else list(v[:1]) if k % 3 == 0 else [])
    return out


@pytest.mark.parametrize("flags", [0, 32, 64, 128, 32 | 64])
def test_repeated_connections(flags, gpu, oracle_lib):
    from sdl_gb300 import synth
    det = repeated(synth.detector("full"))
    events = [synth.make_event(synth.detector("full"), 960, "full", n_pu=500), synth.make_event(synth.detector("full"), 961, "full", n_pu=40)]
    gpu.upload_detector(det)
    gpu.set_events(events)
    gpu.run(4, flags)
    check(gpu, oracle_lib, det, events, flags)


@pytest.mark.parametrize("flags", [0, 3, 32 | 64, 128])
@pytest.mark.parametrize("cuts", [(0,), (1,), (2,), (3,), (0, 1, 2, 3), (1, 3)])
def test_split_runs(cuts, flags, gpu, oracle_lib):
    from sdl_gb300 import synth
    det = synth.detector("full")
    events = [synth.make_event(det, 962, "full", n_pu=350)]
    gpu.upload_detector(det)
    gpu.set_events(events)
    for first, last in zip((0,) + tuple(c + 1 for c in cuts), cuts + (4,)):
        gpu.run_stages(first, last, flags)
    check(gpu, oracle_lib, det, events, flags)


@pytest.mark.parametrize("n_events", [1, 7, 8, 9])
def test_batch_sizes(n_events, gpu, oracle_lib):
    """7 events of the full geometry are 236,068 global modules, 8 are 269,792"""
    from sdl_gb300 import synth
    det = synth.detector("full")
    events = [synth.make_event(det, 970 + k, "full", n_pu=(0, 70, 350)[k % 3], n_signal=5) for k in range(n_events)]
    gpu.upload_detector(det)
    gpu.set_events(events)
    gpu.run(4)
    check(gpu, oracle_lib, det, events, 0)
