"""The launch shapes follow the batch at hand, not the largest that a context
has held: kernels per run and objects of small batches on contexts that held
one above 2^18 hits, with the same and with another number of events, and of
small and large batches in turn."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def world(oracle_lib):
    from sdl_gb300 import build, synth
    build.build()
    det = synth.detector("full")
    ev = synth.make_event(det, 996, "full", n_pu=1500)
    few = synth.make_event(det, 997, "full", n_pu=60)
    n = (1 << 18) // len(ev.x) + 1
    orc = oracle_lib.Oracle(det)
    want = {id(e): [oracle_lib.digest(r) for r in orc.run(e)[0]] for e in (ev, few)}
    return det, [ev] * n, [few] * n, want


def fresh(det):
    from sdl_gb300 import Chain
    ch = Chain(0)
    ch.upload_detector(det)
    return ch


def run(ch, events, want, oracle_lib, flags=0):
    """kernels of a run, its objects checked"""
    ch.set_events(events)
    ch.run(4, flags)
    for e in (0, len(events) - 1):
        assert [oracle_lib.digest(ch.objects(s, e)) for s in range(5)] == want[id(events[e])]
    return ch.launches


@pytest.mark.parametrize("graph", [True, False])
def test_small_after_large(graph, world, oracle_lib):
    from sdl_gb300 import FLAG_NO_GRAPH
    flags = 0 if graph else FLAG_NO_GRAPH
    det, large, small, want = world
    assert sum(len(e.x) for e in large) > 1 << 18 > sum(len(e.x) for e in small)
    alone = {k: run(fresh(det), b, want, oracle_lib, flags) for k, b in (("large", large), ("small", small), ("one", small[:1]))}
    assert alone["small"] < alone["large"]
    ch = fresh(det)
    for k, b in (("large", large), ("small", small), ("large", large), ("small", small), ("one", small[:1]), ("small", small),
                 ("large", large)):
        assert run(ch, b, want, oracle_lib, flags) == alone[k], k
        assert ch.tl_phase_a_check()["mismatches"] == 0


def test_staged_batches_in_turn(world, oracle_lib):
    det, large, small, want = world
    ch = fresh(det)
    order = [large, small, small, large, small]
    ch.set_events(order[0])
    for k, b in enumerate(order):
        ch.run_async(4, 0)
        if k + 1 < len(order):
            ch.stage_events(order[k + 1])
        ch.sync()
        for e in (0, len(b) - 1):
            assert [oracle_lib.digest(ch.objects(s, e)) for s in range(5)] == want[id(b[e])]
