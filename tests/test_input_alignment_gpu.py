"""Pinned input arrays at any address: off a word's boundary (views into packed
records), and word-aligned but not 16-byte aligned above 2^18 hits, where the
copy engines take them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def setup(oracle_lib):
    from sdl_gb300 import Chain, build, synth
    build.build()
    det = synth.detector("full")
    ev = synth.make_event(det, 994, "full", n_pu=200)
    ch = Chain(0)
    ch.upload_detector(det)
    ref, _, _ = oracle_lib.Oracle(det).run(ev)
    return ch, ev, [oracle_lib.digest(r) for r in ref]


def check(setup, oracle_lib, copies, shifts):
    """the event `copies` times, array k starting shifts[k] bytes past its pinned buffer"""
    ch, ev, want = setup
    n = len(ev.x) * copies
    off = np.arange(copies + 1, dtype=np.int64) * len(ev.x)
    mem, at = ch.pinned(5 * (4 * n + 32)), []
    for k, a in enumerate((ev.x, ev.y, ev.z, ev.idx, ev.detid)):
        p = (k * (4 * n + 32) + 15) // 16 * 16 + shifts[k]
        mem[p:p + 4 * n] = np.tile(np.ascontiguousarray(a), copies).view(np.uint8)
        at.append(mem.ctypes.data + p)
    ch.set_events_raw(copies, off.ctypes.data, *at)
    ch.run(4)
    for e in {0, copies // 2, copies - 1}:
        assert [oracle_lib.digest(ch.objects(s, e)) for s in range(5)] == want


@pytest.mark.parametrize("shifts", [(1, 1, 1, 1, 1), (2, 2, 2, 2, 2), (3, 1, 2, 0, 4), (0, 0, 0, 0, 2)])
@pytest.mark.parametrize("copies", [1, 3])
def test_off_a_word(copies, shifts, setup, oracle_lib):
    check(setup, oracle_lib, copies, shifts)


@pytest.mark.parametrize("shifts", [(0, 0, 0, 0, 0), (4, 4, 4, 4, 4), (0, 0, 12, 0, 0), (1, 2, 3, 1, 2)])
def test_many_hits(shifts, setup, oracle_lib):
    copies = (1 << 18) // len(setup[1].x) + 1
    check(setup, oracle_lib, copies, shifts)
