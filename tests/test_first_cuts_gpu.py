"""The single-precision first passes over the mini-doublet and segment
candidates (md_first_cuts; sg_first_cuts and sg_later_cuts) against the whole
algorithms on every candidate of a batch at PU 100, 200 and 300, by the module
map and by the layer pairs, and on the same events moved off their modules
(scaled and turned, so that the candidates meet every cut elsewhere): nothing
they reject is accepted, and they reject most of what is not."""
import numpy as np
import pytest

from test_gpu_parity import run_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from sdl_gb300 import Chain, build
    build.build()
    return Chain(0)


@pytest.fixture(scope="module")
def batch():
    from sdl_gb300 import synth
    det = synth.detector("full")
    return det, [synth.make_event(det, 980 + k, "full", n_pu=n) for k, n in enumerate((3500, 7000, 10500))]


def check(gpu):
    r = gpu.first_cuts_check()
    print(r)
    n = gpu.counts(-1)
    for k, s in enumerate(("MD", "SG")):
        assert r[s]["violations"] == 0, r
        assert r[s]["accepted"] == n[k], (r, n)
        assert r[s]["rejected"] + r[s]["accepted"] <= r[s]["candidates"], r
    return r


@pytest.mark.parametrize("flags", [0, 3])
def test_first_passes_reject_only_what_the_algorithms_reject(flags, gpu, batch):
    det, events = batch
    run_gpu(gpu, det, events, flags)
    r = check(gpu)
    for s in ("MD", "SG"):
        assert r[s]["accepted"] > 0 and r[s]["rejected"] >= 0.8 * (r[s]["candidates"] - r[s]["accepted"]), r


@pytest.mark.parametrize("scale,turn", [(0.2, 0.0), (0.01, 0.3), (3.0, 0.0), (1.0, 0.02)])
def test_first_passes_off_the_modules(scale, turn, gpu, batch):
    """x and y scaled, the upper sensors' hits turned about the beam axis"""
    det, events = batch
    moved = []
    for ev in events[:2]:
        phi = turn * (ev.detid & 1).astype(np.float32)
        x = (scale * (ev.x * np.cos(phi) - ev.y * np.sin(phi))).astype(np.float32)
        y = (scale * (ev.x * np.sin(phi) + ev.y * np.cos(phi))).astype(np.float32)
        moved.append(type(ev)(**{**ev.__dict__, "x": x, "y": y}))
    gpu.upload_detector(det)
    gpu.set_events(moved)
    gpu.run(1, 0)
    check(gpu)


def test_after_the_whole_chain(gpu, batch):
    """The check makes the connection sums over the mini-doublets again"""
    det, events = batch
    gpu.upload_detector(det)
    gpu.set_events(events[:1])
    gpu.run(1, 0)
    want = gpu.first_cuts_check()
    for flags in (0, 64, 128):
        gpu.run(4, flags)
        assert gpu.first_cuts_check() == want
