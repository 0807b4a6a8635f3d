"""Mini-doublet candidates of tilted pairs whose pixel hit lies a millimetre from
the beam axis while the shifted strip hit is 60 cm out: the directions' cross
product is then the difference of products a thousand times larger, and the cut
is small (the asin term vanishes with the pixel hit's rt), so that its rounding
is larger than the cut's margin at larger radii.  Against the CPU restatement."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def near_axis_event(rng, slope, lower, upper, n=256):
    """n upper (pixel) hits within 1.5 mm of the axis, their direction off the strips' by about the cut (asin(r k), with
    the first layer's scattering and vertex terms), n lower (strip) hits whose projections on the strips' lines through
    them lie 60 cm out"""
    from sdl_gb300 import synth
    r = rng.uniform(0.05, 0.15, n)
    cut = np.arcsin(r * 2.99792458e-3 * 3.8 / 2) + np.hypot(3 * 0.0052, 0.1 / 21.8)
    phi = np.arctan(slope) + rng.choice([-1, 1], n) * (cut - rng.uniform(-5e-5, 1e-4, n)) * (1 - r / 60)
    up = np.stack([r * np.cos(phi), r * np.sin(phi)], axis=1)
    t = np.array([1.0, slope]) / np.hypot(1.0, slope)
    lo = rng.uniform(55.0, 65.0, (n, 1)) * t + rng.uniform(-5.0, 5.0, (n, 1)) * np.array([-t[1], t[0]])
    p = np.concatenate([lo, up]).astype(np.float32)
    z = np.concatenate([rng.uniform(40.0, 40.5, n), rng.uniform(40.6, 41.0, n)]).astype(np.float32)
    ids = np.repeat(np.array([lower, upper], dtype=np.uint32), n)
    return synth.Event(p[:, 0].copy(), p[:, 1].copy(), z, np.arange(2 * n, dtype=np.int32), ids)


def events(n=24):
    from sdl_gb300 import module_info, synth
    det = synth.detector("full")
    slopes = {int(r[0]): r[2] for r in det.tilted_rows}
    rng = np.random.default_rng(17)
    out = []
    for d in sorted(slopes):
        m = module_info(d)
        # a strip sensor (1) below a pixel sensor (0), its line neither along x nor along y
        if m["isLower"] and m["moduleLayerType"] == 1 and module_info(m["partnerDetId"])["moduleLayerType"] == 0 and \
                0.2 < abs(slopes[d]) < 5 and len(out) < n:
            out.append(near_axis_event(rng, slopes[d], d, m["partnerDetId"]))
    return det, out


def test_pixel_hits_near_the_axis(oracle_lib):
    from sdl_gb300 import Chain, build
    build.build()
    det, evs = events()
    assert len(evs) == 24
    gpu = Chain(0)
    gpu.upload_detector(det)
    gpu.set_events(evs)
    gpu.run(0)
    orc = oracle_lib.Oracle(det)
    total = lost = 0
    for e, ev in enumerate(evs):
        ref, _, _ = orc.run(ev, stop_after=0)
        extra, missing = oracle_lib.multiset_diff(gpu.objects(0, e), ref[0])
        assert len(extra) == 0
        lost += len(missing)
        total += len(ref[0])
    assert lost == 0 and total > 10_000, (lost, total)
