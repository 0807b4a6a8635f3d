"""Phase B1 of the tracklets where its betaIn threshold is above pi / 2: inner
segments from the barrel to the endcap with an rt step below 0.08 cm
(asin(...) + 0.02 / step) and outer anchors past 120 cm, against the CPU
restatement.  The segments' directions differ by more than a right angle from
their dPhiChange, and the pair is a tracklet."""
import numpy as np
import pytest

from test_gpu_parity import describe

pytestmark = pytest.mark.gpu

ANCHORS = np.array([(92.5385818, 0.0, 115.57547), (92.4359741, 4.52619553, 131.0), (122.129112, -61.8187904, 153.213913),
                    (132.612854, -91.5498657, 185.0)])
SPREAD = np.array([(0.3, 0.0, 0.5), (0.0, 0.3, 0.0), (1.0, 1.0, 0.3), (1.0, 1.0, 0.0)])


def chain_of_modules():
    """A 2S barrel module connected to one of the endcap, that to the next, and that to a third: (lower, upper) each"""
    from sdl_gb300 import synth
    mods = []
    lo, up = synth.sensor_bits(synth.is_inverted(5, 3, 6, 2))
    mods.append((synth.barrel_detid(6, 3, 1, 2, lo), synth.barrel_detid(6, 3, 1, 2, up)))
    for layer in (1, 2, 4):
        lo, up = synth.sensor_bits(synth.is_inverted(4, 2, layer, 1))
        mods.append((synth.endcap_detid(2, layer, 12, 1, lo), synth.endcap_detid(2, layer, 12, 1, up)))
    det = synth.Detector("chain")
    det.conn = {mods[k][0]: [mods[k + 1][0]] for k in range(3)}
    return det, mods


def steep_event(mods, rng, n_upper=4):
    """Four anchors (lower hits), each with n_upper upper hits around it"""
    from sdl_gb300 import synth
    a = ANCHORS + rng.normal(size=(4, 3)) * SPREAD
    phi = np.arctan2(a[:, 1], a[:, 0])
    r = np.hypot(a[0, 0], a[0, 1]) + rng.uniform(0.005, 0.079)
    a[1, :2] = r * np.cos(phi[1]), r * np.sin(phi[1])
    pts, ids = [], []
    for k in range(4):
        pts.append(a[k])
        ids.append(mods[k][0])
        for _ in range(n_upper):
            if k == 0:  # the barrel's upper sensor, 1.8 mm on
                d = phi[k] + rng.uniform(0.25, 0.5)
                pts.append(a[k] + np.array([0.18 * np.cos(d), 0.18 * np.sin(d), 0.0]))
            else:  # the endcap's, 4 mm on
                d = phi[k] + (rng.uniform(0.0009, 0.0015) if k == 1 else -rng.uniform(0.001, 0.0022))
                rt = np.hypot(a[k, 0], a[k, 1])
                pts.append(np.array([rt * np.cos(d), rt * np.sin(d), a[k, 2] + 0.4]))
            ids.append(mods[k][1])
    p = np.array(pts, dtype=np.float32)
    return synth.Event(p[:, 0].copy(), p[:, 1].copy(), p[:, 2].copy(), np.arange(len(p), dtype=np.int32),
                       np.array(ids, dtype=np.uint32))


def beta_in(ev, tracklets, segments, vals):
    """dPhiChange of the inner segment less the angle from its anchor to the outer end"""
    dpc = {tuple(s): v[3] for s, v in zip(segments, vals)}
    x, y = ev.x.astype(np.float64), ev.y.astype(np.float64)
    a, d = tracklets[:, 0], tracklets[:, 6]
    w = np.arctan2(y[d] - y[a], x[d] - x[a]) - np.arctan2(y[a], x[a])
    return np.array([dpc[tuple(t[:4])] for t in tracklets]) - (np.mod(w + np.pi, 2 * np.pi) - np.pi)


def test_thresholds_past_a_right_angle(oracle_lib):
    from sdl_gb300 import Chain, build
    build.build()
    det, mods = chain_of_modules()
    rng = np.random.default_rng(11)
    events = [steep_event(mods, rng) for _ in range(16)]
    gpu = Chain(0)
    gpu.upload_detector(det)
    gpu.set_events(events)
    gpu.run(4)
    orc = oracle_lib.Oracle(det)
    steep = 0
    for e, ev in enumerate(events):
        ref, _, _, vals = orc.run(ev, vals=True)
        if len(ref[2]):
            steep += int((np.abs(beta_in(ev, ref[2], ref[1], vals[1])) > np.pi / 2).sum())
        for s in range(5):
            got = gpu.objects(s, e)
            assert oracle_lib.digest(got) == oracle_lib.digest(ref[s]), describe(oracle_lib, got, ref[s], s)
    assert steep > 100
    assert gpu.tl_phase_a_check()["mismatches"] == 0
