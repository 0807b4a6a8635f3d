"""The tracklet candidates as the training samples and the phase-A self-check
go through them: the same after a run that went on to the track candidates from
tracklets or triplets, whose connection sums are over those, as after one that
ended with the tracklets."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from sdl_gb300 import Chain, build, synth
    build.build()
    ch = Chain(0)
    det = synth.detector("full")
    ch.upload_detector(det)
    ch.set_events([synth.make_event(det, 992 + k, "full", n_pu=n) for k, n in enumerate((400, 150))])
    return ch


def samples(ch):
    ch.mlp_clear_samples()
    n = ch.mlp_collect(neg_keep=1.0)
    x, y = ch.mlp_samples()
    rows = np.concatenate([x, y[:, None]], axis=1).view(np.uint32)
    return n, rows[np.lexsort(rows.T[::-1])]


@pytest.mark.parametrize("flags", [0, 64, 128])
def test_candidates_after_the_track_candidates(flags, gpu):
    gpu.run(2, 0)
    want_check, (want_n, want) = gpu.tl_phase_a_check(), samples(gpu)
    gpu.run(4, flags)
    check, (n, got) = gpu.tl_phase_a_check(), samples(gpu)
    assert n == want_n > 1000
    assert np.array_equal(got, want)
    assert check == want_check and check["mismatches"] == 0
