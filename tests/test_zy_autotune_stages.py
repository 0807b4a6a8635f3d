"""The autotuner leaves the stages alone that have no candidate-evaluation
kernel to tune: the triplets, and the track candidates except those from
triplets after layer-pair segments."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from sdl_gb300 import Chain, build, synth
    build.build()
    det = synth.detector("full")
    ch = Chain(0)
    ch.upload_detector(det)
    ch.set_events([synth.make_event(det, 999, "full", n_pu=200)])
    return ch


@pytest.mark.parametrize("stop,flags", [(4, 0), (4, 64), (4, 128), (2, 0), (4, 1 | 128)])
def test_untuned_stages_keep_their_shape(stop, flags, gpu):
    shape = gpu.autotune(stop, flags)
    for s in range(5):
        got = (shape["task"][s], shape["ctas_per_sm"][s])
        if s > stop and s >= 3:
            assert got == (0, 0)
        elif s == 3 or (s == 4 and flags != 1 | 128):
            assert got == (256, 8)
        else:
            assert got[0] in (128, 256, 512, 1024) and got[1] in (4, 8, 16)
