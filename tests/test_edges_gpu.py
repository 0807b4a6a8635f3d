"""Sizes where the launch shapes and copies change: gradient samples around the
training tiles and their grid, input copies by alignment and memory kind, and
batches on both sides of 2^18 hits."""
import numpy as np
import pytest

from oracle import mlp as omlp

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    from sdl_gb300 import Chain, build
    build.build()
    return Chain(0)


def digests(gpu, oracle_lib, event, last=4):
    return [oracle_lib.digest(gpu.objects(s, event)) for s in range(last + 1)]


@pytest.mark.parametrize("n", [1, 31, 127, 128, 129, 304 * 128 - 1, 304 * 128 + 1, 2 * 304 * 128 + 130])
def test_gradient_sizes(n, gpu):
    """The gradient against the oracle's.  A hidden unit whose FP32 sum lands on the other side of a BF16
    rounding boundary moves by 2^-8 of itself: at most that share of the gradient where the samples are few
    (4e-3), less than 1e-3 of it among many, and 1e-3 of the loss."""
    p = omlp.init_params(31)
    gpu.mlp_set_params(p, 0.0)
    r = np.random.default_rng(n)
    x = r.normal(0.0, 1.5, size=(n, omlp.N_IN)).astype(np.float32)
    y = (r.random(n) < 0.3).astype(np.float32)
    w = r.uniform(0.5, 2.0, n).astype(np.float32)
    g, loss = gpu.mlp_gradient(x, y, w)
    lr, gr = omlp.loss_and_grad(p, x, y, w)
    assert abs(loss - lr) <= 1e-3 * (1 + abs(lr))
    assert np.linalg.norm(g - gr) <= (4e-3 if n < 1000 else 1e-3) * np.linalg.norm(gr)


def arrays(ch, ev, pinned, shift):
    """The event's five arrays, `shift` words past the start of their (pinned) buffers"""
    out = []
    for a in (ev.x, ev.y, ev.z, ev.idx, ev.detid):
        a = np.ascontiguousarray(a)
        n = a.size + shift
        buf = (ch.pinned(4 * n) if pinned else np.empty(4 * n, dtype=np.uint8)).view(a.dtype)[:n]
        buf[shift:] = a
        out.append(buf[shift:])
    return out


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("shift", [0, 1, 3])
@pytest.mark.parametrize("n_hits", [1, 255, 1001, 2300])
def test_input_copies(n_hits, shift, pinned, gpu, oracle_lib):
    from sdl_gb300 import synth
    det = synth.detector("barrel_flat")
    ev = synth.make_event(det, 980, "barrel_flat")
    cut = type(ev)(**{**ev.__dict__, **{k: getattr(ev, k)[:n_hits] for k in ("x", "y", "z", "idx", "detid")}})
    gpu.upload_detector(det)
    ref, _, _ = oracle_lib.Oracle(det).run(cut)
    off = np.array([0, len(cut.x)], dtype=np.int64)
    a = arrays(gpu, cut, pinned, shift)
    gpu.set_events_raw(1, off.ctypes.data, *[v.ctypes.data for v in a])
    gpu.run(4)
    assert digests(gpu, oracle_lib, 0) == [oracle_lib.digest(ref[s]) for s in range(5)]


@pytest.mark.parametrize("flags", [0, 32 | 64, 128])
@pytest.mark.parametrize("above", [False, True])
def test_around_two_to_the_eighteenth_hits(above, flags, gpu, oracle_lib):
    """One event many times over: every copy gives the event's objects"""
    from sdl_gb300 import synth
    det = synth.detector("full")
    ev = synth.make_event(det, 981, "full", n_pu=300)
    n = (1 << 18) // len(ev.x) + (1 if above else 0)
    gpu.upload_detector(det)
    ref, _, _ = oracle_lib.Oracle(det).run(ev, mode=flags)
    want = [oracle_lib.digest(ref[s]) for s in range(5)]
    gpu.set_events([ev] * n)
    gpu.run(4, flags)
    assert (n * len(ev.x) > 1 << 18) == above
    for e in (0, n // 2, n - 1):
        assert digests(gpu, oracle_lib, e) == want


@pytest.mark.parametrize("n", [1, 2, 25, 120, 240])
def test_copies_of_an_event(n, gpu, oracle_lib):
    """From a few thousand candidates a stage to millions: candidates judged in place or gathered, exact phases on
    one entry a warp or 32"""
    from sdl_gb300 import synth
    det = synth.detector("full")
    ev = synth.make_event(det, 982, "full", n_pu=700)
    gpu.upload_detector(det)
    ref, cnt, _ = oracle_lib.Oracle(det).run(ev)
    want = [oracle_lib.digest(ref[s]) for s in range(5)]
    gpu.set_events([ev] * n)
    gpu.run(4)
    for e in {0, n // 2, n - 1}:
        assert digests(gpu, oracle_lib, e) == want
        assert np.array_equal(gpu.counters(e), cnt)
