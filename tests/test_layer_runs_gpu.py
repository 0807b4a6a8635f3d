"""Layer-pair segments of detIds that differ in bits the decoding ignores
(endcap bits 21-22, barrel bits 23-24, bits 28-31): a layer's modules are then
many runs of the sorted module table, for the endcap's second layer up to 96
runs of outer modules, against the CPU restatement."""
import copy

import numpy as np
import pytest

from test_joins_gpu import check

pytestmark = pytest.mark.gpu


def spread(det, high):
    """`det` with each detId's ignored bits from its ring or rod (bits 28-29 too where `high`)"""
    def f(d):
        n = (d >> 12) & 3 if (d >> 25) & 7 == 4 else (d >> 10) & 3
        d |= n << (21 if (d >> 25) & 7 == 4 else 23)
        return d | (((d >> 4) & 3) << 28 if high else 0)
    out = copy.copy(det)
    out.tilted_rows = [(f(r[0]),) + tuple(r[1:]) for r in det.tilted_rows]
    out.endcap_rows = [(f(r[0]),) + tuple(r[1:]) for r in det.endcap_rows]
    out.conn = {f(d): [f(e) for e in v] for d, v in det.conn.items()}
    return out, f


@pytest.mark.parametrize("flags", [1, 3, 3 | 128])
@pytest.mark.parametrize("high", [False, True])
def test_layers_of_many_runs(high, flags, oracle_lib):
    from sdl_gb300 import Chain, build, synth
    build.build()
    full = synth.detector("full")
    det, f = spread(full, high)
    events = []
    for seed, n_pu in ((990, 300), (991, 40)):
        ev = synth.make_event(full, seed, "full", n_pu=n_pu)
        ids = np.array([f(int(d)) for d in ev.detid], dtype=np.uint32)
        events.append(type(ev)(**{**ev.__dict__, "detid": ids}))
    gpu = Chain(0)
    gpu.upload_detector(det)
    gpu.set_events(events)
    gpu.run(4, flags)
    check(gpu, oracle_lib, det, events, flags)
    assert gpu.counts(-1)[1] > 1000
