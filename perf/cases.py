"""What is measured: the work that a user of the segment-linking chain has it do, through
:class:`sdl_gb300.Chain`.

Events are pile-up overlays on the synthetic detectors of :mod:`sdl_gb300.synth`, mixed from a library of
sub-events as experiments mix theirs (20 pile-up units each, plus a signal event of 20 helices); every hit has
an idx of its own in its batch.  A state holds a context with the geometry loaded, the batch in pinned host
memory and pinned memory for the results; the context has run the batch's sizes before, as a program that
processes a stream of events has.  The order of the objects of one module is not specified, so the tuples are
returned in the order of a hash of their rows, at the head of an array of the case's size (the rest is -1).
"""
import math
import os

import numpy as np
import torch

import sdl_gb300
from sdl_gb300 import mlp, synth

SUB_PU = 20          # pile-up units of one library sub-event
N_SUB = 30           # library: up to 600 pile-up units in one event
N_SIGNAL = 8
N_FLAT = 24
HITS_PER_PU = 485.0  # hits of the generator per pile-up unit
FLAT_HITS = 2340

# objects per event of the plain chain at these pile-ups (this generator, rounded up), by stage
PU_GRID = (20, 40, 60, 100, 140, 200, 250, 300, 400)
PER_EVENT = ((3000, 5950, 8900, 15000, 21500, 31000, 38500, 48500, 67000),
             (2700, 6200, 10700, 23000, 39500, 75500, 108000, 172000, 360000),
             (1450, 3500, 6800, 18000, 37500, 100000, 175000, 405000, 1300000),
             (2700, 7200, 14200, 39000, 81000, 204000, 335000, 680000, 2100000),
             (330, 900, 1800, 6400, 17000, 61500, 123000, 385000, 1600000))
FLAT_PER_EVENT = (700, 720, 380, 880, 125)

_tables, _library = {}, {}


def listed():
    return [
        # one barrel-only event of 100 helices and 1,000 noise hits: the smallest call, launches and latency
        dict(name="flat_event", kind="chain", geometry="barrel_flat", events=1, pu_lo=0, pu_hi=0, flags=0),
        # one event at PU 200, the plain chain: an event display, a trigger study, one event at a time
        dict(name="pu200_event", kind="chain", geometry="full", events=1, pu_lo=200, pu_hi=200, flags=0),
        # events of uneven size one after the other, the next one's hits and the last one's candidates
        # copied while one runs: an online farm's loop, with the learned pre-filter
        dict(name="event_stream", kind="stream", geometry="full", events=6, pu_lo=60, pu_hi=260, flags=sdl_gb300.FLAG_MLP),
        # the create* calls one by one with the objects and per-layer counters of each: the reference's C++
        # calling sequence
        dict(name="stage_by_stage", kind="stages", geometry="full", events=1, pu_lo=60, pu_hi=60, flags=0),
        # 100 barrel-only events in one batch with the pre-filter trained for them
        dict(name="flat_batch", kind="chain", geometry="barrel_flat", events=100, pu_lo=0, pu_hi=0, flags=sdl_gb300.FLAG_MLP),
        # 64 events of uneven size, the plain chain: offline reprocessing with the reference's objects
        dict(name="uneven_batch", kind="chain", geometry="full", events=64, pu_lo=50, pu_hi=250, flags=0),
        # 128 dense events with the pre-filter: the benchmark's workload, the largest; a filter farm that takes
        # the per-layer counters of every event and the candidates of one in eight
        dict(name="dense_batch", kind="chain", geometry="full", events=128, pu_lo=150, pu_hi=300, flags=sdl_gb300.FLAG_MLP,
             read_every=8),
        # the layer-pair variants (createSegments, createTracklets) on sparse events, where their all-pairs
        # candidate spaces are affordable
        dict(name="layer_pairs", kind="chain", geometry="full", events=5, pu_lo=20, pu_hi=40,
             flags=sdl_gb300.FLAG_SG_LAYERS | sdl_gb300.FLAG_TL_LAYERS),
        # tracklets via navigation, track candidates from tracklets
        dict(name="navigation_batch", kind="chain", geometry="full", events=13, pu_lo=100, pu_hi=220,
             flags=sdl_gb300.FLAG_TL_NAV | sdl_gb300.FLAG_TC_FROM_TL),
        # track candidates from triplets
        dict(name="triplet_candidates", kind="chain", geometry="full", events=3, pu_lo=100, pu_hi=200,
             flags=sdl_gb300.FLAG_TC_FROM_TP),
        # mini-doublets alone from and to the caller's device memory, without allocation
        dict(name="mini_doublets_device", kind="static", geometry="full", events=1, pu_lo=180, pu_hi=180, flags=0),
        # forward and backward pass of the pre-filter's training over one large batch
        dict(name="prefilter_gradient", kind="gradient", samples=262144),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def pus(lo, hi):
        a, b = sorted(rng.uniform(lo, hi) for _ in range(2))
        return dict(pu_lo=round(a, 1), pu_hi=round(b, 1))

    kind = rng.choice(["event", "event", "batch", "batch", "batch", "stream", "stages", "flat", "variant", "static", "gradient"])
    mlp_flag = rng.choice([0, sdl_gb300.FLAG_MLP])
    if kind == "event":
        pu = round(math.exp(rng.uniform(math.log(20), math.log(300))), 1)
        return dict(kind="chain", geometry="full", events=1, pu_lo=pu, pu_hi=pu, flags=mlp_flag)
    if kind == "batch":
        return dict(kind="chain", geometry="full", events=log_int(2, 100), **pus(40, 260), flags=mlp_flag,
                    read_every=rng.choice([1, 8]))
    if kind == "stream":
        return dict(kind="stream", geometry="full", events=rng.randint(2, 8), **pus(40, 280), flags=mlp_flag)
    if kind == "stages":
        pu = round(rng.uniform(20, 200), 1)
        return dict(kind="stages", geometry="full", events=1, pu_lo=pu, pu_hi=pu, flags=0)
    if kind == "flat":
        return dict(kind="chain", geometry="barrel_flat", events=log_int(1, 200), pu_lo=0, pu_hi=0, flags=mlp_flag)
    if kind == "variant":
        flags, hi, n = rng.choice([(sdl_gb300.FLAG_SG_LAYERS | sdl_gb300.FLAG_TL_LAYERS, 40, 8), (sdl_gb300.FLAG_TL_LAYERS, 60, 8),
                                   (sdl_gb300.FLAG_TL_NAV, 260, 32), (sdl_gb300.FLAG_TC_FROM_TL, 200, 16),
                                   (sdl_gb300.FLAG_TC_FROM_TP, 200, 6)])
        return dict(kind="chain", geometry="full", events=rng.randint(1, n), **pus(20, hi), flags=flags)
    if kind == "static":
        pu = round(math.exp(rng.uniform(math.log(20), math.log(240))), 1)
        return dict(kind="static", geometry="full", events=1, pu_lo=pu, pu_hi=pu, flags=0)
    return dict(kind="gradient", samples=log_int(3000, 600000))


# ---------------------------------------------------------------- inputs
def _detector_tables(geometry):
    if geometry not in _tables:
        _tables[geometry] = synth.detector(geometry).tables()
    return _tables[geometry]


def _sub_event(what, k):
    """Sub-event k of the library as device tensors (x, y, z, detid)."""
    if (what, k) not in _library:
        with np.errstate(all="ignore"):
            det = synth.detector("barrel_flat" if what == "flat" else "full")
            if what == "flat":
                e = synth.make_event(det, 70000 + k, "barrel_flat")
            elif what == "signal":
                e = synth.make_event(det, 71000 + k, "full", n_pu=0, n_signal=20)
            else:
                e = synth.make_event(det, 72000 + k, "full", n_pu=35 * SUB_PU, n_signal=0)
        _library[what, k] = [torch.from_numpy(a).cuda() for a in (e.x, e.y, e.z, e.detid.astype(np.int32))]
    return _library[what, k]


def _batch(case, rng, gen, n_events):
    """(offsets, [x, y, z, idx, detid]) of n_events events: host offsets, device tensors."""
    parts, sizes = [], []
    for _ in range(n_events):
        if case["geometry"] == "barrel_flat":
            picks = [("flat", int(rng.integers(N_FLAT)))]
        else:
            pu = rng.uniform(case["pu_lo"], case["pu_hi"]) if case["pu_hi"] > case["pu_lo"] else case["pu_lo"]
            n = max(1, min(N_SUB, int(round(pu / SUB_PU))))
            picks = [("pileup", int(k)) for k in rng.permutation(N_SUB)[:n]] + [("signal", int(rng.integers(N_SIGNAL)))]
        subs = [_sub_event(*p) for p in picks]
        parts += subs
        sizes.append(sum(len(s[0]) for s in subs))
    off = np.zeros(n_events + 1, dtype=np.int64)
    off[1:] = np.cumsum(sizes)
    total = int(off[-1])
    ev = torch.repeat_interleave(torch.arange(n_events, device="cuda"), torch.tensor(sizes, device="cuda"))
    order = torch.argsort(ev + torch.rand(total, generator=gen, device="cuda", dtype=torch.float64) * 0.999)
    x, y, z, det = (torch.cat([p[k] for p in parts])[order] for k in range(4))
    return off, [x, y, z, torch.arange(total, device="cuda", dtype=torch.int32), det]


def _to_pinned(chain, arrays):
    n = len(arrays[0])
    mem = chain.pinned(max(1, 20 * n))
    views = []
    for k, a in enumerate(arrays):
        v = mem[4 * n * k:4 * n * (k + 1)].view(a.cpu().numpy().dtype)
        v[:] = a.cpu().numpy()
        views.append(v)
    return views


def _chain(case):
    chain = sdl_gb300.Chain(0)
    chain.upload_tables(*_detector_tables(case["geometry"]))
    if case["flags"] & sdl_gb300.FLAG_MLP:
        name = "tl_mlp_flat.npz" if case["geometry"] == "barrel_flat" else "tl_mlp_pu.npz"
        params, threshold, _ = mlp.load(os.path.join(mlp.WEIGHTS, name))
        chain.mlp_set_params(params, threshold)
    return chain


def _result_buffer(chain, stage, rows):
    width = sdl_gb300.WIDTH[stage]
    return chain.pinned(max(1, rows) * width * 4).view(np.int32).reshape(-1, width)


def _gradient_inputs(case, seed):
    """Feature rows of the pre-filter's ranges with labels that depend on them, weights as training gives
    them (positives four times)."""
    r = np.random.default_rng(seed)
    n = case["samples"]
    x = np.empty((n, sdl_gb300.MLP_FEATURES), dtype=np.float32)
    for k, (m, s) in enumerate(((0.4, 0.2), (0.0, 0.6), (0.8, 0.2), (0.0, 0.9), (0.0, 0.6), (0.0, 0.5), (0.0, 0.5), (0.0, 0.4),
                                (0.0, 0.4), (0.0, 1.0), (0.0, 0.8))):
        x[:, k] = r.normal(m, s, n)
    x[:, 11] = r.integers(0, 13, n) * 0.125
    y = (np.abs(x[:, 7] - x[:, 8]) + 0.5 * np.abs(x[:, 9]) + r.normal(0, 0.2, n) < 0.45).astype(np.float32)
    return x, y, np.where(y > 0, np.float32(4), np.float32(1))


def _rows(case, stage):
    """Size of the result array of a stage: the fitted number of objects with some room."""
    n = -(-case["events"] // case.get("read_every", 1))
    if case["geometry"] == "barrel_flat":
        return int(1.2 * n * FLAT_PER_EVENT[stage] + 4 * FLAT_PER_EVENT[stage]) + 64
    pu = SUB_PU * np.maximum(1, np.round(np.linspace(case["pu_lo"], case["pu_hi"], 101) / SUB_PU))
    per = np.exp(np.interp(np.log(pu), np.log(PU_GRID), np.log(PER_EVENT[stage])))
    many = 8.0 if case["flags"] & sdl_gb300.FLAG_TC_FROM_TP and stage == 4 else 1.6 if case["flags"] & (
        sdl_gb300.FLAG_TC_FROM_TL | sdl_gb300.FLAG_SG_LAYERS) else 1.0
    if case["kind"] == "stream":  # one event to an array
        return int(3 * many * per.max()) + 64
    # single events spread widely about the fit, batches less so
    batch = min(n * per.max(), n * per.mean() + 3 * math.sqrt(n) * per.std())
    return int(1.1 * many * (batch + 2 * math.sqrt(n) * per.mean())) + 64


def prepare(case, seed):
    if case["kind"] == "gradient":
        params, threshold, _ = mlp.load(os.path.join(mlp.WEIGHTS, "tl_mlp_pu.npz"))
        chain = sdl_gb300.Chain(0)
        chain.mlp_set_params(params, threshold)
        return dict(case=case, chain=chain, inputs=_gradient_inputs(case, seed))
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    chain = _chain(case)
    state = dict(case=case, chain=chain)
    if case["kind"] == "static":
        off, arrays = _batch(case, rng, gen, 1)
        n = int(off[1])
        state.update(inputs=arrays, stream=torch.cuda.Stream(), n=n,
                     pairs=torch.empty((_rows(case, 0), 2), dtype=torch.int32, device="cuda"),
                     count=torch.zeros(1, dtype=torch.int64, device="cuda"),
                     status=torch.zeros(1, dtype=torch.int32, device="cuda"))
        torch.cuda.synchronize()
        return state
    batches = [_batch(case, rng, gen, 1) for _ in range(case["events"])] if case["kind"] == "stream" else [
        _batch(case, rng, gen, case["events"])]
    state["inputs"] = []
    for off, arrays in batches:
        views = _to_pinned(chain, arrays)
        state["inputs"].append((len(off) - 1, off.ctypes.data, *[v.ctypes.data for v in views], off, views))
    wanted = range(5) if case["kind"] == "stages" else (4,)
    state["out"] = [{s: _result_buffer(chain, s, _rows(case, s)) for s in wanted} for _ in batches]
    for _ in range(2):  # the capacities and the captured graph of these sizes
        for b in state["inputs"]:
            chain.set_events_raw(*b[:7])
            chain.run(4, case["flags"])
    return state


# ---------------------------------------------------------------- a pass
_multipliers = {}


def _by_hash(rows):
    """(device rows, order): the order of the rows by a 64-bit hash."""
    t = torch.from_numpy(rows).cuda() if isinstance(rows, np.ndarray) else rows
    w = t.shape[1] // 2
    if w not in _multipliers:
        r = np.random.default_rng(w)
        _multipliers[w] = torch.from_numpy(r.integers(-2**62, 2**62, w) * 2 + 1).cuda()
    return t, torch.sort((t.view(torch.int64) * _multipliers[w]).sum(1)).indices


def _padded(t, order, size, fill):
    out = torch.full((size, t.shape[1]), fill, dtype=t.dtype, device=t.device)
    torch.index_select(t, 0, order, out=out[:len(order)])
    return out


def _tuples(rows, size):
    return _padded(*_by_hash(rows), size, -1)


def run(state):
    case, chain = state["case"], state["chain"]
    flags = case.get("flags", 0)
    if case["kind"] == "gradient":
        x, y, w = state["inputs"]
        grad, loss = chain.mlp_gradient(x, y, w)
        return {"gradient": grad, "loss": loss, "logits": chain.mlp_score(x)}
    if case["kind"] == "static":
        s = state["stream"]
        with torch.cuda.stream(s):
            p = [a.data_ptr() for a in state["inputs"]]
            chain.mini_doublets_static(state["n"], *p, state["pairs"].data_ptr(), len(state["pairs"]),
                                       state["count"].data_ptr(), state["status"].data_ptr(), s.cuda_stream)
            n = int(state["count"].item())
            return {"count": n, "pairs": _tuples(state["pairs"][:n], len(state["pairs"]))}
    if case["kind"] == "stream":
        batches = state["inputs"]
        found = []
        chain.set_events_raw(*batches[0][:7])
        for k in range(len(batches)):
            chain.run_async(4, flags)
            if k + 1 < len(batches):
                chain.stage_events_raw(*batches[k + 1][:7])
            chain.sync()
            found.append(chain.objects_async(4, -1, state["out"][k][4]))
        chain.wait_objects()
        return [_tuples(out[4][:n], len(out[4])) for out, n in zip(state["out"], found)]
    chain.set_events_raw(*state["inputs"][0][:7])
    if case["kind"] == "stages":
        result = {}
        for s in range(5):
            chain.run_stages(s, s, flags)
            out = state["out"][0][s]
            t, order = _by_hash(chain.objects(s, 0, out=out))
            result["objects%d" % s] = _padded(t, order, len(out), -1)
            if s < 2:  # the floats that mini-doublets and segments keep
                result["values%d" % s] = _padded(torch.from_numpy(chain.links(s, 0)[2]).cuda(), order, len(out), 0.0)
        result["counters"] = chain.counters(0).astype(np.int64)
        return result
    chain.run(4, flags)
    counts = chain.counts(-1)
    out = state["out"][0][4]
    every = case.get("read_every", 1)
    if every == 1:
        return {"counts": counts, "track_candidates": _tuples(chain.objects(4, -1, out=out), len(out))}
    counters = np.stack([chain.counters(e) for e in range(case["events"])]).astype(np.int64)
    n = 0
    for e in range(0, case["events"], every):
        n += len(chain.objects(4, e, out=out[n:]))
    return {"counts": counts, "counters": counters, "track_candidates": _tuples(out[:n], len(out))}


# ---------------------------------------------------------------- work and exact values
def work(case):
    """Hits read (20 bytes each) and results written once; about twelve operations for the first cut of every
    tracklet candidate, or the network's multiply-adds."""
    if case["kind"] == "gradient":
        n = case["samples"]
        return {"bytes": n * 4.0 * (sdl_gb300.MLP_FEATURES + 3), "flops": 8.0 * n * (12 * 64 + 64 * 64 + 64)}
    n = case["events"]
    if case["geometry"] == "barrel_flat":
        return {"bytes": n * (20.0 * FLAT_HITS + 64 * FLAT_PER_EVENT[4]), "flops": 12.0 * n * 8000}
    pu = np.linspace(case["pu_lo"], case["pu_hi"], 101)
    hits = n * HITS_PER_PU * float(pu.mean())
    stages = {"static": (0,), "stages": range(5)}.get(case["kind"], (4,))
    found = n * sum(4 * sdl_gb300.WIDTH[s] * float(np.exp(np.interp(np.log(pu), np.log(PU_GRID), np.log(PER_EVENT[s]))).mean())
                    for s in stages)
    pairs = n * (97.0 * float(pu.mean()) if case["kind"] == "static" else 6.4e6 * float(((pu / 200) ** 3).mean()))
    return {"bytes": 20 * hits + found / case.get("read_every", 1), "flops": 12 * pairs}


def exact(case, seed):
    """The pre-filter's gradient, loss and logits in 64 bits, with the network's own roundings (its weights and
    first hidden layer are BF16 by definition); the objects are whole numbers."""
    if case["kind"] != "gradient":
        return None
    params, _, _ = mlp.load(os.path.join(mlp.WEIGHTS, "tl_mlp_pu.npz"))
    x, y, w = (torch.from_numpy(a) for a in _gradient_inputs(case, seed))

    def r(a):
        return a.float().bfloat16().double()

    p = torch.from_numpy(params)
    w1, b1, w2, b2, w3 = (r(v) for v in torch.split(p[:-1], [768, 64, 4096, 64, 64]))
    w1, w2, b3 = w1.view(64, 12), w2.view(64, 64), float(p[-1])
    x1, y, w = r(x), y.double(), w.double()
    h1 = r((x1 @ w1.T + b1).clamp_min(0))
    h2 = (h1 @ w2.T + b2).clamp_min(0)
    z = h2 @ w3 + b3
    loss = float((w * (torch.nn.functional.softplus(z) - y * z)).mean())
    dz = w * (torch.sigmoid(z) - y) / len(y)
    d2 = (h2 > 0) * torch.outer(dz, w3)
    d1 = (h1 > 0) * (d2 @ w2)
    g = torch.cat([(d1.T @ x1).reshape(-1), d1.sum(0), (d2.T @ h1).reshape(-1), d2.sum(0), dz @ h2, dz.sum()[None]])
    return {"gradient": g.numpy(), "loss": loss, "logits": z.numpy()}
