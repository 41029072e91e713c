"""What is timed: the work users of trax_gb300 have it do, through its public entry points.

A case is one of six kinds:

  batch   a resident batch of events through the whole chain (trax_seed_batch, graph replay or the host-synced
          per-event path), triplets and tracks read back -- the program that seeds one batch after the other
  stages  the same chain through the seven stage calls, in the order of the reference's buildTriplets()
  stream  groups of events that differ in size, each uploaded from page-locked memory, seeded and read back through
          one context -- the event loop of a reconstruction job
  link    connectivity, circle fit and cellular automaton on a caller's triplets
  fit     the differentiable triplet fit: chi2 (forward) or chi2 and its gradient (backward) at given layer shifts
  scan    the allocation-free prefix sum on device memory

Events are the workloads of trax_gb300.events, generated on the GPU from the seed; a program
holds them as host columns, as its event loader leaves them.
"""
import ctypes
import math

import numpy as np
import torch

from trax_gb300 import capi, events

# The event shapes and their workload in trax_gb300.events; "tracks" is the mean number of tracks per event (per
# vertex for pileup), "hits" the hits per track, and a + n / b + (n / c)^2 the triplets per track of an event of n
# tracks (combinations grow with the tracks that share an event), about a tenth above the mean.
SHAPES = {
    "muons": {"config": 0, "tracks": 10, "hits": 2.97, "triplets": (1.0, math.inf, math.inf)},
    "multimuon": {"config": 1, "tracks": 200, "hits": 4.73, "triplets": (1.1, 2000.0, math.inf)},
    "ttbar": {"config": 2, "tracks": 1650, "hits": 5.7, "triplets": (2.4, 800.0, math.inf)},
    "pileup": {"config": 3, "tracks": 1000, "hits": 6.24, "triplets": (3.0, math.inf, 2050.0)},
}
VERTICES = {"pileup": 20}
# grids each shape is run with: its own, and others close to it (the autotuner's candidates)
GRIDS = {
    "muons": [(20, 20), (50, 8), (40, 40)],
    "multimuon": [(40, 100), (50, 48), (100, 64)],
    "ttbar": [(250, 48), (200, 64), (300, 48), (150, 64), (50, 128)],
    "pileup": [(80, 256), (150, 128), (200, 64)],
}


def listed():
    return [
        # ten muons in three pixel layers, ten events: the smallest batch there is, launches and latency
        _batch("muons_10", "muons", 10, (20, 20)),
        # a test-beam sized sample: 200 tracks per event, four layers, noise
        _batch("multimuon_100", "multimuon", 100, (40, 100)),
        # one event as it comes, through the stage calls with a host-read count after each (the reference's structure)
        dict(_batch("event_by_stages", "ttbar", 1, (250, 48)), kind="stages"),
        # an online buffer of a few dozen collisions
        _batch("ttbar_37", "ttbar", 37, (250, 48)),
        # the offline batch (the benchmark's workload)
        _batch("ttbar_1000", "ttbar", 1000, (250, 48)),
        # high occupancy as first run, nothing chosen for it
        _batch("pileup_3", "pileup", 3, (80, 256)),
        # high occupancy in bulk, with the finer z grid that the autotuner finds for it
        _batch("pileup_16_fine", "pileup", 16, (80, 256), fine=8),
        # an event loop: four groups of two dozen events, no two of the same size, one context
        {"name": "stream_4x24", "kind": "stream", "shape": "ttbar", "groups": 4, "events": 24, "tracks": 1650,
         "n_z": 250, "n_phi": 48},
        # linking stages on triplets made elsewhere
        {"name": "link_40", "kind": "link", "events": 40, "tracks": 1650},
        # one gradient of the detector alignment over a thousand events (an optimiser's step)
        {"name": "fit_gradient_1000", "kind": "fit", "grad": True, "params": False, "events": 1000, "tracks": 1650},
        # the fit's per-triplet parameters of a small sample (monitoring)
        {"name": "fit_params_20", "kind": "fit", "grad": False, "params": True, "events": 20, "tracks": 1650},
        # a compaction's offsets inside another framework's memory pool
        {"name": "scan_1m", "kind": "scan", "n": 1000003},
    ]


def _batch(name, shape, n_events, grid, fine=0, graph=True, linking=True, tracks=None):
    return {"name": name, "kind": "batch", "shape": shape, "events": n_events,
            "tracks": tracks or SHAPES[shape]["tracks"], "n_z": grid[0], "n_phi": grid[1], "fine": fine,
            "graph": graph, "linking": linking}


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["batch"] * 6 + ["stages", "stream", "link", "fit", "fit", "scan"])
    if kind == "scan":
        return {"kind": "scan", "n": spread(1000, 16000000)}
    if kind == "link":
        return {"kind": "link", "events": spread(2, 120), "tracks": spread(300, 2500)}
    if kind == "fit":
        grad = rng.random() < 0.7
        return {"kind": "fit", "grad": grad, "params": not grad and rng.random() < 0.5,
                "events": spread(5, 900), "tracks": spread(300, 1650)}
    shape = rng.choice(["muons", "multimuon", "ttbar", "ttbar", "ttbar", "pileup"])
    tracks = {"muons": spread(3, 30), "multimuon": spread(40, 400), "ttbar": spread(300, 2500),
              "pileup": spread(200, 1000)}[shape]
    most = {"muons": 200, "multimuon": 300, "ttbar": min(700, int(8e5 / tracks)), "pileup": 8}[shape]
    grid = rng.choice(GRIDS[shape])
    if kind == "stream":
        return {"kind": "stream", "shape": shape, "groups": rng.randint(2, 5),
                "events": spread(1, min(most, 40)), "tracks": tracks, "n_z": grid[0], "n_phi": grid[1]}
    c = _batch("", shape, spread(1, min(most, 20) if kind == "stages" else most), grid,
               fine=rng.choice([0, 4, 8]) if shape == "pileup" else 0, graph=rng.random() < 0.85,
               linking=rng.random() < 0.85, tracks=tracks)
    del c["name"]
    c["kind"] = kind
    return c


# ------------------------------------------------------------------ events
def _tracks_of(shape, n_events, mean, group=0):
    """Tracks of every event: a fixed number, or Poisson with the mean spread tenfold between events (ttbar-like).
    They go by the case alone, so that one size of read-back array holds the results of any seed."""
    if shape != "ttbar":
        return np.full(n_events, mean * VERTICES.get(shape, 1), dtype=np.int64)
    rng = np.random.default_rng([n_events, mean, group])
    return rng.poisson(rng.uniform(mean * 2 / 11, mean * 20 / 11, n_events) if n_events > 1 else [mean])


def _triplets_of(shape, tracks):
    a, b, c = SHAPES[shape]["triplets"]
    n = np.asarray(tracks, dtype=np.float64)
    return float((n * (a + n / b + (n / c) ** 2)).sum())


def _make_events(shape, n_events, mean_tracks, seed, group=0, config=None):
    """An EventBatch of helical tracks through barrel layers (the model of trax_gb300.events, drawn on the GPU), and
    per track and layer the index of its hit (-1: none)."""
    w = events.workload(SHAPES[shape]["config"] if config is None else config, n_events)
    gen = torch.Generator(device="cuda").manual_seed(int(seed) * 16 + group)
    f64 = {"dtype": torch.float64, "device": "cuda"}

    def uniform(n, lo=0.0, hi=1.0):
        return lo + (hi - lo) * torch.rand(n, generator=gen, **f64)

    def normal(n, sigma):
        return sigma * torch.randn(n, generator=gen, **f64)

    L, E = len(w.radii), w.n_events
    per_event = torch.as_tensor(_tracks_of(shape, n_events, mean_tracks, group), device="cuda")
    n = int(per_event.sum())
    ev = torch.repeat_interleave(torch.arange(E, device="cuda"), per_event)
    first = torch.cumsum(per_event, 0) - per_event
    number = torch.arange(n, device="cuda") - first[ev]  # of the track in its event
    vertex = ev * w.n_vertices + number % w.n_vertices
    nv = E * w.n_vertices
    vx, vy, vz = normal(nv, w.vertex_sigma_xy)[vertex], normal(nv, w.vertex_sigma_xy)[vertex], \
        normal(nv, w.vertex_sigma_z)[vertex]
    u = uniform(n)
    if w.pt_dist == "loguniform":
        pt = torch.exp(math.log(w.pt_range[0]) + u * math.log(w.pt_range[1] / w.pt_range[0]))
    elif w.pt_dist == "exp":
        pt = w.pt_range[0] - torch.log1p(-u)
    else:  # pt^-3 above the lower end
        pt = w.pt_range[0] * (1.0 - u) ** -0.5
    eta, phi0 = uniform(n, -w.eta_max, w.eta_max), uniform(n, -math.pi, math.pi)
    q = torch.where(uniform(n) < 0.5, -1.0, 1.0).to(torch.float64)
    R = pt / (0.299792458 * w.b_field) * 100.0  # cm
    cx, cy = vx + q * R * torch.sin(phi0), vy - q * R * torch.cos(phi0)
    d, psi = torch.hypot(cx, cy), torch.atan2(cy, cx)
    th0 = torch.atan2(vy - cy, vx - cx)
    cols = {k: [] for k in ("x", "y", "z", "group", "track", "slot")}

    def add(x, y, z, e, layer, track, slot):
        for k, v in zip(("x", "y", "z", "group", "track", "slot"), (x, y, z, e * L + layer, track, slot)):
            cols[k].append(v)

    for layer in range(L):
        half = events.half_length(w.radii[layer])
        r = w.radii[layer] + uniform(n, -w.stagger, w.stagger)
        arg = (r * r - d * d - R * R) / (2.0 * R * d)
        ok = arg.abs() <= 1.0
        dth = torch.arccos(arg.clamp(-1.0, 1.0))
        alpha = torch.minimum(torch.remainder((th0 - (psi + dth)) * q, 2 * math.pi),
                              torch.remainder((th0 - (psi - dth)) * q, 2 * math.pi))
        th = th0 - q * alpha
        x, y, z = cx + R * torch.cos(th), cy + R * torch.sin(th), vz + R * alpha * torch.sinh(eta)
        ok &= (alpha < math.pi) & (z.abs() < half) & (uniform(n) < w.efficiency)
        ph, along = torch.atan2(y, x), normal(n, w.sigma_rphi)
        x, y, z = x - torch.sin(ph) * along, y + torch.cos(ph) * along, z + normal(n, w.sigma_z)
        keep = torch.nonzero(ok)[:, 0]
        add(x[keep], y[keep], z[keep], ev[keep], layer, number[keep] + 1, keep * L + layer)
        if w.noise_fraction:
            noise = torch.round(w.noise_fraction * torch.bincount(ev[keep], minlength=E)).to(torch.int64)
            e = torch.repeat_interleave(torch.arange(E, device="cuda"), noise)
            m = e.numel()
            r, ph = w.radii[layer] + uniform(m, -w.stagger, w.stagger), uniform(m, -math.pi, math.pi)
            add(r * torch.cos(ph), r * torch.sin(ph), uniform(m, -half + 0.01, half - 0.01), e, layer,
                torch.zeros_like(e), torch.full_like(e, -1))
    c = {k: torch.cat(v) for k, v in cols.items()}
    # by event and layer, shuffled inside a layer
    key = (c["group"] << 31) + torch.randint(1 << 31, c["group"].shape, generator=gen, device="cuda")
    order = torch.sort(key, stable=True)[1]
    c = {k: v[order] for k, v in c.items()}
    hit_of = torch.full((n * L,), -1, dtype=torch.int64, device="cuda")
    real = torch.nonzero(c["slot"] >= 0)[:, 0]
    hit_of[c["slot"][real]] = real
    layer, event = c["group"] % L, c["group"] // L
    module = torch.floor((torch.atan2(c["y"], c["x"]) + math.pi) * (64 / (2 * math.pi))).to(torch.int64) % 64
    layer_hits = torch.bincount(c["group"], minlength=E * L).reshape(E, L).cpu().numpy().astype(np.uint32)
    offsets = np.cumsum(layer_hits, axis=1, dtype=np.uint32) - layer_hits
    totals = layer_hits.sum(axis=1, dtype=np.uint32)

    def column(v, dtype):
        out = capi.pinned_empty(v.shape, dtype)  # page-locked, as a program that uploads often keeps its columns
        out[...] = v.to(torch.float32 if dtype == np.float32 else torch.int32).cpu().numpy().view(dtype)
        return out

    batch = events.EventBatch(
        x=column(c["x"], np.float32), y=column(c["y"], np.float32), z=column(c["z"], np.float32),
        layer=column(layer + 1, np.uint32), det_id=column((layer + 1) * 100000 + module, np.uint32),
        hit_id=column(c["track"], np.uint32), event=column(event, np.uint32),
        event_offsets=np.ascontiguousarray(np.cumsum(totals, dtype=np.uint32) - totals),
        layer_hits=layer_hits, layer_offsets=np.ascontiguousarray(offsets),
        min_r=np.array([r - w.stagger for r in w.radii], np.float32),
        max_r=np.array([r + w.stagger for r in w.radii], np.float32),
        lts=w.lts, n_z=w.n_z, n_phi=w.n_phi, min_pt=w.min_pt, d_eta_cut=w.d_eta_cut, workload=w)
    return batch, hit_of.reshape(n, L), ev


def _track_triplets(batch, hit_of, ev, fakes, most, seed):
    """The first `most` triplets of consecutive layers (hits of one track, not straight; with `fakes`, a share of them
    again with the third hit of another track of the event), grouped by event and layer triplet and ordered by second
    and first hit, as the filter leaves them.  Returns h1, h2, h3 and the 0-based layer triplet, on the GPU."""
    gen = torch.Generator(device="cuda").manual_seed(seed + 77)
    parts = []
    pos = torch.stack([torch.as_tensor(np.asarray(v), device="cuda").double() for v in (batch.x, batch.y, batch.z)], 1)
    for k in range(len(batch.lts)):
        t = torch.nonzero((hit_of[:, k:k + 3] >= 0).all(1))[:, 0]
        p = pos[hit_of[t, k:k + 3]]
        t = t[_fit_model(p, torch.zeros_like(p), strict=True)["usable"]]
        a, b, c, e = hit_of[t, k], hit_of[t, k + 1], hit_of[t, k + 2], ev[t]
        parts.append((e, a, b, c, k))
        if fakes:
            i = torch.nonzero(torch.rand(t.numel(), generator=gen, device="cuda") < fakes)[:, 0]
            j = (i + 1 + torch.randint(16, i.shape, generator=gen, device="cuda")).clamp(max=max(t.numel() - 1, 0))
            i, j = i[e[i] == e[j]], j[e[i] == e[j]]
            parts.append((e[i], a[i], b[i], c[j], k))
    e, a, b, c = (torch.cat([p[i] for p in parts]) for i in range(4))
    lt = torch.cat([torch.full_like(p[0], p[4]) for p in parts])
    o = torch.sort(c, stable=True)[1]
    for key in (a, b, e * len(batch.lts) + lt):  # a stable sort by each, the leading one last
        o = o[torch.sort(key[o], stable=True)[1]]
    return a[o][:most], b[o][:most], c[o][:most], lt[o][:most]


# ------------------------------------------------------------------ states
class State:
    def __init__(self, case):
        self.case = case
        self.ctx = None

    def __del__(self):
        if self.ctx is not None:
            self.ctx.close()


def _zeros(n):
    a = capi.pinned_empty((n,), np.uint32)
    a[...] = 0
    return a


def _result_buffers(ctx, room):
    """Page-locked arrays for `room` triplets with their segments' offsets, and for their tracks."""
    st = ctx.stats()
    if max(st.n_triplets, st.n_track_entries) > room:
        raise RuntimeError(f"{st.n_triplets} triplets, {st.n_track_entries} track entries: room for {room}")
    return [_zeros(n) for n in (room, room, room, ctx.n_events * ctx.n_lt + 1)], \
        [_zeros(n) for n in (room, room, room + 1)]


def _room(case, group=0):
    return 256 + int(1.3 * _triplets_of(case["shape"], _tracks_of(case["shape"], case["events"], case["tracks"], group)))


def _n_caller_triplets(case):
    """Triplets of the link and fit kinds: a number that the tracks of every seed give."""
    tracks = _tracks_of("ttbar", case["events"], case["tracks"]).sum()
    return int(tracks * (3.0 if case["kind"] == "link" else 2.0))


def _shifts(n_layers, seed):
    rng = np.random.default_rng([seed, 5])
    return np.stack([rng.normal(0.0, 0.005, n_layers), rng.normal(0.0, 0.005, n_layers),
                     rng.normal(0.0, 20e-6, n_layers)], axis=1)


SIGMA_TIP = [0.01, 0.015, 0.03, 0.04, 0.05, 0.06, 0.07, 0.08]  # cm, per layer triplet of the alignment workload
SIGMA_Z = 0.002


def prepare(case, seed):
    s = State(case)
    if case["kind"] == "scan":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        s.data = torch.randint(0, 60, (case["n"],), generator=gen, device="cuda", dtype=torch.int32)
        s.out = torch.empty_like(s.data)
        s.scan = capi.load().trax_prefix_sum_noalloc
        s.scan.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint64, ctypes.c_void_p, ctypes.c_char_p,
                           ctypes.c_size_t]
        s.scan.restype = ctypes.c_int
        s.message = ctypes.create_string_buffer(256)
        return s
    s.ctx = capi.Context(0)
    if case["kind"] in ("link", "fit"):
        return _prepare_triplets(s, case, seed)
    n_groups = case["groups"] if case["kind"] == "stream" else 1
    s.batches = []
    for g in range(n_groups):
        b, _, _ = _make_events(case["shape"], case["events"], case["tracks"], seed, group=g)
        b.n_z, b.n_phi = case["n_z"], case["n_phi"]
        s.batches.append(b)
    s.ctx.upload(s.batches[0])
    if case.get("fine"):
        s.ctx.set_fine_rows(case["fine"])
    s.linking = case.get("linking", True)
    s.buffers = []
    for g, b in enumerate(s.batches):  # a first run: the context keeps its buffers and its graph
        if n_groups > 1:
            s.ctx.upload_hits(b)
        s.ctx.seed_batch(use_graph=case.get("graph", True), run_linking=s.linking, d_eta_cut=b.d_eta_cut)
        s.buffers.append(_result_buffers(s.ctx, _room(case, g)))
    return s


def _prepare_triplets(s, case, seed):
    fit = case["kind"] == "fit"
    b, hit_of, ev = _make_events("ttbar", case["events"], case["tracks"], seed, config=4 if fit else 2)
    n = _n_caller_triplets(case)
    a = _track_triplets(b, hit_of, ev, 0.0 if fit else 0.5, n, seed)
    s.ctx.upload(b)
    s.ctx.set_tracklets(*(v.to(torch.int32).cpu().numpy().view(np.uint32) for v in a[:3]))
    if fit:
        s.ctx.fit_prepare(sigma_z=SIGMA_Z, sigma_tip=SIGMA_TIP, truth_only=True)
        s.shifts = _shifts(b.n_layers, seed)
    else:
        s.cut = b.d_eta_cut
        s.buffers = [_zeros(k) for k in (n, 3 * n, n + 1)]
    return s


# --------------------------------------------------------------------- run
def run(s):
    kind, ctx = s.case["kind"], s.ctx
    if kind == "scan":
        rc = s.scan(s.data.data_ptr(), s.out.data_ptr(), s.data.numel(), torch.cuda.current_stream().cuda_stream,
                    s.message, len(s.message))
        if rc:
            raise RuntimeError(s.message.value.decode())
        return s.out
    if kind == "fit":
        if s.case["grad"]:
            chi2, grad, _, diag = ctx.fit_backward(s.shifts, squares=True)
            return {"chi2": chi2, "grad": grad, "diag": diag}
        chi2, params = ctx.fit_forward(s.shifts, params=s.case["params"])
        return {"chi2": chi2, "params": params} if s.case["params"] else {"chi2": chi2}
    if kind == "link":
        ctx.connectivity(s.cut)
        ctx.circle_fit()
        ctx.cellular_automaton()
        eta, pt = ctx.eta_pt()
        ctx.tracks(out=s.buffers)
        return {"eta": eta, "pt": pt, "tracks": [v.view(np.int32) for v in s.buffers]}
    out = []
    for b, (trip, track) in zip(s.batches, s.buffers):
        if kind == "stream":
            ctx.upload_hits(b)
        if kind == "stages":
            ctx.grid_build()
            ctx.pair_gen()
            ctx.triplet_predict()
            ctx.triplet_filter()
            if s.linking and ctx.connectivity(b.d_eta_cut):
                ctx.circle_fit()
                ctx.cellular_automaton()
        else:
            ctx.seed_batch(use_graph=s.case.get("graph", True), run_linking=s.linking, d_eta_cut=b.d_eta_cut)
        ctx.triplets(out=trip)
        if s.linking:
            ctx.tracks(out=track)
        out.append([v.view(np.int32) for v in (trip + track if s.linking else trip)])
    return out


def work(case):
    """Bytes of the inputs and of the results, each once; operations of the windows and fits, in 32 bits."""
    if case["kind"] == "scan":
        return {"bytes": 8.0 * case["n"], "flops": float(case["n"])}
    if case["kind"] in ("link", "fit"):
        hits = SHAPES["ttbar"]["hits"] * case["events"] * case["tracks"]
        t = _n_caller_triplets(case)
        if case["kind"] == "fit":
            return {"bytes": 12.0 * hits + 12.0 * t + (16.0 * t if case["params"] else 0.0),
                    "flops": (550.0 if case["grad"] else 200.0) * t}
        # positions, triplets; eta and pt, states, chains and their offsets
        return {"bytes": 12.0 * hits + 12.0 * t + 20.0 * t, "flops": 80.0 * t}
    total = {"bytes": 0.0, "flops": 0.0}
    for g in range(case["groups"] if case["kind"] == "stream" else 1):
        tracks = _tracks_of(case["shape"], case["events"], case["tracks"], g)
        t = _triplets_of(case["shape"], tracks)
        # seven columns per hit; three hits per triplet, and its state, chain and offset
        total["bytes"] += 28.0 * SHAPES[case["shape"]]["hits"] * float(tracks.sum()) \
            + (24.0 if case.get("linking", True) else 12.0) * t
        total["flops"] += 600.0 * t
    return total


# ------------------------------------------------------------- exact values
def exact(case, seed):
    """chi2, gradient and per-triplet parameters of the fit, and the pseudorapidity of caller triplets, in 64 bits.
    The seeding chain's results are whole numbers."""
    if case["kind"] not in ("link", "fit"):
        return None
    fit = case["kind"] == "fit"
    b, hit_of, ev = _make_events("ttbar", case["events"], case["tracks"], seed, config=4 if fit else 2)
    h1, h2, h3, lt = _track_triplets(b, hit_of, ev, 0.0 if fit else 0.5, _n_caller_triplets(case), seed)
    pos = torch.stack([torch.as_tensor(np.asarray(v), device="cuda").double() for v in (b.x, b.y, b.z)], 1)
    if not fit:
        p = pos[h3] - pos[h1]
        eta = torch.asinh(p[:, 2] / torch.hypot(p[:, 0], p[:, 1]))
        return {"eta": eta.cpu().numpy(), "pt": None, "tracks": None}
    o = torch.sort(lt, stable=True)[1]  # the fit's rows run by layer triplet, then by event
    rows, lt = torch.stack([h1, h2, h3], 1)[o], lt[o]
    layer = lt[:, None] + torch.arange(3, device="cuda")
    w_tip = torch.as_tensor([1.0 / np.float64(np.float32(v)) ** 2 for v in SIGMA_TIP], device="cuda")[lt]
    w_z = 1.0 / float(np.float32(SIGMA_Z)) ** 2
    L = b.n_layers
    total = {"chi2": 0.0, "grad": torch.zeros(L, 3, dtype=torch.float64, device="cuda"),
             "diag": torch.zeros(L, 3, dtype=torch.float64, device="cuda")}
    params = []
    shifts = torch.as_tensor(_shifts(L, seed), device="cuda")
    for i in range(0, rows.shape[0], 1 << 20):  # in parts, for memory
        lay, wt = layer[i:i + (1 << 20)], w_tip[i:i + (1 << 20)]
        p = pos[rows[i:i + (1 << 20)]]
        a = shifts[lay].requires_grad_(case["grad"])
        m = _fit_model(p, a)
        used = m["usable"]
        chi2 = (wt * m["d0"] ** 2 + w_z * (m["e"] ** 2).sum(1))[used]
        total["chi2"] += float(chi2.detach().sum())
        params.append(torch.where(used[:, None], torch.stack([1 / m["R"], m["d0"], m["z0"], m["t"]], 1),
                                  torch.nan).detach())
        if case["grad"]:
            g = torch.autograd.grad(chi2.sum(), a, retain_graph=True)[0]
            h = torch.autograd.grad(m["d0"][used].sum(), a)[0]
            sss = (m["ds"] ** 2).sum(1, keepdim=True)
            pkk = w_z * (2.0 / 3.0 - m["ds"] ** 2 / sss)
            tq = m["t"][:, None] / torch.sqrt(1.0 - m["x"] ** 2)
            diag = torch.stack([wt[:, None] * h[..., 0] ** 2 + tq ** 2 * pkk, pkk, wt[:, None] * h[..., 2] ** 2], 2)
            for k, v in (("grad", g), ("diag", diag.detach())):
                total[k].index_add_(0, lay[used].reshape(-1), v[used].reshape(-1, 3))
    if case["grad"]:
        return {"chi2": total["chi2"], "grad": total["grad"].cpu().numpy(), "diag": total["diag"].cpu().numpy()}
    if case["params"]:
        return {"chi2": total["chi2"], "params": torch.cat(params).cpu().numpy()}
    return {"chi2": total["chi2"]}


def _fit_model(p, a, strict=False):
    """The circle and line through the triplets p [n, 3 hits, xyz] at shifts a [n, 3 hits, (dr, dz, dphi)], and where
    they can be used (with `strict`, at nearby shifts and in 32 bits too)."""
    x, y = p[..., 0], p[..., 1]
    r = torch.hypot(x, y)
    f, c, s = 1.0 + a[..., 0] / r, torch.cos(a[..., 2]), torch.sin(a[..., 2])
    X, Y, Z = f * (x * c - y * s), f * (x * s + y * c), p[..., 2] + a[..., 1]
    u2, v2, u3, v3 = X[:, 1] - X[:, 0], Y[:, 1] - Y[:, 0], X[:, 2] - X[:, 0], Y[:, 2] - Y[:, 0]
    q2, q3 = u2 * u2 + v2 * v2, u3 * u3 + v3 * v3
    D = 2.0 * (u2 * v3 - u3 * v2)
    ca, cb = (v3 * q2 - v2 * q3) / D, (u2 * q3 - u3 * q2) / D
    R = torch.hypot(ca, cb)
    X1, Y1 = X[:, 0], Y[:, 0]
    d0 = (X1 * X1 + Y1 * Y1 + 2.0 * (X1 * ca + Y1 * cb)) / (torch.hypot(X1 + ca, Y1 + cb) + R)
    rho = r + a[..., 0]
    xs = (rho / (2.0 * R[:, None])).clamp(max=1.0)
    arc = 2.0 * R[:, None] * torch.asin(xs)
    ds = arc - arc.mean(1, keepdim=True)
    dz = Z - Z.mean(1, keepdim=True)
    t = (ds * dz).sum(1) / (ds * ds).sum(1)
    e = dz - t[:, None] * ds
    z0 = Z.mean(1) - t * arc.mean(1)
    usable = (rho < (1.7 if strict else 1.8) * R[:, None]).all(1) & torch.isfinite(d0) \
        & (D.abs() > (1e-4 if strict else 1e-7) * torch.sqrt(q2 * q3))
    return {"R": R, "d0": d0, "t": t, "z0": z0, "e": e, "ds": ds, "x": xs, "usable": usable}
