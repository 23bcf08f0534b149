"""Workloads of the search, the track fit and the doublet network, for timing.

Every case is one call sequence a user's program makes through the public
entry points: the C ABI of include/velo_search.h, through the ctypes binding
cl_forward_gb300.native.  Events follow the synthetic VELO generator of
cl_forward_gb300.generator (same geometry, acceptance and distributions),
drawn here on the GPU so that thousands of events take milliseconds.

A search emits an event's tracks in no fixed order, and reserves the events'
output rows in the order in which they finish.  A program that wants
reproducible results therefore orders them by event and first hit (no two
tracks of an event start with the same hit) before it goes on; so does run().
"""
import ctypes
import functools
import math
import os

import numpy as np
import torch

from cl_forward_gb300 import learned, native
from cl_forward_gb300.events import TRACK_DTYPE
from cl_forward_gb300.generator import HALF_OVERLAP, MODULE_Z, N_MODULES, R_MAX, R_MIN, SIGMA_XY

WEIGHTS = os.path.join(os.path.dirname(native.__file__), "weights", "doublet_mlp.npz")

# Hits and tracks per primary vertex in this geometry (20 tracks per vertex).
HITS_PER_PV, TRACKS_PER_PV = 152.7, 20.3
MLP_MACS = 10 * 32 + 32 * 32 + 32 * 2
WIDTH_WEIGHT = 0.1


# ------------------------------------------------------------------ cases --
def _search(kind, events, pv=7.6, pv_spread=0.0, eff=0.98, noise=0.005, y_lanes=4, per_event=False):
    """`pv`: mean primary vertices per event; `pv_spread`: the mean itself is uniform in pv -+ pv_spread."""
    return {"kind": kind, "events": events, "pv": pv, "pv_spread": pv_spread, "eff": eff, "noise": noise,
            "y_lanes": y_lanes, "per_event": per_event}


def listed():
    return [
        # a trigger node or an event display searching one event as it arrives
        dict(_search("call", 1), name="one_event"),
        # the small sample of the reference's own runs: 100 events, one call on pinned buffers
        dict(_search("in_place", 100), name="hundred_events"),
        # an ordinary buffer of events through the default options (copied to the device and back)
        dict(_search("copied", 1003), name="copied_batch"),
        # the flagship workload: 10,000 events end to end, read and written in place
        dict(_search("in_place", 10000), name="scale_10k"),
        # events already on the device: search, fetch the tracks, fit them
        dict(_search("resident_fit", 10000), name="search_and_fit"),
        # very uneven pile-up, about 200 to 8,000 hits per event
        dict(_search("in_place", 10000, pv=16.0, pv_spread=14.0), name="uneven_10k"),
        # four times the pile-up, noisier and less efficient
        dict(_search("in_place", 4000, pv=30.0, eff=0.96, noise=0.02), name="dense_4k"),
        # events as the detector writes them: x-sort on the device, then the search
        dict(_search("unsorted", 5000), name="unsorted_5k"),
        # seeding pruned by the trained network
        dict(_search("learned", 5000), name="learned_5k"),
        # events and results in the caller's own device memory (no allocation by the library)
        dict(_search("device", 90), name="device_arrays"),
        # training the network: batches of 4,096 doublets, forward, backward, Adam
        {"name": "train", "kind": "train", "samples": 300000, "batch": 4096, "steps": 60},
        # scoring held-out doublets to calibrate the cuts
        {"name": "score", "kind": "score", "samples": 1000000},
    ]


def _most(case, per_pv):
    """Room for a case's hits or tracks, whatever the seed: eight standard deviations above the mean."""
    pvs = case["events"] * case["pv"]
    spread = case["events"] * case["pv_spread"] ** 2 / 3
    return int(per_pv * (pvs + 8 * math.sqrt(pvs + spread) + 20))


# each kind's largest drawn batch, in events of the ordinary pile-up
KIND_EVENTS = {"call": 8, "in_place": 10000, "copied": 10000, "resident_fit": 10000, "unsorted": 10000,
               "learned": 8000, "device": 90}


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["call", "in_place", "in_place", "in_place", "copied", "resident_fit", "unsorted", "learned",
                       "device", "train", "score"])
    if kind == "train":
        batch = _log_int(rng, 100, 8192)
        return {"kind": kind, "samples": _log_int(rng, 2000, 300000), "batch": batch,
                "steps": rng.randint(5, min(60, 60 * 4096 // batch))}
    if kind == "score":
        return {"kind": kind, "samples": _log_int(rng, 50, 1000000)}
    pv = rng.choice([2.0, 4.0, 7.6, 7.6, 12.0, 20.0, 30.0])
    spread = rng.choice([0.0, 0.0, 0.5 * pv]) if kind in ("in_place", "copied") else 0.0
    eff, noise = rng.choice([(0.98, 0.005), (0.96, 0.02)])
    most = min(KIND_EVENTS[kind], int(KIND_EVENTS[kind] * 7.6 / pv))
    return _search(kind, _log_int(rng, 1, max(1, most)), pv, spread, eff, noise, rng.choice([4, 4, 4, 1, 2, 3]),
                   kind == "in_place" and rng.random() < 0.2)


def work(case):
    kind, n = case["kind"], case.get("samples", 0)
    if kind == "train":
        seen = case["batch"] * case["steps"]
        return {"bytes": 48.0 * min(n, seen) + 8.0 * native.MLP_PARAMS, "flops": 6.0 * MLP_MACS * seen}
    if kind == "score":
        return {"bytes": 48.0 * n, "flops": 2.0 * MLP_MACS * n}
    hits, tracks = case["pv"] * HITS_PER_PV, case["pv"] * TRACKS_PER_PV
    per = 8 + 12 * N_MODULES + 16 * hits + 8 + 100 * tracks
    if kind == "resident_fit":
        per += 20 * tracks
    if kind == "unsorted":
        per += 8 + 12 * N_MODULES + 16 * hits   # the sorted events come back too
    return {"bytes": per * case["events"], "flops": 0.0}   # a search: comparisons, not a contraction


# ----------------------------------------------------------------- events --
def _events_on_gpu(case, seed, sort):
    """(words int32, word offset of each event, words of each event, hits of each event), on the GPU.

    The generator's physics: straight tracks from vertices near the beam line,
    a scattering kick after each crossed module, hit losses, smear, noise."""
    dev = torch.device("cuda")
    g = torch.Generator(dev).manual_seed(seed * 1000003 + 17)

    def uniform(n, lo, hi):
        return torch.rand(n, generator=g, device=dev, dtype=torch.float64) * (hi - lo) + lo

    def normal(n, sigma):
        return torch.randn(n, generator=g, device=dev, dtype=torch.float64) * sigma

    n = case["events"]
    events = torch.arange(n, device=dev)
    lam = uniform(n, case["pv"] - case["pv_spread"], case["pv"] + case["pv_spread"])
    n_pv = torch.poisson(lam, generator=g).long()
    pv_event = torch.repeat_interleave(events, n_pv)
    pvs = pv_event.numel()
    pv_x, pv_y, pv_z = normal(pvs, 0.05), normal(pvs, 0.05), normal(pvs, 50.0)
    n_trk = torch.poisson(torch.full((pvs,), 20.0, device=dev), generator=g).long()
    pv_of = torch.repeat_interleave(torch.arange(pvs, device=dev), n_trk)
    t = pv_of.numel()
    trk_event = pv_event[pv_of]
    first_trk = torch.searchsorted(trk_event, events)   # particle keys count from 1 in each event
    forward = uniform(t, 0.0, 1.0) < 0.85
    eta = torch.where(forward, uniform(t, 1.6, 5.0), uniform(t, -4.0, -2.0))
    phi = uniform(t, 0.0, 2.0 * math.pi)
    scatter = 0.5e-3 / (0.3 - 5.0 * torch.log1p(-uniform(t, 0.0, 1.0)))   # mrad GeV / p
    tan = torch.tan(2.0 * torch.atan(torch.exp(-eta)))
    tx, ty = tan * torch.cos(phi), tan * torch.sin(phi)
    x, y, z = pv_x[pv_of], pv_y[pv_of], pv_z[pv_of]
    zs = torch.tensor(MODULE_Z, device=dev)
    step = torch.where(forward, 1, -1)
    start = torch.where(forward, torch.searchsorted(zs, z, right=True), torch.searchsorted(zs, z) - 1)
    got = []
    for k in range(N_MODULES):
        m = start + k * step
        alive = (m >= 0) & (m < N_MODULES)
        m = m.clamp(0, N_MODULES - 1)
        zm = torch.where(alive, zs[m], z)
        x, y, z = x + tx * (zm - z), y + ty * (zm - z), zm
        r2 = x * x + y * y
        side = torch.where(m % 2 == 0, x < HALF_OVERLAP, x > -HALF_OVERLAP)
        crossed = alive & side & (r2 >= R_MIN * R_MIN) & (r2 <= R_MAX * R_MAX)
        at = torch.nonzero(crossed & (uniform(t, 0.0, 1.0) < case["eff"])).squeeze(1)
        got.append((at, m[at], x[at] + normal(at.numel(), SIGMA_XY), y[at] + normal(at.numel(), SIGMA_XY)))
        kick = torch.where(crossed, scatter, torch.zeros_like(scatter))
        tx, ty = tx + normal(t, 1.0) * kick, ty + normal(t, 1.0) * kick
    trk, mod, hx, hy = (torch.cat([c[i] for c in got]) for i in range(4))
    group = trk_event[trk] * N_MODULES + mod
    key = trk - first_trk[trk_event[trk]] + 1
    # noise: uniform over the module's half ring, as many as the share of its hits says
    real = torch.bincount(group, minlength=n * N_MODULES)
    n_noise = torch.poisson(case["noise"] * real.double(), generator=g).long()
    noise_group = torch.repeat_interleave(torch.arange(n * N_MODULES, device=dev), n_noise)
    q = noise_group.numel()
    r = torch.sqrt(uniform(q, R_MIN * R_MIN, R_MAX * R_MAX))
    a = uniform(q, -0.5 * math.pi, 0.5 * math.pi) + torch.where(noise_group % N_MODULES % 2 == 0, math.pi, 0.0)
    group = torch.cat([group, noise_group])
    key = torch.cat([key, (1 << 23) + torch.arange(q, device=dev)])
    hx, hy = (torch.cat([u, v]).float() for u, v in ((hx, r * torch.cos(a)), (hy, r * torch.sin(a))))
    order = torch.argsort(hx, stable=True) if sort else torch.arange(group.numel(), device=dev)
    order = order[torch.argsort(group[order], stable=True)]
    group, key, hx, hy = group[order], key[order], hx[order], hy[order]
    # pack: header, module tables, then IDs, x, y, z; events at 16-byte boundaries
    num = torch.bincount(group, minlength=n * N_MODULES).view(n, N_MODULES)
    hits = num.sum(1)
    size = 2 + 3 * N_MODULES + 4 * hits
    room = (size + 3) // 4 * 4
    off = torch.cumsum(room, 0) - room
    words = torch.zeros(int(room.sum()), dtype=torch.int32, device=dev)
    words[off], words[off + 1] = N_MODULES, hits.int()
    column = torch.arange(N_MODULES, device=dev)
    for k, table in enumerate((zs.trunc().int().expand(n, -1), (torch.cumsum(num, 1) - num).int(), num.int())):
        words[(off + 2 + k * N_MODULES).unsqueeze(1) + column] = table
    ev = group // N_MODULES
    before = torch.cumsum(hits, 0) - hits
    at = off[ev] + 2 + 3 * N_MODULES + torch.arange(group.numel(), device=dev) - before[ev]
    mod = group % N_MODULES
    ids = ((key << 8) | mod).to(torch.int32)
    for k, v in enumerate((ids, hx.view(torch.int32), hy.view(torch.int32), zs.float()[mod].view(torch.int32))):
        words[at + k * hits[ev]] = v
    return words, off, size, hits


class _State:
    """Buffers, options and handle of one search case."""


def _pinned(shape, dtype):
    return torch.zeros(shape, dtype=dtype, pin_memory=True)


@functools.lru_cache(maxsize=None)
def _context(with_network=False):
    """The handle a program keeps for its calls, one without and one with the network's weights."""
    ctx = native.Context(0)
    if with_network:
        w = np.load(WEIGHTS)
        ctx.set_mlp(w["weights"], float(w["keep_threshold"]), float(w["window_margin"]), float(w["min_keep_rate"]),
                    int(w["max_event_hits"]))
    return ctx


def _doublets(n, seed, labelled):
    """Doublet features in the ranges the seeding produces, and labels and width targets from a smooth rule."""
    g = torch.Generator().manual_seed(seed * 1000003 + 29)
    slope = torch.randn(n, 2, generator=g).clamp(-3.5, 3.5) * 0.6
    rest = torch.rand(n, 8, generator=g)
    x = torch.cat([slope, 0.12 + 0.88 * rest[:, :1] ** 2, 2 * rest[:, 1:2] - 1, (rest[:, 2:3] * 48).floor() / 52 + 4 / 52,
                   2 * rest[:, 3:5] - 1, -0.25 - 0.25 * (rest[:, 5:6] > 0.8).float(), (rest[:, 6:7] ** 2 * 40).floor() / 32,
                   rest[:, 7:8]], 1)
    if not labelled:
        return x.numpy()
    odds = 2.5 - 4.0 * (x[:, 0] * x[:, 3].cos() - x[:, 5]).abs() - 3.0 * (x[:, 1] * x[:, 3].sin() - x[:, 6]).abs()
    label = (torch.rand(n, generator=g) < torch.sigmoid(odds)).float()
    target = label * (0.05 + 0.1 * torch.rand(n, generator=g) * (1 + x[:, 0].abs()))
    return x.numpy(), label.numpy(), target.numpy()


def prepare(case, seed):
    s = _State()
    s.kind = kind = case["kind"]
    if kind == "train":
        s.x, s.label, s.target = _doublets(case["samples"], seed, True)
        s.weights = learned.init_weights(seed)
        s.steps, s.batch, s.seed = case["steps"], case["batch"], seed
        return s
    if kind == "score":
        s.x = _doublets(case["samples"], seed, False)
        s.weights = np.load(WEIGHTS)["weights"]
        return s
    words, off, size, hits = _events_on_gpu(case, seed, sort=kind != "unsorted")
    n, total = case["events"], int(hits.sum())
    rows = hits.clamp(min=1)
    s.base = torch.cumsum(rows, 0) - rows   # a row per (event, hit): the order of the results
    # where the ordered results go on the GPU, the rest left zero
    most = _most(case, TRACKS_PER_PV)
    s.ordered = [torch.zeros((most, 25), dtype=torch.int32, device="cuda")]
    s.n, s.y_lanes = n, case["y_lanes"]
    s.offsets, s.sizes = (4 * off).cpu().numpy().astype(np.uint64), (4 * size).cpu().numpy().astype(np.uint64)
    if kind == "device":
        s.words, s.total_hits, s.max_hits = words, total, int(hits.max())
        s.d_off, s.d_size = 4 * off, 4 * size
        s.d_tracks = torch.zeros((total + n, 25), dtype=torch.int32, device="cuda")
        s.d_counts, s.d_first, s.d_status = (torch.zeros(n, dtype=d, device="cuda")
                                             for d in (torch.int32, torch.int64, torch.int32))
        return s
    s.words = torch.empty(words.shape, dtype=torch.int32, pin_memory=True)
    s.words.copy_(words)
    s.events = s.words.numpy().view(np.uint8)
    if kind == "call":
        s.most = most
        s.blobs = [s.events[int(o):int(o) + int(z)].tobytes() for o, z in zip(s.offsets, s.sizes)]
    else:
        s.tracks = torch.empty((most, 25), dtype=torch.int32, pin_memory=True)
        s.counts, s.first, s.status = (_pinned(n, d) for d in (torch.int32, torch.int64, torch.int32))
        s.out = (s.tracks.numpy().reshape(-1).view(TRACK_DTYPE), s.counts.numpy().view(np.uint32),
                 s.first.numpy().view(np.uint64), s.status.numpy().view(np.uint32))
    s.ctx = _context(kind == "learned")
    options = {"y_lanes": case["y_lanes"]}
    if kind in ("in_place", "learned"):
        options["host_direct"] = 1
    if kind == "learned":
        options["learned"] = 1
    if case["per_event"]:   # the reference's launch style: a 256-thread group per event
        options.update(launch_mode=native.LAUNCH_PER_EVENT, threads_per_event=256)
    s.options = native.default_options(**options)
    if kind == "resident_fit":
        s.ctx = native.Context(0)   # it holds the staged events
        s.ctx.stage(s.events, s.offsets, s.sizes)
        s.fits = torch.empty((most, 5), dtype=torch.float32, pin_memory=True)
        s.ordered.append(torch.zeros((most, 5), dtype=torch.float32, device="cuda"))
    if kind == "unsorted":
        room = n * (2 + 3 * N_MODULES + 4) + 4 * _most(case, 1.1 * HITS_PER_PV)
        s.sorted = _pinned(room, torch.int32)
    return s


# ------------------------------------------------------------------- runs --
def _ordered(s, total, tracks, counts, first, *more):
    """The results on the GPU, by event and first hit."""
    by_first = torch.argsort(first)
    event = torch.repeat_interleave(by_first, counts[by_first], output_size=total)
    order = torch.argsort((s.base[event] + tracks[:, 1]).int())
    for out, v in zip(s.ordered, (tracks, *more)):
        torch.index_select(v, 0, order, out=out[:total])
    return s.ordered


def _fetched(s, *more):
    """As _ordered, for results in pinned host memory."""
    total = int(s.out[1].sum())
    tracks, counts, first, *more = (v.to("cuda", non_blocking=True)
                                    for v in (s.tracks[:total], s.counts, s.first, *(m[:total] for m in more)))
    return _ordered(s, total, tracks, counts, first, *more)


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _run_device(s):
    stream = torch.cuda.current_stream().cuda_stream
    st = native.load().velo_search_device_static(_ptr(s.words), _ptr(s.d_off), _ptr(s.d_size), s.n, s.total_hits,
                                                 s.max_hits, s.y_lanes, _ptr(s.d_tracks), s.d_tracks.shape[0],
                                                 _ptr(s.d_counts), _ptr(s.d_first), _ptr(s.d_status),
                                                 ctypes.c_void_p(stream))
    if st != native.OK:
        raise native.VeloError(st, "velo_search_device_static")
    total = int(s.d_counts.sum())
    return [*_ordered(s, total, s.d_tracks[:total], s.d_counts, s.d_first), s.d_counts, s.d_status]


def _check(s, st, what):
    if st != native.OK:
        raise native.VeloError(st, what)


def run(s):
    if s.kind == "train":
        return native.mlp_train(s.x, s.label, s.target, s.weights, s.steps, s.batch, 1e-3, s.seed)
    if s.kind == "score":
        return native.mlp_forward(s.weights, s.x)
    if s.kind == "device":
        return _run_device(s)
    if s.kind == "call":
        per_event, status = s.ctx.search(s.blobs, s.options)
        per_event = [t[np.argsort(t["hits"][:, 0])] for t in per_event]
        out = np.zeros((s.most, 25), np.int32)
        found = np.concatenate(per_event)
        out[:len(found)] = found.view(np.int32).reshape(-1, 25)
        return [out, np.array([len(t) for t in per_event], np.int32), status.view(np.int32)]
    if s.kind == "resident_fit":
        s.ctx.run(s.options)
        s.ctx.fetch_into(*s.out)
        _check(s, native.load().velo_fit_tracks(s.ctx._h, _ptr(s.fits), s.fits.shape[0]), "velo_fit_tracks")
        return [*_fetched(s, s.fits), s.counts, s.status]
    if s.kind == "unsorted":
        s.ctx.stage(s.events, s.offsets, s.sizes)
        s.ctx.sort_staged()
        s.ctx.run(s.options)
        s.ctx.fetch_into(*s.out)
        # the tracks' hits index the sorted events
        _check(s, native.load().velo_fetch_staged(s.ctx._h, _ptr(s.sorted), 4 * s.sorted.numel()), "velo_fetch_staged")
        return [*_fetched(s), s.counts, s.status, s.sorted]
    s.ctx.search_packed_into(s.events, s.offsets, s.sizes, s.options, *s.out)
    return [*_fetched(s), s.counts, s.status]


# ------------------------------------------------------------------ exact --
def _sample_order(n, count, seed):
    """The documented sampling without replacement per epoch: a Fisher-Yates shuffle driven by splitmix64."""
    mask, s, order, out = (1 << 64) - 1, seed, list(range(n)), []
    while len(out) < count:
        for i in range(n - 1, 0, -1):
            s = (s + 0x9E3779B97F4A7C15) & mask
            z = ((s ^ (s >> 30)) * 0xBF58476D1CE4E5B9) & mask
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
            j = (z ^ (z >> 31)) % (i + 1)
            order[i], order[j] = order[j], order[i]
        out += order[:count - len(out)]
    return np.array(out, np.int64)


def _layers(w):
    return w[:320].view(32, 10), w[320:352], w[352:1376].view(32, 32), w[1376:1408], w[1408:1472].view(2, 32), w[1472:]


def _outputs(w, x):
    a, b, c, d, e, f = _layers(w)
    return torch.relu(torch.relu(x @ a.T + b) @ c.T + d) @ e.T + f


def exact(case, seed):
    """The network's outputs in 64 bits.  The searches return whole numbers and, with the fit, lines through
    tracks that only a search can give: there is no value to state without it."""
    if case["kind"] == "score":
        s = prepare(case, seed)
        return _outputs(torch.tensor(s.weights).double().cuda(), torch.tensor(s.x).double().cuda())
    if case["kind"] != "train":
        return None
    s = prepare(case, seed)
    x, label, target = (torch.tensor(v).double().cuda() for v in (s.x, s.label, s.target))
    index = torch.tensor(_sample_order(len(s.x), s.steps * s.batch, s.seed)).cuda().view(s.steps, s.batch)
    w = torch.tensor(s.weights).double().cuda()
    m, v = torch.zeros_like(w), torch.zeros_like(w)
    beta1, beta2, lr, eps = (float(np.float32(c)) for c in (0.9, 0.999, 1e-3, 1e-8))
    losses = []
    for k in range(s.steps):
        w.requires_grad_(True)
        xb, yb, tb = x[index[k]], label[index[k]], target[index[k]]
        o = _outputs(w, xb)
        loss = (torch.nn.functional.binary_cross_entropy_with_logits(o[:, 0], yb, reduction="none")
                + yb * WIDTH_WEIGHT * (o[:, 1] - tb) ** 2).mean()
        grad, = torch.autograd.grad(loss, w)
        w = w.detach()
        m, v = beta1 * m + (1 - beta1) * grad, beta2 * v + (1 - beta2) * grad * grad
        w = w - lr * (m / (1 - beta1 ** (k + 1))) / (torch.sqrt(v / (1 - beta2 ** (k + 1))) + eps)
        losses.append(float(loss.detach()))
    return w, torch.tensor(losses, dtype=torch.float64)
