"""The calls whose speed matters to a user of this package, with their inputs.

A program that uses the package packs hit records on the device, runs the
reconstruction of the batch and gathers the global tracks; it may prune the
YZ stage with the combination scorer, continue to vertices, dimuons and
histograms, write the reference's output rows, convert drift times with the
R-T calibration, and score or train the scorer's network.  Each listed case
is one such call on seeded events of the generator's workloads:

  dimuon   one opposite-sign muon pair and Poisson(150) noise per event;
  uneven   0-3 muons, log-normal noise (median 300, sigma 0.8) per event:
           a few events hold most of the combinations;
  high     two muons, Poisson(1000) noise and after-pulses: the event
           reducer rejects every event.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "e1039-gpu_gb300"))

from orgpu import GEOMETRY_E906, _lib, learned, pipeline  # noqa: E402
from orgpu import layout as L  # noqa: E402
from orgpu import synth as S  # noqa: E402

DATA = os.path.dirname(GEOMETRY_E906)
CALIBRATION = os.path.join(DATA, "calibration_e906.txt")

# distinct events generated for a batch; a larger batch draws from them
POOL = 4096

# per event of each workload: hit records, XZ tracklets kept as track
# records, FP32 operations of the reference's fits and chi2 sums
PER_EVENT = {"dimuon": (213, 8, 1.5e5), "uneven": (480, 15, 2.3e6), "high": (1170, 0, 0.0)}

MLP_FLOPS = 2 * (16 * 64 + 64 * 64 + 64)
TRAIN_BATCH = 8192


def listed():
    return [
        # an online monitor that looks at a single triggered event
        {"name": "event_1", "call": "chain", "events": "dimuon", "n": 1},
        # the smallest batch the event server runs
        {"name": "spill_256", "call": "chain", "events": "dimuon", "n": 256},
        # a small uneven batch: some warps get far more work than others
        {"name": "uneven_333", "call": "chain", "events": "uneven", "n": 333},
        # a full batch of the reference program (its structs hold 10,000 events)
        {"name": "dimuon_10000", "call": "chain", "events": "dimuon", "n": 10000},
        # the throughput workload: a resident batch of 100,000 uneven events
        {"name": "uneven_100000", "call": "chain", "events": "uneven", "n": 100000},
        # high-occupancy running, where the packer and the event reducer are all there is
        {"name": "high_20000", "call": "chain", "events": "high", "n": 20000},
        # the chain with the combination scorer pruning the YZ stage
        {"name": "scored_10000", "call": "scored", "events": "uneven", "n": 10000},
        # what follows global tracking: selection, vertices, dimuons, histograms
        {"name": "physics_10000", "call": "physics", "events": "dimuon", "n": 10000},
        # the reference program as a whole, to its output rows
        {"name": "program_2000", "call": "program", "events": "dimuon", "n": 2000},
        # packing with the drift distances from the R-T calibration
        {"name": "pack_rt_16001", "call": "pack_rt", "events": "uneven", "n": 16001},
        # the scorer's network alone, on a table of rows
        {"name": "score_1000003", "call": "score", "n": 1000003},
        # one epoch of the scorer's training (forward, backward, Adam)
        {"name": "train_40000", "call": "train", "n": 40000},
    ]


def draw(rng):
    call = rng.choice(["chain", "chain", "chain", "chain", "scored", "physics", "program", "pack_rt", "score", "train"])
    lo, hi = {"chain": (1, 60000), "scored": (100, 20000), "physics": (100, 20000), "program": (10, 4000),
              "pack_rt": (100, 20000), "score": (1000, 4000000), "train": (TRAIN_BATCH, 80000)}[call]
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if call in ("score", "train"):
        return {"call": call, "n": n}
    events = rng.choice(["dimuon", "uneven", "uneven", "high"] if call in ("chain", "pack_rt") else ["dimuon", "uneven"])
    return {"call": call, "events": events, "n": min(n, 20000) if events == "high" else n}


def _records(geo, events, n, seed):
    """Hit records (uint8) and event offsets of n seeded events, on the GPU."""
    m = min(n, POOL)
    cfg = {"dimuon": S.config_small, "uneven": S.config_uneven, "high": S.config_high_occupancy}[events](m, seed)
    rec, off, _ = S.generate(geo, cfg)
    rec, off = S.cap_records(rec, off)
    d_rec = torch.from_numpy(rec.view(np.uint8)).cuda()
    d_off = torch.from_numpy(off).cuda()
    if n > m:
        gen = torch.Generator().manual_seed(seed)
        pick = torch.randint(0, m, (n,), generator=gen).cuda()
        length = (d_off[1:] - d_off[:-1])[pick]
        new = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
        new[1:] = torch.cumsum(length, 0)
        at = torch.repeat_interleave(d_off[pick] - new[:-1], length)
        at += torch.arange(at.numel(), device="cuda")
        d_rec = d_rec.view(torch.int32).view(-1, 4)[at].reshape(-1).view(torch.uint8)
        d_off = new
    return d_rec, d_off


def _hits(b):
    return {"nhits_cham": b.nhits_cham, "hits_cham": b.hits_cham, "nhits_hodo": b.nhits_hodo,
            "hits_hodo": b.hits_hodo, "nhits_prop": b.nhits_prop, "hits_prop": b.hits_prop}


def _tracks(b):
    return {"ntracks": b.ntracks, "tracks": b.tracks, "ntracklets": b.ntracklets, "toomany": b.toomany,
            "nhits_cham": b.nhits_cham, "nhits_hodo": b.nhits_hodo, "nhits_prop": b.nhits_prop}


def _scorer_rows(n, seed, sp):
    """Feature rows with the spread of the rows the scorer was trained on."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(n, L.NFEAT, generator=gen, device="cuda")
    return x / torch.from_numpy(sp.inv_std).cuda() + torch.from_numpy(sp.mean).cuda()


def _train_inputs(n, seed, sp):
    x = _scorer_rows(n, seed, sp)
    gen = torch.Generator(device="cuda").manual_seed(seed + 1)
    labels = (torch.rand(n, generator=gen, device="cuda") < 0.02).to(torch.uint8)
    return x, labels, learned.ScorerParams.init(sp.mean, sp.inv_std, seed)


def prepare(case, seed):
    call, n = case["call"], case["n"]
    plane, wp = _lib.geometry_load(GEOMETRY_E906)
    if call in ("score", "train"):
        rc = pipeline.Reconstruction(plane, 0, max_events=1)
        sp = learned.ScorerParams.load(learned.MODEL_COMBO_E906)
        s = {"call": call, "n": n, "rc": rc, "learned": learned.Learned(rc)}
        if call == "score":
            s["model"] = learned.DeviceModel(sp)
            s["rows"] = _scorer_rows(n, seed, sp).reshape(-1)
            s["scores"] = torch.zeros(n, device="cuda")
        else:
            x, labels, start = _train_inputs(n, seed, sp)
            s["trainer"] = learned.Trainer(s["learned"], start, x.reshape(-1), labels, batch=TRAIN_BATCH, pos_weight=20.0)
            s["rng"] = np.random.default_rng(seed)
        return s
    geo = S.Geometry(plane, wp)
    rec, off = _records(geo, case["events"], n, seed)
    # the default context is sized for 100,000 events; smaller ones by their largest batch
    rc = pipeline.Reconstruction(plane, 0, max_events=None if n > 50000 else max(n, 256))
    b = pipeline.DeviceBatch(n, with_tracks=call != "pack_rt")
    for t in _hits(b).values():
        t.zero_()
    s = {"call": call, "n": n, "rc": rc, "b": b, "rec": rec, "off": off,
         "wp": torch.from_numpy(geo.wire_pos_f32().reshape(-1)).cuda()}
    if call == "chain":
        s["rows"] = torch.zeros(max(64, 4 * n) * L.COLLECT_STRIDE, device="cuda")
        s["count"] = torch.zeros(1, dtype=torch.int64, device="cuda")
    elif call == "scored":
        s["scorer"] = learned.ComboScorer(rc)
        s["sp"] = learned.ScorerParams.load(learned.MODEL_COMBO_E906)
        s["model"] = learned.DeviceModel(s["sp"])
        s["outer"] = learned.OuterRows(n, max_rows=max(100000, 600 * n))
    elif call == "pack_rt":
        s["rt"] = pipeline.rt_to_device(_lib.rt_load(CALIBRATION, plane)[0])
    if call in ("physics", "program"):
        s["dimuons"] = pipeline.DeviceDimuons(n)
        s["hists"] = pipeline.DeviceHists()
        s["trigger"] = torch.from_numpy(S.trigger_bits(n, seed)).cuda()
    if call == "program":
        # row tables of its own, as the C interface takes them
        s["caps"] = {"events": n, "hits": n * 512, "tracks": n * 8, "track_hits": n * 8 * L.MAXHITS_PER_TRACK, "dimuons": n * 4}
        widths = {"events": L.OUT_EV_FIELDS, "hits": L.OUT_HIT_FIELDS, "tracks": L.OUT_TRACK_FIELDS,
                  "track_hits": L.OUT_TRACKHIT_FIELDS, "dimuons": L.OUT_DIMUON_FIELDS}
        s["tables"] = {k: torch.zeros(s["caps"][k] * w, dtype=torch.int64 if k == "events" else torch.float32, device="cuda")
                       for k, w in widths.items()}
        s["tables"]["counts"] = torch.zeros(5, dtype=torch.int64, device="cuda")
    if call == "physics":
        rc.pack(b, rec, off, s["wp"])
        rc.run_batch(b)
        rc.sync()
    return s


def _output_rows(s):
    rc, b, d = s["rc"], s["b"], s["dimuons"]
    v = L.OrOutputView()
    v.counts = s["tables"]["counts"].data_ptr()
    for k, cap in s["caps"].items():
        setattr(v, k, s["tables"][k].data_ptr())
        setattr(v, "cap_" + k, cap)
    _lib.check(rc.lib.or_output_rows(rc.ctx, b.hits_view(), b.tracks_view(), d.view(), b.toomany.data_ptr(), None, None,
                                     7.0, v, b.n, torch.cuda.current_stream().cuda_stream), "or_output_rows")


def run(s):
    call, rc, b = s["call"], s["rc"], s.get("b")
    if call == "score":
        s["learned"].score(s["model"], s["rows"], s["n"], s["scores"])
        return {"scores": s["scores"]}
    if call == "train":
        t = s["trainer"]
        loss = t.epoch(s["rng"])
        return {"loss": loss, "param": t.param, "m1": t.m1, "m2": t.m2}
    if call == "pack_rt":
        rc.pack_rt(b, s["rec"], s["off"], s["wp"], s["rt"])
        return _hits(b)
    if call != "physics":
        rc.pack(b, s["rec"], s["off"], s["wp"])
    if call == "chain":
        rc.run_batch(b)
        rc.collect(b, s["rows"], s["count"])
        out = dict(_tracks(b), count=s["count"])
        if s["n"] <= 256:  # the row order of larger batches is not fixed
            out["rows"] = s["rows"]
        return out
    if call == "scored":
        s["scorer"].run_batch(b, s["outer"], s["model"], s["sp"].t_keep, s["sp"].t_unc)
        return dict(_tracks(b), rows=s["outer"].rows, uncertain=s["outer"].uncertain)
    if call == "program":
        rc.run_batch(b)
    rc.selection(b)
    s["hists"].zero_counts()
    rc.run_physics(b, s["dimuons"], s["hists"], s["trigger"])
    out = {"ndimuons": s["dimuons"].ndimuons, "dimuons": s["dimuons"].dimuons,
           "hists": s["hists"].buf[L.OrHists.values.offset:].view(torch.float32)}
    if call == "program":
        _output_rows(s)
        out.update(s["tables"])
    else:
        out.update(tracks=b.tracks)
    return out


def work(case):
    call, n = case["call"], case["n"]
    if call == "score":
        return {"bytes": n * (64 + 4), "flops": n * MLP_FLOPS}
    if call == "train":
        rows = n // TRAIN_BATCH * TRAIN_BATCH
        return {"bytes": rows * (64 + 1 + 8) + 3 * 2 * 4 * L.MLP_NPARAM, "flops": rows * 3 * MLP_FLOPS}
    hits, tracklets, flops = PER_EVENT[case["events"]]
    packed = n * (8 + 16 * hits + 20 * hits + 4 * 54)  # records in, hit slots and their counts out
    if call == "pack_rt":
        return {"bytes": packed, "flops": n * hits * 6}
    tracks = n * (4 * L.NTRKPARAM * tracklets + 64 + 5)  # records, slot counts, flags
    swim = n * 2e4
    if call == "physics":
        return {"bytes": tracks, "flops": swim}
    if call == "program":
        return {"bytes": packed + tracks + n * 20 * hits, "flops": n * flops + swim}
    return {"bytes": packed + tracks, "flops": n * flops}


# -- the same in 64 bits -----------------------------------------------------

def _spline(t, r):
    """Piece coefficients of the cubic spline through (t, r) with zero end slopes."""
    n = len(t)
    h, dd = np.diff(t), np.diff(r) / np.diff(t)
    a = np.zeros((n, n))
    rhs = np.zeros(n)
    a[0, 0] = a[-1, -1] = 1.0
    for k in range(1, n - 1):
        a[k, k - 1], a[k, k], a[k, k + 1] = h[k], 2 * (h[k - 1] + h[k]), h[k - 1]
        rhs[k] = 3 * (h[k] * dd[k - 1] + h[k - 1] * dd[k])
    s = np.linalg.solve(a, rhs)
    return s[:-1], (3 * dd - 2 * s[:-1] - s[1:]) / h, (s[:-1] + s[1:] - 2 * dd) / h ** 2


def _calibration():
    out = {}
    with open(CALIBRATION) as f:
        lines = [x.split() for x in f if x.strip()]
    i = 0
    while i < len(lines):
        det, nbin, tmin, tmax = int(lines[i][0]), int(lines[i][1]), float(lines[i][2]), float(lines[i][3])
        pts = np.array([[float(v) for v in x[1:3]] for x in lines[i + 1:i + 1 + nbin]])
        i += 1 + nbin
        if nbin > 1 and (det <= 30 or det > 46):
            out[det] = (tmin, tmax, pts[:, 0], pts[:, 1]) + _spline(pts[:, 0], pts[:, 1])
    return out


def _exact_pack_rt(case, seed):
    plane, wp = _lib.geometry_load(GEOMETRY_E906)
    n = case["n"]
    rec, off = _records(S.Geometry(plane, wp), case["events"], n, seed)
    words = rec.view(torch.int32).view(-1, 4)
    det = (words[:, 0] & 0xFFFF).long()
    elem = words[:, 0].long() >> 16
    tdc = words[:, 1].contiguous().view(torch.float32).double()
    drift = words[:, 2].contiguous().view(torch.float32).double()
    flag = words[:, 3].double()
    for d, (tmin, tmax, t, r, b, c, e) in _calibration().items():
        at = torch.nonzero(det == d).reshape(-1)
        x = tdc[at]
        t, r, b, c, e = (torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (t, r, b, c, e))
        k = (torch.searchsorted(t, x) - 1).clamp(0, len(t) - 2)
        dx = x - t[k]
        v = r[k] + dx * (b[k] + dx * (c[k] + dx * e[k]))
        v = torch.where(x > tmax, torch.zeros_like(v), v)
        drift[at] = torch.where(x < tmin, torch.full_like(v, 0.5 * float(plane.cellwidth[d])), v)
    event = torch.repeat_interleave(torch.arange(n, device="cuda"), off[1:] - off[:-1])
    key = event * 55 + det
    count = torch.bincount(key, minlength=n * 55).view(n, 55)
    first = torch.zeros(n * 55 + 1, dtype=torch.int64, device="cuda")
    first[1:] = torch.cumsum(count.reshape(-1), 0)
    rank = torch.arange(len(key), device="cuda") - first[key]
    pos = torch.from_numpy(wp.astype(np.float32).astype(np.float64)).cuda()[det, elem]
    out = {}
    for name, lo, hi, cap in (("cham", 1, 30, 200), ("hodo", 31, 46, 60), ("prop", 47, 54, 120)):
        out["nhits_" + name] = None
        hits = torch.zeros(n * (hi - lo + 1) * 5 * cap, dtype=torch.float64, device="cuda")
        at = torch.nonzero((det >= lo) & (det <= hi)).reshape(-1)
        c = count.view(-1)[key[at]]
        base = (event[at] * (hi - lo + 1) + det[at] - lo) * 5 * cap + rank[at]
        for f, v in enumerate((elem.double(), pos, tdc, flag, drift)):
            hits[base + f * c] = v[at]
        out["hits_" + name] = hits
    return out


def _network(p, x):
    w1, b1, w2, b2, w3, b3 = p
    return torch.relu(torch.relu(x @ w1.T + b1) @ w2.T + b2) @ w3 + b3


def _unpack(v):
    sizes = [(64, 16), (64,), (64, 64), (64,), (64,), ()]
    out, o = [], 0
    for s in sizes:
        m = int(np.prod(s))
        out.append(v[o:o + m].reshape(s))
        o += m
    return out


def exact(case, seed):
    """Selections of hits follow FP32 cuts, so only the calls without them have a 64-bit answer."""
    call, n = case["call"], case["n"]
    if call == "pack_rt":
        return _exact_pack_rt(case, seed)
    if call not in ("score", "train"):
        return None
    z = np.load(learned.MODEL_COMBO_E906)
    sp = learned.ScorerParams.load(learned.MODEL_COMBO_E906)
    mean, inv_std = (torch.from_numpy(z[k].astype(np.float64)).cuda() for k in ("mean", "inv_std"))
    if call == "score":
        p = _unpack(torch.from_numpy(z["params"].astype(np.float64)).cuda())
        x = _scorer_rows(n, seed, sp).double()
        return {"scores": torch.cat([torch.sigmoid(_network(p, (c - mean) * inv_std)) for c in x.split(1 << 19)])}
    x, labels, start = _train_inputs(n, seed, sp)
    x, y = (x.double() - mean) * inv_std, labels.double()
    param = torch.from_numpy(start.params.astype(np.float64)).cuda()
    m1, m2 = torch.zeros_like(param), torch.zeros_like(param)
    perm = torch.from_numpy(np.random.default_rng(seed).permutation(n)).cuda()
    total, steps = 0.0, n // TRAIN_BATCH
    for k in range(steps):
        i = perm[k * TRAIN_BATCH:(k + 1) * TRAIN_BATCH]
        v = param.clone().requires_grad_(True)
        out = _network(_unpack(v), x[i])
        sp_pos, sp_neg = torch.nn.functional.softplus(out, threshold=60), torch.nn.functional.softplus(-out, threshold=60)
        loss = (20.0 * y[i] * sp_neg + (1 - y[i]) * sp_pos).mean()
        g = torch.autograd.grad(loss, v)[0]
        m1 = 0.9 * m1 + 0.1 * g
        m2 = 0.999 * m2 + 0.001 * g * g
        param = param - 1e-3 * (m1 / (1 - 0.9 ** (k + 1))) / ((m2 / (1 - 0.999 ** (k + 1))).sqrt() + 1e-8)
        total += float(loss)
    return {"loss": total / steps, "param": param, "m1": m1, "m2": m2}
