"""Histograms, vertexing and dimuons of batches where few events or none have
anything to do: all rejected, all without tracks, one live event among many,
with stale tracks and dimuons in the rejected ones, against the oracle."""
import numpy as np
import pytest

from helpers import Snapshots, mixed_events, track_mismatches

pytestmark = pytest.mark.gpu

COPIES = 12


@pytest.fixture(scope="module")
def setup(geometry):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from oracle import pyoracle as O
    from orgpu import layout as L, pipeline, synth as S
    plane, wp = geometry
    _, _, _, hits0 = mixed_events(plane, wp, 90, 30, seed=53)
    snap = Snapshots(plane, hits0)
    st = O.OracleState(hits0.n)
    st.toomany[:] = snap.toomany_xz
    vertexed = snap.tracks_sel.copy()
    O.vertexing(plane, vertexed, st)
    dims = L.HostDimuons(hits0.n)
    O.dimuons(plane, vertexed, dims, st)
    return dict(plane=plane, snap=snap, n=hits0.n, vertexed=vertexed, dims=dims,
                rc=pipeline.Reconstruction(plane, 0, max_events=256),
                trig=np.tile(S.trigger_bits(hits0.n, seed=5), COPIES))


def _flags(s, what):
    """Rejected events of COPIES copies of the batch."""
    n = s["n"] * COPIES
    live = np.zeros(n, bool)
    pick = np.nonzero(s["dims"].ndimuons)[0]
    if what == "first":
        live[pick[0]] = True
    elif what == "last":
        live[(COPIES - 1) * s["n"] + pick[-1]] = True
    elif what == "some":
        live[np.random.default_rng(3).choice(n, 40, replace=False)] = True
    live &= np.tile(s["snap"].toomany_xz, COPIES) == 0
    return (~live).astype(np.uint8)


def _batch(s, tracks, toomany):
    import torch
    from orgpu import pipeline
    b = pipeline.DeviceBatch(s["n"] * COPIES)
    b.ntracks.copy_(torch.from_numpy(tracks.ntracks.view(np.int16)).repeat(COPIES))
    b.tracks.copy_(torch.from_numpy(tracks.tracks).repeat(COPIES))
    b.toomany.copy_(torch.from_numpy(toomany))
    return b


@pytest.mark.parametrize("what", ["none", "first", "last", "some"])
@pytest.mark.parametrize("tracks", [True, False])
def test_histograms(setup, what, tracks):
    import torch
    from oracle import pyoracle as O
    from orgpu import layout as L, pipeline
    s = setup
    toomany = _flags(s, what)
    want = O.hist_table()
    for c in range(COPIES):
        st = O.OracleState(s["n"])
        st.toomany[:] = toomany[c * s["n"]:(c + 1) * s["n"]]
        t, d = s["vertexed"].copy(), L.HostDimuons(s["n"])
        if tracks:
            d.ndimuons[:], d.dimuons[:] = s["dims"].ndimuons, s["dims"].dimuons
        else:
            t.ntracks[:] = 0
        O.fill_histograms(t, d, want, np.ascontiguousarray(s["trig"][c * s["n"]:(c + 1) * s["n"]]), st)
    b = _batch(s, s["vertexed"], toomany)
    d = pipeline.DeviceDimuons(b.n)
    if tracks:
        d.ndimuons.copy_(torch.from_numpy(s["dims"].ndimuons.view(np.int16)).repeat(COPIES))
        d.dimuons.copy_(torch.from_numpy(s["dims"].dimuons).repeat(COPIES))
    else:
        b.ntracks.zero_()
    h = pipeline.DeviceHists()
    s["rc"].fill_histograms(b, d, h, torch.from_numpy(s["trig"]).cuda())
    s["rc"].sync()
    got = h.download().values_array()
    np.testing.assert_array_equal(got, want.values_array())
    assert (got.sum() > 0) == (tracks and what != "none")


# events whose tracks go beyond what a warp lists at a time: tracks per event
# from a multiple of the largest group on, in a batch large enough for it
# (some 9,100 events on 152 SMs)
BATCH = 9200
DENSE = {0: [3], 160: [100] * 16, 320: [512, 0, 512, 1, 0, 300, 40, 0, 0, 224, 223, 225, 256, 2, 0, 512], 9199: [40]}


def _dense(s, stid, opposite):
    """The events of DENSE from vertexed tracks of the batch, their charges
    negative in `opposite` of each event's and among them records below
    `stid`."""
    from orgpu import layout as L
    pool = np.array([r for e in range(s["n"]) if not s["snap"].toomany_xz[e]
                     for _, _, r in s["vertexed"].records(e) if r[L.TRK_STID] == 7], np.float32)
    assert len(pool) > 50
    rng = np.random.default_rng(61)
    at = [p + i for p, c in DENSE.items() for i in range(len(c))]
    counts = [m for c in DENSE.values() for m in c]
    t = L.HostTracks(len(at))
    T = t.tracks.reshape(len(at), L.NSLOTS, L.SLOTCAP, L.NTRKPARAM)
    for e, m in enumerate(counts):
        r = pool[rng.integers(0, len(pool), m)]
        r[:, L.TRK_CHARGE] = 1.0
        r[rng.permutation(m)[:opposite], L.TRK_CHARGE] = -1.0
        r[:, L.TRK_STID] = np.where(rng.random(m) < 0.05, 3.0, stid)
        # slot after slot, or spread over the slots
        slot, k = (np.arange(m) // L.SLOTCAP, np.arange(m) % L.SLOTCAP) if e % 2 else (np.arange(m) % L.NSLOTS, np.arange(m) // L.NSLOTS)
        T[e, slot, k] = r
        t.ntracks[e * L.NSLOTS:(e + 1) * L.NSLOTS] = np.bincount(slot, minlength=L.NSLOTS)
    return np.array(at), t


def _dense_batch(at, t):
    import torch
    from orgpu import layout as L, pipeline
    b = pipeline.DeviceBatch(BATCH)
    idx = torch.from_numpy(at).cuda()
    b.ntracks.view(BATCH, L.NSLOTS)[idx] = torch.from_numpy(t.ntracks.view(np.int16)).view(-1, L.NSLOTS).cuda()
    b.tracks.view(BATCH, -1)[idx] = torch.from_numpy(t.tracks).view(len(at), -1).cuda()
    return b, idx


def test_vertexing_of_dense_events(setup):
    from oracle import pyoracle as O
    from orgpu import layout as L
    s = setup
    at, t = _dense(s, 6.0, 4)
    b, idx = _dense_batch(at, t)
    s["rc"].vertexing(b)
    s["rc"].sync()
    got = L.HostTracks(len(at))
    got.ntracks[:] = t.ntracks
    got.tracks[:] = b.tracks.view(BATCH, -1)[idx].cpu().numpy().reshape(-1)
    st = O.OracleState(len(at))
    O.vertexing(s["plane"], t, st)
    assert track_mismatches(got, t) == []
    assert (t.tracks.reshape(-1, L.NTRKPARAM)[:, L.TRK_STID] == 7).sum() > 2000


def test_dimuons_of_dense_events(setup):
    import golden_io as G
    from oracle import pyoracle as O
    from orgpu import layout as L, pipeline
    s = setup
    at, t = _dense(s, 7.0, 4)
    b, idx = _dense_batch(at, t)
    d = pipeline.DeviceDimuons(BATCH)
    d.ndimuons.fill_(5)
    s["rc"].dimuons(b, d)
    s["rc"].sync()
    st = O.OracleState(len(at))
    want, got = L.HostDimuons(len(at)), L.HostDimuons(len(at))
    O.dimuons(s["plane"], t, want, st)
    counts = d.ndimuons.cpu().numpy().view(np.uint16)
    assert not np.delete(counts, at).any()
    got.ndimuons[:] = counts[at]
    got.dimuons[:] = d.dimuons.view(BATCH, -1)[idx].cpu().numpy().reshape(-1)
    no = np.zeros(len(at), np.uint8)
    r = G.compare_dimuons(G.compact_dimuons(got, no), G.compact_dimuons(want, no), 0.0, phi_ulps=4)
    assert r["count_mismatch"] == [] and r["value_mismatch"] == [], r
    assert want.ndimuons.sum() > 20
