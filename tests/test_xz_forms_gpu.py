"""XZ tracklets where its forms change: a CTA or a warp per event (by the
batch's size), x-plane hits beyond shared memory, heavy events whose warps
find more tracklets than they keep, events the bins reject -- hits as packed
or after the event reducer, against the oracle bit for bit."""
import numpy as np
import pytest

from orgpu import layout as L
from orgpu import synth as S

pytestmark = pytest.mark.gpu


def make_records(geo, n_events, noise, gates, seed):
    """Events whose prop-tube and hodoscope hits are thinned to a share
    `gates`, so that dense chambers do not pass every candidate."""
    rec, off, _ = S.generate(geo, S.EventConfig(n_events, seed, (0.0, 0.0, 0.2, 0.4, 0.4), "poisson", noise))
    rng = np.random.default_rng(seed)
    ev = np.repeat(np.arange(n_events), np.diff(off))
    keep = (rec["det"] <= L.NCHAM) | (rng.random(len(rec)) < gates)
    off = np.concatenate(([0], np.cumsum(np.bincount(ev[keep], minlength=n_events)))).astype(np.int64)
    return S.cap_records(rec[keep], off)


# (noise hits, share of gate hits, reduced first, events, copies of them)
@pytest.mark.parametrize("noise,gates,reduce,n_events,copies", [
    (1900.0, 0.15, False, 24, 1), (2200.0, 0.1, False, 24, 1), (2200.0, 0.2, False, 24, 60),
    (450.0, 1.0, True, 60, 1), (350.0, 1.0, True, 60, 25), (0.0, 1.0, True, 3, 1)])
def test_xz_forms(geometry, noise, gates, reduce, n_events, copies):
    import torch
    from oracle import pyoracle as O
    from orgpu import pipeline
    plane, wp = geometry
    geo = S.Geometry(plane, wp)
    rec, off = make_records(geo, n_events, noise, gates, 4000 + int(noise))
    hits = S.pack(rec, off, geo.wire_pos_f32())
    st = O.OracleState(n_events)
    if reduce:
        O.event_reduce(hits, st)
    ref = L.HostTracks(n_events)
    given = st.toomany.copy()
    O.xz(plane, hits, ref, st)
    rc = pipeline.Reconstruction(plane, 0, max_events=256)
    b = pipeline.DeviceBatch(n_events * copies)
    for dst, src in zip((b.nhits_cham, b.hits_cham, b.nhits_hodo, b.hits_hodo, b.nhits_prop, b.hits_prop), hits.arrays()):
        dst.copy_(torch.from_numpy(src.view(np.int32) if src.dtype == np.uint32 else src).repeat(copies))
    b.toomany.copy_(torch.from_numpy(given).repeat(copies))
    rc.xz_tracking(b)
    rc.sync()
    got = b.download_tracks()
    assert np.array_equal(b.toomany.cpu().numpy(), np.tile(st.toomany, copies))
    assert np.array_equal(got.ntracks, np.tile(ref.ntracks, copies))
    T = got.tracks.reshape(copies, n_events, L.NSLOTS, L.SLOTCAP, L.NTRKPARAM).view(np.uint32)
    R = ref.tracks.reshape(n_events, L.NSLOTS, L.SLOTCAP, L.NTRKPARAM).view(np.uint32)
    valid = np.arange(L.SLOTCAP)[None, None, :] < ref.ntracks.reshape(n_events, L.NSLOTS)[:, :, None]
    assert valid.any()
    for c in range(copies):
        assert np.array_equal(T[c][valid], R[valid])
