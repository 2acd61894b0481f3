"""YZ and global tracking when their lists of work do not fit the context
(sized for small batches, given a large one): every slot is visited instead,
with the same results.  YZ's list has room for 70 slots per unit of the queue's
capacity (65,536 at least).  All but the first events are rejected, so hits and
tracks are there for those alone; flags and counts for all."""
import numpy as np
import pytest

from helpers import Snapshots, mixed_events, track_mismatches

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1400, 70 * 65536 // 32 + 140])
def test_large_batch_on_a_small_context(geometry, n):
    import torch
    from orgpu import _lib, layout as L, pipeline
    plane, wp = geometry
    _, _, _, hits0 = mixed_events(plane, wp, 120, 60, seed=59)
    snap = Snapshots(plane, hits0)
    m = hits0.n

    def padded(a, per):
        t = torch.zeros(n * per, dtype=torch.int16 if a.dtype == np.uint16 else torch.int32, device="cuda")
        t[:m * per].copy_(torch.from_numpy(a.view(np.int16 if a.dtype == np.uint16 else np.int32)))
        return t

    h, t0 = snap.hits_er, snap.tracks_xz
    counts = [padded(h.nhits_cham, L.NCHAM), padded(h.nhits_hodo, L.NHODO), padded(h.nhits_prop, L.NPROP)]
    hits = [torch.from_numpy(x).cuda() for x in (h.hits_cham, h.hits_hodo, h.hits_prop)]
    ntracks, tracks = padded(t0.ntracks, L.NSLOTS), torch.from_numpy(t0.tracks).cuda()
    toomany = torch.ones(n, dtype=torch.uint8, device="cuda")
    toomany[:m].copy_(torch.from_numpy(snap.toomany_xz))
    hv, tv = L.OrHitsView(), L.OrTracksView()
    hv.nhits_cham, hv.nhits_hodo, hv.nhits_prop = (x.data_ptr() for x in counts)
    hv.hits_cham, hv.hits_hodo, hv.hits_prop = (x.data_ptr() for x in hits)
    tv.ntracks, tv.tracks = ntracks.data_ptr(), tracks.data_ptr()
    rc = pipeline.Reconstruction(plane, 0, max_events=32)
    st = rc._stream(None)

    def got():
        rc.sync()
        t = L.HostTracks(m)
        t.ntracks[:] = ntracks[:m * L.NSLOTS].cpu().numpy().view(np.uint16)
        t.tracks[:] = tracks.cpu().numpy()
        return t

    _lib.check(rc.lib.or_yz(rc.ctx, hv, tv, toomany.data_ptr(), n, st), "or_yz")
    assert track_mismatches(got(), snap.tracks_yz, snap.toomany_xz) == []
    _lib.check(rc.lib.or_back_clean(rc.ctx, tv, toomany.data_ptr(), n, st), "or_back_clean")
    assert track_mismatches(got(), snap.tracks_clean, snap.toomany_xz) == []
    _lib.check(rc.lib.or_global(rc.ctx, hv, tv, toomany.data_ptr(), n, st), "or_global")
    assert track_mismatches(got(), snap.tracks_global, snap.toomany_xz) == []
    rc.close()
