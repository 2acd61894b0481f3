"""or_xz on its own, given planes that state more hits than the reference's
scratch arrays hold: the event is refused from the counts alone (a view's
stride is the stated count, so its hits would lie past the slot, for the last
event past the collection), in both forms of the kernel (a CTA or a warp per
event), and the other events are untouched by it.  The chamber collection ends
right after the last event's slots."""
import numpy as np
import pytest

from helpers import Snapshots, mixed_events, track_mismatches

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [1, 30])
@pytest.mark.parametrize("planes,count", [((28,), 201), ((27, 28), 700), ((15, 16), 100000), ((21,), 2 ** 31 - 1)])
def test_refused_from_the_counts(geometry, planes, count, copies):
    import torch
    from orgpu import layout as L, pipeline
    plane, wp = geometry
    _, _, _, hits0 = mixed_events(plane, wp, 30, 20, seed=47)
    snap = Snapshots(plane, hits0)
    n = hits0.n
    b = pipeline.DeviceBatch(n * copies)
    for dst, src in zip((b.nhits_cham, b.hits_cham, b.nhits_hodo, b.hits_hodo, b.nhits_prop, b.hits_prop),
                        snap.hits_er.arrays()):
        dst.copy_(torch.from_numpy(src.view(np.int32) if src.dtype == np.uint32 else src).repeat(copies))
    b.toomany.copy_(torch.from_numpy(snap.toomany_er).repeat(copies))
    bad = [e for e in (0, n - 1) if not snap.toomany_er[e]] + [n * copies - 1]
    counts = b.nhits_cham.view(n * copies, L.NCHAM)
    for e in bad:
        for p in planes:
            counts[e, p - 1] = count
    b.toomany[n * copies - 1] = 0
    b.ntracklets.fill_(7)
    b.ntracks.fill_(3)
    rc = pipeline.Reconstruction(plane, 0, max_events=256)
    rc.xz_tracking(b)
    rc.sync()
    want = np.tile(snap.toomany_xz, copies)
    want[bad] = 1
    assert np.array_equal(b.toomany.cpu().numpy(), want)
    got = b.download_tracks()
    for e in bad:
        assert int(b.ntracklets[e]) == 0 and not got.ntracks[e * L.NSLOTS:(e + 1) * L.NSLOTS].any()
    # every copy of the other events as the oracle has them
    per = L.EVT_TRK_FLOATS
    for c in range(copies):
        one = L.HostTracks(n)
        one.ntracks[:] = got.ntracks[c * n * L.NSLOTS:(c + 1) * n * L.NSLOTS]
        one.tracks[:] = got.tracks[c * n * per:(c + 1) * n * per]
        assert track_mismatches(one, snap.tracks_xz, want[c * n:(c + 1) * n]) == []
    rc.close()
