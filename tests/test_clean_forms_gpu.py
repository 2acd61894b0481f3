"""Back-track cleaning on track records of every form: YZ-like ones (one hit
per plane, planes 13..30, channels 1..255) take the kernel's byte form, the
others its general one; both against the oracle, bit for bit."""
import numpy as np
import pytest

from orgpu import layout as L

pytestmark = pytest.mark.gpu


def make_tracks(rng, n_events, per_slot, form):
    """Random track collections in which many tracks share hits."""
    t = L.HostTracks(n_events)
    n = rng.integers(0, per_slot + 1, (n_events, L.NSLOTS))
    t.ntracks[:] = n.reshape(-1).astype(np.uint16)
    T = t.tracks.reshape(n_events, L.NSLOTS, L.SLOTCAP, L.NTRKPARAM)
    for e, s in zip(*np.nonzero(n)):
        for k in range(n[e, s]):
            r = T[e, s, k]
            nh = int(rng.integers(8, 13))
            r[L.TRK_STID] = rng.choice([3.0, 5.0, 5.0, 6.0])
            r[L.TRK_NHITS] = nh
            r[L.TRK_CHI2] = rng.uniform(1.0, 50.0)
            det = np.sort(rng.choice(np.arange(13, 31), nh, replace=False))
            chan = rng.integers(1, 4, nh)
            if form == "repeated" and rng.random() < 0.5:
                det[1] = det[0]
            elif form == "planes" and rng.random() < 0.5:
                det[:2] = (1, 2)
            elif form == "channels" and rng.random() < 0.5:
                chan[0] = rng.choice([0, 256, 300])
            elif form == "few":
                r[L.TRK_NHITS] = rng.choice([0.0, 4.0, 18.0])
            r[L.TRK_HIT_DETID:L.TRK_HIT_DETID + nh] = det
            r[L.TRK_HIT_CHAN:L.TRK_HIT_CHAN + nh] = chan
    return t


@pytest.mark.parametrize("form,n_events,per_slot", [("yz", 1, 16), ("yz", 33, 3), ("yz", 200, 1), ("repeated", 20, 3),
                                                    ("planes", 20, 3), ("channels", 20, 3), ("few", 20, 3)])
@pytest.mark.parametrize("warps", [4, 16])
def test_clean_forms(geometry, form, n_events, per_slot, warps):
    from oracle import pyoracle as O
    from orgpu import autotune, pipeline
    plane = geometry[0]
    t = make_tracks(np.random.default_rng(len(form) + n_events), n_events, per_slot, form)
    ref, st = t.copy(), O.OracleState(n_events)
    O.back_clean(ref, st)
    rc = pipeline.Reconstruction(plane, 0, max_events=256)
    autotune.set_launch(rc, "back_clean", warps)
    b = pipeline.DeviceBatch(n_events)
    b.upload_tracks(t)
    rc.back_track_cleaning(b)
    rc.sync()
    got = b.download_tracks()
    assert np.array_equal(got.tracks.view(np.uint32), ref.tracks.view(np.uint32))
    assert np.any(ref.tracks != t.tracks) or form == "few"
