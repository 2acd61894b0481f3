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
