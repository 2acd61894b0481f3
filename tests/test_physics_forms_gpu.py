"""Vertexing and dimuon swims at the ends of the ranges where their double
statements are decided by other arithmetic (momenta, slopes, distances and
charges outside it take the double expressions), and histogram tables whose
bins are not in order, against the oracle.  Tolerances: none for the tracks
(the results are the same bits; from some 6,000 GeV on the energy-loss
polynomial runs away and the momentum is not a number in either, whose sign
and payload IEEE 754 leaves to the machine); those of the physics stages for
the rest."""
import numpy as np
import pytest

from helpers import Snapshots, mixed_events, track_mismatches

pytestmark = pytest.mark.gpu

N = 96


@pytest.fixture(scope="module")
def setup(geometry):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from oracle import pyoracle as O
    from orgpu import pipeline, synth as S
    plane, _ = geometry
    geo, rec, off, hits0 = mixed_events(plane, geometry[1], N, 600, seed=29)
    snap = Snapshots(plane, hits0)
    st = O.OracleState(hits0.n)
    st.toomany[:] = snap.toomany_xz
    return dict(plane=plane, snap=snap, n=hits0.n, st=st, rc=pipeline.Reconstruction(plane, 0),
                trig=S.trigger_bits(hits0.n, seed=5))


NOT_A_NUMBER = np.float32(-12345.0)


def _nan_marked(a):
    a[np.isnan(a)] = NOT_A_NUMBER


def _altered(s, lo, hi, what):
    """The selected tracks with momenta spread over [lo, hi] GeV."""
    from orgpu import layout as L
    rng = np.random.default_rng(41)
    t = s["snap"].tracks_sel.copy()
    for e in range(s["n"]):
        for _, _, r in t.records(e):
            r[L.TRK_INVP] = 1.0 / np.exp(rng.uniform(np.log(lo), np.log(hi)))
            if what == "straight":
                r[L.TRK_TX] = r[L.TRK_TY] = 0.0
            elif what == "axis":
                r[L.TRK_X0] = r[L.TRK_Y0] = np.float32(rng.uniform(-1e-9, 1e-9))
                r[L.TRK_TY] = 0.0
            elif what == "steep":
                r[L.TRK_TX] = rng.uniform(-2, 2)
                r[L.TRK_TY] = rng.uniform(-2, 2)
            elif what == "far":
                r[L.TRK_X0] = rng.uniform(-1e7, 1e7)
            elif what == "neutral":
                r[L.TRK_CHARGE] = 0.0
    return t


@pytest.mark.parametrize("lo,hi,what", [(3.5, 4.5, ""), (1.0, 140.0, ""), (120.0, 136.0, ""), (1e-3, 1.0, ""),
                                        (200.0, 1e6, ""), (5.0, 120.0, "straight"), (5.0, 120.0, "axis"),
                                        (5.0, 120.0, "steep"), (5.0, 120.0, "far"), (5.0, 120.0, "neutral")])
def test_swims(setup, lo, hi, what):
    import torch
    import golden_io as G
    from oracle import pyoracle as O
    from orgpu import layout as L, pipeline
    s = setup
    t = _altered(s, lo, hi, what)
    want = t.copy()
    O.vertexing(s["plane"], want, s["st"])
    b = pipeline.DeviceBatch(s["n"])
    b.upload_hits(s["snap"].hits_er)
    b.upload_tracks(t)
    b.toomany.copy_(torch.from_numpy(s["snap"].toomany_xz))
    s["rc"].vertexing(b)
    s["rc"].sync()
    got, ref = b.download_tracks(), want.copy()
    _nan_marked(got.tracks)
    _nan_marked(ref.tracks)
    assert track_mismatches(got, ref, s["snap"].toomany_xz) == []
    dims = L.HostDimuons(s["n"])
    O.dimuons(s["plane"], want, dims, s["st"])
    d = pipeline.DeviceDimuons(s["n"])
    b.upload_tracks(want)
    s["rc"].dimuons(b, d)
    s["rc"].sync()
    got = d.download()
    _nan_marked(got.dimuons)
    _nan_marked(dims.dimuons)
    r = G.compare_dimuons(G.compact_dimuons(got, s["snap"].toomany_xz),
                          G.compact_dimuons(dims, s["snap"].toomany_xz), 0.0, phi_ulps=4)
    assert r["count_mismatch"] == [] and r["value_mismatch"] == [], r


def test_histogram_bins_out_of_order(setup):
    import torch
    import golden_io as G
    from oracle import pyoracle as O
    from orgpu import layout as L, pipeline
    s = setup
    tv = s["snap"].tracks_sel.copy()
    O.vertexing(s["plane"], tv, s["st"])
    dims = L.HostDimuons(s["n"])
    O.dimuons(s["plane"], tv, dims, s["st"])
    want = O.hist_table()
    x = np.ctypeslib.as_array(want.xpts).reshape(-1, L.OrHists.xpts.size // 4 // len(np.ctypeslib.as_array(want.nbins).reshape(-1)))
    nb = np.ctypeslib.as_array(want.nbins).reshape(-1)
    rng = np.random.default_rng(3)
    for i in range(0, len(nb), 2):  # every second table
        x[i, :nb[i]] = rng.permutation(x[i, :nb[i]])
    h = pipeline.DeviceHists()
    h.buf.copy_(torch.from_numpy(np.frombuffer(want.to_bytes(), np.uint8).copy()))
    O.fill_histograms(tv, dims, want, s["trig"], s["st"])
    b = pipeline.DeviceBatch(s["n"])
    b.upload_hits(s["snap"].hits_er)
    b.upload_tracks(tv)
    b.toomany.copy_(torch.from_numpy(s["snap"].toomany_xz))
    d = pipeline.DeviceDimuons(s["n"])
    d.ndimuons.copy_(torch.from_numpy(dims.ndimuons.view(np.int16)))
    d.dimuons.copy_(torch.from_numpy(dims.dimuons))
    s["rc"].fill_histograms(b, d, h, torch.from_numpy(s["trig"]).cuda())
    s["rc"].sync()
    got = h.download()
    np.testing.assert_array_equal(got.values_array(), want.values_array())
    assert got.values_array().sum() > 100
