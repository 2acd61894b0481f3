"""The event reducer on planes that ascend and planes that do not, with hits
on one channel, clusters of every length, channels past the map's ends, full
planes and empty ones, against the oracle: the kept hits are equal."""
import numpy as np
import pytest

from helpers import hit_mismatches

pytestmark = pytest.mark.gpu

N = 120


def _events(kind, seed):
    """Hits of N events: `kind` says how a plane's channels lie."""
    from orgpu import layout as L
    rng = np.random.default_rng(seed)
    h = L.HostHits(N)
    for e in range(N):
        most = (3, 12, 31, 33, 70, 200)[e % 6]
        for det in range(1, L.NDET):
            t, k, _, cap = L.slot_of(det)
            n = int(min(cap, rng.integers(0, most + 1)))
            if e % 6 == 5 and det % 3 == 0:
                n = cap
            ch = rng.integers(0, 202, n)
            if kind == "runs":  # neighbours and repeats: clusters of many lengths
                ch = np.cumsum(rng.choice([0, 1, 1, 1, 2, 7], n)) % 202
            elif kind == "ends":
                ch = rng.choice([-3, -1, 0, 1, 200, 201, 202, 250, 1000], n)
            if kind != "shuffled":
                ch = np.sort(ch)
            if kind == "one late" and n > 1:
                ch[-1] = ch[0]
            a = np.zeros((5, n), np.float32)
            a[0] = ch
            a[1] = ch * np.float32(1.0 if rng.random() < 0.3 else 2.0)
            a[2] = rng.choice([1600, 1604, 1608, 1590, 1700], n) + rng.integers(0, 12, n)
            a[3] = np.where(rng.random(n) < 0.9, 2, 0) + rng.integers(0, 2, n)
            a[4] = rng.choice([0.0, 0.2, 0.45, 0.5, 0.9], n) * np.float32(rng.random())
            cnt = (h.nhits_cham, h.nhits_hodo, h.nhits_prop)[t]
            buf = (h.hits_cham, h.hits_hodo, h.hits_prop)[t]
            per = (L.NCHAM, L.NHODO, L.NPROP)[t]
            ef = (L.EVT_CHAM_FLOATS, L.EVT_HODO_FLOATS, L.EVT_PROP_FLOATS)[t]
            cnt[e * per + k] = n
            at = e * ef + k * 5 * cap
            buf[at:at + 5 * n] = a.reshape(-1)
    return h


@pytest.mark.parametrize("kind", ["ascending", "runs", "ends", "shuffled", "one late"])
def test_event_reducer_forms(geometry, kind):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from oracle import pyoracle as O
    from orgpu import pipeline
    hits = _events(kind, 61)
    want = hits.copy()
    st = O.OracleState(N)
    O.event_reduce(want, st)
    rc = pipeline.Reconstruction(geometry[0], 0)
    b = pipeline.DeviceBatch(N)
    b.upload_hits(hits)
    rc.event_reduce(b)
    rc.sync()
    assert hit_mismatches(b.download_hits(), want) == []
    np.testing.assert_array_equal(b.toomany.cpu().numpy(), st.toomany)
    assert 0 < int(want.nhits_cham.sum()) < int(hits.nhits_cham.sum())
