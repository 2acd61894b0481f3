"""The track gather at the edges of its blocks and clusters, with full, empty
and rejected events and a buffer that is too small, against numpy: the rows
are equal; in order within each 256 events."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 32, 33, 63, 64, 65, 255, 256, 257, 600, 4865])
@pytest.mark.parametrize("short", [False, True])
def test_collect_forms(geometry, n, short):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from orgpu import layout as L, pipeline
    rng = np.random.default_rng(n)
    per = rng.integers(0, L.SLOTCAP + 1, (n, L.NSLOTS)) * (rng.random((n, L.NSLOTS)) < 0.1)
    per[n // 2] = L.SLOTCAP  # one full event
    rc = pipeline.Reconstruction(geometry[0], 0)
    b = pipeline.DeviceBatch(n)
    b.ntracks.copy_(torch.from_numpy(per.reshape(-1).astype(np.int64)).to(b.ntracks.dtype))
    b.tracks.normal_(generator=torch.Generator(device="cuda").manual_seed(n))
    stid = rng.integers(4, 8, (n, L.NSLOTS, L.SLOTCAP)).astype(np.float32)
    b.tracks.view(n, L.NSLOTS, L.SLOTCAP, L.NTRKPARAM)[..., L.TRK_STID] = torch.from_numpy(stid).cuda()
    flag = (rng.random(n) < 0.2).astype(np.uint8)
    flag[n // 2] = 0
    b.toomany.copy_(torch.from_numpy(flag))
    hit = (stid == 6) & (np.arange(L.SLOTCAP) < per[..., None]) & (flag == 0)[:, None, None]
    e, s, k = np.nonzero(hit)
    cap = len(e) // 2 if short else len(e)
    rows = torch.full((cap + 8, L.COLLECT_STRIDE), -1.0, device="cuda")
    cnt = torch.zeros(1, dtype=torch.int64, device="cuda")
    rc.collect(b, rows[:cap], cnt, 6.0)
    rc.sync()
    got = rows.cpu().numpy()
    assert int(cnt.item()) == len(e) and (got[cap:] == -1).all()
    got = got[:cap]
    want = b.tracks.view(n, L.NSLOTS, L.SLOTCAP, L.NTRKPARAM).cpu().numpy()
    ge, gs = got[:, 0].astype(int), got[:, 1].astype(int)
    np.testing.assert_array_equal(got[:, 2:], want[ge, gs // L.SLOTCAP, gs % L.SLOTCAP])
    key = ge * 512 + gs
    assert len(np.unique(key)) == cap and np.isin(key, e * 512 + s * L.SLOTCAP + k).all()
    for g in np.unique(ge // 256):
        assert (np.diff(key[ge // 256 == g]) > 0).all()
    if n <= 256:
        np.testing.assert_array_equal(key, (e * 512 + s * L.SLOTCAP + k)[:cap])
