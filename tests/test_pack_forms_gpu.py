"""The packer on record tables at each alignment a record may have, with
events of no record, one record and more than one group of records in flight,
against the host packer: the hits are equal."""
import numpy as np
import pytest

from helpers import hit_mismatches, make_events

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 4, 8, 12])
def test_pack_record_alignment(geometry, shift):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from orgpu import layout as L, pipeline, synth as S
    plane, wp = geometry
    geo, rec, off, _, _ = make_events(plane, wp, S.config_small(40, 77))
    # events cut to 0, 1, 31, 32, 33, ... records; the last one has all of
    # them (its planes' hits past a slot's capacity are dropped)
    parts, offs = [], [0]
    for e, n in enumerate([0, 1, 31, 32, 33, 127, 128, 129, 1 << 30]):
        r = rec[off[e]:off[e + 1]][:n]
        parts.append(r)
        offs.append(offs[-1] + len(r))
    whole = np.sort(rec, order=["det", "elem", "tdc"])
    first = np.searchsorted(whole["det"], whole["det"], side="left")
    cap = np.array([0] + [L.slot_of(d)[3] for d in range(1, L.NDET)])[whole["det"]]
    fits = whole[np.arange(len(whole)) - first < cap]
    assert 600 < len(fits) < len(whole)
    want = S.pack(np.concatenate(parts + [fits]), np.array(offs + [offs[-1] + len(fits)], np.int64),
                  geo.wire_pos_f32())
    rec, off = np.concatenate(parts + [whole]), np.array(offs + [offs[-1] + len(whole)], np.int64)
    buf = torch.zeros(rec.nbytes + 16, dtype=torch.uint8, device="cuda")
    table = buf[shift:shift + rec.nbytes]
    table.copy_(torch.from_numpy(rec.view(np.uint8)))
    assert table.data_ptr() % 16 == shift
    rc = pipeline.Reconstruction(plane, 0)
    b = pipeline.DeviceBatch(len(off) - 1, 0, with_tracks=False)
    rc.pack(b, table, torch.from_numpy(off).cuda(), torch.from_numpy(geo.wire_pos_f32().reshape(-1)).cuda())
    rc.sync()
    assert hit_mismatches(b.download_hits(), want) == []
