"""or_run_batch when the event reducer's waits give up (or_set_wait_limit 0: no
fault and no hang, the warps wait for their copies and return): the call
reports OR_ERR_TIMEOUT, no tracklet count of an earlier batch is left standing
-- the events of this one are flagged by the caller, so no later stage writes
theirs -- and the context goes on to oracle-exact results."""
import numpy as np
import pytest

from helpers import make_events, track_mismatches

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, 300])
def test_tracklet_counts_are_cleared(geometry, n):
    import torch
    from oracle import pyoracle as O
    from orgpu import _lib, layout as L, pipeline, synth as S
    plane, wp = geometry
    geo, rec, off, hits, _ = make_events(plane, wp, S.config_small(n, 906110))
    rc = pipeline.Reconstruction(plane, 0, max_events=256)
    b = pipeline.DeviceBatch(n)
    b.upload_hits(hits)
    b.ntracklets.fill_(9)
    b.toomany.fill_(1)
    _lib.check(rc.lib.or_set_wait_limit(rc.ctx, 0), "or_set_wait_limit")
    rc.run_batch(b)
    with pytest.raises(_lib.OrError) as ei:
        rc.sync()
    assert ei.value.status == _lib.OR_ERR_TIMEOUT
    assert int(b.toomany.sum()) == n  # every wait gave up
    assert int(b.ntracklets.abs().sum()) == 0
    _lib.check(rc.lib.or_set_wait_limit(rc.ctx, -1), "or_set_wait_limit")
    b.ntracklets.fill_(9)
    rc.run_batch(b)
    rc.sync()
    ref_h, ref_t, st = hits.copy(), L.HostTracks(n), O.OracleState(n)
    O.run_all(plane, ref_h, ref_t, st)
    assert np.array_equal(b.toomany.cpu().numpy(), st.toomany)
    assert np.array_equal(b.ntracklets.cpu().numpy(), st.ntracklets)
    assert track_mismatches(b.download_tracks(), ref_t, st.toomany) == []
    rc.close()
