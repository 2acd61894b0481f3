"""or_mlp_score with the model on a 16-byte boundary and on the 4-byte ones
between, from one row to several tiles per CTA: the same bits."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 127, 128, 129, 20000, 300001])
@pytest.mark.parametrize("shift", [4, 8, 12])
def test_model_address(geometry, n, shift):
    import torch
    from orgpu import _lib, layout as L, learned, pipeline
    rc = pipeline.Reconstruction(geometry[0], 0, max_events=1)
    model = learned.DeviceModel(learned.ScorerParams.load(learned.MODEL_COMBO_E906))
    assert model.ptr() % 16 == 0
    room = torch.zeros(C.sizeof(L.OrMlp) + 16, dtype=torch.uint8, device="cuda")
    room[shift:shift + model.bytes.numel()].copy_(model.bytes)
    rng = np.random.default_rng(n)
    x = torch.from_numpy(rng.normal(0, 1.5, n * L.NFEAT).astype(np.float32)).cuda()
    want = torch.full((n + 3,), -1.0, device="cuda")
    got = want.clone()
    learned.Learned(rc).score(model, x, n, want)
    _lib.check(rc.lib.or_mlp_score(rc.ctx, room.data_ptr() + shift, x.data_ptr(), n, got.data_ptr(),
                                   rc._stream(None)), "or_mlp_score")
    rc.sync()
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))
    assert bool((got[n:] == -1.0).all()) and bool((got[:n] >= 0).all())  # written, and no further
    rc.close()
