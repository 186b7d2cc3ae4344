"""GPU: a skipping grid built on one stream and read on another.  The first
stream is kept busy ahead of the build, and nothing but the library orders the
second behind it: its frame has to end after that work, and be the frame
rendered alone."""
import numpy as np
import pytest

from ivr_gb300 import api, synth
from ivr_gb300.state import orbit_state

pytestmark = pytest.mark.gpu

KEPT = 128  # grids a volume keeps: later builds go into an old one, without an allocation
BUSY = 200_000_000  # clock cycles, some 0.1 s


@pytest.mark.parametrize("skip", [api.SKIP_GRID, api.SKIP_LEARNED], ids=["grid", "learned"])
@pytest.mark.parametrize("order", [api.TILES_RASTER, api.TILES_COST], ids=["raster", "cost"])
@pytest.mark.parametrize("size", [(120, 96), (1200, 900)])
def test_frame_waits_for_the_build(ctx, skip, order, size):
    import torch
    w, h = size
    v = ctx.load_volume(synth.blob_volume((80, 72, 88), n_blobs=12, seed=31, dtype="u16", zero_fraction=0.6, cell=16))
    scale = 256.0 / 65536.0
    lut = synth.knot_tf(7, zero_first=True)[0]
    clear = lut.copy()
    clear[:, 3] = 0.0
    tf = ctx.transfer_function().set_lut(lut, 0, scale)
    mlp = None
    if skip == api.SKIP_LEARNED:
        mlp = ctx.mlp(3)
        mlp.add_samples(v, tf)
        mlp.train(2, batch_rows=512)
        v.set_mlp(mlp, mlp.calibrate(0.02)[0], certify=True)
    views = [ctx.view().set(v, orbit_state(30.0, 20.0, w, h), api.config_params(skip=skip, tiles=order))
             for _ in range(2)]
    outs = [torch.empty((h, w, 4), dtype=torch.uint8, device="cuda") for _ in range(3)]
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    began, ended = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    try:
        for view, s in zip(views, (a, b)):  # (their scratch is there afterwards)
            view.render(tf, None, outs[0].data_ptr(), s.cuda_stream)
            torch.cuda.synchronize()
        want = outs[0].cpu()
        assert want.any()
        for _ in range(KEPT + 1):  # every kept grid takes all cells as transparent
            tf.set_lut(clear, 0, scale)
            views[0].render(tf, None, outs[0].data_ptr(), a.cuda_stream)
            torch.cuda.synchronize()
        assert not outs[0].any()
        for _ in range(2):
            tf.set_lut(lut, 0, scale)
            for o in outs:
                o.fill_(9)
            torch.cuda.synchronize()
            with torch.cuda.stream(a):
                torch.cuda._sleep(BUSY)
            began.record(a)
            views[0].render(tf, None, outs[0].data_ptr(), a.cuda_stream)
            views[1].render(tf, None, outs[1].data_ptr(), b.cuda_stream)
            views[1].render(tf, None, outs[2].data_ptr(), b.cuda_stream)
            ended.record(b)
            assert not began.query()  # the build had not run when the second stream was given its frames
            torch.cuda.synchronize()
            assert began.elapsed_time(ended) >= 0.0
            for o in outs:
                assert torch.equal(o.cpu(), want)
            tf.set_lut(clear, 0, scale)
            views[0].render(tf, None, outs[0].data_ptr(), a.cuda_stream)
            torch.cuda.synchronize()
    finally:
        for view in views:
            view.free()
        v.set_mlp(None)
        if mlp is not None:
            mlp.free()
        tf.free()
        v.free()
