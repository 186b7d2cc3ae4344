"""GPU: the REF march against the restatement, bitwise, where its sampler
changes: brick edges at 0 seen from an eye on the axis planes (rays the packed
divisions leave to the general sampler), extents and dims that are no powers
of two, sample counts that leave every remainder, windows that cut blocks."""
import numpy as np
import pytest

from ivr_gb300 import api, synth
from ivr_gb300.state import orbit_state

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


@pytest.mark.parametrize("dtype", ["u8", "u16", "f32"])
@pytest.mark.parametrize("mode", [api.TF_SEISMIC, api.TF_MED, api.TF_SEISMIC2, api.TF_CHEM, api.TF_BLEND])
@pytest.mark.parametrize("shape,bricks,az,el,dist,win,max_samples", [
    ((32, 32, 32), 2, 0.0, 0.0, 5.0, (37, 29), 256),     # edges and eye at 0
    ((19, 30, 23), 3, 31.0, 17.0, 5.0, (50, 33), 255),   # odd extents and dims
    ((32, 16, 64), 1, 90.0, 0.0, 5.0, (16, 8), 1),       # one sample, one block
    ((24, 24, 24), 2, 200.0, -40.0, 0.3, (21, 40), 6)])  # the eye in the box
def test_matches_the_oracle(ctx, oracle_mod, dtype, mode, shape, bricks, az, el, dist, win, max_samples):
    import torch
    vol = synth.blob_volume(shape, n_blobs=5, seed=12, dtype="u8", noise=0.1)
    vol = vol.astype({"u8": np.uint8, "u16": np.uint16, "f32": np.float32}[dtype])
    if dtype == "f32":
        vol += np.random.default_rng(3).uniform(0.0, 0.9, shape).astype(np.float32)
    lut = synth.ramp_tf(256)
    st = orbit_state(az, el, win[0], win[1], dist=dist, alpha=0.7)
    ref = oracle_mod.render(vol, st, lut, 0, mode, procdims=(bricks,) * 3, max_samples=max_samples)
    v = ctx.load_volume(vol)
    if bricks > 1:
        v.bricks(bricks, bricks, bricks)
    tf = ctx.transfer_function().set_lut(lut, 0, 1.0, mode)
    p = api.ref_params()
    p.max_samples = max_samples
    view = ctx.view().set(v, st, p)
    try:
        o32 = torch.full((win[1], win[0], 4), -7.0, device="cuda")
        o8 = torch.full((win[1], win[0], 4), 7, dtype=torch.uint8, device="cuda")
        view.render(tf, o32.data_ptr(), o8.data_ptr())
        torch.cuda.synchronize()
        assert np.array_equal(bits(o32.cpu().numpy()), bits(ref["rgba32"]))
        assert np.array_equal(o8.cpu().numpy(), ref["rgba8"])
        x, y = 5, 3  # a tile whose blocks start inside the window
        tile = torch.zeros((win[1] - y, win[0] - x, 4), device="cuda")
        view.render_tile(tf, x, y, win[0] - x, win[1] - y, tile.data_ptr())
        torch.cuda.synchronize()
        assert np.array_equal(bits(tile.cpu().numpy()), bits(np.ascontiguousarray(ref["rgba32"][y:, x:])))
    finally:
        view.free()
        tf.free()
        v.free()
