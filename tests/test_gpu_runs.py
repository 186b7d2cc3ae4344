"""GPU: the CONFIG march's runs of opaque samples, where they are cut: more
runs than a lane holds, runs longer than it looks ahead, runs that are no
multiple of the samples taken at once, windows of fewer tiles than the
launch has warps, frames of one view in a row, tiles and single bricks."""
import numpy as np
import pytest

from ivr_gb300 import api, synth
from ivr_gb300.state import orbit_state

pytestmark = pytest.mark.gpu


def spiky(dtype, n, period, seed=5):
    """Opaque 4-voxel cells every `period` cells in a transparent volume
    (period 1: every cell opaque), with a little noise in them."""
    rng = np.random.default_rng(seed)
    c = np.indices((n, n, n)) // 4
    on = (c.sum(axis=0) % period) == 0
    v = np.where(on, rng.uniform(60.0, 130.0, (n, n, n)), 0.0)
    if dtype == "u16":
        return (v * 256.0).astype(np.uint16)
    return v.astype(np.uint8 if dtype == "u8" else np.float32)


def thin_tf():
    """Opacities small enough that rays cross the whole volume."""
    lut = synth.ramp_tf(256)
    lut[:, 3] *= np.float32(0.02)
    return lut


@pytest.mark.parametrize("dtype", ["u8", "u16", "f32"])
@pytest.mark.parametrize("period,cell,step,win,bricks", [
    (3, 4, 0.25, (33, 21), 1),   # many short runs: more than a lane holds
    (2, 4, 0.07, (9, 5), 2),     # runs of some 60 samples, several bricks
    (1, 16, 0.05, (40, 23), 1),  # one run of thousands of samples
    (5, 4, 0.5, (1, 1), 1),      # one pixel
    (3, 8, 1.7, (130, 97), 2)])  # steps over a voxel: runs shorter than K
def test_runs_match_the_oracle(ctx, oracle_mod, dtype, period, cell, step, win, bricks):
    import torch
    vol = spiky(dtype, 48, period)
    lut, scale = thin_tf(), 256.0 / 65536.0 if dtype == "u16" else 1.0
    st = orbit_state(31.0, 17.0, win[0], win[1])
    ref = oracle_mod.render(vol, st, lut, 0, 6, preset=1, procdims=(bricks,) * 3, step=step, lut_scale=scale)
    v = ctx.load_volume(vol).macrocell(cell)
    if bricks > 1:
        v.bricks(bricks, bricks, bricks)
    tf = ctx.transfer_function().set_lut(lut, 0, scale, api.TF_F2B)
    try:
        for skip in (True, False):
            for quads in (True, False):
                v.quads(quads)
                view = ctx.view().set(v, st, api.config_params(step=step, skip=skip))
                for _ in range(3):  # launches of one view share its ticket counter
                    o32 = torch.full((win[1], win[0], 4), -7.0, device="cuda")
                    o8 = torch.full((win[1], win[0], 4), 7, dtype=torch.uint8, device="cuda")
                    view.render(tf, o32.data_ptr(), o8.data_ptr())
                    torch.cuda.synchronize()
                    assert np.array_equal(o32.cpu().numpy().view(np.uint32), ref["rgba32"].view(np.uint32))
                    assert np.array_equal(o8.cpu().numpy(), ref["rgba8"])
                x, y = win[0] // 2, win[1] // 3
                w, h = win[0] - x, win[1] - y
                o32 = torch.zeros((h, w, 4), device="cuda")
                view.render_tile(tf, x, y, w, h, o32.data_ptr())
                torch.cuda.synchronize()
                assert np.array_equal(o32.cpu().numpy(), ref["rgba32"][y:, x:])
                view.free()
    finally:
        tf.free()
        v.free()
