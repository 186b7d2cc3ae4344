"""GPU: the costliest-first order of a frame's tiles, in frames that have
enough of them for it (8 a resident warp): the frame of the row order, bit for
bit, with every pixel written."""
import numpy as np
import pytest

from ivr_gb300 import api, synth
from ivr_gb300.state import orbit_state

pytestmark = pytest.mark.gpu


def least_tiles():
    import torch
    return 8 * 5 * 4 * torch.cuda.get_device_properties(0).multi_processor_count


def tiles(w, h):
    return (w + 7) // 8 * ((h + 3) // 4)


@pytest.fixture(scope="module")
def scene(ctx):
    vol = synth.blob_volume((64, 64, 64), n_blobs=8, seed=5, dtype="f32", zero_fraction=0.5, cell=8)
    v = ctx.load_volume(vol).bricks(2, 2, 2)
    tf = ctx.transfer_function().set_lut(synth.ramp_tf(256), 0, 1.0, api.TF_F2B)
    yield v, tf
    tf.free()
    v.free()


def frames(ctx, v, tf, st, size, order, window=None, stream=None):
    """The frame's and the window's floats and bytes."""
    import torch
    w, h = size
    view = ctx.view().set(v, st, api.config_params(tiles=order))
    out = [torch.full((h, w, 4), -7.0, device="cuda"), torch.full((h, w, 4), 7, dtype=torch.uint8, device="cuda")]
    view.render(tf, out[0].data_ptr(), out[1].data_ptr(), stream)
    if window:
        x, y, ww, wh = window
        out.append(torch.full((wh, ww, 4), -7.0, device="cuda"))
        view.render_tile(tf, x, y, ww, wh, out[2].data_ptr(), None, stream)
    torch.cuda.synchronize()
    view.free()
    return [o.cpu().numpy() for o in out]


@pytest.mark.parametrize("alpha", [1.0, 0.0])
def test_cost_order_is_the_row_order_frame(ctx, scene, alpha):
    v, tf = scene
    size = (1211, 997)  # ragged tiles at both edges
    window = (13, 9, 1203 - 13, 991 - 9)
    assert tiles(*window[2:]) >= least_tiles()
    st = orbit_state(30, 20, *size, fovy=30.0, alpha=alpha)
    rows, cost = (frames(ctx, v, tf, st, size, o, window) for o in (api.TILES_RASTER, api.TILES_COST))
    for a, b in zip(rows, cost):
        assert np.array_equal(a.view(np.uint8), b.view(np.uint8))
    assert not (cost[0] == -7.0).any() and not (cost[2] == -7.0).any()
    assert cost[0].any() == (alpha > 0.0)


@pytest.mark.parametrize("more", [-1, 0, 1])
def test_around_the_least_number_of_tiles(ctx, scene, more):
    v, tf = scene
    size = (8 * 160, 4 * (least_tiles() // 160 + more))
    assert tiles(*size) == least_tiles() + 160 * more
    st = orbit_state(-40, 35, *size, fovy=30.0)
    rows, cost = (frames(ctx, v, tf, st, size, o) for o in (api.TILES_RASTER, api.TILES_COST))
    for a, b in zip(rows, cost):
        assert np.array_equal(a.view(np.uint8), b.view(np.uint8))


def test_in_a_captured_graph(ctx, scene):
    import torch
    v, tf = scene
    w, h = 1211, 997
    st = orbit_state(30, 20, w, h, fovy=30.0)
    want = frames(ctx, v, tf, st, (w, h), api.TILES_RASTER)[0]
    view = ctx.view().set(v, st, api.config_params(tiles=api.TILES_COST))
    out = torch.zeros((h, w, 4), device="cuda")
    view.render(tf, out.data_ptr())  # (the order's buffers)
    torch.cuda.synchronize()
    s, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        view.render(tf, out.data_ptr(), None, torch.cuda.current_stream().cuda_stream)
    out.fill_(-7.0)
    g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy().view(np.uint32), want.view(np.uint32))
    view.free()
