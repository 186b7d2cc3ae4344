"""CPU: what the library's launches are ordered behind when a program renders
on several streams without waiting in between: no frame, of whatever skip
mode, tile order or size, may read a skipping grid (or a tile order) whose
build on another stream may still be running."""
import random

import numpy as np
import pytest

from host import HostContext, load
from ivr_gb300 import api, synth
from ivr_gb300.state import orbit_state

SKIPS = [api.SKIP_GRID, api.SKIP_LEARNED, api.SKIP_NONE]
ORDERS = [api.TILES_RASTER, api.TILES_COST]
SIZES = [(120, 96), (1200, 900)]  # below and above the cost order's least number of tiles
OUT = 0x1000  # an address that nothing follows


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return load(tmp_path_factory.mktemp("host"))


@pytest.fixture
def scene(lib):
    lib.fake_reset()
    ctx = HostContext(lib)
    v = ctx.load_volume(np.arange(24 * 20 * 28, dtype=np.uint16).reshape(24, 20, 28)).bricks(2, 1, 1)
    mlp = ctx.mlp(1)
    v.set_mlp(mlp, 0.1)
    lut = synth.knot_tf(1, zero_first=True)[0]
    tf = ctx.transfer_function().set_lut(lut, 0, 1.0)
    yield ctx, v, tf, lut
    v.set_mlp(None)
    v.free()
    mlp.free()
    tf.free()
    ctx.close()


def view_of(ctx, v, skip, order, size):
    return ctx.view().set(v, orbit_state(20, 10, *size), api.config_params(skip=skip, tiles=order))


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("order", ORDERS)
@pytest.mark.parametrize("skip", SKIPS)
@pytest.mark.parametrize("census", [False, True])
def test_frame_on_a_second_stream(lib, scene, skip, order, size, census):
    ctx, v, tf, lut = scene
    a, b = ctx.stream(), ctx.stream()
    one, two = (view_of(ctx, v, skip, order, size) for _ in range(2))
    for _ in range(3):
        lib.cudaDeviceSynchronize()  # a TF that frames still read is not edited
        tf.set_lut(lut, 0, 1.0)  # the next frame builds new grids
        one.render(tf, None, OUT, a)
        if census:
            two.census(tf, b)
        two.render(tf, None, OUT, b)
        two.render(tf, None, OUT, b)
        assert lib.fake_races() == 0, lib.fake_first_race()
    one.free()
    two.free()


def test_many_streams_views_and_edits(lib, scene):
    """Frames of every kind on four streams in any order, edits in between,
    a batch now and then; each view stays on its stream."""
    ctx, v, tf, lut = scene
    rng = random.Random(5)
    tfs = [tf] + [ctx.transfer_function().set_lut(lut, 0, 1.0) for _ in range(3)]
    streams = [0] + [ctx.stream() for _ in range(3)]
    views = [(view_of(ctx, v, skip, order, size), s) for s in streams for skip in SKIPS for order in ORDERS
             for size in SIZES]
    batch = ctx.batch(4)
    for n in range(600):
        if rng.random() < 0.06:
            lib.cudaDeviceSynchronize()
            rng.choice(tfs).set_lut(lut, 0, 1.0)
        if rng.random() < 0.03:
            batch.clear()
            batch.add(next(w for w, _ in views if w is not None), rng.choice(tfs), OUT)
            batch.render(False, rng.choice(streams))
        w, s = rng.choice(views)
        w.render(rng.choice(tfs), None, OUT, s)
        assert lib.fake_races() == 0, (n, lib.fake_first_race())
    assert lib.fake_early() > 100  # plain frames still overlap
    batch.free()
    for w, _ in views:
        w.free()
    for t in tfs[1:]:
        t.free()
