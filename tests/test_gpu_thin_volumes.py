"""GPU: volumes of narrow rows and low slabs: the gradient against numpy, and
that it takes no longer than a cube's of as many voxels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DTYPES = {"u8": np.uint8, "u16": np.uint16, "f32": np.float32}


def volume(shape, dtype, seed=1):
    rng = np.random.default_rng(seed)
    if dtype == "f32":
        return rng.uniform(-50.0, 200.0, shape).astype(np.float32)
    return rng.integers(0, np.iinfo(DTYPES[dtype]).max + 1, shape).astype(DTYPES[dtype])


def device_us(fn, runs=9):
    """Median time of fn's work on the current stream."""
    import torch
    fn()
    took = []
    for _ in range(runs):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        fn()
        b.record()
        b.synchronize()
        took.append(1e3 * a.elapsed_time(b))
    return float(np.median(took))


@pytest.mark.parametrize("dtype", ["u8", "u16", "f32"])
@pytest.mark.parametrize("shape", [(2, 2, 2), (130, 2, 2), (65, 3, 3), (9, 5, 4), (7, 40, 5), (3, 33, 9), (5, 4, 17),
                                   (4, 17, 31), (6, 9, 32), (2, 300, 33), (257, 2, 8), (3, 6, 129), (5, 2, 300)])
def test_gradient(ctx, dtype, shape):
    import torch
    vol = volume(shape, dtype)
    v = ctx.load_volume(vol)
    out = torch.full((*shape, 4), -7.0, device="cuda")
    v.gradient(out.data_ptr())
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    v.free()
    f = vol.astype(np.float32)
    want = np.empty((*shape, 4), np.float32)
    for a in range(3):  # z, y, x
        n = shape[a]
        hi, lo = np.minimum(np.arange(n) + 1, n - 1), np.maximum(np.arange(n) - 1, 0)
        want[..., 2 - a] = (np.take(f, hi, a) - np.take(f, lo, a)) / np.float32(2.0)
    x, y, z = (want[..., k] for k in range(3))
    want[..., 3] = np.sqrt(x * x + y * y + z * z)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("shape", [(2048, 2048, 2), (1024, 1024, 8), (500000, 4, 4)])
def test_gradient_takes_no_longer(ctx, shape):
    import torch
    out = torch.empty((256, 256, 128, 4), device="cuda")
    us = {}
    for s in ((256, 256, 128), shape):
        v = ctx.load_volume(np.zeros(s, np.uint8))
        us[s] = device_us(lambda: v.gradient(out.data_ptr()))
        v.free()
    assert us[shape] < 2.0 * us[(256, 256, 128)], us


@pytest.mark.parametrize("dtype", ["u8", "u16", "f32"])
@pytest.mark.parametrize("shape,bricks", [((2, 2, 2), (1, 1, 1)), ((70, 2, 2), (1, 1, 2)), ((65, 4, 3), (2, 1, 1)),
                                          ((9, 5, 6), (2, 2, 1)), ((7, 40, 5), (1, 1, 1)), ((33, 35, 33), (1, 1, 1)),
                                          ((5, 3, 34), (1, 1, 1)), ((6, 38, 66), (1, 2, 1)), ((2, 260, 9), (3, 1, 1))])
def test_corner_packed_copies(ctx, dtype, shape, bricks):
    """Frames from the copies are those from the voxels."""
    import torch
    from ivr_gb300 import api, synth
    from ivr_gb300.state import orbit_state
    v = ctx.load_volume(volume(shape, dtype)).bricks(*bricks)
    tf = ctx.transfer_function().set_lut(synth.ramp_tf(256), 0, 256.0 / 65536.0 if dtype == "u16" else 1.0)
    frames = []
    for on in (True, False):
        v.quads(on)
        assert (v.quad_bytes() > 0) == on
        view = ctx.view().set(v, orbit_state(35.0, 25.0, 160, 120), api.config_params(step=0.1, term_alpha=2.0))
        out = torch.full((120, 160, 4), -7.0, device="cuda")
        view.render(tf, out.data_ptr())
        torch.cuda.synchronize()
        frames.append(out.cpu().numpy().view(np.uint32))
        view.free()
    v.free()
    tf.free()
    assert frames[1].any() and np.array_equal(*frames)


def test_corner_packed_copies_take_no_longer(ctx):
    """What the copies add to the set-up of a thin brick, against a cube's."""
    import time
    import torch
    added = {}
    for shape in ((512, 512, 128), (4096, 4096, 2)):
        v = ctx.load_volume(np.zeros(shape, np.uint8))
        took = {}
        for on in (True, False):
            v.quads(on)
            t = []
            for _ in range(9):
                torch.cuda.synchronize()
                a = time.perf_counter()
                v.bricks(1, 1, 1)  # (ends with a synchronisation)
                t.append(1e6 * (time.perf_counter() - a))
            took[on] = np.median(t)
        added[shape] = took[True] - took[False]
        v.free()
    assert added[(4096, 4096, 2)] < 2.0 * added[(512, 512, 128)] + 100.0, added
