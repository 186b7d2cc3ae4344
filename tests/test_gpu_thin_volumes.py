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
