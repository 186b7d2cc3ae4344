"""GPU: the passes over a whole volume (min/max, histogram) at the sizes
where their vector loads, bin ranges and counter copies change."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def volume(dtype, shape, top, seed=1):
    """Uniform values up to `top` with half the voxels background and the
    extremes present; f32 values have fractions and a fractional minimum."""
    rng = np.random.default_rng(seed)
    v = rng.uniform(0.0, top, shape) * (rng.uniform(size=shape) < 0.5)
    v.reshape(-1)[-1] = top
    if dtype == "f32":
        return (v + 0.25).astype(np.float32)
    return v.astype(np.uint8 if dtype == "u8" else np.uint16)


# shapes whose voxel count leaves every remainder of a 16-byte load, one
# smaller than a load, and one with more than one trip per thread; voxels per
# bin on both sides of the shared counters' rule (128); and for the shared
# ones 32, 2 and 1 copies, one range, two ranges, and more bins than two hold
@pytest.mark.parametrize("dtype,shape,top", [
    ("u8", (2, 2, 2), 255), ("u8", (5, 7, 11), 255), ("u8", (16, 16, 16), 3), ("u8", (32, 32, 31), 255),
    ("u8", (32, 32, 32), 255), ("u8", (160, 170, 181), 255), ("u16", (3, 3, 5), 65535), ("u16", (63, 64, 65), 896),
    ("u16", (31, 33, 35), 28671), ("u16", (130, 130, 113), 14335), ("u16", (205, 205, 204), 65535),
    ("f32", (3, 3, 3), 255.0), ("f32", (97, 101, 103), 255.0), ("f32", (40, 40, 40), 57343.0),
    ("f32", (196, 195, 194), 57343.0), ("f32", (245, 245, 246), 114687.0), ("f32", (245, 246, 247), 114688.0),
    ("f32", (48, 40, 44), 1.0e6)])
def test_minmax_and_histogram_match_the_oracle(ctx, oracle_mod, dtype, shape, top):
    vol = volume(dtype, shape, top)
    omn, omx, ohist = oracle_mod.minmax_histogram(vol)
    v = ctx.load_volume(vol)
    try:
        assert v.minmax() == (omn, omx)
        assert np.array_equal(v.histogram(len(ohist)), ohist)
        few = max(1, len(ohist) // 3)  # values above the last bin are not counted
        assert np.array_equal(v.histogram(few), ohist[:few])
        more = v.histogram(len(ohist) + 300000)
        assert np.array_equal(more[:len(ohist)], ohist) and not more[len(ohist):].any()
    finally:
        v.free()


def test_minmax_and_histogram_with_nan_and_infinite_voxels(ctx):
    """NaNs are no minimum or maximum and count as the bin (int)(NaN) = 0;
    an infinite voxel leaves every bin."""
    vol = volume("f32", (9, 9, 9), 100.0)
    vol[0, 0, :4] = np.nan
    vol[1, 1, 1] = np.inf
    v = ctx.load_volume(vol)
    try:
        mn, mx = v.minmax()
        assert mn == np.float32(0.25) and mx == np.inf
        fin = vol[np.isfinite(vol)]
        want = np.bincount((fin - np.float32(0.25)).astype(np.int64), minlength=200)[:200]
        want[0] += 4
        assert np.array_equal(v.histogram(200), want)
    finally:
        v.free()
