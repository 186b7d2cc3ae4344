"""GPU: histograms of volumes with few voxels: every kernel's side of the
limits in voxels, bins and voxels a bin, against the counts themselves; and
voxels that crowd in one bin take no longer than spread ones."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DTYPES = {"u8": np.uint8, "u16": np.uint16, "f32": np.float32}


def expected(vol, hsize):
    b = (vol.astype(np.float32) - np.float32(vol.min())).astype(np.int64).ravel()
    return np.bincount(b[(b >= 0) & (b < hsize)], minlength=hsize)


@pytest.mark.parametrize("dtype,top", [("u8", 255), ("u16", 12287), ("u16", 12288), ("u16", 65535), ("f32", 999),
                                       ("f32", 12287), ("f32", 12288)])
@pytest.mark.parametrize("shape", [(2, 2, 2), (3, 5, 7), (8, 8, 8), (31, 33, 35), (117, 114, 118), (136, 136, 134),
                                   (136, 136, 135)])
def test_counts(ctx, dtype, top, shape):
    rng = np.random.default_rng(top + shape[0])
    vol = rng.integers(3, top + 1, shape)
    vol[rng.random(shape) < 0.4] = top  # a crowded bin that is not the minimum's
    vol = vol.astype(DTYPES[dtype])
    if dtype == "f32":
        vol += rng.uniform(0.0, 0.9, shape).astype(np.float32)
    v = ctx.load_volume(vol)
    try:
        for hsize in (1, 2, top // 3, top - 2, top + 5):
            assert np.array_equal(v.histogram(hsize), expected(vol, hsize)), hsize
    finally:
        v.free()


@pytest.mark.parametrize("n,top", [(48, 1023), (80, 4095), (112, 12287)])
def test_crowded_voxels_take_no_longer(ctx, n, top):
    """Fewer than 128 voxels a bin, 60% of them of the largest value: counted
    one by one in global memory they took up to seven times as long a call."""
    rng = np.random.default_rng(n)
    spread = rng.integers(0, top + 1, (n, n, n)).astype(np.uint16)
    crowded = spread.copy()
    crowded[rng.random(spread.shape) < 0.6] = top
    times = {}
    for name, vol in (("spread", spread), ("crowded", crowded)):
        v = ctx.load_volume(vol)
        assert np.array_equal(v.histogram(top + 1), np.bincount(vol.ravel(), minlength=top + 1))
        took = []
        for _ in range(60):
            t = time.perf_counter()
            v.histogram(top + 1)
            took.append(time.perf_counter() - t)
        times[name] = np.median(took)
        v.free()
    assert times["crowded"] < 2.0 * times["spread"], times
