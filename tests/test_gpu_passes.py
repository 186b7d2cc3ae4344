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


@pytest.mark.parametrize("dtype,n", [("u8", 70), ("u16", 140), ("f32", 80)])
def test_histogram_of_plateaus(ctx, oracle_mod, dtype, n):
    """Stretches of one value, longer and shorter than a 16-byte load and at
    every offset in one: background, saturated and in between."""
    rng = np.random.default_rng(11)
    top = 255 if dtype != "u16" else 16383  # 140^3 voxels: shared counters, one copy
    vals = rng.choice([0, 1, top // 3, top], 400000)
    vol = np.repeat(vals, rng.integers(1, 41, vals.size))[:n ** 3]
    vol = np.resize(vol, n ** 3).reshape(n, n, n).astype({"u8": np.uint8, "u16": np.uint16, "f32": np.float32}[dtype])
    vol.reshape(-1)[:2] = (0, top)
    _, _, ohist = oracle_mod.minmax_histogram(vol)
    v = ctx.load_volume(vol)
    try:
        assert np.array_equal(v.histogram(len(ohist)), ohist)
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


@pytest.mark.parametrize("dtype", ["u8", "u16", "f32"])
@pytest.mark.parametrize("shape,cell,bricks", [
    ((17, 18, 129), 16, 1),   # scalar rows: one column past a 128-column segment
    ((20, 33, 128), 16, 1),   # 16-byte rows: one whole f32 segment
    ((9, 34, 544), 32, 1),    # two segments of u8, the edge between two cells
    ((35, 19, 272), 4, 1),    # the smallest cells
    ((2, 3, 2), 16, 1),       # the smallest volume
    ((40, 37, 66), 8, 2)])    # bricks with halos: odd rows
def test_grids_gradient_and_copies_match_brute_force(ctx, oracle_mod, dtype, shape, cell, bricks):
    """The exact skipping grid shows each macrocell's min and max (a LUT that
    is opaque in one value range only); the gradient and a frame through the
    corner-packed copies, against the oracle."""
    import torch
    from ivr_gb300 import api, synth
    from ivr_gb300.state import orbit_state
    vol = volume(dtype, shape, 255 if dtype != "u16" else 65535, seed=7)
    scale = 256.0 / 65536.0 if dtype == "u16" else 1.0
    v = ctx.load_volume(vol).macrocell(cell)
    try:
        if bricks > 1:
            v.bricks(bricks, bricks, bricks)
        for lo in (0, 100, 250):
            lut = np.zeros((256, 4), np.float32)
            lut[lo:lo + 3, 3] = 0.5
            tf = ctx.transfer_function().set_lut(lut, 0, scale, api.TF_F2B)
            if bricks == 1:
                got = v.skip_grid(tf)
                idx = (vol.astype(np.float32) * np.float32(scale)).astype(np.int64)
                for z, y, x in np.ndindex(got.shape):
                    part = idx[z * cell:(z + 1) * cell + 1, y * cell:(y + 1) * cell + 1, x * cell:(x + 1) * cell + 1]
                    opaque = lut[max(part.min() - 1, 0):min(part.max() + 1, 255) + 1, 3].any()
                    assert (got[z, y, x] == 0) == opaque, (z, y, x)
            st = orbit_state(25.0, -35.0, 61, 47)
            ref = oracle_mod.render(vol, st, lut, 0, 6, preset=1, procdims=(bricks,) * 3, lut_scale=scale)
            view = ctx.view().set(v, st, api.config_params())
            o32 = torch.zeros((47, 61, 4), device="cuda")
            view.render(tf, o32.data_ptr())
            torch.cuda.synchronize()
            assert np.array_equal(o32.cpu().numpy().view(np.uint32), ref["rgba32"].view(np.uint32))
            view.free()
            tf.free()
        out = torch.full(shape + (4,), -1.0, device="cuda")
        v.gradient(out.data_ptr())
        torch.cuda.synchronize()
        want = oracle_mod.gradient(vol.astype(np.float32))
        assert np.array_equal(out.cpu().numpy().view(np.uint32), np.ascontiguousarray(want, np.float32).view(np.uint32))
    finally:
        v.free()


@pytest.mark.parametrize("n,shift_in,shift_out", [(1, 0, 0), (7, 0, 0), (4096, 0, 0), (4099, 0, 0), (1000, 1, 0),
                                                  (1001, 0, 1), (1002, 4, 4), (3000003, 0, 0)])
def test_quantize_at_any_length_and_alignment(ctx, oracle_mod, n, shift_in, shift_out):
    import torch
    rng = np.random.default_rng(n)
    x = rng.uniform(-0.2, 1.2, n + shift_in).astype(np.float32)
    x[::97] = np.nan
    x[1::89] = np.inf
    src = torch.from_numpy(x).cuda()
    dst = torch.full((n + shift_out + 8,), 77, dtype=torch.uint8, device="cuda")
    ctx.quantize(src.data_ptr() + 4 * shift_in, dst.data_ptr() + shift_out, n)
    torch.cuda.synchronize()
    got = dst.cpu().numpy()
    assert np.array_equal(got[shift_out:shift_out + n], oracle_mod.quantize(np.nan_to_num(x[shift_in:], nan=0.0)))
    assert (got[:shift_out] == 77).all() and (got[shift_out + n:] == 77).all()
