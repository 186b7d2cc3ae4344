"""CPU: the bounds within which the REF march takes its packed divisions
(ref_fast in ivr_march.cu, read from there) against IEEE division, operation
for operation in C: the divisions at the ends of the range that the bounds
leave, and the sampler's cell and weight along an axis, with positions next to
brick edges and cell corners."""
import ctypes
import os
import re
import subprocess

import numpy as np
import pytest

from ivr_gb300 import build

SRC = r"""
#include <math.h>
#include <string.h>
typedef struct { float c, h, l; } fixed_div;
static fixed_div fd(float c) { const float h = 1.0f / c; return (fixed_div){c, h, fmaf(-c, h, 1.0f) * h}; }
static float quot(fixed_div d, float x)
{
    const float q = fmaf(x, d.h, x * d.l);
    return fmaf(fmaf(q, -d.c, x), d.h, q);
}
long quotients(const float *x, long n, float c)
{
    long bad = 0;
    const fixed_div d = fd(c);
    for (long i = 0; i < n; i++) {
        const float got = quot(d, x[i]), want = x[i] / c;
        bad += memcmp(&got, &want, 4) != 0;
    }
    return bad;
}
static int cell_of(float r, int dim)
{
    int c = r >= 2147483648.0f ? 2147483647 : r <= -2147483648.0f ? -2147483647 - 1 : (int) r;
    c = c < dim - 2 ? c : dim - 2;
    return c > 0 ? c : 0;
}
/* positions u along an axis: cells and weights that differ */
long axis(const float *u, long n, float bmin, float extent, int dim)
{
    long bad = 0;
    const fixed_div e = fd(extent), d = fd((float) dim);
    for (long i = 0; i < n; i++) {
        const int c = cell_of((float) dim * ((u[i] - bmin) / extent), dim);
        const float want = (fabsf((u[i] + fabsf(bmin)) - (float) c * extent / (float) dim) * extent) / (float) dim;
        const int cf = cell_of((float) dim * quot(e, u[i] + -bmin), dim);
        const float mu0 = quot(d, (float) cf * -extent);
        const float got = fabsf(quot(d, ((u[i] + fabsf(bmin)) + mu0) * extent));
        bad += c != cf || memcmp(&got, &want, 4) != 0;
    }
    return bad;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("ref_divisions")
    src, so = os.path.join(d, "d.c"), os.path.join(d, "d.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.run(["gcc", "-O2", "-shared", "-fPIC", "-ffp-contract=off", src, "-o", so, "-lm"], check=True)
    lib = ctypes.CDLL(so)
    lib.quotients.restype = lib.axis.restype = ctypes.c_long
    lib.quotients.argtypes = [ctypes.c_void_p, ctypes.c_long, ctypes.c_float]
    lib.axis.argtypes = [ctypes.c_void_p, ctypes.c_long, ctypes.c_float, ctypes.c_float, ctypes.c_int]
    return lib


@pytest.fixture(scope="module")
def bounds():
    with open(os.path.join(build.CSRC, "ivr_march.cu")) as f:
        src = f.read()
    b = {k: float(re.search(r"\b%s = ([0-9.e+-]+)f" % k, src).group(1)) for k in ("kRefNear", "kRefFar", "kRefThin")}
    b["kRefDim"] = 1 << int(re.search(r"\bkRefDim = 1 << (\d+);", src).group(1))
    return b


def dense(lo, hi, n, rng):
    """Floats of [lo, hi]: random ones, the ends, and mantissas next to powers of two."""
    e = np.arange(np.ceil(np.log2(lo)), np.floor(np.log2(hi)) + 1)
    x = np.concatenate([np.exp2(rng.uniform(np.log2(lo), np.log2(hi), n)), np.exp2(e), [lo, hi]]).astype(np.float32)
    x = np.concatenate([x, np.nextafter(x, np.float32(np.inf)), np.nextafter(x, np.float32(0))])
    return np.ascontiguousarray(x[(x >= np.float32(lo)) & (x <= np.float32(hi))])


def test_divisions_over_the_range(lib, bounds):
    """The smallest dividend is a difference of positions, a multiple of the
    last place of an edge or a corner, times the smallest extent."""
    rng = np.random.default_rng(2)
    thin, far, near, dim = (bounds[k] for k in ("kRefThin", "kRefFar", "kRefNear", "kRefDim"))
    corner = thin / dim
    difference = min(near * 1e-6 / 2, near / 2 * 2.0 ** -23, corner / 2 * 2.0 ** -23)
    low, high = difference * min(thin, 1.0), 2.0 * far * 2.0 ** 17 * far
    assert low >= 2.0 ** -73 and high <= 2.0 ** 98  # (what FixedDiv's comment takes for granted)
    x = dense(2.0 ** -73, 2.0 ** 98, 60000, rng)
    x = np.ascontiguousarray(np.concatenate([x, -x, np.zeros(1, np.float32)]))
    for c in np.concatenate([dense(thin, far, 60, rng)[::3], dense(2.0, dim, 20, rng).round(), [3, 5, 7, 65535]]):
        assert lib.quotients(x.ctypes.data, len(x), float(c)) == 0, float(c)


@pytest.mark.parametrize("seed", range(4))
def test_cells_and_weights(lib, bounds, seed):
    rng = np.random.default_rng(seed)
    thin, far, near, top = (bounds[k] for k in ("kRefThin", "kRefFar", "kRefNear", "kRefDim"))
    for _ in range(300):
        dim = int(np.exp2(rng.uniform(1, np.log2(top)))) if rng.random() < 0.9 else int(rng.choice([2, 3, top - 1, top]))
        extent = np.float32(np.exp2(rng.uniform(np.log2(thin), 3))) if rng.random() < 0.9 else np.float32(
            rng.choice([thin, far]))
        edge = rng.random()
        if edge < 0.3:
            bmin = np.float32(0.0)
        else:
            bmin = np.float32(-extent / 2 if edge < 0.6 else rng.choice([-1, 1]) * np.exp2(rng.uniform(np.log2(near), 3)))
        # next to the edges and corners, by a few last places, and anywhere
        at = np.concatenate([rng.integers(0, dim + 1, 300) * (float(extent) / dim), [0.0, float(extent)]])
        for edge_sign in (1.0, -1.0):
            u = np.concatenate([edge_sign * float(bmin) + at, -abs(float(bmin)) + at]).astype(np.float32)
            u = np.concatenate([u, np.nextafter(u, np.float32(9)), np.nextafter(u, np.float32(-9)),
                                rng.uniform(-2, 2, 200).astype(np.float32) * extent])
            if bmin == 0.0:  # seen from o = 0, or from a float's last place of an o of kRefNear and more
                u = u[(u == 0.0) | (np.abs(u) >= min(near * 1e-6, near / 2 * 2.0 ** -23))]
            u = np.ascontiguousarray(u)
            assert lib.axis(u.ctypes.data, len(u), float(bmin), float(extent), dim) == 0, (bmin, extent, dim)
