"""CPU: the division by a fixed divisor that the REF march uses (FixedDiv in
ivr_march.cu: two-word reciprocal, one remainder step) against IEEE division,
operation for operation in C."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

SRC = r"""
#include <math.h>
#include <stdint.h>
#include <string.h>
/* number of x in [0, n) whose quotient by d differs in any bit */
long mismatches(const float *x, long n, float d)
{
    const float h = 1.0f / d, l = fmaf(-d, h, 1.0f) * h;
    long bad = 0;
    for (long i = 0; i < n; i++) {
        const float q = fmaf(x[i], h, x[i] * l);
        const float got = fmaf(fmaf(-q, d, x[i]), h, q), want = x[i] / d;
        bad += memcmp(&got, &want, 4) != 0;
    }
    return bad;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("fixed_div")
    src, so = os.path.join(d, "d.c"), os.path.join(d, "d.so")
    with open(src, "w") as f:
        f.write(SRC)
    subprocess.run(["gcc", "-O2", "-shared", "-fPIC", "-ffp-contract=off", src, "-o", so, "-lm"], check=True)
    lib = ctypes.CDLL(so)
    lib.mismatches.restype = ctypes.c_long
    lib.mismatches.argtypes = [ctypes.c_void_p, ctypes.c_long, ctypes.c_float]
    return lib


def test_equals_ieee_division(lib):
    """Divisors: brick extents (2 w / max), dims, mantissas next to a power
    of two and random ones; dividends: positions and cell offsets, mantissas
    next to a power of two, the ends of the range the sampler lets through,
    and zero."""
    rng = np.random.default_rng(1)
    one, two = np.float32(1.0), np.float32(2.0)
    near = [np.nextafter(one, two), np.nextafter(two, one), np.nextafter(np.nextafter(two, one), one)]
    d = [np.float32(n) for n in (2, 3, 7, 17, 85, 128, 181, 255, 301, 384, 1023, 1024, 1025, 4095, 65535)]
    d += [np.float32(2.0) * np.float32(a) / np.float32(b) for a, b in ((3, 7), (5, 6), (223, 301), (260, 301), (1, 3))]
    d += near + [np.float32(2.0 ** -60), np.float32(2.0 ** 60)]
    d += list(np.exp2(rng.uniform(-32, 32, 40)).astype(np.float32))
    x = np.concatenate([rng.uniform(-8, 8, 40000), rng.uniform(0, 1e-3, 20000), np.exp2(rng.uniform(-60, 60, 40000)),
                        -np.exp2(rng.uniform(-60, 60, 20000)), rng.integers(0, 4096, 10000),
                        np.exp2(np.arange(-60, 60)), np.array(near), [0.0, 2.0 ** -60, 2.0 ** 60]]).astype(np.float32)
    x = np.concatenate([x, np.nextafter(x, np.float32(np.inf)), np.nextafter(x, np.float32(-np.inf))])
    x = np.ascontiguousarray(x[(np.abs(x) >= 2.0 ** -60) | (np.signbit(x) == 0) & (x == 0)].astype(np.float32))
    for c in d:
        assert lib.mismatches(x.ctypes.data, len(x), float(c)) == 0, float(c)
