"""The LUT entries that a macrocell's samples can index: the rule itself on the
CPU, over the ends of the ints, and frames of volumes with values beyond them
(infinities among them) on the GPU."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from ivr_gb300 import api, build, synth
from ivr_gb300.state import orbit_state

INT_MIN, INT_MAX = -2 ** 31, 2 ** 31 - 1
SRC = r"""
#include <stdio.h>
#include "ivr_internal.h"
int main(void)
{
    int x0, x1, off, n;
    while (scanf("%d %d %d %d", &x0, &x1, &off, &n) == 4) {
        const ivr::LutRange r = ivr::lut_range(x0, x1, off, n);
        printf("%d %d %d\n", r.lo, r.hi, ivr::lut_index(x0, off));
    }
    return 0;
}
"""


def test_range_holds_every_index_of_the_cell(tmp_path):
    """Against exact integers; no signed overflow anywhere (the sanitiser
    ends the program at one)."""
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "r.cpp", tmp_path / "r"
    src.write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-O2", "-fsanitize=undefined", "-fno-sanitize-recover=all",
                    "-I" + os.path.join(build.ROOT, "include"), "-I" + build.CSRC, "-I" + build.CUDA_INC, str(src), "-o",
                    str(exe)], check=True)
    xs = [INT_MIN, INT_MIN + 1, -70000, -256, -2, -1, 0, 1, 2, 254, 255, 256, 70000, INT_MAX - 1, INT_MAX]
    cases = [(a, b, off, n) for a in xs for b in xs if a <= b for off in (INT_MIN, -300, -7, 0, 5, 255, INT_MAX)
             for n in (1, 2, 256, 1 << 24)]
    out = subprocess.run([str(exe)], input="".join("%d %d %d %d\n" % c for c in cases), capture_output=True, text=True,
                         check=True).stdout.split()
    got = np.array(out, dtype=np.int64).reshape(-1, 3)

    def index(x, off, n):  # what a sample of the value reads
        i = (x - off + 2 ** 31) % 2 ** 32 - 2 ** 31
        return i, min(max(i, 0), n - 1)

    for (a, b, off, n), (lo, hi, i) in zip(cases, got):
        assert i == index(a, off, n)[0]
        for x in {a, b, (a + b) // 2, min(a + 1, b), max(b - 1, a), min(max(off, a), b)}:
            assert 0 <= lo <= index(x, off, n)[1] <= hi < n, (a, b, off, n, x)
        if INT_MIN <= a - off and b - off <= INT_MAX:  # no wider than one entry at each end
            assert lo == min(max(a - off - 1, 0), n - 1) and hi == min(max(b - off + 1, 0), n - 1)


@pytest.mark.gpu
@pytest.mark.parametrize("off", [0, 5, -7])
@pytest.mark.parametrize("top", [3.0e9, 1.0e30, float("inf")])
def test_frames_of_values_beyond_the_ints(ctx, top, off):
    """With a skipping grid, exact or learned, as without one; infinities (whose
    neighbourhood samples NaN) under a LUT that has no transparent entry."""
    import torch
    vol = synth.blob_volume((48, 40, 56), n_blobs=6, seed=9, dtype="f32", noise=0.02, zero_fraction=0.5, cell=8)
    vol[20:24, 16:19, 30:40] = top
    vol[40, 5, 5] = -top
    lut = synth.ramp_tf(256)
    if np.isinf(top):
        lut[:, 3] = np.maximum(lut[:, 3], 0.01)
    v = ctx.load_volume(vol)
    tf = ctx.transfer_function().set_lut(lut, off, 1.0)
    mlp = ctx.mlp(2)
    try:
        mlp.add_samples(v, tf)
        v.set_mlp(mlp, 0.05, certify=True)
        for quads in (True, False):
            v.quads(quads)
            frames = []
            for skip in (api.SKIP_NONE, api.SKIP_GRID, api.SKIP_LEARNED):
                view = ctx.view().set(v, orbit_state(25.0, 15.0, 160, 120), api.config_params(skip=skip))
                out = torch.full((120, 160, 4), -7.0, device="cuda")
                view.render(tf, out.data_ptr())
                torch.cuda.synchronize()
                frames.append(out.cpu().numpy().view(np.uint32))
                view.free()
            assert np.array_equal(frames[0], frames[1])
            assert np.array_equal(frames[0], frames[2])
    finally:
        v.set_mlp(None)
        mlp.free()
        tf.free()
        v.free()
