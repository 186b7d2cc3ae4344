"""GPU: frames in a row on one stream (a launch may begin while the one
before it ends): one buffer, several views, sizes, skip modes and transfer
functions in turn, new grids in between, on several streams, and in a
captured graph; every frame is the one rendered alone."""
import numpy as np
import pytest

from ivr_gb300 import api, synth
from ivr_gb300.state import orbit_state

pytestmark = pytest.mark.gpu


def scene(ctx):
    v = ctx.load_volume(synth.blob_volume((60, 70, 64), n_blobs=6, seed=3, dtype="u16", noise=0.05)).bricks(2, 2, 2)
    scale = 256.0 / 65536.0
    tfs = [ctx.transfer_function().set_lut(synth.knot_tf(s, zero_first=True)[0], 0, scale) for s in range(3)]
    jobs = []
    for n, (w, h) in enumerate([(64, 48), (400, 300), (33, 21), (1200, 900), (256, 256), (8, 4)]):
        for skip in (api.SKIP_GRID, api.SKIP_NONE):
            st = orbit_state(25.0 * n, 10.0 * n - 30.0, w, h)
            jobs.append((ctx.view().set(v, st, api.config_params(skip=skip)), tfs[n % 3], w, h))
    return v, tfs, jobs


def test_frames_in_a_row_equal_frames_alone(ctx):
    import torch
    v, tfs, jobs = scene(ctx)
    try:
        alone = []
        for view, tf, w, h in jobs:
            out = torch.zeros((h, w, 4), device="cuda")
            view.render(tf, out.data_ptr())
            torch.cuda.synchronize()
            alone.append(out.cpu().numpy())
        streams = [torch.cuda.current_stream(), torch.cuda.Stream(), torch.cuda.Stream()]
        for s in streams:
            # all into one buffer, each copied out behind its launch; then
            # without the copies, the last frame stands
            big = torch.zeros(1200 * 900 * 4, device="cuda")
            with torch.cuda.stream(s):
                got = []
                for view, tf, w, h in jobs * 2:
                    view.render(tf, big.data_ptr(), None, s.cuda_stream)
                    got.append(big[:w * h * 4].clone())
                for view, tf, w, h in jobs * 2:
                    view.render(tf, big.data_ptr(), None, s.cuda_stream)
                last = big.clone()
            s.synchronize()
            for k, g in enumerate(got):
                assert np.array_equal(g.cpu().numpy(), alone[k % len(jobs)].reshape(-1)), k
            full = np.zeros(1200 * 900 * 4, np.float32)
            for a in alone * 2:
                full[:a.size] = a.reshape(-1)
            assert np.array_equal(last.cpu().numpy()[:full.size], full)
    finally:
        v.free()


def test_edits_between_frames(ctx):
    """A new grid before every frame, and the same grid built through one
    stream and read on another."""
    import torch
    v, tfs, jobs = scene(ctx)
    view, _, w, h = jobs[2]
    scale = 256.0 / 65536.0
    try:
        luts = [synth.knot_tf(50 + k, zero_first=True)[0] for k in range(8)]
        want = []
        for lut in luts:
            tfs[0].set_lut(lut, 0, scale)
            out = torch.zeros((h, w, 4), device="cuda")
            view.render(tfs[0], out.data_ptr())
            torch.cuda.synchronize()
            want.append(out.cpu().numpy())
        other = torch.cuda.Stream()
        for _ in range(2):
            outs = []
            for k, lut in enumerate(luts):
                tfs[0].set_lut(lut, 0, scale)
                for s in (torch.cuda.current_stream(), other) if k % 2 else (other, torch.cuda.current_stream()):
                    out = torch.empty((h, w, 4), device="cuda")
                    s.wait_stream(torch.cuda.current_stream())
                    with torch.cuda.stream(s):
                        for _ in range(3):
                            view.render(tfs[0], out.data_ptr(), None, s.cuda_stream)
                    s.synchronize()  # one view's launches are ordered
                    outs.append((k, out))
            for k, out in outs:
                assert np.array_equal(out.cpu().numpy(), want[k]), k
    finally:
        v.free()


def test_frames_in_a_captured_graph(ctx):
    import torch
    v, tfs, jobs = scene(ctx)
    try:
        picks = [jobs[0], jobs[2], jobs[5], jobs[8]]
        outs = [torch.zeros((h, w, 4), device="cuda") for _, _, w, h in picks]
        want = []
        for (view, tf, w, h), o in zip(picks, outs):
            view.render(tf, o.data_ptr())
            view.render(tf, o.data_ptr())
            torch.cuda.synchronize()
            want.append(o.cpu().numpy())
            o.zero_()
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            for (view, tf, w, h), o in zip(picks, outs):
                view.render(tf, o.data_ptr(), None, torch.cuda.current_stream().cuda_stream)
        g.replay()
        torch.cuda.synchronize()
        for o, w_ in zip(outs, want):
            assert np.array_equal(o.cpu().numpy(), w_)
    finally:
        v.free()
