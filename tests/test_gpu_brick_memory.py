"""GPU: what a memory budget admits of a brick layout: its arrays in order,
the corner-packed copies only where they fit, refusals that leave nothing
behind; and layouts that follow one another in a volume's memory."""
import numpy as np
import pytest

from ivr_gb300 import api, synth
from ivr_gb300._lib import IvrError
from ivr_gb300.state import orbit_state

pytestmark = pytest.mark.gpu

N, CELL = 40, 8


def layout_arrays():
    """(bytes, optional) of each array of the 2x2x2 layout of an N^3 u8 volume
    with a halo of one, in the order in which they are admitted."""
    out = []
    for r in range(8):
        d = [N // 2 if last else N // 2 + 1 for last in (r % 2, r // 2 % 2, r // 4)]
        cells = np.prod([(x - 2) // CELL + 1 for x in d])
        out += [(int(np.prod(d)), False), (int(cells) * 8, False), ((d[0] - 1) * (d[1] - 1) * d[2] * 4, True)]
    return out


@pytest.mark.parametrize("room", [0, 1, 3, 8, 20, None])
def test_budget_admits_the_arrays_in_order(room):
    vol = np.random.default_rng(3).integers(0, 256, (N, N, N)).astype(np.uint8)
    arrays = layout_arrays()
    with api.Context(0, hbm_budget=1 << 30) as small:
        v = small.load_volume(vol)
        v.quads(False)
        v.macrocell(CELL)
        base = small.mem_used - int(np.prod([(N - 2) // CELL + 1] * 3)) * 8  # without the layout's arrays
        v.free()
    must = sum(b for b, opt in arrays if not opt)
    quads = [b for b, opt in arrays if opt]
    budget = base + (must + sum(quads[:room]) if room is not None else must - 1)
    # the arrays that fit, one after the other
    used, packed, refused = base, 0, False
    for b, opt in arrays:
        if used + b > budget:
            if not opt:
                refused = True
                break
            continue
        used += b
        packed += b if opt else 0
    with api.Context(0, hbm_budget=budget) as small:
        before = small.mem_used
        v = small.load_volume(vol)
        v.macrocell(CELL)
        if refused:
            with pytest.raises(IvrError) as e:
                v.bricks(2, 2, 2)
            assert e.value.code == -3
            assert small.mem_used == base
        else:
            v.bricks(2, 2, 2)
            assert small.mem_used == used and v.quad_bytes() == packed
        v.bricks(1, 1, 1)
        v.free()
        assert small.mem_used == before


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.float32])
def test_layouts_in_turn_render_as_new_volumes(ctx, dtype):
    """The corner-packed copies of one layout lie where those of the one
    before lay, also with frames still running, switched off and on between."""
    import torch
    vol = (np.random.default_rng(5).integers(0, 256, (37, 41, 33)) * (255 if dtype == np.uint16 else 1)).astype(dtype)
    tf = ctx.transfer_function()
    tf.set_lut(synth.ramp_tf(256), 0, 1.0 / 255.0 if dtype == np.uint16 else 1.0, api.TF_F2B)
    cam = orbit_state(37, 21, 150, 110, fovy=30.0, alpha=1.0, dist=5.0)
    params = api.config_params(step=0.3, skip=api.SKIP_GRID)
    stream = torch.cuda.Stream()

    def frame(v, view):
        out = torch.zeros((110, 150, 4), dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        view.set(v, cam, params)
        view.render(tf, None, out.data_ptr(), stream.cuda_stream)
        return out

    layouts = [(1, 1, 1), (2, 2, 2), (1, 1, 4), None, (3, 1, 2), (1, 1, 1)]
    v, view, got = ctx.load_volume(vol), ctx.view(), []
    for k in layouts:
        if k is None:
            v.quads(False)
            assert v.quad_bytes() == 0
            v.quads(True)
        else:
            v.bricks(*k)
        assert v.quad_bytes() > 0
        got.append(frame(v, view))
    used = ctx.mem_used
    v.bricks(2, 2, 2)
    v.bricks(1, 1, 1)
    torch.cuda.synchronize()
    assert ctx.mem_used <= used  # (the layout's skipping grids are gone)
    v.free()
    for i, k in enumerate(layouts):
        fresh = ctx.load_volume(vol)
        fresh.bricks(*(k or layouts[i - 1]))
        want = frame(fresh, ctx.view())
        torch.cuda.synchronize()
        assert torch.equal(got[i], want), (i, k)
        fresh.free()
