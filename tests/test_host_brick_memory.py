"""CPU: brick set-up on a device that runs out of memory, allocation by
allocation and at every capacity, and with launches that fail: what is needed
is placed while it fits, the corner-packed copies are left out where they do
not, a refusal leaves nothing behind, and no call reports another's failure."""
import ctypes

import numpy as np
import pytest

from host import HostContext, load
from ivr_gb300 import api, synth
from ivr_gb300._lib import IvrError
from ivr_gb300.state import orbit_state

N = 40
VOL = np.zeros((N, N, N), np.float32)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return load(tmp_path_factory.mktemp("host"))


def try_bricks(v, grid):
    try:
        v.bricks(*grid)
        return 0
    except IvrError as e:
        return e.code


def frame(ctx, v):
    """A frame renders (and reports nothing that an earlier call left)."""
    tf = ctx.transfer_function().set_lut(synth.ramp_tf(16), 0, 1.0)
    view = ctx.view()
    try:
        view.set(v, orbit_state(10, 10, 32, 32), api.config_params()).render(tf, None, 0x1000)
    finally:
        view.free()
        tf.free()


def needed(grid):
    """Bytes of a layout's voxels and macrocells, and of its copies."""
    must = copies = 0
    py, px, pz = grid
    for r in range(py * px * pz):
        at, n = (r % px, r // px % py, r // (py * px)), (px, py, pz)
        d = [N // n[a] + (N % n[a] if at[a] == n[a] - 1 else 1) for a in range(3)]
        must += (int(np.prod(d)) * 4 if py * px * pz > 1 else 0) + int(np.prod([(x - 2) // 16 + 1 for x in d])) * 8
        copies += (d[0] - 1) * (d[1] - 1) * d[2] * 16
    return must, copies


@pytest.mark.parametrize("grid", [(1, 1, 1), (2, 2, 2), (1, 3, 4)])
@pytest.mark.parametrize("first", [0, 1, 2, 3])
@pytest.mark.parametrize("more", [0, 1, 2, 40])
def test_allocations_that_fail(lib, grid, first, more):
    """The first-th allocation of the set-up fails, and with `more` as many of
    those behind it."""
    lib.fake_reset()
    ctx = HostContext(lib)
    v = ctx.load_volume(VOL)
    empty = ctx.mem_used - sum(needed((1, 1, 1)))
    m, copies = needed(grid)
    lib.fake_fail_malloc(first)
    lib.fake_fail_more(more)
    rc = try_bricks(v, grid)
    lib.fake_fail_malloc(-1)
    assert lib.cudaGetLastError() == 0
    if rc:
        assert rc == -3 and first == 0 and more > 0  # the arrays that must be, block and one by one
        assert ctx.mem_used == empty
        assert try_bricks(v, grid) == 0
    elif first + more == 0:  # (the kept copies' block is given back, and asked for again)
        assert v.quad_bytes() == copies
    assert ctx.mem_used == empty + m + v.quad_bytes()
    frame(ctx, v)
    v.free()
    ctx.close()
    assert lib.fake_in_use() == 0


@pytest.mark.parametrize("grid", [(2, 2, 2), (1, 1, 4), (3, 1, 2)])
def test_every_capacity(lib, grid):
    lib.fake_reset()
    must, copies = needed(grid)
    served = 0
    for extra in range(0, copies + copies // 4, 4096):
        lib.fake_capacity(1 << 40)
        ctx = HostContext(lib)
        base = lib.fake_in_use() + VOL.nbytes
        v = ctx.load_volume(VOL)
        lib.fake_capacity(base + must + extra)
        rc = try_bricks(v, grid)
        assert lib.cudaGetLastError() == 0
        # what must be fits (but for the arrays' alignment)
        if extra >= 512 * 2 * np.prod(grid):
            assert rc == 0, extra
        if rc == 0:
            got = v.quad_bytes()
            assert served <= got <= extra  # more room, more copies
            served = got if got == copies else 0
            assert ctx.mem_used <= lib.fake_in_use()
        lib.fake_capacity(1 << 40)
        if rc == 0:
            frame(ctx, v)
        v.free()
        ctx.close()
        assert lib.fake_in_use() == 0
    assert served == copies


@pytest.mark.parametrize("n", range(25))
def test_launches_that_fail(lib, n):
    """The set-up of eight bricks has 24 launches: one fails, no brick is left
    that was not filled, and the next set-up is whole."""
    lib.fake_reset()
    ctx = HostContext(lib)
    v = ctx.load_volume(VOL)
    empty = ctx.mem_used - sum(needed((1, 1, 1)))
    lib.fake_fail_launch(n)
    rc = try_bricks(v, (2, 2, 2))
    lib.fake_fail_launch(-1)
    assert (rc != 0) == (n < 24)
    if rc:
        assert rc == -2 and ctx.mem_used == empty and v.quad_bytes() == 0
        with pytest.raises(IvrError):
            frame(ctx, v)
        assert try_bricks(v, (2, 2, 2)) == 0
    assert ctx.mem_used == empty + sum(needed((2, 2, 2)))
    frame(ctx, v)
    v.free()
    ctx.close()
    assert lib.fake_in_use() == 0
