"""CPU: what training takes of a memory budget: its losses stay, the bias
corrections of an epoch only while it runs, so that a budget which served a
training and what follows it goes on serving them."""
import numpy as np
import pytest

from host import HostContext, load
from ivr_gb300 import synth
from ivr_gb300._lib import IvrError


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return load(tmp_path_factory.mktemp("host"))


def predictor(ctx):
    v = ctx.load_volume(np.zeros((40, 40, 40), np.uint8))
    v.macrocell(4)
    tf = ctx.transfer_function().set_lut(synth.ramp_tf(16), 0, 1.0)
    m = ctx.mlp(1)
    return v, tf, m, m.add_samples(v, tf)


@pytest.mark.parametrize("epochs", [1, 2])
def test_under_a_budget(lib, epochs):
    lib.fake_reset()
    budget = 1 << 30
    for _ in range(2):  # the second time with what the first one needed
        ctx = HostContext(lib, budget)
        v, tf, m, n = predictor(ctx)
        used, cap, peak = ctx.mem_used, 0, 0
        for rows in (512, 64, 512, 24):
            nb = -(-n // rows)
            if nb > cap:
                grown = max(nb, 2 * cap)
                peak = max(peak, used + 4 * grown)  # (the old losses go once the new ones are there)
                used += 4 * (grown - cap)
                cap = grown
            peak = max(peak, used + 8 * nb)
            m.train(epochs, batch_rows=rows)
            assert ctx.mem_used == used
        budget = peak
        for h in (m, tf, v):
            h.free()
        ctx.close()
        assert lib.fake_in_use() == 0
    ctx = HostContext(lib, peak - 1)
    v, tf, m, n = predictor(ctx)
    with pytest.raises(IvrError) as e:
        for rows in (512, 64, 512, 24):
            m.train(epochs, batch_rows=rows)
    assert e.value.code == -3
    for h in (m, tf, v):
        h.free()
    ctx.close()
    assert lib.fake_in_use() == 0


def test_without_a_budget_the_corrections_are_kept(lib):
    lib.fake_reset()
    ctx = HostContext(lib)
    v, tf, m, n = predictor(ctx)
    m.train(1, batch_rows=64)
    before = lib.fake_mallocs()
    for rows in (64, 512):
        m.train(2, batch_rows=rows)
    assert lib.fake_mallocs() == before
    for h in (m, tf, v):
        h.free()
    ctx.close()
    assert lib.fake_in_use() == 0
