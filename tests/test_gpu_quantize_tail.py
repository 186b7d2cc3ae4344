"""GPU: quantising a number of floats that is no multiple of four: every
remainder, and no second launch for it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6, 1021, 1022, 1023, 1244673, 1244674, 1244675])
def test_remainders(ctx, oracle_mod, n):
    import torch
    x = np.random.default_rng(n).uniform(-0.1, 1.1, n).astype(np.float32)
    src, dst = torch.from_numpy(x).cuda(), torch.full((n + 8,), 77, dtype=torch.uint8, device="cuda")
    ctx.quantize(src.data_ptr(), dst.data_ptr(), n)
    torch.cuda.synchronize()
    got = dst.cpu().numpy()
    assert np.array_equal(got[:n], oracle_mod.quantize(x)) and (got[n:] == 77).all()


def test_a_remainder_takes_no_longer(ctx):
    import torch
    src, dst = torch.zeros(1024, device="cuda"), torch.zeros(1024, dtype=torch.uint8, device="cuda")

    def us(n, calls=400):
        took = []
        for _ in range(9):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(calls):
                ctx.quantize(src.data_ptr(), dst.data_ptr(), n)
            b.record()
            b.synchronize()
            took.append(1e3 * a.elapsed_time(b) / calls)
        return np.median(took)

    us(1024)
    assert us(1023) < 1.6 * us(1024)
