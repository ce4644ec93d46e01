"""Device arrays that the default stream is still writing when pg_learned_make_pairs or pg_learned_loss is called:
the context's stream does not order itself behind them, the call has to."""
import numpy as np
import pytest

from plategpu import learned, workloads

pytestmark = pytest.mark.gpu


def late(torch, values):
    """A device tensor whose values arrive some 20 ms after this returns, NaN until then."""
    t = torch.full(values.shape, float("nan"), dtype=values.dtype, device="cuda")
    torch.cuda.synchronize()
    torch.cuda._sleep(40_000_000)
    t.copy_(values)
    return t


def test_pairs_wait_for_the_default_stream(gpu_ctx):
    import torch
    wl = workloads.plate_q4(20, 3, edges="fixed", name="plate_q4_20_inputs")
    ls = learned.LearnedSolver(gpu_ctx, wl, seed=3)
    rng = np.random.default_rng(1)
    free = wl.cons_mask == 0
    xs = torch.from_numpy(rng.standard_normal((3, wl.n_dof)) * free).cuda()
    F = torch.from_numpy(np.stack([wl.F] * 3).astype(np.float32)).cuda()
    zero = torch.zeros_like(xs)
    out = [torch.zeros_like(F) for _ in range(4)]
    torch.cuda.synchronize()
    ls.learned.make_pairs(3, F.data_ptr(), xs.data_ptr(), zero.data_ptr(), out[0].data_ptr(), out[1].data_ptr())
    x2 = late(torch, xs)
    ls.learned.make_pairs(3, F.data_ptr(), x2.data_ptr(), zero.data_ptr(), out[2].data_ptr(), out[3].data_ptr())
    assert torch.equal(out[0], out[2]) and torch.equal(out[1], out[3])
    want = ls.learned.loss(3, out[0].data_ptr(), out[1].data_ptr())
    r2 = late(torch, out[0])
    got = ls.learned.loss(3, r2.data_ptr(), out[1].data_ptr())
    ls.close()
    assert np.all(np.isfinite(want)) and np.allclose(got, want, rtol=1e-6, atol=0)  # the loss's sums by atomics
