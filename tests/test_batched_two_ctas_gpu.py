"""GPU: batches with two CTAs per SM.  In the FP64 mode items whose W and U
take more than half of an SM's shared memory are factored without keeping U
(with wide blocks, test_batched_wide_blocks_gpu.py, in a panel that may be
narrower than planned): same pivots as the oracle's,
backward error below 20 n eps.  A workspace of the size that one CTA per SM
needs is still accepted."""
import ctypes

import numpy as np
import pytest

from common import backward_error, kkt_matrix, uniform_symmetric

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


def _run(bbk, sizes, block_sizes=None, mode="fp64", bytes_of=None):
    plan = bbk.BatchedPlan(sizes, block_sizes=block_sizes)
    if bytes_of is not None:
        plan.bytes = bytes_of(plan)
    mats = [kkt_matrix(n, max(1, (3 * n) // 4), n + k) if k % 2 else uniform_symmetric(n, n + k)
            for k, n in enumerate(sizes)]
    rhs = [np.random.default_rng(k).standard_normal(n) for k, n in enumerate(sizes)]
    a, x = plan.pack(mats, rhs)
    perm, pt, _ = bbk.batched_factor_solve(plan, a, x, mode=mode)
    return plan, mats, rhs, a.cpu().numpy(), x.cpu().numpy(), perm.cpu().numpy(), pt.cpu().numpy()


def _check(port, plan, mats, rhs, x, perm, pt):
    for k, m in enumerate(mats):
        want = port.factor(m, int(plan.block_sizes[k]))
        assert np.array_equal(plan.vector(pt, k), want.pivot_types), (k, m.shape)
        assert np.array_equal(plan.vector(perm, k), want.perm), (k, m.shape)
        assert backward_error(m, plan.vector(x, k), rhs[k]) < 20 * m.shape[0] * EPS, (k, m.shape)


@pytest.mark.parametrize("sizes,blocks", [
    ([195, 196, 197, 255, 256], None),                  # around half the shared memory, one slot per thread
    ([257, 300, 383, 500, 511, 512], None),             # two
    ([513, 700, 1023, 1024, 16, 33], None),             # four
    ([256, 128, 96, 64, 65, 1], [64] * 6),              # wide blocks
    ([512, 256, 31], [32, 64, 48, 48, 24, 12]),         # the tuned table
])
def test_two_ctas_per_sm_pivot_like_the_oracle(cuda, bbk, port, sizes, blocks):
    plan, mats, rhs, a, x, perm, pt = _run(bbk, sizes, blocks)
    _check(port, plan, mats, rhs, x, perm, pt)


@pytest.mark.parametrize("sizes", [
    [16 + k % 25 for k in range(300)],             # two CTAs per SM finish sooner
    [256, 200, 192] + [16] * 200,                  # the largest would hold the others up
])
def test_one_or_two_ctas_per_sm_give_the_same_bits(cuda, bbk, sizes):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count

    def one(plan):
        moved, n = 132, max(sizes)
        stride = -(-(2 * moved * n + 3 * n + 2 * moved * 66 + moved) // 32) * 32
        return plan.bytes - sms * stride * ctypes.sizeof(ctypes.c_double)

    got, want = _run(bbk, sizes), _run(bbk, sizes, bytes_of=one)
    for g, w in zip(got[3:], want[3:]):
        assert np.array_equal(g, w)


def test_workspace_for_one_cta_per_sm_is_still_accepted(cuda, bbk, port):
    import torch
    sizes = [512, 300, 64, 17]
    sms = torch.cuda.get_device_properties(0).multi_processor_count

    def one(plan):
        moved, n = 132, max(sizes)
        stride = -(-(2 * moved * n + 3 * n + 2 * moved * 66 + moved) // 32) * 32
        return plan.bytes - sms * stride * ctypes.sizeof(ctypes.c_double)

    plan, mats, rhs, a, x, perm, pt = _run(bbk, sizes, bytes_of=one)
    _check(port, plan, mats, rhs, x, perm, pt)
    with pytest.raises(bbk.BbkError):
        _run(bbk, sizes, bytes_of=lambda p: one(p) - 8)
