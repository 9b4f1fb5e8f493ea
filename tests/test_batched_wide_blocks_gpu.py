"""GPU: batched orders whose block is cut to what shared memory held when the
blocks were bounded, and takes a little more as it is laid out now: 245 to 251
(blocks 49 and 50) and 629 to 638 (block 18).  They run in every mode and with
a workspace for one CTA per SM, with the planned block."""
import ctypes

import numpy as np
import pytest

from common import backward_error, uniform_symmetric

pytestmark = pytest.mark.gpu
SIZES = [245, 246, 247, 251, 629, 633, 638]


@pytest.mark.parametrize("mode,small", [("fp64_ordered", False), ("fp32", False), ("fp64", False), ("fp64", True)])
def test_blocks_cut_to_shared_memory(cuda, bbk, port, mode, small):
    import torch
    plan = bbk.BatchedPlan(SIZES, block_sizes=[64] * 6)
    assert [int(b) for b in plan.block_sizes] == [50, 50, 49, 49, 18, 18, 18]
    if small:  # scratch for one CTA per SM
        sms, moved, n = torch.cuda.get_device_properties(0).multi_processor_count, 132, max(SIZES)
        stride = -(-(2 * moved * n + 3 * n + 2 * moved * 66 + moved) // 32) * 32
        plan.bytes -= sms * stride * ctypes.sizeof(ctypes.c_double)
    mats = [uniform_symmetric(n, n) for n in SIZES]
    rhs = [np.random.default_rng(n).standard_normal(n) for n in SIZES]
    a, x = plan.pack(mats, rhs)
    refine = {"a_orig": a.clone(), "tol": 1e-14, "max_iter": 30} if mode == "fp32" else {}
    perm, pt, _ = bbk.batched_factor_solve(plan, a, x, mode=mode, **refine)
    for k, m in enumerate(mats):
        n = SIZES[k]
        if mode != "fp32":
            want = port.factor(m, int(plan.block_sizes[k]))
            assert np.array_equal(plan.vector(pt.cpu().numpy(), k), want.pivot_types), n
            assert np.array_equal(plan.vector(perm.cpu().numpy(), k), want.perm), n
            if mode == "fp64_ordered":
                f = np.triu(plan.matrix(a.cpu().numpy(), k))
                assert np.array_equal(f, np.triu(want.factors)), n
        assert backward_error(m, plan.vector(x.cpu().numpy(), k), rhs[k]) < 20 * n * 2.0 ** -52, n
