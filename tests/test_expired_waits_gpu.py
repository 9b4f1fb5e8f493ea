"""GPU: wait limits so short that any kernel of a factorization may give up,
at any point.  Each call ends in success or BBK_ERR_TIMEOUT, with nothing of
it still running, and the next one with the usual limit gives the same bits as
the first."""
import numpy as np
import pytest

from common import uniform_symmetric

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["fp64", "bf16x3", "bf16"])
def test_short_wait_limits_leave_the_context_usable(cuda, bbk, mode):
    import torch
    a = torch.from_numpy(uniform_symmetric(2600, 17)).to(cuda)

    def factor():
        f = a.clone()
        perm, pt, _ = bbk.factor_device(f, 256, mode=mode)
        return f.triu().cpu().numpy(), perm.cpu().numpy(), pt.cpu().numpy()

    want = factor()
    for limit in (1, 300, 1000, 3000, 10_000, 30_000, 100_000):
        bbk.set_wait_timeout_ns(limit)
        try:
            got = factor()
        except bbk.BbkError as e:
            assert e.status == bbk.BBK_ERR_TIMEOUT
        else:
            for g, w in zip(got, want):
                assert np.array_equal(g, w)
        finally:
            bbk.set_wait_timeout_ns(5_000_000_000)
    for g, w in zip(factor(), want):
        assert np.array_equal(g, w)
