"""GPU: the solve's groups of eight right-hand sides (up to sixteen side by
side in a launch).  Each right-hand side's solution must not depend on how
many others are solved with it (a group's arithmetic is its own; above 16 blocks
of 64, calls of up to 32 and of more right-hand sides add in another order), its
backward error stays below 20 n eps, and an infinite entry of a right-hand
side reaches exactly the entries that substitution takes it to."""
import numpy as np
import pytest

from common import backward_error, kkt_matrix, uniform_symmetric

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("n", [1, 31, 33, 64, 65, 96, 97, 161, 700])
@pytest.mark.parametrize("nrhs", [1, 8, 9, 33, 128, 129])
def test_groups_solve_each_right_hand_side_alike(cuda, bbk, n, nrhs):
    import torch
    a = kkt_matrix(n, max(1, (3 * n) // 4), n) if n > 60 else uniform_symmetric(n, n) + 2.0 * np.eye(n)
    rhs = np.random.default_rng(n + nrhs).standard_normal((nrhs, n))
    f = torch.from_numpy(a).to(cuda)
    perm, pt, _ = bbk.factor_device(f, 32)
    x = bbk.solve_device(f, perm, pt, torch.from_numpy(rhs).to(cuda)).cpu().numpy()
    assert backward_error(a, x.T, rhs.T) < 20 * n * EPS
    for k in (0, nrhs // 2, nrhs - 1):
        one = bbk.solve_device(f, perm, pt, torch.from_numpy(rhs[k:k + 1].copy()).to(cuda)).cpu().numpy()
        assert np.array_equal(one[0], x[k]), k


def test_infinity_stays_where_substitution_takes_it(cuda, bbk):
    import torch
    n = 200  # block diagonal: 8 x 8 blocks, so L couples nothing across them
    a = np.zeros((n, n))
    for k in range(0, n, 8):
        a[k:k + 8, k:k + 8] = uniform_symmetric(8, k) + 20.0 * np.eye(8)  # diagonally dominant: no interchanges
    f = torch.from_numpy(a).to(cuda)
    perm, pt, _ = bbk.factor_device(f, 32)
    assert np.array_equal(perm.cpu().numpy(), np.arange(n))
    rhs = np.ones((1, n))
    rhs[0, 77] = np.inf
    x = bbk.solve_device(f, perm, pt, torch.from_numpy(rhs).to(cuda)).cpu().numpy()[0]
    # L's zeros times the infinity are NaN below it, in both sweeps all rows
    # above the first NaN fold zeros of L times it: what substitution gives
    ref = rhs[0].copy()
    L = np.eye(n) + np.triu(f.cpu().numpy(), 1).T
    d = np.diag(f.cpu().numpy())
    with np.errstate(invalid="ignore"):
        for k in range(n):
            ref[k + 1:] -= L[k + 1:, k] * ref[k]
        ref /= d
        for k in range(n - 1, -1, -1):
            ref[:k] -= L[k, :k] * ref[k]
    assert np.array_equal(np.isfinite(x), np.isfinite(ref))
