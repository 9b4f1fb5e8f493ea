"""GPU: the error of the solve's sums over many columns.  Beyond 32 right-hand
sides the backward sweep keeps the sums of sixteen blocks apart, so the mean
backward error stays near that of sums taken block by block; around the edges
of that window (16 and 17 blocks of 64, the last one short) and of the count (32,
33) nothing else changes."""
import numpy as np
import pytest

from common import backward_error, uniform_symmetric

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


def test_mean_backward_error_of_many_right_hand_sides(cuda, bbk):
    import torch
    n = 5000
    g = torch.Generator(device=cuda)
    g.manual_seed(1)
    a = torch.empty(n, n, dtype=torch.float64, device=cuda).uniform_(-1.0, 1.0, generator=g)
    a = torch.triu(a) + torch.triu(a, 1).T
    f = a.clone()
    perm, pt, _ = bbk.factor_device(f, 128)
    b = torch.randn(64, n, generator=g, dtype=torch.float64, device=cuda)
    x = bbk.solve_device(f, perm, pt, b.clone())
    r = (b - x @ a).abs().amax(1) / (a.abs().sum(1).max() * x.abs().amax(1) + b.abs().amax(1))
    # block by block 1.00e-15, one running sum 1.37e-15 (the mean's own spread is 2 %)
    assert float(r.mean()) < 1.15e-15


@pytest.mark.parametrize("n", [1000, 1024, 1025, 1088, 1089, 2049, 2111])
@pytest.mark.parametrize("nrhs", [32, 33, 40])
def test_windows_of_the_backward_sweep(cuda, bbk, n, nrhs):
    import torch
    a = uniform_symmetric(n, n)
    rhs = np.random.default_rng(n + nrhs).standard_normal((nrhs, n))
    f = torch.from_numpy(a).to(cuda)
    perm, pt, _ = bbk.factor_device(f, 64)
    x = bbk.solve_device(f, perm, pt, torch.from_numpy(rhs).to(cuda)).cpu().numpy()
    assert backward_error(a, x.T, rhs.T) < 20 * n * EPS
    one = bbk.solve_device(f, perm, pt, torch.from_numpy(rhs[-1:].copy()).to(cuda)).cpu().numpy()
    assert np.abs(one[0] - x[-1]).max() <= 1e-9 * np.abs(one).max()  # (sums apart: other roundings)
