"""GPU: the tcgen05 BF16 update's tile edges: panels that end between two
64- or 128-row blocks, a last tile of two rows or columns, block sizes whose k
chunks end inside a chunk of 16, and enough tiles that each CTA goes round its
four accumulators.

A three-term update carries 24 bits of each operand, as FP32 does, so the
bound on the reconstruction is that of an FP32 factorization: n u32 times the
growth of the factors, 5e-5 on these matrices (u32 = 6e-8, n <= 1026; growth
below 1); the pivots are the FP64 factorization's, whose decisions on uniform
random entries are further apart than that."""
import numpy as np
import pytest

from common import reconstruct, relative_error, uniform_symmetric

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,b", [(130, 64), (258, 100), (386, 33), (514, 127), (1026, 65)])
def test_tile_edges(cuda, bbk, n, b):
    import torch
    a = uniform_symmetric(n, 7 * n + b)
    f = torch.from_numpy(a).to(cuda)
    perm, pt, _ = bbk.factor_device(f, b, mode="bf16x3")
    g = torch.from_numpy(a).to(cuda)
    perm64, pt64, _ = bbk.factor_device(g, b, mode="fp64")
    assert torch.equal(pt, pt64) and torch.equal(perm, perm64)
    fh = f.cpu().numpy()
    assert relative_error(reconstruct(fh, perm.cpu().numpy(), pt.cpu().numpy()), a) < 5e-5
    # the strict lower triangle is nobody's
    assert np.array_equal(np.tril(fh, -1), np.tril(a, -1))


def test_accumulators_in_turn(cuda, bbk):
    """990 tiles in the first update, six or seven per CTA; the solution's
    error is the update's, against the FP64 factors' solution."""
    import torch
    n, b = 5700, 64
    a = torch.from_numpy(uniform_symmetric(n, 5)).to(cuda)
    rhs = torch.from_numpy(np.random.default_rng(2).standard_normal((1, n))).to(cuda)
    f = a.clone()
    perm, pt, _ = bbk.factor_device(f, b, mode="bf16x3")
    x = bbk.solve_device(f, perm, pt, rhs.clone())
    r = rhs - x @ a
    be = float(r.abs().max() / (a.abs().sum(1).max() * x.abs().max() + rhs.abs().max()))
    assert be < 1e-5, be
