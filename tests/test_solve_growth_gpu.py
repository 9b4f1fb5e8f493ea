"""GPU: the solve where the inverses of the triangle's diagonal blocks grow.
Bunch-Kaufman does not bound L, so such blocks have to be substituted through:
every right-hand side's backward error stays that of substitution in FP64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


def _triangle(kind, n):
    rng = np.random.default_rng(n)
    if kind == "couplings":  # 2x2 pivots, one of them across every block boundary
        l = np.tril(rng.uniform(-1.5, 1.5, (n, n)), -1) * 10.0 ** rng.integers(-3, 1, (n, 1))
    elif kind == "bidiagonal":
        l = np.diag(np.full(n - 1, -1.3), -1)
    elif kind == "columns":  # a few large columns: growth in step with the triangle's own
        l = np.tril(rng.uniform(-0.1, 0.1, (n, n)), -1)
        l[:, ::19] *= 500.0
        l = np.tril(l, -1)
    else:
        l = np.tril(np.full((n, n), float(kind)), -1)
        k = np.arange(n)
        l[np.abs(k[:, None] - k[None, :]) > 40] = 0.0  # (growth within blocks, not over all of n)
    return l + np.eye(n)


def _errors(l, d, x, b):
    wide = np.longdouble
    r = l.astype(wide) @ (d.astype(wide) @ (l.T.astype(wide) @ x.astype(wide))) - b
    a = l @ d @ l.T
    return np.abs(r).max(0) / (np.abs(a).sum(1).max() * np.abs(x).max(0) + np.abs(b).max(0))


def _substituted(l, d, b):
    n = l.shape[0]
    x = b.copy()
    for k in range(n):
        x[k + 1:] -= l[k + 1:, k:k + 1] * x[k]
    x = np.linalg.solve(d, x)
    for k in range(n - 1, 0, -1):
        x[:k] -= l[k, :k][:, None] * x[k]
    return x


@pytest.mark.parametrize("kind", ["-0.1", "-0.12", "-0.15", "-0.3", "-0.5", "-1", "0.7", "bidiagonal", "columns",
                                  "couplings"])
@pytest.mark.parametrize("n", [32, 64, 75, 200])
def test_backward_error_is_substitutions(cuda, bbk, kind, n):
    import torch
    rng = np.random.default_rng(1)
    l = _triangle(kind, n)
    d, pt = np.diag(rng.choice([-1.0, 1.0], n) * rng.uniform(1.0, 2.0, n)), np.ones(n, np.int32)
    if kind == "couplings":
        for k in range(3, n - 1, 10):  # 63 among them
            d[k, k + 1] = d[k + 1, k] = 3.0
            l[k + 1, k] = 0.0
            pt[k], pt[k + 1] = 2, -2
    f = np.triu(l.T, 1) + np.triu(d)
    x = 10.0 ** rng.uniform(-6.0, 0.0, (n, 20)) * rng.choice([-1.0, 1.0], (n, 20))
    b = np.hstack([rng.standard_normal((n, 20)), l @ (d @ (l.T @ x)), l @ rng.standard_normal((n, 20))])
    got = bbk.solve_device(torch.from_numpy(f).to(cuda), torch.arange(n, dtype=torch.int32, device=cuda),
                           torch.from_numpy(pt).to(cuda), torch.from_numpy(b.T.copy()).to(cuda)).cpu().numpy().T
    assert np.isfinite(got).all()
    want = _errors(l, d, _substituted(l, d, b), b).reshape(3, 20).max(1)
    # a few roundings apart: fused products, another order of sums
    assert (_errors(l, d, got, b).reshape(3, 20).max(1) <= 4.0 * want + 4.0 * EPS).all()
