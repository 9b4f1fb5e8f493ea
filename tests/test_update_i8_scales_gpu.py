"""GPU: the digit update where the entries of an operand row differ in scale.
A row's digits are fixed-point, so entries of C whose products are all far
below their row's and column's largest have to come from the FP64 tensor
cores: every entry of A is to be reproduced to a few units of its own
|L| |D| |L^T|, as in the reference's order, not of the largest one's."""
import numpy as np
import pytest

from common import uniform_symmetric

pytestmark = pytest.mark.gpu


def _residual_by_entry(a, f, perm, pt, rows):
    """max over rows `rows` (positions) of |P A P^T - L D L^T| / (|L| |D| |L^T|)."""
    n = a.shape[0]
    two = np.where(pt == 2)[0]
    lt = np.triu(f, 1)
    lt[two, two + 1] = 0.0
    lt[np.diag_indices(n)] = 1.0
    l = lt[:, rows].T
    d, off = np.diag(f), f[two, two + 1]

    def product(l, lt, d, off):
        ld = l * d
        ld[:, two] += l[:, two + 1] * off
        ld[:, two + 1] += l[:, two] * off
        return ld @ lt

    wide = [v.astype(np.longdouble) for v in (l, lt, d, off)]
    r = np.abs(a[np.ix_(perm[rows], perm)] - product(*wide))
    size = product(*(np.abs(v) for v in (l, lt, d, off)))  # (in double: it needs no more)
    assert not r[size == 0.0].any()
    return float((r[size > 0.0] / size[size > 0.0]).max())


def _factor(bbk, cuda, a, b, mode):
    import torch
    f = torch.from_numpy(a).to(cuda)
    perm, pt, _ = bbk.factor_device(f, b, mode=mode)
    return f, perm, pt


def _two_sets(n, scale):
    # two index sets, of size `scale` and 1, coupled by entries of size 1
    a = uniform_symmetric(n, 21) + np.diag(np.random.default_rng(1).uniform(2.0, 4.0, n))
    big = np.random.default_rng(2).random(n) < 0.5
    return np.where(np.outer(big, big), scale, 1.0) * a


def _few_rows(n, scale):
    # three rows that all but one of the first panel's pivots hardly touch
    a = uniform_symmetric(n, 22)
    a[:300, :300] += 40.0 * np.eye(300)  # these stay the first pivots
    for x in (900, 1500, 2200):
        a[x, :300] /= scale
        a[x, 7] = 1.0
        a[:300, x] = a[x, :300]
    return a


def _flat(n, scale):
    # pivots that do not couple, then rows of entries close to the largest that
    # the leading digit holds, all of one sign: the digits' sums are at their largest
    rng = np.random.default_rng(23)
    a = uniform_symmetric(n, 23)
    h = 1000
    a[:h, :h] = np.diag(np.full(h, 10.0))
    a[:h, h:] = rng.uniform(0.9925, 0.9955, (h, n - h))
    a[h:, :h] = a[:h, h:].T
    a[h:, h:] += a[h:, :h] @ a[:h, h:] / 10.0  # (what the update takes off again)
    return a


@pytest.mark.parametrize("kind,scale,n,b", [
    ("flat", 1.0, 2100, 1000), ("flat", 1.0, 2200, 500),
    ("two", 1.0, 2304, 256), ("two", 1e2, 2304, 256), ("two", 1e4, 2304, 256), ("two", 1e6, 2304, 256),
    ("two", 1e10, 2304, 256), ("two", 1e5, 2450, 305), ("two", 1e6, 3000, 600), ("two", 1e6, 2200, 1000),
    ("two", 1e6, 8300, 64), ("few", 1e4, 2304, 256), ("few", 1e8, 2304, 256),
])
def test_every_entry_is_as_accurate_as_in_the_references_order(cuda, bbk, kind, scale, n, b):
    a = {"two": _two_sets, "few": _few_rows, "flat": _flat}[kind](n, scale)
    got = []
    for mode in ("fp64", "fp64_ordered"):
        f, perm, pt = (t.cpu().numpy() for t in _factor(bbk, cuda, a, b, mode))
        rows = np.random.default_rng(3).choice(n, 24 if n < 4000 else 4, replace=False)
        if kind == "few":
            rows[:3] = np.flatnonzero(np.isin(perm, (900, 1500, 2200)))
        got.append(_residual_by_entry(a, f, perm, pt, rows))
    # units of 2^-53: the reference's order leaves 1.3 to 3.4, the FP64 tensor
    # cores up to 5.4 (the panel's reassociated sums); an entry in digits is
    # off by at most 16, a bound that rounding errors of either sign stay far below
    assert got[0] <= max(2.0 * got[1], 8 * 2.0 ** -53), got


@pytest.mark.parametrize("power", [0, 4, 8, 12, 16])
def test_scaled_solution_where_large_rows_couple_to_half_of_a_panel(cuda, bbk, power):
    # A = D M D, M well conditioned; 60 rows of scale 10^power; the second half
    # of the first panel's pivots couples neither to them nor to the first half
    import torch
    n, b = 2304, 256
    m = uniform_symmetric(n, 31) * (6.0 / np.sqrt(n)) + 14.0 * np.eye(n)
    m[128:256, :128] = m[:128, 128:256] = 0.0
    m[128:256, n - 60:] = m[n - 60:, 128:256] = 0.0
    d = np.ones(n)
    d[n - 60:] = 10.0 ** power
    a = m * d[:, None] * d[None, :]
    y = np.random.default_rng(5).uniform(0.5, 1.0, n)
    rhs = ((m.astype(np.longdouble) @ y) * d).astype(np.float64)
    err = []
    for mode in ("fp64", "fp64_ordered"):
        f, perm, pt = _factor(bbk, cuda, a, b, mode)
        x = bbk.solve_device(f, perm, pt, torch.from_numpy(rhs[None, :].copy()).to(cuda)).cpu().numpy()[0]
        err.append(float(np.abs(x * d - y).max()))
    assert err[0] <= 4.0 * err[1], err
