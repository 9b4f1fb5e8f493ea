"""GPU: the FP64 trailing update on the integer tensor cores (order times
block at least 2^19, even leading dimension).  The factors must have the
oracle's pivots and a residual no larger than twice its own (both are a few
n eps / 10; the digit sums round less than FP64 ones), whatever the scale of
the matrix, and entries that the digits cannot hold must give what the FP64
tensor cores give."""
import numpy as np
import pytest

from common import kkt_matrix, uniform_symmetric

pytestmark = pytest.mark.gpu


def _factor(bbk, cuda, a, b, mode="fp64", pad=0):
    import torch
    n = a.shape[0]
    buf = torch.zeros(n, n + pad, dtype=torch.float64, device=cuda)
    buf[:, :n] = torch.from_numpy(a).to(cuda)
    f = buf[:, :n]
    perm, pt, ends = bbk.factor_device(f, b, mode=mode)
    return f, perm, pt, ends


def _residual(bbk, a, f, perm, pt):
    r = bbk.reconstruct_device(f, perm, pt).cpu().numpy()
    return np.linalg.norm(r - a) / np.linalg.norm(a)


def _scaled(a, spread, seed):
    s = 10.0 ** np.random.default_rng(seed).uniform(-spread, spread, a.shape[0])
    return a * s[:, None] * s[None, :]


@pytest.mark.parametrize("n,b,pad,kind", [
    (2306, 256, 0, "random"),   # one panel above the line, a tile column of two
    (2432, 255, 0, "random"),   # odd width: k padded inside a chunk
    (2559, 257, 1, "random"),   # odd order, even leading dimension, k in nine chunks
    (1664, 512, 2, "kkt"),
    (2100, 900, 0, "random"),   # a wide panel: k = 900
    (2200, 1000, 0, "random"),  # nearly the widest, k = 1000
    (4400, 130, 0, "kkt"),
    (2306, 256, 0, "scaled3"),  # rows and columns spread over 10^+-3, 10^+-30
    (2306, 256, 0, "scaled30"),
])
def test_digit_update_has_the_oracles_pivots_and_residual(cuda, bbk, port, n, b, pad, kind):
    a = kkt_matrix(n, int(0.75 * n), 7) if kind == "kkt" else uniform_symmetric(n, 11)
    if kind.startswith("scaled"):
        a = _scaled(a, float(kind[6:]), 3)
    want = port.factor(a, b)
    launches = [bbk.kernel_launch_count()]
    f, perm, pt, ends = _factor(bbk, cuda, a, b, pad=pad)
    launches.append(bbk.kernel_launch_count())
    assert np.array_equal(pt.cpu().numpy(), want.pivot_types)
    assert np.array_equal(perm.cpu().numpy(), want.perm)
    assert np.array_equal(ends.cpu().numpy(), want.panel_end)
    fo, po, to, _ = _factor(bbk, cuda, a, b, mode="fp64_ordered", pad=pad)
    launches.append(bbk.kernel_launch_count())
    # the digit kernels ran: four launches more for each panel above the line
    above = [m for m in range(n - b + 1, b, -b) if m >= 1024 and m * b >= 1 << 19]
    assert above and launches[1] - launches[0] == launches[2] - launches[1] + 4 * len(above)
    assert _residual(bbk, a, f, perm, pt) <= 2.0 * _residual(bbk, a, fo, po, to)


def test_scales_the_digits_cannot_hold_go_to_the_fp64_kernel(cuda, bbk):
    # a power of two beyond the digit kernel's range (2^400) scales every FP64
    # result exactly; the pivot tests square the entries, so it stays below 2^510
    n, b, k = 2306, 256, 440
    a = uniform_symmetric(n, 5)
    f1, perm1, pt1, _ = _factor(bbk, cuda, a, b)
    f2, perm2, pt2, _ = _factor(bbk, cuda, np.ldexp(a, k), b)
    assert np.array_equal(pt1.cpu().numpy(), pt2.cpu().numpy())
    assert np.array_equal(perm1.cpu().numpy(), perm2.cpu().numpy())
    r1 = _residual(bbk, a, f1, perm1, pt1)
    fd = f2.clone()  # undo the scale on D
    d = fd.diagonal()
    d.mul_(2.0 ** -k)
    first = np.flatnonzero(pt2.cpu().numpy() == 2)
    fd[first, first + 1] *= 2.0 ** -k
    assert _residual(bbk, a, fd, perm2, pt2) <= 4.0 * r1


@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_entries_that_are_not_finite_stay_where_fp64_puts_them(cuda, bbk, port, value):
    n, b = 2306, 256
    a = uniform_symmetric(n, 9)
    a[n - 1, n - 3] = a[n - 3, n - 1] = value  # in the last panels: the updates before it carry it
    a[5, n - 2] = a[n - 2, 5] = value          # in the first panel's rows
    want = port.factor(a, b)
    f, perm, pt, _ = _factor(bbk, cuda, a, b)
    got = np.triu(f.cpu().numpy())
    assert np.array_equal(perm.cpu().numpy(), want.perm)
    assert np.array_equal(pt.cpu().numpy(), want.pivot_types)
    assert np.array_equal(np.isfinite(got), np.isfinite(np.triu(want.factors)))
