"""GPU: panels on one thread-block cluster (up to 3584 active columns).  In
the ordered mode the factors are the oracle's bit for bit, in the FP64 mode
the pivots are and the residual is within the reference's 1e-10; at the
orders where the cluster grows (64 columns per CTA), where the first panels
run on the grid and the last ones on a cluster, and with panels wider than a
cluster's shared memory takes."""
import os
import subprocess
import sys

import numpy as np
import pytest

from common import kkt_matrix, reconstruct, relative_error, uniform_symmetric

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CASES = [(1, 1), (2, 1), (3, 2), (64, 16), (65, 16), (66, 64), (129, 32), (257, 31), (513, 48), (1025, 64),
         (1300, 255),  # the first panel's rows do not fit a cluster
         (700, 350), (2049, 100)]


def _check(bbk, cuda, a, b, mode, want):
    import torch
    f = torch.from_numpy(a).to(cuda)
    perm, pt, ends = bbk.factor_device(f, b, mode=mode)
    assert np.array_equal(pt.cpu().numpy(), want.pivot_types)
    assert np.array_equal(perm.cpu().numpy(), want.perm)
    assert np.array_equal(ends.cpu().numpy(), want.panel_end)
    return np.triu(f.cpu().numpy()), perm.cpu().numpy(), pt.cpu().numpy()


@pytest.mark.parametrize("n,b", CASES)
@pytest.mark.parametrize("kind", ["random", "kkt"])
def test_cluster_panels_are_the_oracles(cuda, bbk, port, n, b, kind):
    a = kkt_matrix(n, max(1, (3 * n) // 4), n + b) if kind == "kkt" else uniform_symmetric(n, n + b)
    want = port.factor(a, b)
    f, _, _ = _check(bbk, cuda, a, b, "fp64_ordered", want)
    assert np.array_equal(f, np.triu(want.factors), equal_nan=True)
    f, perm, pt = _check(bbk, cuda, a, b, "fp64", want)
    if n <= 700:
        assert relative_error(reconstruct(f, perm, pt), a) < 1e-10


def test_grid_panels_then_cluster_panels(cuda, bbk, port):
    n, b = 3650, 64  # 3 584 columns are active at the second panel
    a = uniform_symmetric(n, 8)
    want = port.factor(a, b)
    f, _, _ = _check(bbk, cuda, a, b, "fp64_ordered", want)
    assert np.array_equal(f, np.triu(want.factors), equal_nan=True)
    _check(bbk, cuda, a, b, "fp64", want)


@pytest.mark.parametrize("value", [0.0, np.nan, np.inf])
def test_cluster_panels_with_degenerate_entries(cuda, bbk, port, value):
    n, b = 300, 32
    a = uniform_symmetric(n, 4)
    a[40:90, :] = a[:, 40:90] = 0.0  # zero rows: zero pivots
    a[10, 200] = a[200, 10] = value
    a[250, 250] = value
    want = port.factor(a, b)
    f, _, _ = _check(bbk, cuda, a, b, "fp64_ordered", want)
    assert np.array_equal(f, np.triu(want.factors), equal_nan=True)


def test_an_expired_wait_in_a_cluster_is_reported_and_the_context_survives(cuda, bbk):
    import torch
    for ctas in (1, 2, 8):  # a grid's and a cluster's exchange that can never complete
        assert bbk.probe_bounded_wait(ctas, 20_000_000) == bbk.BBK_ERR_TIMEOUT
    a = uniform_symmetric(900, 3)
    bbk.set_wait_timeout_ns(1)  # (whether a wait is this long is left to the device)
    try:
        try:
            bbk.factor_device(torch.from_numpy(a).to(cuda), 64)
        except bbk.BbkError as e:
            assert e.status == bbk.BBK_ERR_TIMEOUT
    finally:
        bbk.set_wait_timeout_ns(5_000_000_000)
    f = torch.from_numpy(a).to(cuda)
    perm, pt, _ = bbk.factor_device(f, 64)
    r = bbk.reconstruct_device(f, perm, pt).cpu().numpy()
    assert relative_error(r, a) < 1e-10


@pytest.mark.parametrize("slots", [97, 129, 288])
def test_many_slots_per_cta_split_the_rows(cuda, bbk, slots):
    # the grid panel's kernel for 97 to 288 slots per CTA at full width, its rows
    # split between shared and global memory (block 256 beyond 90 slots or so):
    # a permutation and the solution's backward error
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = slots * sms
    g = torch.Generator(device=cuda)
    g.manual_seed(slots)
    a = torch.empty(n, n, dtype=torch.float64, device=cuda).uniform_(-1.0, 1.0, generator=g)
    a = torch.triu(a) + torch.triu(a, 1).T
    f = a.clone()
    perm, pt, ends = bbk.factor_device(f, 256)
    p = perm.cpu().numpy()
    assert np.array_equal(np.sort(p), np.arange(n))
    b = torch.randn(2, n, dtype=torch.float64, device=cuda, generator=g)
    x = bbk.solve_device(f, perm, pt, b.clone())
    r = (b.T - a @ x.T).abs().amax(0)
    berr = r / (a.abs().sum(1).amax() * x.T.abs().amax(0) + b.T.abs().amax(0))
    assert float(berr.max()) < 1e-13


SLOTS = """
import sys
import numpy as np
import torch
import blockedbunchkaufmanldlt_b200 as bbk
slots, b = int(sys.argv[1]), int(sys.argv[2])
n = slots * (-(-3700 // slots))  # beyond a cluster's columns at first
rng = np.random.default_rng(slots)
a = np.triu(rng.uniform(-1.0, 1.0, (n, n)))
a = torch.from_numpy(a + np.triu(a, 1).T).cuda()
out = []
for mode in ("fp64", "fp64_ordered"):
    f = a.clone()
    out.append((f,) + bbk.factor_device(f, b, mode=mode))
for k in (1, 2, 3):
    assert torch.equal(out[0][k], out[1][k]), ("perm", "pivot types", "panel ends")[k - 1]
u, w = (torch.triu(o[0]) for o in out)
assert float((u - w).norm() / w.norm()) < 1e-10
"""


@pytest.mark.parametrize("slots,b", [(96, 64), (97, 64), (224, 128), (257, 64), (288, 64), (288, 300), (289, 64)])
def test_slots_per_cta_pivot_as_the_ordered_mode(cuda, bbk, slots, b):
    # fewer CTAs, so that each has as many slots at an order where the pivots
    # can be compared: 96 and 97, 257 and 288 (nine chunks), 289 (one thread per
    # slot again), rows in shared and (block 300) in global memory
    env = {**os.environ, "BBK_PANEL_COLS": str(slots), "PYTHONPATH": ROOT}
    run = subprocess.run([sys.executable, "-c", SLOTS, str(slots), str(b)], env=env, capture_output=True, text=True,
                         timeout=300)
    assert run.returncode == 0, run.stderr[-2000:]
