"""Systems outside the range of the fast elementary functions."""
import numpy as np
import pytest

from cbc_b200 import scenes
from cbc_b200.ensemble import Ensemble

pytestmark = pytest.mark.gpu

KEYS = ("state", "t", "h", "event", "status", "steps", "rejected", "conv_ok", "conv_fail", "lin_iters")


def timed(sc, cap):
    """Milliseconds of a solve of `cap` steps (best of five) and its results."""
    import torch
    e = Ensemble.from_scene(sc).to_device()
    e.solve(10)
    best = np.inf
    for _ in range(5):
        e.reset_device()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        a.record()
        e.solve(cap)
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b))
    return best, e.to_host()


@pytest.mark.parametrize("K", [1, 2, 4, 8])
def test_systems_outside_are_evaluated_once(cuda, K):
    """Phases past 2^50 in every system: an attempt is evaluated with the general
    functions alone.  Evaluated with both it would take at least twice as long as
    within the range, since the general functions are no faster than the fast ones;
    alone they take at most about 1.5 times as long."""
    ns, cap = {1: 20000, 2: 10000, 4: 4000, 8: 1200}[K], 300
    sc = scenes.uniform(K, ns=ns, periods=50.0, seed=400 + K, pa_hi=1.0)
    inside, _ = timed(sc, cap)
    sc.PS = sc.PS + 5e14          # times pi
    outside, _ = timed(sc, cap)
    assert outside < 1.9 * inside, f"K = {K}: {inside:.2f} ms inside, {outside:.2f} ms outside"


@pytest.mark.parametrize("K", [1, 2, 4, 8, 11, 16, 20])
def test_far_end_time_is_no_slower(cuda, K):
    """An end time of 1e30 with a step cap: the same results as a near one, bit
    for bit, at the same speed (the general functions take 1.1 to 1.3 times as
    long from K = 11 down; runs of one batch differ by about 1 %)."""
    ns = {1: 20000, 2: 10000, 4: 4000, 8: 1200, 11: 400, 16: 400, 20: 200}[K]
    sc = scenes.uniform(K, ns=ns, periods=50.0, seed=400 + K, pa_hi=1.0 if K <= 8 else 0.6,
                        x_range=(-0.25, 0.25) if K <= 8 else (-0.5, 0.5))
    near, a = timed(sc, 300)
    sc.t_end[:] = 1e30
    far, b = timed(sc, 300)
    for k in KEYS:
        x, y = a[k], b[k]
        same = (x == y) | (np.isnan(x) & np.isnan(y)) if x.dtype.kind == "f" else (x == y)
        assert np.all(same), f"{k}: {np.count_nonzero(~same)} mismatches"
    assert far < 1.05 * near, f"K = {K}: {near:.2f} ms near, {far:.2f} ms far"
