"""Time slices, resumed solves, step caps, traces, sparse warps and latency
lanes for every kernel form (one system per lane, one lane per bubble, padded
and exact, two lanes per bubble), in one batch with backfill grids.  Every
output equals that of one uninterrupted solve bit for bit."""
import numpy as np
import pytest

from cbc_b200 import scenes
from cbc_b200.ensemble import Ensemble, WorkList, make_work_list

pytestmark = pytest.mark.gpu

# bubbles per system: (systems, span); two or more blocks of each, so that a
# start share below one leaves a backfill grid
BATCH = {1: (700, 0.6), 8: (70, 0.2), 11: (41, 0.06), 16: (41, 0.06), 20: (13, 0.04), 32: (13, 0.04)}
KEYS = ("state", "t", "h", "event", "status", "steps", "rejected", "conv_ok", "conv_fail", "lin_iters",
        "dense_index", "dense_time", "dense_state")


def batch():
    parts = [scenes.uniform(K, ns=ns, periods=span, seed=300 + K, pa_hi=1.2, x_range=(-0.5, 0.5))
             for K, (ns, span) in BATCH.items()]
    return Ensemble.from_scene(scenes.concat(*parts), ndo=3).to_device()


def compare(a, b, keys=KEYS):
    for k in keys:
        x, y = a[k], b[k]
        same = (x == y) | (np.isnan(x) & np.isnan(y)) if x.dtype.kind == "f" else (x == y)
        assert np.all(same), f"{k}: {np.count_nonzero(~same)} mismatches"


@pytest.fixture(scope="module")
def single(cuda):
    """One uninterrupted solve, to the end and to 30 steps."""
    import torch
    out = {}
    for cap in (100_000, 30):
        e = batch()
        e.solve(cap)
        torch.cuda.synchronize()
        out[cap] = e.to_host()
    return out


@pytest.mark.parametrize("cap", [100_000, 30])
def test_slices_until_done_equal_one_solve(single, cap):
    """The first slices are over before any block starts."""
    import torch
    e = batch()
    e.enable_trace()
    wl = make_work_list(e.host["K"], e.host["t_end"] - e.host["t"])
    assert wl.share is not None and np.all(wl.share < 1.0)
    calls = 0
    for budget in [1] * 4 + [20_000] + [200_000] * 2000:
        e.solve(cap, work=wl, budget_ns=budget, steps_total=True)
        calls += 1
        st, steps = e.dev["status"].cpu().numpy(), e.dev["steps"].cpu().numpy()
        if not np.any(((st == 0) | (st == -1)) & (steps < cap)):
            break
    torch.cuda.synchronize()
    assert calls > 6
    got = e.to_host()
    assert np.all(got["steps"] <= cap)
    compare(got, single[cap])
    assert np.all(got["trace_load_ns"] > 0) and np.all(got["trace_done_ns"] >= got["trace_load_ns"])


@pytest.mark.parametrize("slots", ["one", "half"])
def test_sparse_warps_equal_one_solve(single, slots):
    import torch
    e = batch()
    wl = make_work_list(e.host["K"], e.host["t_end"])
    wl.slots = np.asarray([1 if slots == "one" else max(1, 16 // int(k)) for k in wl.bucket_K], np.int32)
    e.solve(100_000, work=wl)
    torch.cuda.synchronize()
    compare(e.to_host(), single[100_000])


@pytest.mark.parametrize("budget_ns", [0, 400_000])
def test_latency_lanes_of_every_form_equal_one_solve(single, budget_ns):
    """Two exclusive SMs per bubble count, the rest in ordinary buckets."""
    import torch
    e = batch()
    K = e.host["K"]
    order, bk, ex = [], [], []
    for k in sorted(BATCH):
        ids = np.nonzero(K == k)[0].astype(np.int32)
        n = max(5, ids.size // 3)
        order += [ids[:n], ids[n:]]
        bk += [k, k]
        ex += [2, 0]
    wl = WorkList(order=np.concatenate(order), bucket_K=np.asarray(bk, np.int32),
                  bucket_begin=np.concatenate([[0], np.cumsum([o.size for o in order])]).astype(np.int32),
                  exclusive=np.asarray(ex, np.int32))
    for _ in range(2000):
        e.solve(100_000, work=wl, budget_ns=budget_ns, steps_total=True)
        st = e.dev["status"].cpu().numpy()
        if not np.any((st == 0) | (st == -1)):
            break
    torch.cuda.synchronize()
    compare(e.to_host(), single[100_000])
