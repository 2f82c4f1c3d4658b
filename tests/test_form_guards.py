"""Every kernel form at arguments where the fast elementary functions give other
bits than the general ones, against the CPU oracle bit for bit: phases past the
range in no system and in some, radii, positions and denominators past the
range in some systems of a batch."""
import numpy as np
import pytest

from cbc_b200 import scenes
from cbc_b200.ensemble import Ensemble

from _parity import assert_bit_exact, run_pair
from test_parity_ensemble import compare, oracle_ragged

FORMS = [1, 2, 3, 4, 5, 6, 7, 8, 9, 11, 16, 17, 24, 32]
FIELDS = [("SW_A", 2), ("SW_N", 2), ("CONST", 3)]
TWO_OVER_PI = float.fromhex("0x1.45f306dc9c883p-1")
MAGIC = 1.5 * 2.0 ** 52


def quadrants(x):
    """Quadrant of a phase in the fast form (low bits of the rounded sum) and in
    the general one (rounded product)."""
    v = np.asarray(x) * TWO_OVER_PI
    return (v + MAGIC).view(np.int64) & 3, np.rint(v).astype(np.int64) & 3


def scene(K, ac, nk, ns, marked, periods):
    sc = scenes.uniform(K, ns=ns, periods=periods, seed=500 + 7 * K + nk, pa_hi=1.2, ac=ac, x_range=(-0.5, 0.5))
    pick = [0, 1, 0][:nk]
    sc.PA, sc.FR, sc.PS = sc.PA[pick].copy(), sc.FR[pick].copy(), sc.PS[pick].copy()
    if marked:
        far = 3e16 + 64.0 * np.arange(4096)                     # times pi
        fast, general = quadrants(far * np.pi)
        far = far[fast != general]
        assert far.size > ns
        sc.PS[-1, 1::3] = far[:sc.PS[-1, 1::3].size]
    return sc


def test_marked_phases_differ_between_the_forms():
    """The phases as the kernels get them."""
    for K in (1, 16):
        sc = scene(K, "SW_A", 2, 9, True, 0.1)
        e = Ensemble.from_scene(sc)
        ph = e.host["control_params"][1::3, 5]
        fast, general = quadrants(ph)
        assert np.mean(fast != general) > 0.5
        inside = e.host["control_params"][0::3, 5]
        fast, general = quadrants(inside)
        assert np.all(fast == general)


@pytest.mark.gpu
@pytest.mark.parametrize("marked", [False, True])
@pytest.mark.parametrize("ac,nk", FIELDS)
@pytest.mark.parametrize("K", FORMS)
def test_phases_reference_layout(cuda, K, ac, nk, marked):
    sc = scene(K, ac, nk, 2 * (32 // K) + 1, marked, 0.02 if K > 8 else 0.1)
    gpu, ref = run_pair(sc, max_steps=120, kernel_steps=60)
    assert_bit_exact(gpu, ref)


@pytest.mark.gpu
@pytest.mark.parametrize("K", FORMS)
def test_states_outside(cuda, K):
    """Finite states past the guards in one system of four, so that warps hold
    them beside systems within the range.  (Positions: past 2^32, with phases below
    2^63, where the quadrant of the general sincos is defined.)"""
    import torch
    cap = 40
    outside = [(0, 2.0 ** -400), (0, 2.0 ** 400), (0, 2.0 ** -66), (0, 2.0 ** 66), (1, 2.0 ** 50), (1, -2.0 ** 33),
               (2, 1.0e308), (2, -1.0e200), (0, -1.0)]
    sc = scene(K, "SW_A", 2, 4 * len(outside) + 1, False, 0.2)
    ens, models = Ensemble.from_scene(sc, return_models=True)
    (sel, model), = models.values()
    assert np.array_equal(sel, np.arange(sc.ns))
    for i, (c, v) in enumerate(outside):
        s, bubble = 4 * i + 1, i % K
        ens.host["state"][ens.host["bubble_offset"][s] + bubble, c] = v
        model.runtime.host_buffers.state.actual_state[c, s, bubble] = v
    ens.to_device()
    ens.solve(cap)
    torch.cuda.synchronize()
    got, ref = ens.to_host(), oracle_ragged(models, ens.host, cap, ens.solver_spec)
    compare(got, ref)
    assert np.all(got["steps"][0::4] > 10)
