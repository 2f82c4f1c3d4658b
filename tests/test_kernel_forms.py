"""The kernel form chosen by the bubble count, against the CPU oracle bit for
bit, at the edges of each form's range: smallest, largest and odd bubble counts,
field types and harmonic counts with and without their own compiled right-hand
side, batches that do not fill the last warp, both entry points.

One system in three has a phase past the range of the fast elementary functions,
so its warp evaluates with the general ones; the results are the same.
No tolerance: every output equals the oracle's."""
import numpy as np
import pytest

from cbc_b200 import scenes
from cbc_b200.ensemble import Ensemble
from cbc_b200.models import SolverSpec

from _parity import assert_bit_exact, run_pair
from test_parity_ensemble import compare, oracle_ragged

pytestmark = pytest.mark.gpu

FORMS = [1, 2, 3, 4, 5, 6, 7, 8, 9, 11, 15, 16, 17, 24, 31, 32]
FIELDS = [("SW_A", 2), ("SW_N", 2), ("CONST", 2), ("SW_A", 1), ("SW_N", 3), ("SW_A", 4)]


def scene(K, ac, nk, ns, periods, samples_per_period=0):
    sc = scenes.uniform(K, ns=ns, periods=periods, seed=100 + 7 * K + nk, pa_hi=1.2, ac=ac,
                        samples_per_period=samples_per_period, x_range=(-0.5, 0.5))
    pick = [0, 1, 0, 1][:nk]
    sc.PA, sc.FR, sc.PS = sc.PA[pick].copy(), sc.FR[pick].copy(), sc.PS[pick].copy()
    sc.PS[-1, 1::3] = 5e14          # times pi: above 2^50
    return sc


@pytest.mark.parametrize("ac,nk", FIELDS)
@pytest.mark.parametrize("K", FORMS)
def test_form_reference_layout(cuda, K, ac, nk):
    sc = scene(K, ac, nk, ns=2 * (32 // K) + 1, periods=0.02 if K > 8 else 0.2)
    gpu, ref = run_pair(sc)
    assert_bit_exact(gpu, ref)


@pytest.mark.parametrize("ac,nk", [("SW_A", 2), ("CONST", 3)])
@pytest.mark.parametrize("K", FORMS)
def test_form_batched(cuda, K, ac, nk):
    """Refilled slots (more systems than one warp holds) and both dense modes."""
    import torch
    sc = scene(K, ac, nk, ns=3 * (32 // K) + 2, periods=0.04 if K > 8 else 0.2, samples_per_period=50)
    for mode in ("reference", "grid"):
        ens, models = Ensemble.from_scene(sc, return_models=True, solver_spec=SolverSpec(dense_mode=mode))
        ens.to_device()
        ens.solve(100_000)
        torch.cuda.synchronize()
        compare(ens.to_host(), oracle_ragged(models, ens.host, 100_000, ens.solver_spec))
