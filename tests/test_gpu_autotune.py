"""igapgpu_batch_autotune tunes what a whole assembly launches: entries of the
schedule that no launch reads stay as they were, and the FP64 time is that of
the kernel that runs."""
import numpy as np
import pytest

import igap4_gb300 as ig

pytestmark = pytest.mark.gpu

ODD = {"grab_fp64": 3, "ctas_per_sm_fp64": 1, "grab_tc": 5, "order": 1}  # none of the candidates' grabs


def tuned(prec, nquad, frac, law=ig.LAW_LINGRAD):
    B = ig.BatchAssembly(ig.batch_instances(4, nx=(8, 20), nyz=(3, 6)), law=law, nquad=nquad)
    B.set_precision(prec)
    U = np.random.default_rng(0).uniform(-1e-2, 1e-2, B.ndof)
    R0, K0 = B.residual(U), B.tangent(U)
    B.schedule = ODD
    best, t64, ttc = B.autotune(reps=1, frac=frac)
    assert best == B.schedule
    np.testing.assert_array_equal(B.residual(U), R0)
    np.testing.assert_array_equal(B.tangent(U), K0)
    return best, t64, ttc


@pytest.mark.parametrize("frac", [0.1, 1.0])
def test_exact_route_has_no_schedule(frac):
    best, t64, ttc = tuned(ig.PREC_FP64, 4, frac)
    assert best == ODD and t64 > 0 and ttc == 0


@pytest.mark.parametrize("frac", [0.1, 1.0])
def test_split_residual_has_no_schedule(frac):
    best, t64, ttc = tuned(ig.PREC_SPLIT, 4, frac)
    assert (best["grab_fp64"], best["ctas_per_sm_fp64"]) == (3, 1)
    assert best["grab_tc"] in (1, 2, 4, 8) and t64 > 0 and ttc > 0


@pytest.mark.parametrize("frac", [0.1, 1.0])
@pytest.mark.parametrize("nquad,law", [(3, ig.LAW_LINGRAD), (4, ig.LAW_GRADELAST)])
def test_queue_kernel_is_tuned(frac, nquad, law):
    best, t64, ttc = tuned(ig.PREC_FP64, nquad, frac, law)
    assert best["grab_fp64"] in (1, 2, 4, 8) and best["grab_tc"] == 5 and t64 > 0 and ttc == 0
