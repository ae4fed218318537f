"""Error words of the kernels with bounded waits: a failure that one kernel
left behind does not spoil the next assembly, and the FP64 tensor-core
kernel's failure is reported once, also by a solve that rejects its initial
iterate.  The words are preset from the host; no wait runs out."""
import numpy as np
import pytest

import igap4_gb300 as ig

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def beam():
    bct, neu = ig.clamp_bc((0,), traction_face=1, traction=(0.0, 0.0, -1e-3))
    knots, w, X = ig.beam_mesh((5, 4, 3), (4.0, 1.0, 1.0))
    A = ig.Assembly((5, 4, 3), knots, w, X, law=ig.LAW_LINGRAD, bc_type=bct, neumann=neu)
    U = A.impose_dirichlet(np.random.default_rng(0).uniform(-1e-2, 1e-2, A.ndof))
    return A, U


def on_device(A, U):
    """residual and tangent through device pointers, without a synchronisation by the library"""
    Ud = torch.tensor(U, device="cuda")
    R, K = Ud.new_zeros(A.ndof), Ud.new_zeros(A.nnz)
    torch.cuda.synchronize()
    A.assemble(Ud, R, K)
    torch.cuda.synchronize()
    return R.cpu().numpy(), K.cpu().numpy()


def test_stale_word_does_not_spoil_the_next_assembly():
    A, U = beam()
    R0, K0 = on_device(A, U)
    A.debug_set_error(2)
    R, K = on_device(A, U)
    np.testing.assert_array_equal(R, R0)
    np.testing.assert_array_equal(K, K0)


def test_failure_is_reported_once():
    A, U = beam()
    on_device(A, U)
    A.synchronize()
    A.debug_set_error(2)
    on_device(A, U)  # a later launch does not clear it
    A.set_precision(ig.PREC_SPLIT)
    on_device(A, U)  # nor does another kernel's
    with pytest.raises(ig.IgapGpuError, match="wait expired"):
        A.synchronize()
    A.synchronize()
    A.set_precision(ig.PREC_FP64)
    assert np.isfinite(A.tangent(U)).all()


@pytest.mark.parametrize("graphs", [0, 1])
def test_rejecting_solve_reports_it(graphs):
    A, U = beam()
    on_device(A, U)
    A.synchronize()
    st = A.solve(U.copy(), snes_f0_max=1e-30, use_graphs=graphs)
    assert st["converged"] == 0 and st["newton_its"] == 0
    A.debug_set_error(2)
    with pytest.raises(ig.IgapGpuError, match="wait expired"):
        A.solve(U.copy(), snes_f0_max=1e-30, use_graphs=graphs)
    A.solve(U.copy(), snes_f0_max=1e-30, use_graphs=graphs)


def test_batch_reports_it():
    inst = ig.batch_instances(3, nx=(4, 6), nyz=(2, 3))
    A = ig.BatchAssembly(inst)
    U = np.random.default_rng(0).uniform(-1e-2, 1e-2, A.ndof)
    R0 = A.residual(U)
    A.debug_set_error(2)
    with pytest.raises(ig.IgapGpuError, match="wait expired"):
        A.residual(U)
    np.testing.assert_array_equal(A.residual(U), R0)
