"""Device memory that the FP64 assembly takes for itself: how much, and when."""
import numpy as np
import pytest

import igap4_gb300 as ig

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

MB = 1 << 20


def beam(nelem, law=ig.LAW_LINGRAD):
    bct, neu = ig.clamp_bc((0,), traction_face=1, traction=(0.0, 0.0, -1e-3))
    knots, w, X = ig.beam_mesh(nelem, (4.0, 1.0, 1.0))
    return ig.Assembly(nelem, knots, w, X, law=law, bc_type=bct, neumann=neu)


def free_bytes():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_residual_alone_takes_no_element_matrices():
    A = beam((32, 8, 8))
    nel = 32 * 8 * 8
    slices = nel * (8 * 33792 + 256 * 8 + 88 * 2)
    U = np.zeros(A.ndof)
    f0 = free_bytes()
    A.residual(U)
    f1 = free_bytes()
    assert slices - 4 * MB <= f0 - f1 <= slices + 81 * 8 * nel + 8 * MB
    out = torch.zeros(A.nnz, dtype=torch.float64, device="cuda")
    f1 = free_bytes()
    A.tangent(torch.zeros(A.ndof, dtype=torch.float64, device="cuda"), out)
    f2 = free_bytes()
    assert 378 * 9 * 8 * nel - 4 * MB <= f1 - f2 <= 378 * 9 * 8 * nel + 8 * MB


def leave_free(nbytes):
    """a tensor that leaves about nbytes of device memory"""
    torch.cuda.empty_cache()
    try:
        return torch.empty(free_bytes() - nbytes, dtype=torch.uint8, device="cuda")
    except torch.OutOfMemoryError:
        pytest.skip("the free memory is not available in one piece")


def test_caches_take_at_most_a_quarter(monkeypatch):
    nelem = (64, 16, 16)  # 4.5 GB of slices
    U = np.zeros(3 * 66 * 18 * 18)
    A, B = beam(nelem), beam(nelem)
    hold = leave_free(12 << 30)
    f0 = free_bytes()
    R = A.residual(U)
    assert f0 - free_bytes() < 1 << 30  # the residual buffer only
    del hold
    torch.cuda.empty_cache()
    monkeypatch.setenv("IGAPGPU_TC_EXACT", "0")
    np.testing.assert_array_equal(B.residual(U), R)


def test_caches_make_room_for_the_krylov_basis():
    A = beam((32, 8, 8))
    U = np.random.default_rng(0).uniform(-1e-2, 1e-2, A.ndof)
    K = A.tangent(U)  # 0.56 GB of slices, 56 MB of element matrices
    A.tangent_internal(U)
    b, x = np.ones(A.ndof), np.zeros(A.ndof)
    hold = leave_free(300 * MB)
    its, rn = A.ksp_solve(b, x, ksp_restart=4000, ksp_max_it=2, ksp_rtol=1e-30)  # 0.65 GB
    assert its == 2 and np.isfinite(rn)
    assert np.linalg.norm(A.tangent(U) - K) <= 4e-15 * np.linalg.norm(K)  # through the scatter
    del hold
    torch.cuda.empty_cache()


def test_refused_allocation_and_solve_afterwards():
    A = beam((16, 4, 4))
    U = np.zeros(A.ndof)
    st = A.solve(U)  # graphs hold the caches' addresses
    assert st["converged"] == 1
    A.tangent_internal(U)
    f0 = free_bytes()
    with pytest.raises(ig.IgapGpuError, match="does not fit"):
        A.ksp_solve(np.ones(A.ndof), np.zeros(A.ndof), ksp_restart=20_000_000)
    assert free_bytes() - f0 > -400 * MB
    V = np.zeros(A.ndof)
    st2 = A.solve(V)
    assert st2["converged"] == 1 and st2["newton_its"] == st["newton_its"]
    assert np.linalg.norm(U - V) <= 1e-9 * np.linalg.norm(U)


def test_a_callers_graph_keeps_the_caches():
    A = beam((16, 4, 4))
    U = torch.tensor(np.random.default_rng(0).uniform(-1e-2, 1e-2, A.ndof), device="cuda")
    R, K = U.new_zeros(A.ndof), U.new_zeros(A.nnz)
    torch.cuda.synchronize()
    A.assemble(U, R, K)
    A.synchronize()
    want = R.clone(), K.clone()
    A.tangent_internal(U)
    s = torch.cuda.Stream()
    A.set_stream(s.cuda_stream)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        A.assemble(U, R, K)
    with pytest.raises(ig.IgapGpuError, match="does not fit"):
        A.ksp_solve(torch.ones_like(U), torch.zeros_like(U), ksp_restart=20_000_000)
    R.zero_()
    K.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(R, want[0]) and torch.equal(K, want[1])


def test_caches_make_room_for_another_precision():
    A = beam((32, 8, 8))
    U = np.random.default_rng(0).uniform(-1e-2, 1e-2, A.ndof)
    K = A.tangent(U)
    hold = leave_free((4 << 30) + 200 * MB)
    A.set_precision(ig.PREC_OZAKI)  # 0.37 GB of slices of its own, beside 4 GB
    Kq = A.tangent(U)
    del hold
    torch.cuda.empty_cache()
    err = np.linalg.norm(Kq - K) / np.linalg.norm(K)
    assert 1e-14 < err < 1e-9  # from the BF16 slices, not from the FP64 kernel
