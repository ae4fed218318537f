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
