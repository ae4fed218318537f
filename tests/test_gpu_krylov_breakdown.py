"""GMRES that breaks down inside a cycle (the product of a unit vector
overflows in its norm) is an error and leaves the caller's x as it was."""
import numpy as np
import pytest

import igap4_gb300 as ig

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("restart", [1, 5, 200, 201])
def test_breakdown_leaves_x(restart):
    bct, neu = ig.clamp_bc((0,), traction_face=1, traction=(0.0, 0.0, -1e-3))
    knots, w, X = ig.beam_mesh((4, 3, 2), (4.0, 1.0, 1.0))
    A = ig.Assembly((4, 3, 2), knots, w, X, law=ig.LAW_LINGRAD, par=[1e170, 1e170, 0.1], bc_type=bct, neumann=neu)
    A.tangent_internal(np.zeros(A.ndof))
    b = torch.ones(A.ndof, dtype=torch.float64, device="cuda")
    x = torch.zeros_like(b)
    torch.cuda.synchronize()
    with pytest.raises(ig.IgapGpuError):
        A.ksp_solve(b, x, ksp_restart=restart, ksp_max_it=10, ksp_rtol=1e-12, pc=0)
    torch.cuda.synchronize()
    assert not x.any()
