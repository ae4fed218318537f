"""igapgpu_set_neumann is complete on return: an assembly on a stream set
afterwards sees the new load, also when the old stream was busy."""
import numpy as np
import pytest

import igap4_gb300 as ig

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("porder", [2, 3])
def test_neumann_before_a_stream_change(porder):
    bct, neu = ig.clamp_bc((0,), traction_face=1, traction=(0.0, 0.0, -1e-3))
    knots, w, X = ig.beam_mesh((5, 4, 3), (4.0, 1.0, 1.0), porder=porder)
    A = ig.Assembly((5, 4, 3), knots, w, X, law=ig.LAW_LINGRAD, bc_type=bct, neumann=neu, porder=porder)
    U = torch.zeros(A.ndof, dtype=torch.float64, device="cuda")
    R, want = torch.zeros_like(U), torch.zeros_like(U)
    torch.cuda.synchronize()
    A.residual(U, R)  # one-time set-up
    A.synchronize()
    table = neu.copy()
    table[6 + 2] = -7e-3
    busy, other = torch.cuda.Stream(), torch.cuda.Stream()
    A.set_stream(busy.cuda_stream)
    with torch.cuda.stream(busy):
        torch.cuda._sleep(100_000_000)  # about 50 ms
    A.set_neumann(table)
    A.set_stream(other.cuda_stream)
    A.residual(U, R)
    torch.cuda.synchronize()
    A.residual(U, want)
    A.synchronize()
    assert torch.equal(R, want) and want.norm() > 0
