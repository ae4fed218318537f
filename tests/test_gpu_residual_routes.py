"""The linear law's FP64 residual alone with one to three Gauss points per
direction: the quadrature loop (slower through the element matrices), so the
bits of the kernel without them; beside the tangent and with 64 points from
the element matrices."""
import numpy as np
import pytest

import igap4_gb300 as ig

pytestmark = pytest.mark.gpu


def single(nquad):
    bct, neu = ig.clamp_bc((0,), traction_face=1, traction=(0.0, 0.0, -1e-3))
    knots, w, X = ig.beam_mesh((7, 3, 4), (4.0, 1.0, 1.0), perturb=True)
    return ig.Assembly((7, 3, 4), knots, w, X, law=ig.LAW_LINGRAD, bc_type=bct, neumann=neu, nquad=nquad)


def batch(nquad):
    return ig.BatchAssembly(ig.batch_instances(3, nx=(4, 7), nyz=(2, 4)), nquad=nquad)


# 4e-15: both sides round 64 x 36 products a pair in 53 bits
@pytest.mark.parametrize("make", [single, batch])
@pytest.mark.parametrize("nquad", [1, 2, 3, 4])
def test_residual_alone(monkeypatch, make, nquad):
    out = []
    for flag in ("1", "0"):
        monkeypatch.setenv("IGAPGPU_TC_EXACT", flag)
        A = make(nquad)
        U = np.random.default_rng(0).uniform(-1e-2, 1e-2, A.ndof)
        R = A.residual(U)
        RR, K = np.zeros(A.ndof), np.zeros(A.nnz)
        A.assemble(U, RR, K)
        np.testing.assert_array_equal(A.residual(U), R)  # whatever ran in between
        out.append((R, RR))
        A.close()
    (R, RR), (Rq, RRq) = out
    assert np.array_equal(R, Rq) == (nquad < 4)
    assert np.linalg.norm(R - Rq) <= 4e-15 * np.linalg.norm(Rq)
    assert np.linalg.norm(RR - RRq) <= 4e-15 * np.linalg.norm(RRq)
