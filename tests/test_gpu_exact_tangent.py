"""FP64 tangent of the linear law from exact BF16 slices (csrc/tc_exact.cu)
against the CPU oracle: the sizes of the smallest lattice, fewer and more
elements than SMs, partial chunks (27 points), length scales that put the
gradient or the Hessian rows in front, rational weights, distorted elements."""
import numpy as np
import pytest

import igap4_gb300 as ig
import pyoracle as po

pytestmark = pytest.mark.gpu


def both(monkeypatch, nelem, par, nquad=4, perturb=False, weights=False, seed=0):
    bct, neu = ig.clamp_bc((0,), traction_face=1, traction=(0.0, 0.0, -1e-3))
    knots, w, X = ig.beam_mesh(nelem, (4.0, 1.0, 1.0), perturb=perturb)
    if weights:
        w = np.random.default_rng(seed).uniform(0.8, 1.25, w.size)
    out = []
    for flag in ("1", "0"):
        monkeypatch.setenv("IGAPGPU_TC_EXACT", flag)
        A = ig.Assembly(nelem, knots, w, X, law=ig.LAW_LINGRAD, par=par, bc_type=bct, neumann=neu, nquad=nquad)
        U = np.random.default_rng(seed).uniform(-1e-2, 1e-2, A.ndof)
        K = A.tangent(U)
        np.testing.assert_array_equal(A.tangent(U), K)  # deterministic
        out.append(K)
        A.close()
    return out


# 4e-15: both sides round 64 x 36 products a pair in 53 bits
@pytest.mark.parametrize("nelem,par,nquad,perturb,weights", [
    ((2, 2, 2), [1.0, 1.0, 0.1], 4, False, False),
    ((5, 3, 4), [0.7, 1.9, 0.02], 4, True, True),
    ((7, 6, 5), [1.3, 0.5, 0.5], 3, False, True),
    ((19, 4, 4), [1.0, 0.4, 10.0], 4, True, False),
    ((3, 2, 2), [2.0, 1.0, 0.1], 2, False, False),
    ((3, 2, 2), [2.0, 1.0, 0.1], 5, False, False)])
def test_matches_fp64_kernel(monkeypatch, nelem, par, nquad, perturb, weights):
    K, Kf = both(monkeypatch, nelem, par, nquad, perturb, weights)
    assert np.linalg.norm(K - Kf) <= 4e-15 * np.linalg.norm(Kf)
    assert np.abs(K - Kf).max() <= 4e-15 * np.abs(Kf).max()
    assert np.array_equal(K, Kf) == (nquad == 5)  # more than 64 points keep the FP64 kernel


def test_matches_oracle():
    bct, neu = po.clamp_bc((0,), 1, (0.0, 0.0, -1e-3))
    prob = po.Problem(nelem=(9, 5, 4), L=(4.0, 1.0, 1.0), law=po.LAW_LINGRAD, bc_type=bct, neumann=neu, perturb=True)
    U = po.random_state(prob, 2)
    knots, w, X = ig.beam_mesh(prob.nelem, prob.L, perturb=True)
    A = ig.Assembly(prob.nelem, knots, w, X, law=prob.law, par=prob.params(), bc_type=bct, neumann=neu)
    A.set_state(U)
    Ko = po.OracleCase(prob).tangent(U)
    assert np.linalg.norm(A.tangent() - Ko) <= 1e-14 * np.linalg.norm(Ko)


# 496 elements: three or four per SM; 1, 4 and 8 chunks (fewer than, as many as
# and more than the copy stages).  Tolerance as above.
@pytest.mark.parametrize("nquad", [2, 3, 4])
def test_several_elements_per_block(monkeypatch, nquad):
    K, Kf = both(monkeypatch, (31, 4, 4), [0.9, 1.2, 0.1], nquad, True, True)
    assert np.linalg.norm(K - Kf) <= 4e-15 * np.linalg.norm(Kf)
    assert np.abs(K - Kf).max() <= 4e-15 * np.abs(Kf).max()
