"""FP64 tangent of the reference's laws by sum factorisation (csrc/sumfac.cu)
against the direct contraction (IGAPGPU_LAW_PRECOMPUTE=0: the law inside the
element kernel): the smallest lattice, uneven sizes, rational weights and
distorted elements, both laws; 27 points keep the direct form."""
import numpy as np
import pytest

import igap4_gb300 as ig

pytestmark = pytest.mark.gpu


# 1e-13: 64 x 100 products of each pair in 53 bits, and the two forms of the law (1e-13 apart in their own test)
@pytest.mark.parametrize("law", [ig.LAW_GRADELAST, ig.LAW_GRADELASTTIME])
@pytest.mark.parametrize("nelem,perturb,weights,nquad", [((2, 2, 2), False, False, 4), ((5, 3, 4), True, True, 4),
                                                         ((3, 9, 2), True, False, 4), ((4, 2, 3), False, True, 3)])
def test_matches_direct_form(monkeypatch, law, nelem, perturb, weights, nquad):
    bct, neu = ig.clamp_bc((0,), traction_face=1, traction=(0.0, 0.0, -1e-3))
    knots, w, X = ig.beam_mesh(nelem, (4.0, 1.0, 1.0), perturb=perturb)
    rng = np.random.default_rng(3)
    if weights:
        w = rng.uniform(0.8, 1.25, w.size)
    par = list(ig.LAW_DEFAULT_PAR[law])
    if law == ig.LAW_GRADELASTTIME:
        par[5], par[6] = 1.3, 0.7  # inertia and damping: the value slots' term
    out = []
    for flag in ("1", "0"):
        monkeypatch.setenv("IGAPGPU_LAW_PRECOMPUTE", flag)
        A = ig.Assembly(nelem, knots, w, X, law=law, par=par, bc_type=bct, neumann=neu, nquad=nquad)
        r = np.random.default_rng(4)
        for lvl in range(A.torder + 1):
            A.set_history(lvl, r.uniform(-2e-2, 2e-2, A.ndof))
        RR, K = np.zeros(A.ndof), np.zeros(A.nnz)
        A.assemble(None, RR, K)
        np.testing.assert_array_equal(A.tangent(), A.tangent())  # deterministic
        np.testing.assert_array_equal(A.residual(), A.residual())
        out.append((RR, K))
        A.close()
    for a, b in zip(*out):
        assert np.linalg.norm(a - b) <= 1e-13 * np.linalg.norm(b)
        assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()
