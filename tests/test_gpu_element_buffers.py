"""The colour-by-colour scatter, which runs where the element buffers have no
room (IGAPGPU_ELEMENT_BUFFERS=0), against the buffers and their gather: the
same bits from the same element kernel, with Dirichlet rows and sizes that the
colours do not divide, for every law, in FP64 and in the split mode."""
import numpy as np
import pytest

import igap4_gb300 as ig

pytestmark = pytest.mark.gpu


def assembled(monkeypatch, buffers, nelem, law, prec, env):
    monkeypatch.setenv("IGAPGPU_ELEMENT_BUFFERS", buffers)
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    bct, neu = ig.clamp_bc((0, 3), traction_face=1, traction=(0.0, 0.0, -1e-3))
    knots, w, X = ig.beam_mesh(nelem, (4.0, 1.0, 1.0), perturb=True)
    w = np.random.default_rng(2).uniform(0.8, 1.25, w.size)
    A = ig.Assembly(nelem, knots, w, X, law=law, bc_type=bct, neumann=neu)
    A.set_precision(prec)
    r = np.random.default_rng(4)
    for lvl in range(A.torder + 1):
        A.set_history(lvl, r.uniform(-2e-2, 2e-2, A.ndof))
    RR, K = np.zeros(A.ndof), np.zeros(A.nnz)
    A.assemble(None, RR, K)
    out = A.residual(), A.tangent(), RR, K
    A.close()
    return out


LAWS = [ig.LAW_LINGRAD, ig.LAW_GRADELAST, ig.LAW_GRADELASTTIME]


@pytest.mark.parametrize("law", LAWS)
@pytest.mark.parametrize("nelem", [(2, 2, 2), (5, 3, 4), (7, 2, 3)])
def test_same_bits_fp64(monkeypatch, law, nelem):
    env = {"IGAPGPU_TC_EXACT": "0", "IGAPGPU_LAW_PRECOMPUTE": "0"}  # the element kernel on both sides
    for a, b in zip(*(assembled(monkeypatch, f, nelem, law, ig.PREC_FP64, env) for f in "10")):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("law", LAWS[1:])
def test_same_bits_split(monkeypatch, law):
    got, want = (assembled(monkeypatch, f, (5, 3, 4), law, ig.PREC_SPLIT, {}) for f in "10")
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)


# 1e-13: 64 x 100 products of each pair in 53 bits, as between the library's other routes
@pytest.mark.parametrize("law", LAWS)
@pytest.mark.parametrize("prec", [ig.PREC_FP64, ig.PREC_OZAKI])
def test_default_routes_agree(monkeypatch, law, prec):
    got, want = (assembled(monkeypatch, f, (7, 2, 3), law, prec, {}) for f in "10")
    for a, b in zip(got, want):
        assert np.linalg.norm(a - b) <= 1e-13 * np.linalg.norm(b)
