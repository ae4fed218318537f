"""FP64 residual of the linear law from the element matrices (csrc/tc_exact.cu)
against the quadrature kernel: smooth, affine, bending and translated states,
alone and beside the tangent, rational weights, several elements per block and
partial chunks; and the context whose digits leave the exactness bound, which
keeps the quadrature kernel and its bits."""
import numpy as np
import pytest

import igap4_gb300 as ig

pytestmark = pytest.mark.gpu


def state(kind, X, rng):
    x, y, z = X.reshape(-1, 3).T
    if kind == "random":
        U = rng.uniform(-1e-2, 1e-2, (x.size, 3))
    elif kind == "affine":
        U = 1e-2 * np.stack([0.3 * x + 0.1 * y, 0.2 * z - 0.4 * y, 0.5 * x + 0.7 * z], -1)
    elif kind == "bending":
        U = 1e-2 * np.stack([-2.0 * x * (z - 0.5), 0.0 * x, x * x], -1)
    else:
        U = 1e-2 * np.stack([np.sin(x), np.cos(2.0 * y + x), np.sin(z * x)], -1)
    return U.reshape(-1)


def make(monkeypatch, flag, nelem, par=(1.0, 1.0, 0.1), nquad=4, perturb=False, weights=False, clamp=True):
    monkeypatch.setenv("IGAPGPU_TC_EXACT", flag)
    bct, neu = ig.clamp_bc((0,), traction_face=1, traction=(0.0, 0.0, -1e-3)) if clamp else (None, None)
    knots, w, X = ig.beam_mesh(nelem, (4.0, 1.0, 1.0), perturb=perturb)
    if weights:
        w = np.random.default_rng(5).uniform(0.8, 1.25, w.size)
    return ig.Assembly(nelem, knots, w, X, law=ig.LAW_LINGRAD, par=list(par), bc_type=bct, neumann=neu, nquad=nquad), X


# 2e-14: the quadrature loop itself is off by up to 3e-15 on bending states at
# these length scales, most of it from the geometry's cancellation between the
# 64 points; twice that for the two sides, and a factor of three for rational weights
@pytest.mark.parametrize("kind", ["random", "affine", "bending", "smooth"])
@pytest.mark.parametrize("nelem,nquad,perturb,weights", [
    ((2, 2, 2), 4, False, False), ((5, 3, 4), 4, True, True), ((31, 4, 4), 4, True, True), ((31, 4, 4), 3, False, True),
    ((31, 4, 4), 2, True, False)])
def test_matches_quadrature(monkeypatch, kind, nelem, nquad, perturb, weights):
    out = []
    for flag in ("1", "0"):
        A, X = make(monkeypatch, flag, nelem, nquad=nquad, perturb=perturb, weights=weights)
        U = state(kind, X, np.random.default_rng(0))
        RR, K = np.zeros(A.ndof), np.zeros(A.nnz)
        A.assemble(U, RR, K)
        out.append((A.residual(U), RR))
        A.close()
    for a, b in zip(*out):
        assert np.linalg.norm(a - b) <= 2e-14 * np.linalg.norm(b)


def test_translations_drop_out(monkeypatch):
    """Displacements that are multiples of 2^-40, so that adding 5 is exact: the
    same bits (the quadrature loop's residual moves by about 2e-13)."""
    A, X = make(monkeypatch, "1", (9, 4, 5), perturb=True, clamp=False)
    U = np.round(state("random", X, np.random.default_rng(0)) * 0.1 * 2.0 ** 40) / 2.0 ** 40
    np.testing.assert_array_equal(A.residual(U + 5.0), A.residual(U))


def both_routes(monkeypatch, nelem, ell):
    out = []
    for flag in ("1", "0"):
        A, X = make(monkeypatch, flag, nelem, par=(1.0, 1.0, ell))
        U = state("random", X, np.random.default_rng(0))
        RR, K = np.zeros(A.ndof), np.zeros(A.nnz)
        A.assemble(U, RR, K)
        out.append((A.residual(U), A.tangent(U), RR, K))
        A.close()
    return zip(*out)


# regular meshes whose largest digit norms, taken together over an element's rows,
# exceed what sums exactly in FP32, and no pair of rows does: still the tensor-core
# route, with its accuracy (4e-15: both sides round 64 x 36 products a pair in 53 bits)
@pytest.mark.parametrize("nelem,ell", [((16, 4, 5), 0.1778), ((4, 4, 6), 0.1857), ((7, 6, 5), 0.1828),
                                       ((30, 3, 4), 0.1044), ((24, 13, 24), 0.1755)])
def test_bound_holds_entry_by_entry(monkeypatch, nelem, ell):
    for a, b in both_routes(monkeypatch, nelem, ell):
        assert not np.array_equal(a, b)
        assert np.linalg.norm(a - b) <= 4e-15 * np.linalg.norm(b)


def test_digits_beyond_the_bound_keep_the_quadrature_kernel(monkeypatch):
    """A mesh where a pair of rows does exceed it: the FP64 kernel and its bits."""
    for a, b in both_routes(monkeypatch, (20, 10, 3), 0.09793557511207801):
        np.testing.assert_array_equal(a, b)
