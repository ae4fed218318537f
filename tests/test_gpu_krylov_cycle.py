"""GMRES restart cycles in one cooperative kernel (csrc/krylov_cycle.cu):
fixed numbers of iterations against GMRES(m) with modified Gram-Schmidt in
numpy on the same matrix, at restarts and iteration limits that end inside,
at and after a cycle, and against the launch-by-launch path (restarts above
the kernel's limit of 200)."""
import numpy as np
import pytest

import igap4_gb300 as ig

pytestmark = pytest.mark.gpu
sp = pytest.importorskip("scipy.sparse")


def system(nelem, seed=0):
    bct, neu = ig.clamp_bc((0,), traction_face=1, traction=(0.0, 0.0, -1e-3))
    knots, w, X = ig.beam_mesh(nelem, (4.0, 1.0, 1.0))
    A = ig.Assembly(nelem, knots, w, X, law=ig.LAW_LINGRAD, bc_type=bct, neumann=neu)
    U = A.impose_dirichlet(np.random.default_rng(seed).uniform(-1e-2, 1e-2, A.ndof))
    b = -A.residual(U.copy())
    vals = A.tangent(U.copy())
    A.tangent_internal(U.copy())
    rowptr, cols = A.pattern()
    return A, sp.csr_matrix((vals, cols, rowptr), shape=(A.ndof, A.ndof)), b


def preconditioner(K, nelem, pc):
    if pc == 0:
        return lambda v: v
    if pc == 1:
        d = K.diagonal()
        return lambda v: v / d
    nb = [n + 2 for n in nelem]
    groups = {}
    for cp in range(K.shape[0] // 3):
        i = (cp // (nb[1] * nb[2]), (cp // nb[2]) % nb[1], cp % nb[2])
        groups.setdefault(cp if pc == 2 else tuple(v // 2 for v in i), []).extend(3 * cp + e for e in range(3))
    inv = [(g, np.linalg.inv(K[g][:, g].toarray())) for g in groups.values()]

    def apply(v):
        z = np.empty_like(v)
        for g, B in inv:
            z[g] = B @ v[g]
        return z

    return apply


def gmres(K, b, M, m, max_it):
    x, its = np.zeros_like(b), 0
    while its < max_it:
        r = b - K @ x
        beta = np.linalg.norm(r)
        V, Z, steps = [r / beta], [], min(m, max_it - its)
        H = np.zeros((steps + 1, steps))
        for j in range(steps):
            Z.append(M(V[j]))
            w = K @ Z[j]
            for i in range(j + 1):
                H[i, j] = V[i] @ w
                w = w - H[i, j] * V[i]
            H[j + 1, j] = np.linalg.norm(w)
            V.append(w / H[j + 1, j])
        e = np.zeros(steps + 1)
        e[0] = beta
        x = x + np.linalg.lstsq(H, e, rcond=None)[0] @ np.array(Z)
        its += steps
    return x, np.linalg.norm(b - K @ x)


# 1e-9: condition number (up to 1e5) x 1e-16 x 60 iterations, plus what the
# reference's own iterate moves by when the right-hand side changes in its last
# bit (without a preconditioner the iterate of an unconverged cycle is that
# sensitive: 2e-5 at 2x2x2 after 30 steps), in the iterate and its residual norm
@pytest.mark.parametrize("nelem,m,max_it,pc", [
    ((2, 2, 2), 1, 3, 1), ((2, 2, 2), 30, 30, 0), ((5, 3, 4), 7, 20, 1), ((5, 3, 4), 33, 33, 2),
    ((9, 2, 3), 32, 40, 3), ((16, 4, 4), 60, 60, 1), ((23, 5, 4), 200, 37, 3)])
def test_cycle_matches_numpy(nelem, m, max_it, pc):
    A, K, b = system(nelem)
    x = np.zeros(A.ndof)
    its, rn = A.ksp_solve(b, x, ksp_restart=m, ksp_max_it=max_it, ksp_rtol=1e-30, pc=pc)
    xr, rr = gmres(K, b, preconditioner(K, nelem, pc), m, max_it)
    assert its == max_it
    # the reference's own spread over last-bit changes of the matrix and the right-hand side
    rng = np.random.default_rng(1)
    dx = dr = 0.0
    for _ in range(16):
        Kp = K.copy()
        Kp.data *= 1.0 + 2.0 ** -52 * rng.standard_normal(K.nnz)
        xm, rm = gmres(Kp, b * (1.0 + 2.0 ** -52 * rng.standard_normal(A.ndof)), preconditioner(K, nelem, pc), m, max_it)
        dx, dr = max(dx, np.linalg.norm(xm - xr)), max(dr, abs(rm - rr))
    assert np.linalg.norm(x - xr) <= 1e-9 * np.linalg.norm(xr) + 4.0 * dx
    assert abs(rn - rr) <= 1e-8 * rr + np.linalg.norm(K @ (x - xr)) + 4.0 * dr


@pytest.mark.parametrize("pc,orth", [(0, 0), (1, 0), (1, 1), (2, 1), (3, 0), (3, 1), (4, 1)])
def test_cycle_and_separate_launches_agree(pc, orth):
    """Newton solves with the cycle kernel (restart 200) and with the separate
    kernels (201): same iteration counts, solutions within the linear tolerance."""
    res = []
    for m in (200, 201):
        A, _, _ = system((7, 3, 3))
        U = np.zeros(A.ndof)
        st = A.solve(U, snes_abstol=1e-12, ksp_rtol=1e-12, ksp_restart=m, pc=pc, orth=orth)
        res.append((U, st))
    (U0, s0), (U1, s1) = res
    assert s0["converged"] == 1 and s1["converged"] == 1, (s0, s1)
    assert s0["newton_its"] == s1["newton_its"]
    assert abs(s0["ksp_its_total"] - s1["ksp_its_total"]) <= 2
    assert np.linalg.norm(U0 - U1) <= 1e-8 * np.linalg.norm(U1)


def test_zero_and_converged_starts():
    A, K, b = system((4, 3, 2))
    x = np.zeros(A.ndof)
    its, rn = A.ksp_solve(np.zeros(A.ndof), x)  # zero right-hand side: no step
    assert its == 0 and rn == 0.0 and not x.any()
    x[:] = 1.0
    its, rn = A.ksp_solve(b, x, ksp_max_it=0)
    assert its == 0 and abs(rn - np.linalg.norm(b - K @ np.ones(A.ndof))) <= 1e-12 * rn
    assert (x == 1.0).all()
