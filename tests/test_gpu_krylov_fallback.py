"""Where the GMRES cycle kernel's grid cannot be resident at once, the separate
launches take the solve; a smaller grid gives the kernel's own result."""
import numpy as np
import pytest

import igap4_gb300 as ig

pytestmark = pytest.mark.gpu


def solves(monkeypatch, blocks):
    if blocks is None:
        monkeypatch.delenv("IGAPGPU_GMRES_CYCLE", raising=False)
    else:
        monkeypatch.setenv("IGAPGPU_GMRES_CYCLE", blocks)
    bct, neu = ig.clamp_bc((0,), traction_face=1, traction=(0.0, 0.0, -1e-3))
    knots, w, X = ig.beam_mesh((7, 3, 3), (4.0, 1.0, 1.0))
    A = ig.Assembly((7, 3, 3), knots, w, X, law=ig.LAW_LINGRAD, bc_type=bct, neumann=neu)
    out = []
    for graphs in (0, 1):
        U = np.zeros(A.ndof)
        st = A.solve(U, snes_abstol=1e-12, ksp_rtol=1e-12, ksp_restart=150, pc=1, use_graphs=graphs)
        assert st["converged"] == 1, st
        out.append((U, st["newton_its"], st["ksp_its_total"]))
    b, x = -A.residual(np.zeros(A.ndof)), np.zeros(A.ndof)
    A.tangent_internal(np.zeros(A.ndof))
    n0 = ig.launch_count()
    its, rn = A.ksp_solve(b, x, ksp_restart=150, ksp_rtol=1e-12, pc=1)
    return out + [(x, its, 0)], ig.launch_count() - n0


# tolerances as in the comparison of restarts 200 and 201
@pytest.mark.parametrize("blocks", ["0", "1", "10", "1000000"])
def test_other_grids_and_separate_launches(monkeypatch, blocks):
    ref, n_ref = solves(monkeypatch, None)
    got, n = solves(monkeypatch, blocks)
    for (U0, nit0, kit0), (U, nit, kit) in zip(ref, got):
        assert abs(nit0 - nit) <= 2 and abs(kit0 - kit) <= 2
        assert np.linalg.norm(U0 - U) <= 1e-8 * np.linalg.norm(U)
    assert n_ref < 20
    assert (n > 1000) == (blocks in ("0", "1000000"))


def test_short_restarts_of_large_systems(monkeypatch):
    """366 k rows in a batch: restarts below the line run as separate launches, the
    others as cycles, with the same residual norms."""
    torch = pytest.importorskip("torch")
    monkeypatch.setenv("IGAPGPU_GEOMETRY_CACHE", "0")
    A = ig.BatchAssembly(ig.batch_instances(24))
    assert A.ndof > 300_000
    U = torch.zeros(A.ndof, dtype=torch.float64, device="cuda")
    b = torch.zeros_like(U)
    torch.cuda.synchronize()
    A.residual(U, b)
    A.tangent_internal(U)
    A.synchronize()
    for m, cycle in ((5, False), (20, True)):
        got = []
        for blocks in (None, "152"):  # the rule, then the cycle kernel whatever it says
            monkeypatch.delenv("IGAPGPU_GMRES_CYCLE", raising=False)
            if blocks:
                monkeypatch.setenv("IGAPGPU_GMRES_CYCLE", blocks)
            x = torch.zeros_like(b)
            torch.cuda.synchronize()
            n0 = ig.launch_count()
            its, rn = A.ksp_solve(b, x, ksp_restart=m, ksp_max_it=m, ksp_rtol=1e-30, pc=1)
            got.append((ig.launch_count() - n0 < 12, rn))
            assert its == m
        assert got[0][0] == cycle and got[1][0]
        assert abs(got[0][1] - got[1][1]) <= 1e-9 * got[0][1]
