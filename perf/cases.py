"""Performance cases: the work a user of the library has it do, through its public entry points.

Kinds
  assembly  residual and/or CSR tangent of one lattice (Assembly.residual / .tangent / .assemble)
  batch     residual and tangent of many uneven beams at once (BatchAssembly.assemble)
  ksp       a budget of GMRES iterations on the assembled matrix (Assembly.ksp_solve)
  newton    a static Newton-Krylov solve from rest (Assembly.solve)
  step      one time step of the transient law (set_neumann, Assembly.solve)
  train     one training step of the Newton predictor (ConvNet.train_step)
  forward   one evaluation of the predictor's network (ConvNet.forward)

Meshes are the box beams of the repository's workloads (beam_mesh), clamped at x = 0 with a traction on
the far face; states are i.i.d. uniform in [-1e-2, 1e-2] per component, as in the assembly sweep.
"""
import math

import numpy as np
import torch

import igap4_gb300 as ig
from igap4_gb300.predictor import NPARAM, ConvNet, init_params

LAWS = {"lingrad": ig.LAW_LINGRAD, "gradelast": ig.LAW_GRADELAST, "gradelasttime": ig.LAW_GRADELASTTIME}
PRECS = {"fp64": ig.PREC_FP64, "split": ig.PREC_SPLIT, "fp64q": ig.PREC_OZAKI}
LENGTH = (4.0, 1.0, 1.0)
TRACTION = 1e-3
DT = 5e-4  # the transient law's default time step


def _asm(name, op, law, prec, nx, ny, nz, perturb=False):
    return {"name": name, "kind": "assembly", "op": op, "law": law, "prec": prec, "nx": nx, "ny": ny, "nz": nz,
            "perturb": perturb}


def listed():
    return [
        # the smallest meshes of the tests: one residual of the reference's static law, as a line search asks for
        _asm("residual_4x2x2", "residual", "gradelast", "fp64", 4, 2, 2),
        # the 16x4x4 cantilever: residual and tangent of one Newton step in the default precision
        _asm("fp64_16x4x4", "assemble", "lingrad", "fp64", 16, 4, 4),
        # the FP64 arm of the assembly sweep on a lattice of odd sizes that fill no tile evenly, distorted elements
        _asm("fp64_63x17x15", "assemble", "lingrad", "fp64", 63, 17, 15, True),
        # the assembly benchmark: the 128x32x32 beam in the FP64-quality mode
        _asm("fp64q_128x32x32", "assemble", "lingrad", "fp64q", 128, 32, 32),
        # the reference's static law in the default precision, on the sweep's first mesh
        _asm("static_32x8x8", "assemble", "gradelast", "fp64", 32, 8, 8),
        # the transient run's Newton step at its workload's size, tangent on the tensor cores
        _asm("transient_64x16x16", "assemble", "gradelasttime", "split", 64, 16, 16),
        # a parameter study: 24 of the seeded uneven beams of the batched workload
        {"name": "batch_24", "kind": "batch", "n": 24, "sizes": 0, "nx0": 8, "nx1": 64, "nyz0": 2, "nyz1": 16},
        # the linear solve of a Newton step when PETSc-like options cap its iterations (Jacobi, MGS)
        {"name": "ksp_32x8x8", "kind": "ksp", "nx": 32, "ny": 8, "nz": 8, "pc": 1, "its": 100},
        # a whole static solve: the 16x4x4 cantilever with the library's default options
        {"name": "newton_16x4x4", "kind": "newton", "nx": 16, "ny": 4, "nz": 4},
        # a whole time step of the transient run (cell-block Jacobi, CGS2, CUDA graphs) at a quarter of its size
        {"name": "step_32x8x8", "kind": "step", "nx": 32, "ny": 8, "nz": 8},
        # training the Newton predictor on trajectories of the 64x16x16 beam
        {"name": "train_66x18x18", "kind": "train", "nx": 66, "ny": 18, "nz": 18, "batch": 8},
        # the predictor's guess for one step of the 128x32x32 beam
        {"name": "forward_130x34x34", "kind": "forward", "nx": 130, "ny": 34, "nz": 34, "batch": 1},
    ]


def _log_int(rng, lo, hi):
    return int(min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def _lattice(rng, most, lo=(4, 2, 2), hi=(128, 32, 32)):
    """Element counts, each spread over its range in the logarithm, at most `most` elements in all."""
    while True:
        n = [_log_int(rng, a, b) for a, b in zip(lo, hi)]
        if n[0] * n[1] * n[2] <= most:
            return n


def draw(rng):
    k = rng.randrange(12)
    if k <= 6:
        law, prec, most = [("lingrad", "fp64", 16000), ("lingrad", "fp64", 16000), ("lingrad", "fp64q", 120000),
                           ("gradelast", "fp64", 2000), ("gradelast", "fp64", 2000), ("gradelasttime", "split", 16000),
                           ("gradelasttime", "split", 16000)][k]
        n = _lattice(rng, most)
        c = _asm("", rng.choice(["residual", "assemble", "assemble", "tangent"]), law, prec, *n,
                 perturb=bool(rng.randrange(2)))
    elif k == 7:
        c = {"kind": "batch", "n": rng.randint(4, 24), "sizes": rng.randrange(1, 1 << 20), "nx0": 8,
             "nx1": rng.randint(12, 60), "nyz0": 2, "nyz1": rng.randint(4, 15)}
    elif k == 8:
        n = _lattice(rng, 2000, lo=(8, 2, 2), hi=(48, 12, 12))
        c = {"kind": "ksp", "nx": n[0], "ny": n[1], "nz": n[2], "pc": rng.choice([1, 2, 3]), "its": rng.randint(30, 100)}
    elif k == 9:
        n = _lattice(rng, 250, lo=(6, 2, 2), hi=(24, 5, 5))
        c = {"kind": "newton", "nx": n[0], "ny": n[1], "nz": n[2]}
    elif k == 10:
        n = _lattice(rng, 2000, lo=(8, 2, 2), hi=(48, 12, 12))
        c = {"kind": "step", "nx": n[0], "ny": n[1], "nz": n[2]}
    else:
        big = rng.randrange(2)
        n = _lattice(rng, 20000 if big else 140000, lo=(8, 4, 4), hi=(130, 34, 34))
        c = {"kind": "train" if big else "forward", "nx": n[0], "ny": n[1], "nz": n[2],
             "batch": rng.randint(1, 8) if big else 1}
    c.pop("name", None)
    return c


# ------------------------------------------------------------------ inputs
def _nelem(case):
    return (case["nx"], case["ny"], case["nz"])


def _bc():
    return ig.clamp_bc((0,), traction_face=1, traction=(0.0, 0.0, -TRACTION))


def _parameters(law, seed):
    """The law's default material with the length scale of the seed's draw."""
    r = np.random.default_rng(seed)
    par = list(ig.LAW_DEFAULT_PAR[LAWS[law]])
    if law == "lingrad":
        par[2] = float(r.uniform(0.05, 0.2))
    return par


def _assembly(law, nelem, par, perturb=False):
    knots, w, X = ig.beam_mesh(nelem, LENGTH, perturb=perturb)
    bct, neu = _bc()
    A = ig.Assembly(nelem, knots, w, X, law=LAWS[law], par=par, bc_type=bct, neumann=neu)
    A.set_stream(torch.cuda.current_stream().cuda_stream)
    return A


def _uniform(n, seed, k=0):
    g = torch.Generator(device="cuda").manual_seed(1000003 * (seed % 1000003) + 7919 * k + 17)
    return (2.0 * torch.rand(n, generator=g, device="cuda", dtype=torch.float64) - 1.0) * 1e-2


def _instances(case, seed):
    """Uneven beams: sizes from the case, material of each from the seed."""
    rs = np.random.default_rng(case["sizes"])
    rp = np.random.default_rng(seed)
    out = []
    for _ in range(case["n"]):
        nx, nyz = int(rs.integers(case["nx0"], case["nx1"] + 1)), int(rs.integers(case["nyz0"], case["nyz1"] + 1))
        par = [float(rp.uniform(0.5, 2.0)), float(rp.uniform(0.5, 2.0)), float(rp.uniform(0.02, 0.2))] + [0.0] * 6
        out.append(((nx, nyz, nyz), par))
    return out


def _smooth_states(nelem, seed):
    """Two consecutive states of a bending beam (u_n, u_{n-1}), zero on the clamped control points."""
    r = np.random.default_rng(seed)
    nb = [n + 2 for n in nelem]
    x = np.maximum((np.arange(nb[0]) - 1.0) / nelem[0], 0.0)[:, None, None]
    y = ((np.arange(nb[1]) - 0.5) / nelem[1])[None, :, None]
    z = ((np.arange(nb[2]) - 0.5) / nelem[2])[None, None, :]
    a = r.uniform(0.5, 1.0, 6) * 1e-3
    u = np.zeros(nb + [3])
    u[..., 0] = a[0] * x ** 2 * (z - 0.5) + a[1] * x ** 3 * (y - 0.5)
    u[..., 1] = a[2] * x ** 2 + a[3] * x ** 3
    u[..., 2] = a[4] * x ** 2 + a[5] * x ** 3
    u[:2] = 0.0
    u = np.ascontiguousarray(u.reshape(-1))
    return u, u * float(r.uniform(0.97, 0.99))


def _net_inputs(case, seed):
    P = case["nx"] * case["ny"] * case["nz"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(case["batch"], P, 9, generator=g, device="cuda")
    t = torch.randn(case["batch"], P, 3, generator=g, device="cuda")
    return x, t, init_params(seed, zero_last=False)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "assembly":
        par = _parameters(case["law"], seed)
        A = _assembly(case["law"], _nelem(case), par, case["perturb"])
        A.set_precision(PRECS[case["prec"]])
        for lvl in range(1, A.torder + 1):
            A.set_history(lvl, _uniform(A.ndof, seed, lvl))
        s = {"A": A, "op": case["op"], "U": _uniform(A.ndof, seed)}
        if case["op"] != "tangent":
            s["RR"] = torch.zeros(A.ndof, dtype=torch.float64, device="cuda")
        if case["op"] != "residual":
            s["K"] = torch.zeros(A.nnz, dtype=torch.float64, device="cuda")
    elif kind == "batch":
        bct, neu = _bc()
        insts = []
        for nelem, par in _instances(case, seed):
            knots, w, X = ig.beam_mesh(nelem, LENGTH)
            insts.append(dict(nelem=nelem, knots=knots, w=w, X=X, par=par, bc_type=bct, neumann=neu))
        A = ig.BatchAssembly(insts, law=ig.LAW_LINGRAD)
        A.set_stream(torch.cuda.current_stream().cuda_stream)
        A.set_precision(ig.PREC_SPLIT)
        s = {"A": A, "op": "assemble", "U": _uniform(A.ndof, seed),
             "RR": torch.zeros(A.ndof, dtype=torch.float64, device="cuda"),
             "K": torch.zeros(A.nnz, dtype=torch.float64, device="cuda")}
    elif kind == "ksp":
        A = _assembly("lingrad", _nelem(case), _parameters("lingrad", seed))
        U = A.impose_dirichlet(_uniform(A.ndof, seed))
        b = torch.zeros(A.ndof, dtype=torch.float64, device="cuda")
        A.residual(U, b)
        A.tangent_internal(U)
        s = {"A": A, "b": b.neg_(), "x": torch.zeros_like(b),
             "opts": dict(pc=case["pc"], ksp_max_it=case["its"], ksp_rtol=1e-30)}
    elif kind == "newton":
        A = _assembly("lingrad", _nelem(case), _parameters("lingrad", seed))
        s = {"A": A, "U": torch.zeros(A.ndof, dtype=torch.float64, device="cuda")}
    elif kind == "step":
        par = list(ig.LAW_DEFAULT_PAR[ig.LAW_GRADELASTTIME])
        par[5], par[7] = 1.0, DT
        A = _assembly("gradelasttime", _nelem(case), par)
        A.set_precision(ig.PREC_SPLIT)
        un, um = (torch.from_numpy(u).cuda() for u in _smooth_states(_nelem(case), seed))
        A.set_history(1, un)
        A.set_history(2, um)
        load = np.zeros(36)
        load[6 + 2] = -TRACTION * float(np.random.default_rng(seed + 1).uniform(0.2, 1.0))
        s = {"A": A, "un": un, "U": torch.zeros_like(un), "load": load,
             "opts": dict(snes_abstol=1e-8, ksp_rtol=1e-5, ksp_restart=100, ksp_max_it=5000, snes_max_it=30,
                          use_graphs=1, pc=3, orth=1)}
    else:
        x, t, params = _net_inputs(case, seed)
        net = ConvNet(_nelem(case), batch_max=case["batch"], params=params)
        s = {"net": net, "x": x, "t": t, "out": torch.zeros_like(t)}
    s["kind"] = kind
    return s


def run(state):
    kind = state["kind"]
    if kind in ("assembly", "batch"):
        A = state["A"]
        if state["op"] == "residual":
            return {"RR": A.residual(state["U"], state["RR"])}
        if state["op"] == "tangent":
            return {"K": A.tangent(state["U"], state["K"])}
        A.assemble(state["U"], state["RR"], state["K"])
        return {"RR": state["RR"], "K": state["K"]}
    if kind == "ksp":
        x = state["x"].zero_()
        state["A"].ksp_solve(state["b"], x, **state["opts"])
        return {"x": x}
    if kind == "newton":
        U = state["U"].zero_()
        state["A"].solve(U)
        return {"U": U}
    if kind == "step":
        A, U = state["A"], state["U"].copy_(state["un"])
        A.set_neumann(state["load"])
        A.solve(U, **state["opts"])
        return {"U": U}
    if kind == "train":
        loss = state["net"].train_step(state["x"], state["t"], 1e-3)
        return {"loss": loss, "grads": state["net"].get_grads()}
    return {"out": state["net"].forward(state["x"], state["out"])}


# -------------------------------------------------------------------- work
def _sizes(nelem):
    nb = [n + 2 for n in nelem]
    nnz = 9
    for m in nb:
        nnz *= sum(min(i + 2, m - 1) - max(i - 2, 0) + 1 for i in range(m))
    return nelem[0] * nelem[1] * nelem[2], 3 * nb[0] * nb[1] * nb[2], nnz


def _assembly_work(nelem, law, op):
    """State, control net and history read once, outputs written once; per element of 64 points the state's
    interpolation and the projection (27 functions, 9 or 10 slots) and the symmetric half of the element matrix:
    a product of 81 rows with 4 terms a point for the linear law, with the law's 30 x 30 moduli for the others."""
    ne, ndof, nnz = _sizes(nelem)
    levels = 3 if law == "gradelasttime" else 1
    b = 8.0 * ndof * levels + 8.0 * ndof * 4 / 3
    f = 0.0
    if op != "tangent":
        b += 8.0 * ndof
        f += ne * 64 * 2.0 * (27 * 27 * levels + 27 * 27)
    if op != "residual":
        b += 8.0 * nnz
        f += ne * 64 * 2.0 * (81 * 82 // 2 * (4 if law == "lingrad" else 10) + (0 if law == "lingrad" else 30 * 81 * 5))
    return b, f


def work(case):
    kind = case["kind"]
    if kind == "assembly":
        b, f = _assembly_work(_nelem(case), case["law"], case["op"])
    elif kind == "batch":
        w = [_assembly_work(n, "lingrad", "assemble") for n, _ in _instances(case, 0)]
        b, f = sum(v[0] for v in w), sum(v[1] for v in w)
    elif kind in ("ksp", "newton", "step"):
        ne, ndof, nnz = _sizes(_nelem(case))
        its = case["its"] if kind == "ksp" else 100
        # the matrix and, on average, half the basis (read for the projection and for the update) an iteration
        b = its * 8.0 * (nnz + ndof * its)
        f = its * 2.0 * (nnz + 2.0 * ndof * its / 2)
        if kind != "ksp":
            law = "lingrad" if kind == "newton" else "gradelasttime"
            ab, af = _assembly_work(_nelem(case), law, "assemble")
            b, f = b + 2 * ab, f + 2 * af
    else:
        pts = case["batch"] * case["nx"] * case["ny"] * case["nz"]
        macs = 27 * (9 * 32 + 32 * 32 * 2 + 32 * 3)
        f = 2.0 * pts * macs * (3 if kind == "train" else 1)
        b = pts * 4.0 * 12 + 4.0 * NPARAM * (7 if kind == "train" else 1)
    return {"bytes": float(b), "flops": float(f)}


# ------------------------------------------------- the same results in 64 bits
SHIFT = 1e-15  # knot-span denominators of the volume basis carry this shift by definition


def _gauss():
    x, w = np.polynomial.legendre.leggauss(4)
    return 0.5 * x + 0.5, 0.5 * w


def _basis(n, shift):
    """[n, 4, 3, 3]: value, first and second derivative of the three quadratic functions of each element of an
    open uniform knot vector at the Gauss points (by element, point, derivative, function)."""
    kn = np.array([0.0, 0.0] + [0.0 if k == 0 else (k * (1.0 / n) if k < n else 1.0) for k in range(n + 1)] + [1.0, 1.0])
    xq, _ = _gauss()
    e = np.arange(n)
    x = (1.0 - xq)[None, :] * kn[e + 2][:, None] + xq[None, :] * kn[e + 3][:, None]
    f = [np.zeros_like(x), np.zeros_like(x), np.ones_like(x), np.zeros_like(x), np.zeros_like(x)]
    d1, d2 = [np.zeros_like(x)] * 5, None
    for q in (1, 2):
        nf, n1, n2 = [], [], []
        for i in range(5 - q):
            k = [kn[e + i + j][:, None] for j in range(q + 2)]
            dl, dr = k[q] - k[0] + shift, k[q + 1] - k[1] + shift
            ok_l, ok_r = dl != 0, dr != 0
            il, ir = np.where(ok_l, 1.0 / np.where(ok_l, dl, 1.0), 0.0), np.where(ok_r, 1.0 / np.where(ok_r, dr, 1.0), 0.0)
            nf.append((x - k[0]) * il * f[i] + (k[q + 1] - x) * ir * f[i + 1])
            n1.append(q * il * f[i] - q * ir * f[i + 1])
            n2.append(q * il * d1[i] - q * ir * d1[i + 1])
        f, d1, d2 = nf, n1, n2
    return np.stack([np.stack(v, -1) for v in (f, d1, d2)], 2)


DERIV = [(0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (2, 0, 0), (1, 1, 0), (1, 0, 1), (0, 2, 0), (0, 1, 1), (0, 0, 2)]
PAIRS = [(0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2)]
SYM = [[0, 1, 2], [1, 3, 4], [2, 4, 5]]


def _control_net(nelem, perturb):
    nb = [n + 2 for n in nelem]
    i, j, k = np.meshgrid(*[np.arange(m) for m in nb], indexing="ij")
    X = np.stack([(v - 0.5) / n * l for v, n, l in zip((i, j, k), nelem, LENGTH)], -1)
    if perturb:
        inner = np.ones(nb)
        for v, m in zip((i, j, k), nb):
            inner *= (v > 2) & (v < m - 2)
        for d, c in enumerate((3, 5, 7)):
            X[..., d] += 0.2 * LENGTH[d] / nb[d] * inner * np.sin(c * (i * k * j))
    return X.reshape(-1, 3)


def _elements(nelem, perturb, chunk=1024):
    """Chunks of elements: control points [E, 27], physical basis [E, 64, 27, 10], weights [E, 64]."""
    dev = "cuda"
    tabs = [torch.from_numpy(_basis(n, SHIFT)).to(dev) for n in nelem]
    nb = [n + 2 for n in nelem]
    X = torch.from_numpy(_control_net(nelem, perturb)).to(dev)
    wq = torch.from_numpy(_gauss()[1]).to(dev)
    w3 = torch.einsum("i,j,k->ijk", wq, wq, wq).reshape(-1) / (nelem[0] * nelem[1] * nelem[2])
    loc = torch.tensor([[(a * nb[1] + b) * nb[2] + c] for a in range(3) for b in range(3) for c in range(3)], device=dev)[:, 0]
    ne = nelem[0] * nelem[1] * nelem[2]
    for e0 in range(0, ne, chunk):
        e = torch.arange(e0, min(ne, e0 + chunk), device=dev)
        ez, ey, ex = e % nelem[2], (e // nelem[2]) % nelem[1], e // (nelem[1] * nelem[2])
        cp = ((ex * nb[1] + ey) * nb[2] + ez)[:, None] + loc[None, :]
        tx, ty, tz = tabs[0][ex], tabs[1][ey], tabs[2][ez]  # [E, 4, 3 derivatives, 3 functions]
        N = torch.stack([torch.einsum("eia,ejb,ekc->eijkabc", tx[:, :, p], ty[:, :, q], tz[:, :, r]).reshape(len(e), 64, 27)
                         for p, q, r in DERIV], -1)
        W = N.sum(2, keepdim=True)  # unit weights: the functions' sum and its derivatives
        R = N / W[..., :1]
        R[..., 1:] = R[..., 1:] - R[..., :1] * W[..., 1:] / W[..., :1]
        for s, (i, j) in enumerate(PAIRS):
            R[..., 4 + s] -= (R[..., 1 + j] * W[..., 1 + i] + R[..., 1 + i] * W[..., 1 + j]) / W[..., 0]
        G = torch.einsum("eqbk,ebd->eqdk", R, X[cp])
        J = G[..., 1:4]
        Ji = torch.linalg.inv(J)
        grad = torch.einsum("eqbj,eqji->eqbi", R[..., 1:4], Ji)
        H = R[..., 4:] - torch.einsum("eqbi,eqis->eqbs", grad, G[..., 4:])
        H = H[..., torch.tensor(SYM, device=dev)]
        H = torch.einsum("eqmi,eqbml,eqlj->eqbij", Ji, H, Ji)
        R = torch.cat([R[..., :1], grad, torch.stack([H[..., i, j] for i, j in PAIRS], -1)], -1)
        yield cp, R, w3[None, :] * torch.linalg.det(J)


def _lin_law(par):
    """Constant 30 x 30 moduli of the linear strain-gradient law: the energy's second derivative."""
    lam, mu, ell = par[:3]
    D = np.zeros((30, 30))

    def add(rows, c):
        v = np.zeros(30)
        for k, a in rows:
            v[k] += a
        D[:] += c * np.outer(v, v)

    def comp(i, j, m):
        return 10 * i + 1 + j if m is None else 10 * i + 4 + SYM[j][m]

    for m, s in ((None, 1.0), (0, ell * ell), (1, ell * ell), (2, ell * ell)):
        add([(comp(i, i, m), 1.0) for i in range(3)], lam * s)
        for i in range(3):
            for j in range(3):
                add([(comp(i, j, m), 0.5), (comp(j, i, m), 0.5)], 2.0 * mu * s)
    return torch.from_numpy(D).cuda()


def _energy(par):
    """The gradient law's stored energy of one point's 30 slots."""
    r, curv = par[0], par[1]
    den = r * r - 2.0 * r * r * curv - r * (4.0 / 3.0 * r - 4.0 / 3.0 * r * curv)
    A, B, C = 2.0 * curv / den, -(4.0 / 3.0 * r - 4.0 / 3.0 * r * curv) / (r * r * den), -1.0 / (r * r * den)
    sym = torch.tensor(SYM, device="cuda")
    eye = torch.eye(3, dtype=torch.float64, device="cuda")

    def psi(u):
        u = u.reshape(3, 10)
        F = eye + u[:, 1:4]
        H = u[:, 4:][:, sym]  # d2 u_k / dx_a dx_m
        E = 0.5 * (F.T @ F - eye)
        g = torch.einsum("ka,kam->am", F, H)  # d E_aa / dx_m
        ev = (E[0, 0] + E[1, 1] + E[2, 2]) / 3 ** 0.5
        e1 = (E[0, 0] - E[1, 1]) / 2 ** 0.5
        e2 = (E[0, 0] + E[1, 1] - 2 * E[2, 2]) / 6 ** 0.5
        g1 = (g[0] - g[1]) / 2 ** 0.5
        g2 = (g[0] + g[1] - 2 * g[2]) / 6 ** 0.5
        q = e1 * e1 + e2 * e2
        return (par[2] * ev * ev + par[3] * (E[0, 1] ** 2 + E[0, 2] ** 2 + E[1, 2] ** 2) + A * q
                + B * (e2 ** 3 - 3 * e1 * e1 * e2) + C * q * q + par[4] ** 2 * ((g1 * g1).sum() + (g2 * g2).sum()))

    return psi


def _law(law, par, u, want_r, want_t):
    """Residual integrand [N, 30] and moduli [N, 30, 30] at states u [N, levels, 30]."""
    from torch.func import grad, hessian, vmap

    psi = _energy(par)
    if law == "gradelast":
        r = vmap(grad(psi), chunk_size=16384)(u[:, 0]) if want_r else None
        return r, vmap(hessian(psi), chunk_size=2048)(u[:, 0]) if want_t else None
    # average-vector-field force between the midpoints m and m + d, its Taylor series in d cut at the third order:
    # the energy is a polynomial of degree 8 in s, so its derivatives at s = 0 come from values at 9 points
    m, d = 0.5 * (u[:, 1] + u[:, 2]), 0.5 * (u[:, 0] - u[:, 2])
    s = np.cos(np.pi * (np.arange(9) + 0.5) / 9)
    inv = np.linalg.inv(np.vander(s, 9, increasing=True))  # rows: Taylor coefficients
    cr, ct = inv[:4].T @ (1.0 / np.arange(1, 5)), 0.5 * inv[:3].T @ (1.0 / np.arange(2, 5))
    r = sum(c * vmap(grad(psi), chunk_size=16384)(m + v * d) for c, v in zip(cr, s)) if want_r else None
    t = sum(c * vmap(hessian(psi), chunk_size=2048)(m + v * d) for c, v in zip(ct, s)) if want_t else None
    rho, damp, dt = par[5], par[6], par[7]
    for k in (0, 10, 20):
        if want_r:
            r[:, k] += damp * (u[:, 0, k] - u[:, 2, k]) / (2 * dt) + rho * (u[:, 0, k] + u[:, 2, k] - 2 * u[:, 1, k]) / dt ** 2
        if want_t:
            t[:, k, k] += damp / (2 * dt) + rho / dt ** 2
    return r, t


def _assembled(nelem, perturb, law, par, U, op):
    """(residual, CSR values) of the clamped beam at the states U [levels, ndof]."""
    dev = "cuda"
    nb = [n + 2 for n in nelem]
    ncp = nb[0] * nb[1] * nb[2]
    lo = [torch.clamp(torch.arange(m, device=dev) - 2, min=0) for m in nb]
    ln = [torch.clamp(torch.arange(m, device=dev) + 2, max=m - 1) - a + 1 for m, a in zip(nb, lo)]
    rowlen = 3 * (ln[0][:, None, None] * ln[1][None, :, None] * ln[2][None, None, :]).reshape(-1)
    start = torch.cumsum(3 * rowlen, 0) - 3 * rowlen  # first CSR slot of a control point's three rows
    want_r, want_t = op != "tangent", op != "residual"
    RR = torch.zeros(3 * ncp, dtype=torch.float64, device=dev)
    K = torch.zeros(int((3 * rowlen).sum()), dtype=torch.float64, device=dev) if want_t else None
    lin = law == "lingrad"
    D0 = _lin_law(par) if lin else None
    three = torch.arange(3, device=dev)
    for cp, R, w in _elements(nelem, perturb, 1024 if lin else 256):
        E = len(cp)
        dof = (3 * cp[:, :, None] + three).reshape(E, 81)
        u = torch.einsum("hebd,eqbk->eqhdk", U[:, dof].reshape(U.shape[0], E, 27, 3), R).reshape(E, 64, U.shape[0], 30)
        if lin:
            rr, D = u[:, :, 0] @ D0, None
        else:
            rr, D = _law(law, par, u.reshape(E * 64, U.shape[0], 30), want_r, want_t)
        if want_r:
            f = torch.einsum("eqdk,eqbk,eq->ebd", rr.reshape(E, 64, 3, 10), R, w)
            RR.index_add_(0, dof.reshape(-1), f.reshape(-1))
        if not want_t:
            continue
        if lin:  # the point weight on one side, the moduli are constant
            M = torch.einsum("dkj,eqbk,eq->ebdqj", D0.reshape(3, 10, 30), R, w).reshape(E, 81, 64, 3, 10)
        else:
            M = torch.einsum("eqdkj,eqbk,eq->ebdqj", D.reshape(E, 64, 3, 10, 30), R, w).reshape(E, 81, 64, 3, 10)
        Rt = R.permute(0, 1, 3, 2).reshape(E, 640, 27)
        Ke = torch.stack([M[:, :, :, e].reshape(E, 81, 640) @ Rt for e in range(3)], -1)  # [E, 81, 27, 3]
        iz, iy, ix = cp % nb[2], (cp // nb[2]) % nb[1], cp // (nb[1] * nb[2])
        pos = ((ix[:, None, :] - lo[0][ix][:, :, None]) * ln[1][iy][:, :, None] + iy[:, None, :] - lo[1][iy][:, :, None]) \
            * ln[2][iz][:, :, None] + iz[:, None, :] - lo[2][iz][:, :, None]
        slot = start[cp][:, :, None, None, None] + three[None, None, :, None, None] * rowlen[cp][:, :, None, None, None] \
            + 3 * pos[:, :, None, :, None] + three
        K.index_add_(0, slot.reshape(-1), Ke.reshape(E, 27, 3, 27, 3).reshape(-1))
    if want_r:  # constant traction on x = L in the face's parameters, plain basis
        ty, tz = (torch.from_numpy(_basis(n, 0.0)[:, :, 0]).to(dev) for n in nelem[1:])
        wq = torch.from_numpy(_gauss()[1]).to(dev)
        face = []
        for t, n in ((ty, nelem[1]), (tz, nelem[2])):
            v = torch.zeros(n + 2, dtype=torch.float64, device=dev)
            for a in range(3):
                v[a:a + n] += torch.einsum("eq,q->e", t[:, :, a], wq) / n
            face.append(v)
        RR.reshape(*nb, 3)[-1, :, :, 2] += TRACTION * face[0][:, None] * face[1][None, :]
        RR.reshape(*nb, 3)[:2] = U[0].reshape(*nb, 3)[:2]  # clamped: both layers at x = 0 hold U - 0
    if want_t:
        row0 = 2 * nb[1] * nb[2]  # control points of the clamped layers come first
        n0 = int(start[row0])
        K[:n0] = 0.0
        for ix in range(4):  # their columns in the rows that reach them: the leading (2 - lo) layers of the stencil
            keep = max(0, 2 - int(lo[0][ix]))
            c = torch.arange(ix * nb[1] * nb[2], (ix + 1) * nb[1] * nb[2], device=dev)
            if ix < 2:
                iz, iy = c % nb[2], (c // nb[2]) % nb[1]
                pos = ((ix - int(lo[0][ix])) * ln[1][iy] + iy - lo[1][iy]) * ln[2][iz] + iz - lo[2][iz]
                for d in range(3):
                    K[start[c] + d * rowlen[c] + 3 * pos + d] = 1.0
            elif keep:
                width = 3 * keep * (ln[1][(c // nb[2]) % nb[1]] * ln[2][c % nb[2]])
                for d in range(3):
                    first = start[c] + d * rowlen[c]
                    k = torch.arange(int(width.max()), device=dev)
                    at = first[:, None] + k[None, :]
                    K[at[k[None, :] < width[:, None]]] = 0.0
    return (RR if want_r else None), K


def _dense(nelem, K):
    """The CSR values as a dense matrix."""
    nb = [n + 2 for n in nelem]
    n = 3 * nb[0] * nb[1] * nb[2]
    A = np.zeros((n, n))
    K, s = K.cpu().numpy(), 0
    for cp in range(n // 3):
        iz, iy, ix = cp % nb[2], (cp // nb[2]) % nb[1], cp // (nb[1] * nb[2])
        r = [range(max(0, i - 2), min(m - 1, i + 2) + 1) for i, m in zip((ix, iy, iz), nb)]
        cols = np.array([3 * ((a * nb[1] + b) * nb[2] + c) + e for a in r[0] for b in r[1] for c in r[2] for e in range(3)])
        for d in range(3):
            A[3 * cp + d, cols] = K[s:s + len(cols)]
            s += len(cols)
    return torch.from_numpy(A).cuda()


def _precondition(A, nelem, pc):
    """Inverse diagonal blocks as a dense block matrix product: Jacobi, control points, 2 x 2 x 2 cells."""
    nb = [n + 2 for n in nelem]
    n = A.shape[0]
    if pc == 1:
        d = A.diagonal().clone()
        return lambda v: v / d
    groups = {}
    for cp in range(n // 3):
        iz, iy, ix = cp % nb[2], (cp // nb[2]) % nb[1], cp // (nb[1] * nb[2])
        groups.setdefault(cp if pc == 2 else (ix // 2, iy // 2, iz // 2), []).extend(3 * cp + e for e in range(3))
    blocks = {}
    for g in groups.values():
        blocks.setdefault(len(g), []).append(g)
    inv = []
    for g in blocks.values():
        ix = torch.tensor(g, device="cuda")
        inv.append((ix, torch.linalg.inv(A[ix[:, :, None], ix[:, None, :]])))

    def apply(v):
        z = torch.empty_like(v)
        for ix, B in inv:
            z[ix] = torch.einsum("gij,gj->gi", B, v[ix])
        return z

    return apply


def _gmres(A, b, M, its):
    """The iterate of right-preconditioned GMRES after `its` steps from zero."""
    V, Z = [b / b.norm()], []
    H = torch.zeros(its + 1, its, dtype=torch.float64, device="cuda")
    for j in range(its):
        Z.append(M(V[j]))
        w = A @ Z[j]
        B = torch.stack(V)
        for _ in range(2):
            h = B @ w
            w = w - h @ B
            H[:j + 1, j] += h
        H[j + 1, j] = w.norm()
        V.append(w / H[j + 1, j])
    e = torch.zeros(its + 1, 1, dtype=torch.float64)
    e[0] = float(b.norm())
    y = torch.linalg.lstsq(H.cpu(), e, driver="gelsd").solution[:, 0].cuda()
    return y @ torch.stack(Z)


def _exact_net(case, seed):
    """Loss and gradients (or outputs) of the network's mathematics with the FP32 master weights."""
    import torch.nn.functional as F

    x, t, params = _net_inputs(case, seed)
    p = torch.from_numpy(params).cuda().double().requires_grad_(case["kind"] == "train")
    o, ws, ci = 0, [], 9
    for co in (32, 32, 32, 3):
        ws.append(p[o:o + co * 27 * ci].reshape(co, 3, 3, 3, ci).permute(0, 4, 1, 2, 3))
        o, ci = o + co * 27 * ci, co
    v = x.double().reshape(case["batch"], *_nelem(case), 9).permute(0, 4, 1, 2, 3)
    for l, w in enumerate(ws):
        bias = p[o:o + w.shape[0]]
        o += w.shape[0]
        v = F.conv3d(v, w, bias, padding=1)
        v = F.relu(v) if l < 3 else v
    out = v.permute(0, 2, 3, 4, 1).reshape(t.shape)
    if case["kind"] == "forward":
        return {"out": out}
    loss = ((out - t.double()) ** 2).mean()
    loss.backward()
    return {"loss": float(loss.detach()), "grads": p.grad}


def exact(case, seed):
    kind = case["kind"]
    if kind == "assembly":
        law, ne = case["law"], case["nx"] * case["ny"] * case["nz"]
        if (law == "gradelast" and ne > 2100) or (law == "gradelasttime" and ne > 400):
            return None
        par = _parameters(law, seed)
        ndof = 3 * (case["nx"] + 2) * (case["ny"] + 2) * (case["nz"] + 2)
        U = torch.stack([_uniform(ndof, seed, k) for k in range(3 if law == "gradelasttime" else 1)])
        RR, K = _assembled(_nelem(case), case["perturb"], law, par, U, case["op"])
        return {k: v for k, v in (("RR", RR), ("K", K)) if v is not None}
    if kind == "batch":
        insts = _instances(case, seed)
        sizes = [_sizes(n)[1] for n, _ in insts]
        U, o, R, K = _uniform(sum(sizes), seed), 0, [], []
        for (nelem, par), nd in zip(insts, sizes):
            r, k = _assembled(nelem, False, "lingrad", par, U[o:o + nd][None], "assemble")
            o += nd
            R.append(r)
            K.append(k)
        return {"RR": torch.cat(R), "K": torch.cat(K)}
    if kind in ("ksp", "newton"):
        nelem = _nelem(case)
        ndof = _sizes(nelem)[1]
        if ndof > 12000:
            return None
        U = torch.zeros(ndof, dtype=torch.float64, device="cuda")
        if kind == "ksp":
            U = _uniform(ndof, seed)
            U[:2 * 3 * (nelem[1] + 2) * (nelem[2] + 2)] = 0.0
        RR, K = _assembled(nelem, False, "lingrad", _parameters("lingrad", seed), U[None], "assemble")
        A = _dense(nelem, K)
        if kind == "newton":
            return {"U": torch.linalg.solve(A, -RR)}
        return {"x": _gmres(A, -RR, _precondition(A, nelem, case["pc"]), case["its"])}
    if kind == "step":
        return None
    return _exact_net(case, seed)
