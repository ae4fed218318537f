"""A caller that captures a context's first FP64 assembly into a graph of its
own: nothing is allocated or built inside the capture (the colour-by-colour
kernels are captured), and the replay gives the assembly.  Also with the
one-time set-up done before, and after a context was used under another
thread's capture."""
import threading

import numpy as np
import pytest

import igap4_gb300 as ig

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def beam(law):
    bct, neu = ig.clamp_bc((0,), traction_face=1, traction=(0.0, 0.0, -1e-3))
    knots, w, X = ig.beam_mesh((5, 4, 3), (4.0, 1.0, 1.0), perturb=True)
    return ig.Assembly((5, 4, 3), knots, w, X, law=law, bc_type=bct, neumann=neu)


# 1e-13: 64 x 100 products of each pair in 53 bits, as between the library's own routes
@pytest.mark.parametrize("law", [ig.LAW_LINGRAD, ig.LAW_GRADELAST])
@pytest.mark.parametrize("op", ["residual", "tangent"])
@pytest.mark.parametrize("mode", ["global", "thread_local", "relaxed"])
def test_first_call_in_a_capture(monkeypatch, law, op, mode):
    if law != ig.LAW_LINGRAD:
        monkeypatch.setenv("IGAPGPU_LAW_PRECOMPUTE", "0")  # the law's output buffers are a first-call allocation too
    ref = beam(law)  # also uploads the constant tables, once per process
    U = torch.tensor(np.random.default_rng(1).uniform(-1e-2, 1e-2, ref.ndof), device="cuda")
    n = ref.ndof if op == "residual" else ref.nnz
    want, out = U.new_zeros(n), U.new_zeros(n)
    torch.cuda.synchronize()
    getattr(ref, op)(U, want)
    ref.synchronize()
    A = beam(law)
    s = torch.cuda.Stream()
    A.set_stream(s.cuda_stream)
    for again in range(2):  # the second capture follows the first plain call
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s, capture_error_mode=mode):
            getattr(A, op)(U, out)
        out.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert (out - want).norm() <= 1e-13 * want.norm()
        getattr(A, op)(U, out)
        A.synchronize()
        assert torch.equal(out, want)


def test_first_call_beside_another_threads_capture():
    ref, A = beam(ig.LAW_LINGRAD), beam(ig.LAW_LINGRAD)
    U = np.random.default_rng(1).uniform(-1e-2, 1e-2, A.ndof)
    want, got, err = ref.tangent(U), [], []
    Ud = torch.tensor(U, device="cuda")
    K, x = Ud.new_zeros(A.nnz), torch.zeros(8, device="cuda")
    torch.cuda.synchronize()

    def work():
        try:
            A.tangent(Ud, K)
        except Exception as e:  # reported below, outside the capture
            err.append(e)

    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):  # mode "global": unsafe calls of any thread are refused
        x += 1.0
        t = threading.Thread(target=work)
        t.start()
        t.join()
    assert not err, err
    A.synchronize()
    torch.cuda.synchronize()
    np.testing.assert_array_equal(K.cpu().numpy(), want)
    g.replay()
    torch.cuda.synchronize()
    assert (x.cpu().numpy() == 1.0).all()
