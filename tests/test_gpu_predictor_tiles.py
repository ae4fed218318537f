"""Tiled input and output layers of the BF16 network (csrc/predictor.cu) where
their tiles of 256 and 512 points can go wrong: one point, a lattice thinner
than the stencil, exactly one tile, one point more, tiles across samples.
6e-2: four layers of BF16 activation rounding, as the other BF16 checks."""
import numpy as np
import pytest

import conv_oracle as co
from igap4_gb300.predictor import ConvNet, init_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lattice,B", [((1, 1, 1), 1), ((2, 3, 1), 2), ((8, 8, 4), 1), ((8, 8, 8), 1), ((19, 9, 3), 1),
                                       ((7, 5, 5), 3)])
def test_tiles_vs_oracle(lattice, B):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(5)
    params = init_params(5, zero_last=False)
    params[-sum(co.COUT):] = rng.standard_normal(sum(co.COUT)).astype(np.float32) * 0.1
    P = int(np.prod(lattice))
    x = rng.standard_normal((B,) + lattice + (9,)).astype(np.float32)
    y = rng.standard_normal((B,) + lattice + (3,)).astype(np.float32)
    net = ConvNet(lattice, batch_max=B, storage="bf16", params=params)
    out = torch.zeros((B, P, 3), dtype=torch.float32, device="cuda")
    net.forward(torch.tensor(x.reshape(B, P, 9), device="cuda"), out)
    loss_ref, grad_ref, y_ref = co.loss_and_grad(params.astype(np.float64), x.astype(np.float64), y.astype(np.float64))
    assert np.linalg.norm(out.cpu().numpy().reshape(y_ref.shape) - y_ref) <= 6e-2 * np.linalg.norm(y_ref)
    loss = net.train_step(torch.tensor(x.reshape(B, P, 9), device="cuda"),
                          torch.tensor(y.reshape(B, P, 3), device="cuda"), 0.0)
    assert abs(loss - loss_ref) <= 6e-2 * loss_ref
    assert np.linalg.norm(net.get_grads() - grad_ref) <= 6e-2 * np.linalg.norm(grad_ref)
