"""The BF16 network's one-output and tiled kernels give the same outputs: a
sample alone and the same sample in a batch that is large enough for the tiles
of both outer layers; and a step's gradients, alone and in such a batch."""
import numpy as np
import pytest

from igap4_gb300.predictor import ConvNet, init_params

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("lattice", [(1, 1, 1), (6, 4, 4), (19, 9, 5), (16, 16, 16), (17, 16, 16)])
def test_sample_alone_and_in_a_batch(lattice):
    P = int(np.prod(lattice))
    B = max(3, 8200 // P + 1)
    net = ConvNet(lattice, batch_max=B, storage="bf16", params=init_params(5, zero_last=False))
    x = torch.tensor(np.random.default_rng(0).standard_normal((B, P, 9)).astype(np.float32), device="cuda")
    whole, one = torch.zeros((B, P, 3), device="cuda"), torch.zeros((1, P, 3), device="cuda")
    net.forward(x, whole)
    for b in (0, B - 1):
        net.forward(x[b:b + 1].contiguous(), one)
        assert torch.equal(one[0], whole[b])


# Four equal samples scale every value by a power of two; what is left is the
# order and the truncation of FP32 sums of up to 10,880 points: 10,880 / 16
# tensor-core steps of 2^-23, 8e-5, and as much again.  No weight changes (rate 0).
@pytest.mark.parametrize("lattice", [(1, 1, 1), (10, 16, 16), (10, 16, 17)])
def test_gradients_alone_and_in_a_batch(lattice):
    P = int(np.prod(lattice))
    net = ConvNet(lattice, batch_max=4, storage="bf16", params=init_params(5, zero_last=False))
    rng = np.random.default_rng(1)
    x = torch.tensor(rng.standard_normal((1, P, 9)).astype(np.float32), device="cuda")
    y = torch.tensor(rng.standard_normal((1, P, 3)).astype(np.float32), device="cuda")
    net.train_step(x, y, 0.0)
    alone = net.get_grads()
    net.train_step(x.repeat(4, 1, 1), y.repeat(4, 1, 1), 0.0)  # the mean over four equal samples
    assert np.linalg.norm(net.get_grads() - alone) <= 2e-4 * np.linalg.norm(alone)
