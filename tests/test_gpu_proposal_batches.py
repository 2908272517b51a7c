"""The proposal network at batch sizes that its kernels divide unevenly: fewer
samples than a block takes (4 and 8 per block in the last convolutions), a
remainder after whole blocks, several samples per weight-gradient block (39 and
more; the first convolution 305 and more) and a last one with fewer.  Loss and
gradients against the FP64 oracle: FP32 sums of up to 2^16 terms and ReLU masks
that may differ where a value is within rounding of zero, 2e-4 relative L2."""
import numpy as np
import pytest
import torch

import emc_gb300 as E
from emc_gb300 import synthetic as S
from oracle import proposal as PO

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def net_data(ctx, cuda):
    prob = S.make_problem(S.Config("prop", 64, 400, 1.5, 12, 400, 3000, (0.5, 1.5), 4, 2, 1,
                                   seed=5))
    net = E.Proposal(ctx, seed=4)
    net.set_data(torch.as_tensor(prob.images, dtype=torch.float32, device=cuda),
                 torch.as_tensor(prob.mask, dtype=torch.int32, device=cuda), 64)
    q = np.random.default_rng(1).normal(size=(400, 4))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    yield net, net.inputs(0, 400).astype(np.float64), q.astype(np.float32)
    net.close()


@pytest.mark.parametrize("batch", [1, 3, 9, 41, 306])
def test_gradients(net_data, cuda, batch):
    net, X, q = net_data
    rows = np.random.default_rng(batch).permutation(400)[:batch].astype(np.int32)
    loss, g = net.loss_grad(rows, torch.as_tensor(q, device=cuda))
    L, want = PO.loss_and_grads(net.params().astype(np.float64), X[rows],
                                q[rows].astype(np.float64))
    assert abs(loss - L) <= 1e-5 * abs(L)
    for o, shape in PO.layout()[0]:
        n = int(np.prod(shape))
        err = np.linalg.norm(g[o:o + n] - want[o:o + n])
        assert err <= 2e-4 * np.linalg.norm(want[o:o + n]), (o, shape)
