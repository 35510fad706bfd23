"""Training gradients at tile counts around the kernels' splits (one tile, an
odd few, more than one slice of the weight gradients) against the oracle, with
the tolerance of the four-tile test: BF16 activations, FP32 sums in another
order."""

import numpy as np
import pytest
import torch

from oracle import cnn_ref
from tests.gpu_util import host
from tests.test_cnn_gpu import ProposalNetwork, load_batch, params, random_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 17])
def test_gradients_match_oracle(cuda, n):
    x0, labels, targets, weights = random_batch(n, 20 + n)
    flat = params(3)
    net = ProposalNetwork(flat)
    load_batch(net, x0)
    net.train_step(n, torch.from_numpy(labels).cuda(), torch.from_numpy(targets).cuda(),
                   torch.from_numpy(weights).cuda(), lr=0.0, weight_decay=0.0)
    got = host(net.grads)
    fwd = cnn_ref.forward(flat, x0)
    loss, dhead = cnn_ref.loss_and_grad(fwd["head"], labels, targets, weights, 4.0)
    want = cnn_ref.backward(flat, fwd, dhead)
    assert abs(float(host(net.loss)[0]) - loss) <= 1e-3 * abs(loss)
    for name, offset, shape in cnn_ref.param_layout():
        size = int(np.prod(shape))
        g, w = got[offset:offset + size].astype(np.float64), want[offset:offset + size]
        assert np.linalg.norm(g - w) <= 2e-2 * np.linalg.norm(w) + 1e-9, name


def test_scratch_off_16_bytes(cuda):
    """A scratch that starts at any float: the same gradients."""
    x0, labels, targets, weights = random_batch(2, 5)
    grads = []
    for offset in (0, 4, 12):
        net = ProposalNetwork(params(4))
        load_batch(net, x0)
        whole = torch.empty(net.scratch.numel() + offset, dtype=torch.uint8, device="cuda")
        net.scratch = whole[offset:]
        net.train_step(2, torch.from_numpy(labels).cuda(), torch.from_numpy(targets).cuda(),
                       torch.from_numpy(weights).cuda(), lr=0.0, weight_decay=0.0)
        grads.append(host(net.grads))
    assert np.array_equal(grads[0], grads[1]) and np.array_equal(grads[0], grads[2])
