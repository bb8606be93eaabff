"""The training step's top-1 accuracy is over the 4,960 triples: a target in the padding columns
is never the greatest, whatever the padding's logits are."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("level", [-100.0, 100.0])
def test_padding_targets_are_no_hits(native_lib, level):
    import torch
    from tdp1375_b200 import order_model as om
    from tdp1375_b200.cases import three_permutation
    rng = np.random.Generator(np.random.PCG64(7))
    rows = 64
    spi, pi, ns = np.zeros((rows, 64), np.uint8), np.zeros((rows, 64), np.uint8), np.zeros(rows, np.uint8)
    for r in range(rows):
        p, s, _ = three_permutation(5, rng)
        spi[r, :15], pi[r, :15], ns[r] = s, p, 15
    d_n = torch.from_numpy(ns).cuda()
    x = om.features(torch.from_numpy(spi).cuda(), torch.from_numpy(pi).cuda(), d_n)
    model = om.OrderModel(seed=3)
    model.bias[3][:om.TRIPLES] = level  # the padding's logits are 0
    logits, _ = model.forward(x)
    best = logits[:, :om.TRIPLES].argmax(dim=1).to(torch.int32)
    target = best.clone()
    target[::2] = om.TRIPLES + torch.arange(rows // 2, dtype=torch.int32, device="cuda")
    _, top1 = model.train_step(x, d_n, target)
    assert top1 == 0.5
