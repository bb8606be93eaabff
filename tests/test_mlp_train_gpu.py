"""The GEMM at the edges of its tiles and output forms, and one whole training step, against plain
PyTorch.

Tolerances.  fp32 accumulation of K products in any order: |err| <= K * 2^-23 * (|A| |B|^T).
A bf16 result adds one rounding, 2^-8 relative.  The training step rounds activations and
gradients to bf16 where the reference below does; a different summation order can flip such a
rounding, one flip is 2^-8 of the element, so a gradient's norm may differ by 2^-8."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

vp = ctypes.c_void_p


@pytest.mark.parametrize("m,n,k,ldo,fp32", [
    (1, 8, 8, 8, True), (127, 64, 72, 64, False), (128, 128, 64, 128, True), (129, 72, 1088, 80, False),
    (129, 200, 64, 204, True),      # row stride a multiple of 16 bytes, N of no tile
    (130, 65, 256, 67, True),       # row stride allows no TMA store
    (257, 40, 128, 41, False), (2500, 1000, 128, 1000, True), (2500, 1000, 128, 1000, False),  # 128-wide tiles
])
def test_gemm_tile_edges_match_torch(native_lib, m, n, k, ldo, fp32):
    import torch
    g = torch.Generator(device="cpu").manual_seed(m + n)
    a = torch.randn(m, k, generator=g).to(torch.bfloat16).cuda()
    b = torch.randn(n, k, generator=g).to(torch.bfloat16).cuda()
    bias = torch.randn(n, generator=g).cuda()
    out = torch.full((m + 1, ldo), 7.0, device="cuda", dtype=torch.float32 if fp32 else torch.bfloat16)
    for relu in (0, 1):
        rc = native_lib.tdp_mlp_gemm(vp(a.data_ptr()), vp(b.data_ptr()), m, n, k, vp(bias.data_ptr()), relu,
                                     vp(out.data_ptr()), int(fp32), ldo, vp(0))
        assert rc == 0
        torch.cuda.synchronize()
        assert native_lib.tdp_mlp_error() == 0
        ref = a.double() @ b.double().T + bias.double()
        if relu:
            ref = torch.relu(ref)
        bound = (k + 1) * 2.0 ** -23 * (a.double().abs() @ b.double().abs().T + bias.abs())
        if not fp32:
            bound = bound + 2.0 ** -8 * ref.abs()
        assert bool(((out[:m, :n].double() - ref).abs() <= bound).all())
        assert bool((out[m:] == 7.0).all()) and bool((out[:, n:] == 7.0).all())  # nothing outside the result


def reference_step(model, x, n, target, lr):
    """One step with torch products in fp32, bf16 where the library stores bf16."""
    import torch
    from tdp1375_b200 import order_model as om
    rows = x.shape[0]
    acts = [x.float()]
    for layer in range(3):
        h = torch.relu(acts[-1] @ model.weight[layer].float().T + model.bias[layer])
        acts.append(h.to(torch.bfloat16).float())
    logits = acts[-1] @ model.weight[3].float().T + model.bias[3]
    last = np.full(om.TRIPLES_PADDED, 255)
    i, j, k = np.nonzero(om.LEX32 >= 0)
    last[om.LEX32[i, j, k]] = k
    valid = torch.from_numpy(last).cuda()[None, :] < n[:, None].long()
    logp = torch.log_softmax(logits.masked_fill(~valid, float("-inf")), dim=1)
    loss = -logp.gather(1, target.long()[:, None])
    top1 = (logits[:, :om.TRIPLES].argmax(dim=1) == target.long()).float().mean()
    grad = logp.exp()
    grad.scatter_add_(1, target.long()[:, None], torch.full_like(loss, -1.0))
    grad = (grad / rows).to(torch.bfloat16).float()
    gw, gb = [None] * 4, [None] * 4
    for layer in (3, 2, 1, 0):
        gw[layer], gb[layer] = grad.T @ acts[layer], grad.sum(0)
        if layer:
            grad = (grad @ model.weight[layer].float()).to(torch.bfloat16).float() * (acts[layer] > 0)
    return float(loss.mean()), float(top1), gw + gb


@pytest.mark.parametrize("rows", [8, 64, 72, 136, 1000, 4096])
def test_train_step_matches_torch(native_lib, rows):
    import torch
    from tdp1375_b200 import order_model as om
    from tdp1375_b200.cases import three_permutation
    torch.backends.cuda.matmul.allow_tf32 = False
    rng = np.random.Generator(np.random.PCG64(rows))
    spi, pi = np.zeros((rows, 64), np.uint8), np.zeros((rows, 64), np.uint8)
    ns, target = np.zeros(rows, np.uint8), np.zeros(rows, np.int32)
    for r in range(rows):
        p, s, _ = three_permutation(int(rng.integers(3, 11)), rng)
        n = len(p)
        spi[r, :n], pi[r, :n], ns[r] = s, p, n
        i, j, k = sorted(int(v) for v in rng.choice(n, 3, replace=False))
        target[r] = om.LEX32[i, j, k]
    d_n, d_t = torch.from_numpy(ns).cuda(), torch.from_numpy(target).cuda()
    x = om.features(torch.from_numpy(spi).cuda(), torch.from_numpy(pi).cuda(), d_n)
    model = om.OrderModel(seed=rows)
    for layer in range(4):
        model.bias[layer].uniform_(-0.1, 0.1)
    want_loss, want_top1, grads = reference_step(model, x, d_n, d_t, 1e-3)
    before = [t.clone() for t in model.master + model.bias]
    loss, top1 = model.train_step(x, d_n, d_t, lr=1e-3)
    assert native_lib.tdp_mlp_error() == 0
    assert abs(loss - want_loss) <= 1e-4 * max(1.0, abs(want_loss))
    assert abs(top1 - want_top1) <= 1.5 / rows  # an argmax between near-equal logits may differ
    after = model.master + model.bias
    for k, g in enumerate(grads):
        got = model.m[k].double() / 0.1  # the first step's moment is a tenth of the gradient
        assert float((got - g.double()).norm()) <= 2.0 ** -8 * float(g.double().norm()) + 1e-12, k
        m, v = model.m[k].double(), model.v[k].double()
        # the update from the moments the library holds
        want = before[k].double() - 1e-3 * (m / (1 - 0.9)) / ((v / (1 - 0.999)).sqrt() + 1e-8)
        if k == 3:
            want[om.TRIPLES:] = 0.0
        assert bool(((after[k].double() - want).abs() <= 1e-6 + 1e-6 * want.abs()).all()), k
    for layer in range(4):
        assert torch.equal(model.weight[layer], model.master[layer].to(torch.bfloat16))


def test_train_step_refuses_rows_of_no_eight(native_lib):
    import torch
    from tdp1375_b200 import order_model as om
    model = om.OrderModel()
    x = torch.zeros(12, om.FEATURES, dtype=torch.bfloat16, device="cuda")
    n = torch.full((12,), 9, dtype=torch.uint8, device="cuda")
    with pytest.raises(RuntimeError, match="multiple of 8"):
        model.train_step(x, n, torch.zeros(12, dtype=torch.int32, device="cuda"))
