"""The element-wise kernels of the C ABI that the training step does not go through, the GEMM's
128-wide tiles with element stores, and the optimiser in the middle of a training, against plain
PyTorch in 64 bits.

Tolerances.  A sum of R fp32 values in any order: |err| <= R * 2^-23 * sum |x|.  A moment is two
products and a sum: 3 * 2^-23 of its terms.  The update divides by bias corrections 1 - beta^step
whose powf is good to 2 ulp, 2^-22 / (1 - beta2^step) <= 2^-18 at the steps below, and takes the
root of half of that; the other operations add a few 2^-23."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

vp = ctypes.c_void_p


def ptr(t):
    return vp(t.data_ptr())


@pytest.mark.parametrize("rows,cols", [(1, 8), (31, 40), (33, 64), (64, 100), (1000, 1088), (129, 5120)])
def test_transpose_and_column_sums(native_lib, rows, cols):
    import torch
    g = torch.Generator(device="cpu").manual_seed(rows + cols)
    a = torch.randn(rows, cols, generator=g).to(torch.bfloat16).cuda()
    out = torch.full((cols * rows + 8,), 7.0, device="cuda", dtype=torch.bfloat16)
    assert native_lib.tdp_mlp_transpose(ptr(a), rows, cols, ptr(out), vp(0)) == 0
    sums = torch.full((cols + 8,), 7.0, device="cuda")
    assert native_lib.tdp_mlp_column_sums(ptr(a), rows, cols, ptr(sums), vp(0)) == 0
    torch.cuda.synchronize()
    assert torch.equal(out[:cols * rows].view(cols, rows), a.T)
    bound = rows * 2.0 ** -23 * a.double().abs().sum(0)
    assert bool(((sums[:cols].double() - a.double().sum(0)).abs() <= bound).all())
    assert bool((out[cols * rows:] == 7.0).all()) and bool((sums[cols:] == 7.0).all())


@pytest.mark.parametrize("count", [1, 255, 257, 1_000_003])
def test_relu_backward(native_lib, count):
    import torch
    g = torch.Generator(device="cpu").manual_seed(count)
    act = torch.relu(torch.randn(count, generator=g)).to(torch.bfloat16).cuda()
    grad = torch.randn(count, generator=g).to(torch.bfloat16).cuda()
    want = torch.where(act > 0, grad, torch.zeros_like(grad))
    assert native_lib.tdp_mlp_relu_backward(ptr(grad), ptr(act), count, vp(0)) == 0
    torch.cuda.synchronize()
    assert torch.equal(grad, want)


def adam_64(w, g, m, v, step, lr=1e-3):
    b1, b2, eps = (float(np.float32(x)) for x in (0.9, 0.999, 1e-8))
    m1 = b1 * m + (1 - b1) * g
    v1 = b2 * v + (1 - b2) * g * g
    return m1, v1, float(np.float32(lr)) * (m1 / (1 - b1 ** step)) / ((v1 / (1 - b2 ** step)).sqrt() + eps)


@pytest.mark.parametrize("count,step", [(1, 100), (1025, 20), (300_001, 1000)])
def test_adam(native_lib, count, step):
    import torch
    gen = torch.Generator(device="cpu").manual_seed(count)
    w, g = (torch.randn(count, generator=gen).cuda() for _ in range(2))
    m, v = torch.randn(count, generator=gen).cuda(), torch.rand(count, generator=gen).cuda()
    low = torch.empty(count, dtype=torch.bfloat16, device="cuda")
    want_m, want_v, update = adam_64(w.double(), g.double(), m.double(), v.double(), step)
    want_w = w.double() - update
    bound_m = 2.0 ** -21 * (m.double().abs() + g.double().abs())
    bound_v = 2.0 ** -21 * (v.double() + g.double() ** 2)
    f = ctypes.c_float
    rc = native_lib.tdp_mlp_adam(ptr(w), ptr(low), ptr(g), ptr(m), ptr(v), count, f(1e-3), f(0.9), f(0.999), f(1e-8),
                                 step, vp(0))
    assert rc == 0
    torch.cuda.synchronize()
    assert bool(((m.double() - want_m).abs() <= bound_m).all())
    assert bool(((v.double() - want_v).abs() <= bound_v).all())
    slack = 2.0 ** -17 * update.abs() + 2.0 ** -17 * 1e-3 * bound_m / 2.0 ** -21 + 2.0 ** -22 * w.double().abs()
    assert bool(((w.double() - want_w).abs() <= slack).all())
    assert torch.equal(low, w.to(torch.bfloat16))


@pytest.mark.parametrize("rows,step", [(136, 100), (1000, 19)])
def test_train_step_in_the_middle_of_a_training(native_lib, rows, step):
    """Moments away from zero: the fused optimiser's decays and bias corrections."""
    import torch
    from tdp1375_b200 import order_model as om
    from tdp1375_b200.cases import three_permutation
    from test_mlp_train_gpu import reference_step
    torch.backends.cuda.matmul.allow_tf32 = False
    rng = np.random.Generator(np.random.PCG64(rows))
    spi, pi = np.zeros((rows, 64), np.uint8), np.zeros((rows, 64), np.uint8)
    ns, target = np.zeros(rows, np.uint8), np.zeros(rows, np.int32)
    for r in range(rows):
        p, s, _ = three_permutation(int(rng.integers(3, 11)), rng)
        n = len(p)
        spi[r, :n], pi[r, :n], ns[r] = s, p, n
        i, j, k = sorted(int(q) for q in rng.choice(n, 3, replace=False))
        target[r] = om.LEX32[i, j, k]
    d_n, d_t = torch.from_numpy(ns).cuda(), torch.from_numpy(target).cuda()
    x = om.features(torch.from_numpy(spi).cuda(), torch.from_numpy(pi).cuda(), d_n)
    model = om.OrderModel(seed=rows)
    model.step = step
    gen = torch.Generator(device="cuda").manual_seed(rows)
    for k in range(8):
        model.m[k] = torch.randn(model.m[k].shape, generator=gen, device="cuda") * 1e-3
        model.v[k] = torch.rand(model.v[k].shape, generator=gen, device="cuda") * 1e-5 + 1e-7
    m0, v0 = [t.double() for t in model.m], [t.double() for t in model.v]
    before = [t.double() for t in model.master + model.bias]
    _, _, grads = reference_step(model, x, d_n, d_t, 1e-3)
    model.train_step(x, d_n, d_t, lr=1e-3)
    assert native_lib.tdp_mlp_error() == 0 and model.step == step + 1
    after = [t.double() for t in model.master + model.bias]
    b1, b2 = float(np.float32(0.9)), float(np.float32(0.999))
    for k, g in enumerate(grads):
        g = g.double()
        m, v = model.m[k].double(), model.v[k].double()
        # a gradient's norm may be off by 2^-8 (bf16 roundings), so its square by twice that times
        # its largest element
        assert float((m - (b1 * m0[k] + (1 - b1) * g)).norm()) <= \
            0.1 * 2.0 ** -8 * float(g.norm()) + 2.0 ** -21 * float(m0[k].norm()), k
        assert float((v - (b2 * v0[k] + (1 - b2) * g * g)).norm()) <= \
            1e-3 * 2.0 ** -6 * float(g.norm()) * float(g.abs().max()) + 2.0 ** -21 * float(v0[k].norm()), k
        update = float(np.float32(1e-3)) * (m / (1 - b1 ** (step + 1))) / ((v / (1 - b2 ** (step + 1))).sqrt() + 1e-8)
        want = before[k] - update
        if k == 3:
            want[om.TRIPLES:] = 0.0
        assert bool(((after[k] - want).abs() <= 2.0 ** -17 * update.abs() + 2.0 ** -22 * before[k].abs()).all()), k


@pytest.mark.parametrize("fp32", [True, False])
def test_wide_gemm_tiles_with_element_stores(native_lib, fp32):
    """128-wide tiles into rows of a stride that TMA does not store."""
    import torch
    m, n, k, ldo = 2500, 1000, 128, 1001
    g = torch.Generator(device="cpu").manual_seed(9)
    a = torch.randn(m, k, generator=g).to(torch.bfloat16).cuda()
    b = torch.randn(n, k, generator=g).to(torch.bfloat16).cuda()
    bias = torch.randn(n, generator=g).cuda()
    out = torch.full((m + 1, ldo), 7.0, device="cuda", dtype=torch.float32 if fp32 else torch.bfloat16)
    assert native_lib.tdp_mlp_gemm(ptr(a), ptr(b), m, n, k, ptr(bias), 1, ptr(out), int(fp32), ldo, vp(0)) == 0
    torch.cuda.synchronize()
    assert native_lib.tdp_mlp_error() == 0
    ref = torch.relu(a.double() @ b.double().T + bias.double())
    bound = (k + 1) * 2.0 ** -23 * (a.double().abs() @ b.double().abs().T + bias.abs())
    if not fp32:
        bound = bound + 2.0 ** -8 * ref.abs()
    assert bool(((out[:m, :n].double() - ref).abs() <= bound).all())
    assert bool((out[m:] == 7.0).all()) and bool((out[:, n:] == 7.0).all())
