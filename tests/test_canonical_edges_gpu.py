"""The canonical form where its lane layout has edges: 2n variants just below, at and above a
group of 32, the largest n, one cycle of all symbols, and symmetric configurations whose
variants tie on the hash (the least variant of equal rows must win)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

vp = ctypes.c_void_p


def rotations(n, step):
    """Symmetric under every rotation by gcd: x -> x + step (mod n)."""
    return [(x + step) % n for x in range(n)]


def configurations():
    out = [[1, 0], [1, 2, 0], [2, 0, 1], [1, 0, 3, 2]]
    for n in (6, 12, 15, 16, 17, 31, 32, 33, 48, 62, 63):
        for step in (1, n - 1, 2, 3, n // 2):
            out.append(rotations(n, step))
    rng = np.random.Generator(np.random.PCG64(63))
    for n in (15, 16, 17, 31, 32, 33, 47, 48, 49, 63):
        q = rng.permutation(n)  # one cycle of all n symbols
        p = [0] * n
        for a, b in zip(q, np.roll(q, -1)):
            p[int(a)] = int(b)
        out.append(p)
    return [p for p in out if all(x != y for x, y in enumerate(p))]


def test_canonical_edges_match_oracle(native_lib, oracle):
    perms = configurations()
    spi, ns = np.zeros((len(perms), 64), np.uint8), np.zeros(len(perms), np.uint8)
    for r, p in enumerate(perms):
        spi[r, :len(p)], ns[r] = p, len(p)
    sig = np.zeros((len(perms), 64), np.float32)
    h, v = np.zeros(len(perms), np.int32), np.zeros(len(perms), np.int32)
    assert native_lib.tdp_canonical(spi.ctypes.data_as(vp), ns.ctypes.data_as(vp), len(perms), sig.ctypes.data_as(vp),
                                    h.ctypes.data_as(vp), v.ctypes.data_as(vp)) == 0
    for r, p in enumerate(perms):
        want_sig, want_h, want_v = oracle.canonical(p)
        assert np.array_equal(sig[r, :len(p)], np.array(want_sig, np.float32)), p
        assert (int(h[r]), int(v[r])) == (want_h, want_v), p
        assert not sig[r, len(p):].any()


def test_canonical_device_marks_bad_rows(native_lib):
    """A bad row beside good ones: variant -1, hash 0 and a zero signature, the others as usual."""
    import torch
    rows = [[1, 2, 0], [1, 0, 2], [1, 1, 0], [64, 0, 1], [255, 2, 0], [1, 2, 0]]
    spi = torch.zeros((len(rows) + 2, 64), dtype=torch.uint8)
    for r, p in enumerate(rows):
        spi[r, :3] = torch.tensor(p, dtype=torch.uint8)
    n = torch.tensor([3] * len(rows) + [1, 64], dtype=torch.uint8)
    d_spi, d_n = spi.cuda(), n.cuda()
    sig = torch.full((len(n), 64), 5.0, device="cuda")
    h = torch.full((len(n),), 5, dtype=torch.int32, device="cuda")
    v = torch.full((len(n),), 5, dtype=torch.int32, device="cuda")
    assert native_lib.tdp_canonical_device(vp(d_spi.data_ptr()), vp(d_n.data_ptr()), len(n), vp(sig.data_ptr()),
                                           vp(h.data_ptr()), vp(v.data_ptr()), vp(0)) == 0
    torch.cuda.synchronize()
    good = torch.tensor([True, False, False, False, False, True, False, False])
    assert ((v.cpu() >= 0) == good).all()
    assert (h.cpu()[~good] == 0).all() and not sig.cpu()[~good].any()
    assert torch.equal(sig[0], sig[5]) and h[0] == h[5] and v[0] == v[5] and bool(sig[0].any())
