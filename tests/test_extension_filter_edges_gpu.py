"""The extension filter at the edges of its tiling (one block per 512 triples of a base, 16-byte
clears): smallest and largest n, one and several blocks per base, cycles of every length,
arbitrary pi, and a keep buffer at an odd address, byte for byte against the oracle."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

vp = ctypes.c_void_p


def base(rng, n, longest, unoriented):
    """One base: pi a random arrangement, spi cycles of 1..longest symbols; unoriented: every
    cycle runs downwards along pi."""
    pi = rng.permutation(n)
    where = np.empty(n, np.int64)
    where[pi] = np.arange(n)
    spi = np.arange(n)
    q, at = rng.permutation(n), 0
    while at < n:
        cyc = q[at:at + int(rng.integers(1, longest + 1))]
        if unoriented:
            cyc = cyc[np.argsort(-where[cyc])]
        spi[cyc] = np.roll(cyc, -1)
        at += len(cyc)
    return spi, pi


@pytest.mark.parametrize("n,longest,unoriented", [(3, 3, False), (4, 4, True), (9, 3, True), (19, 3, True),
                                                  (20, 5, True), (20, 7, False), (33, 3, True), (60, 60, True),
                                                  (60, 4, True)])
def test_extension_filter_edges_match_oracle(native_lib, oracle, n, longest, unoriented):
    import torch
    L = oracle.lib()
    L.oracle_extension_filter.restype = ctypes.c_int64
    rng = np.random.Generator(np.random.PCG64([n, longest, int(unoriented)]))
    count = 2 if n == 60 else 7
    rows = [base(rng, n, longest, unoriented) for _ in range(count)]
    spi, pi = np.zeros((count, 64), np.uint8), np.zeros((count, 64), np.uint8)
    for r, (s, p) in enumerate(rows):
        spi[r, :n], pi[r, :n] = s, p
    per = native_lib.tdp_extension_count(n)
    want = b""
    for r in range(count):
        out = (ctypes.c_uint8 * per)()
        L.oracle_extension_filter(oracle._u8(spi[r, :n]), oracle._u8(pi[r, :n]), n, out)
        want += bytes(out)
    d_spi, d_pi = torch.from_numpy(spi).cuda(), torch.from_numpy(pi).cuda()
    for offset in (0, 1, 15):
        keep = torch.full((count * per + 64,), 7, dtype=torch.uint8, device="cuda")
        rc = native_lib.tdp_extension_filter_device(vp(d_spi.data_ptr()), vp(d_pi.data_ptr()), n, count,
                                                    vp(keep.data_ptr() + offset), vp(0))
        assert rc == 0
        torch.cuda.synchronize()
        got = keep.cpu().numpy()
        assert got[offset:offset + count * per].tobytes() == want
        assert (got[:offset] == 7).all() and (got[offset + count * per:] == 7).all()
