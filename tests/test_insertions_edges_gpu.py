"""tdp_insertion_extensions_device at the edges of its tiling: smallest and largest max_n, rows
shorter and longer than max_n beside full ones, more slots than one block takes, an output buffer that
allows no 16-byte stores, rows of slots that are no extension left untouched.  Every slot
against the definition (positions move by the number of insertions at or before them)."""
import ctypes
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

vp = ctypes.c_void_p


def spi_rows(rng, sizes):
    """Cycles of 2..5 symbols; every second row runs downwards (no 2-move inside a cycle)."""
    rows = []
    for r, n in enumerate(sizes):
        q, at, spi = rng.permutation(n), 0, list(range(n))
        while at < n:
            size = min(int(rng.integers(2, 6)), n - at)
            if n - at - size == 1:
                size += 1
            cyc = [int(v) for v in q[at:at + size]]
            if r % 2:
                cyc.sort(reverse=True)
            for a, b in zip(cyc, cyc[1:] + cyc[:1]):
                spi[a] = b
            at += size
        rows.append(spi)
    return rows


@pytest.mark.parametrize("max_n,sizes,offset", [(3, [2, 3, 3], 0), (4, [4, 2, 3, 4], 0), (16, [16, 15, 6], 0),
                                                (17, [17, 9], 1), (24, [24, 23, 9, 24], 0), (60, [60, 3, 59], 0),
                                                (9, [12, 33, 9], 0)])
def test_insertion_slots_match_the_definition(native_lib, max_n, sizes, offset):
    import torch
    from tdp1375_b200 import extensions
    rng = np.random.Generator(np.random.PCG64(max_n))
    rows = spi_rows(rng, sizes)
    count, slots = len(rows), int(native_lib.tdp_insertion_extension_slots(max_n))
    spi = np.full((count, 64), 201, np.uint8)  # bytes past n are not part of a row
    for r, s in enumerate(rows):
        spi[r, :len(s)] = s
    d_spi, d_n = torch.from_numpy(spi).cuda(), torch.tensor(sizes, dtype=torch.uint8).cuda()
    gates = torch.zeros(count, dtype=torch.int64, device="cuda")
    flags = torch.full((count * slots,), 9, dtype=torch.uint8, device="cuda")
    out = torch.full((count * slots * 64 + 16,), 77, dtype=torch.uint8, device="cuda")
    rc = native_lib.tdp_insertion_extensions_device(vp(d_spi.data_ptr()), vp(d_n.data_ptr()), count, max_n,
                                                    vp(gates.data_ptr()), vp(flags.data_ptr()),
                                                    vp(out.data_ptr() + offset), vp(0))
    assert rc == 0
    torch.cuda.synchronize()
    got_flags = flags.cpu().numpy().reshape(count, slots)
    raw = out.cpu().numpy()
    got = raw[offset:offset + count * slots * 64].reshape(count, slots, 64)
    assert (raw[:offset] == 77).all() and (raw[offset + count * slots * 64:] == 77).all()
    for r, s in enumerate(rows):
        n = len(s)
        gate = extensions.open_gates(s)
        mask = int(gates[r]) & ((1 << 64) - 1)
        assert {a for a in range(64) if (mask >> a) & 1} == gate
        want_flags = np.zeros(slots, np.uint8)
        want = np.full((slots, 64), 77, np.uint8)
        for e, (a, b, c) in enumerate(itertools.combinations_with_replacement(range(max_n), 3)):
            if c >= n or a == c or (gate and not gate & {a, b, c}):
                continue
            want_flags[e] = 1 if gate else 2
            to = [p + (a <= p) + (b <= p) + (c <= p) for p in range(n)]
            want[e] = 0
            want[e, to] = [to[q] for q in s]
            want[e, [c + 2, b + 1, a]] = [b + 1, a, c + 2]
        assert np.array_equal(got_flags[r], want_flags)
        assert np.array_equal(got[r], want)
