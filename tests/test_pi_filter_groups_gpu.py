"""The group kernels of the permutation filter (n <= 16, 120 candidates per thread) against the
general kernels, which take every call with more than 16 triple symbols: the triple padded with
repeats of its first symbol has the same descents.  Covers the tails below five positions, one
and several blocks, several launches, cycles and triples of every length with repeated symbols,
and row limits inside a group."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _u8(seq):
    return (ctypes.c_uint8 * max(1, len(seq)))(*[int(v) for v in seq])


def run(lib, cycle, triple, n, skip, max_rows):
    out = (ctypes.c_uint8 * (max_rows * n + 64))()
    ctypes.memset(out, 255, max_rows * n + 64)
    hits = lib.tdp_pi_filter(_u8(cycle), len(cycle), _u8(triple), len(triple), n, skip, out, max_rows)
    assert hits >= 0
    rows = min(hits, max_rows)
    raw = np.frombuffer(out, np.uint8)
    assert (raw[rows * n:] == 255).all()  # nothing behind the rows
    return hits, raw[:rows * n].tobytes()


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12])
@pytest.mark.parametrize("skip", [0, 1])
def test_groups_match_general_kernels(native_lib, n, skip):
    rng = np.random.Generator(np.random.PCG64([n, skip]))
    forms = [(rng.permutation(n)[:min(n, size)], rng.permutation(n)[:3]) for size in (0, 1, 2, 3, 4, 5, 7, 9, 12)]
    forms += [(rng.integers(0, n, size), rng.integers(0, n, t)) for size, t in ((3, 3), (5, 1), (7, 2), (16, 16), (4, 9))]
    for cycle, triple in forms:
        padded = [triple[0]] * (17 - len(triple)) + list(triple)
        for max_rows in (0, 1, 1000, 1 << 16):
            assert run(native_lib, cycle, triple, n, skip, max_rows) == \
                run(native_lib, cycle, padded, n, skip, max_rows), (cycle, triple, max_rows)


@pytest.mark.parametrize("skip", [0, 1])
def test_several_launches(native_lib, skip):
    """13!/120 groups take several launches.  A symbol that neither cycle nor triple holds may stand
    at any of the other positions: n times as many hits as without it."""
    cycle, triple = [3, 0, 7, 11, 2, 9, 5], [1, 8, 4]
    fewer, _ = run(native_lib, cycle, triple, 12, skip, 1)
    thirteen, _ = run(native_lib, cycle, triple, 13, skip, 1)
    assert thirteen == 12 * fewer
    hits, raw = run(native_lib, cycle, triple, 14, skip, 200_000)
    assert hits == 13 * thirteen
    rows = np.frombuffer(raw, np.uint8).reshape(-1, 14)
    assert (np.sort(rows, axis=1) == np.arange(14)).all() and (rows[:, 0] == 0).all()
    keys = [bytes(r) for r in rows]
    assert all(a < b for a, b in zip(keys, keys[1:]))  # rank order, no repeats


def test_workspace_is_given_back(native_lib):
    """Calls of growing and shrinking sizes reuse one workspace; destroying the slots frees it."""
    want = {n: run(native_lib, [0, 2, 1, 4, 3], [1, 3, 2], n, 0, 5000) for n in (6, 11, 7, 12)}
    native_lib.tdp_destroy_slots()
    for n in (12, 6, 11, 7, 12):
        assert run(native_lib, [0, 2, 1, 4, 3], [1, 3, 2], n, 0, 5000) == want[n]
