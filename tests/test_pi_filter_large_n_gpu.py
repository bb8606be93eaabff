"""The permutation filter's groups at n = 15 and 16 (group numbers above 2^32 at 16): a triple that
fixes the order of all symbols but two leaves (n-1)(n-2) candidates, spread over the ranks, and the
rows are compared with those of the conditions written out in Python."""
import ctypes
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def in_cyclic_order(index, symbols):
    return sum(index[a] > index[b] for a, b in zip(symbols, symbols[1:] + symbols[:1])) <= 1


def has_2_move(index, cycle):
    size = len(cycle)
    for i, j, k in itertools.combinations(range(size), 3):
        if in_cyclic_order(index, [cycle[i], cycle[j], cycle[k]]) and \
                (j - i) % 2 + (k - j) % 2 + (size - k + i) % 2 - size % 2 == 2:
            return True
    return False


def rows_of(n, cycle, order, skip):
    """Rows that hold 0, order[1:], ... in this order and the other symbols anywhere, filtered."""
    free = [s for s in range(n) if s not in order]
    rows = set()
    for at in itertools.permutations(range(1, n), len(free)):
        row = [None] * n
        for p, s in zip(at, free):
            row[p] = s
        rest = iter(order)
        rows.add(tuple(next(rest) if s is None else s for s in row))
    kept = []
    for row in sorted(rows):
        index = {s: p for p, s in enumerate(row)}
        reverse = {s: n - 1 - p for p, s in enumerate(row)}
        if not in_cyclic_order(reverse, cycle) and (skip or not has_2_move(index, cycle)):
            kept.append(row)
    return kept


@pytest.mark.parametrize("n", [15, 16])
@pytest.mark.parametrize("kind,cycle", [("down", [0, 3, 6, 4, 2]), ("up", [6, 3, 5, 2, 4]), ("mixed", [1, 7, 3, 9, 5, 8])])
def test_rows_at_the_largest_groups(native_lib, n, kind, cycle):
    rng = np.random.Generator(np.random.PCG64(n))
    order = list(range(1, n))
    if kind == "down":
        order.reverse()  # ranks near (n-1)!
    elif kind == "mixed":
        order = [int(v) for v in rng.permutation(order)]
    order = [0] + [s for s in order if s not in (cycle[1], cycle[4])]
    for skip in (0, 1):
        want = rows_of(n, cycle, order, bool(skip))
        out = (ctypes.c_uint8 * (1000 * n))()
        hits = native_lib.tdp_pi_filter((ctypes.c_uint8 * len(cycle))(*cycle), len(cycle),
                                        (ctypes.c_uint8 * len(order))(*order), len(order), n, skip, out, 1000)
        got = np.frombuffer(out, np.uint8).reshape(-1, n)[:max(0, hits)]
        assert hits == len(want)
        assert [tuple(int(v) for v in row) for row in got] == want
        assert skip == 0 or hits > 0
