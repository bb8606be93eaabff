"""Device memory that finished calls of the permutation filter leave for later ones: bounded over all
threads, given back by tdp_destroy_slots, and no reason for a call to fail."""
import ctypes
import threading

import pytest

pytestmark = pytest.mark.gpu

CYCLE, TRIPLE = [0, 2, 1, 4, 3, 6, 5], [1, 3, 2]
MB = 1 << 20


def run(lib, max_rows, n=12, out=None):
    c = (ctypes.c_uint8 * len(CYCLE))(*CYCLE)
    t = (ctypes.c_uint8 * 3)(*TRIPLE)
    return lib.tdp_pi_filter(c, len(CYCLE), t, 3, n, 0, out, max_rows)


def leave_idle(lib, max_rows):
    """Calls from eight threads at once."""
    hits = []

    def worker():
        for _ in range(20):
            hits.append(run(lib, max_rows))

    threads = [threading.Thread(target=worker) for _ in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(set(hits)) == 1 and hits[0] > 0
    return hits[0]


def free_bytes():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("max_rows", [1 << 20, 3_000_000, 5_000_000])  # 18, 42 and 66 MB a call
def test_idle_memory_is_bounded_and_given_back(native_lib, max_rows):
    run(native_lib, 1, n=6)  # the module is loaded
    native_lib.tdp_destroy_slots()
    before = free_bytes()
    leave_idle(native_lib, max_rows)
    held = before - free_bytes()
    assert 0 < held <= 96 * MB + 16 * MB  # 16: each set's 2-MB granules, pinned staging
    native_lib.tdp_destroy_slots()
    assert free_bytes() >= before - 2 * MB


def test_idle_memory_does_not_make_a_call_fail(native_lib):
    """Two idle sets of 42 MB and 40 MB free: 104 MB of rows fit once both sets are given back."""
    import torch
    native_lib.tdp_destroy_slots()
    hits = leave_idle(native_lib, 3_000_000)
    filler = []
    try:
        for step in (1 << 30, 64 * MB, 8 * MB):
            while free_bytes() > 40 * MB + step:
                filler.append(torch.empty(max(step, (free_bytes() - 40 * MB) // step * step), dtype=torch.uint8,
                                          device="cuda"))
        assert run(native_lib, 8_700_000) == hits
        # out of memory all the same: an error of this call alone
        assert run(native_lib, 39_916_800) == -4  # 479 MB
        assert b"memory" in native_lib.tdp_last_error()
        assert run(native_lib, 1000) == hits
    finally:
        del filler[:]
        torch.cuda.empty_cache()
        native_lib.tdp_destroy_slots()
