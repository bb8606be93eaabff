"""Searches on two slots at once: a launch that gets only part of the SMs, because another slot's
search holds the rest, finishes with the blocks it has.  Every launch has a time limit of a few
seconds, so no wait outlasts it."""
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

R1375 = float(np.float32(2) / np.float32(1.375))
R145 = float(np.float32(2) / np.float32(1.45))


@pytest.fixture(scope="module")
def slots(native_lib):
    """Slots of this module alone: other modules destroy and create theirs."""
    from tdp1375_b200 import GPUSortingSearch
    GPUSortingSearch(1, 2, 256 << 20, 1 << 21)
    yield
    GPUSortingSearch.destroySlots()


def config(slot, blocks, limit, per_instance=0):
    from tdp1375_b200 import api
    cfg = api.engine_config(slot)
    cfg.blocks_per_sm, cfg.time_limit_s, cfg.warps_per_instance = blocks, limit, per_instance
    api.set_engine_config(slot, cfg)


def small_cases():
    from tdp1375_b200.cases import three_permutation
    rng = np.random.Generator(np.random.PCG64(11))
    return [three_permutation(m, rng) for m in (3, 4, 5, 5, 6, 6)] + [three_permutation(11, rng)]  # the last: n = 33


def verdicts(oracle, cases, depths):
    return [oracle.search_gpu_rule(list(map(int, pi)), list(map(int, spi)), even, R1375, depth, True, dedup=True,
                                   tight=True)[0] for (pi, spi, even), depth in zip(cases, depths)]


@pytest.mark.parametrize("blocks", [1, 2])
@pytest.mark.parametrize("per_instance", [0, 4096])
def test_small_searches_finish_beside_a_long_one(slots, oracle, blocks, per_instance):
    from tdp1375_b200 import GPUSortingSearch, make_instances, search_batch
    from tdp1375_b200.cases import three_permutation
    cases = small_cases()
    depths = [8] * 6 + [3]
    want = verdicts(oracle, cases, depths)
    config(0, blocks, 20.0)
    config(1, 0, 4.0, per_instance)
    pi, spi, even = three_permutation(10, np.random.Generator(np.random.PCG64(11)))
    # the slot's buffers grow to their size first: freeing memory waits for the whole device
    search_batch(1, make_instances(cases[:1] * 120, 8, True), 120, R1375)
    ended = []

    def long_search():
        try:
            GPUSortingSearch.searchForSortingSeq(list(pi), list(spi), even, R145, 14, True, 0)
            ended.append("finished")
        except RuntimeError as exc:
            ended.append(str(exc))

    t = threading.Thread(target=long_search)
    t.start()
    try:
        time.sleep(0.3)
        got, whole = [], []
        for case, depth in zip(cases, depths):
            got.append(search_batch(1, make_instances([case], depth, True), 1, R1375)[0].status)
        for _ in range(3):
            whole.append([r.status for r in search_batch(1, make_instances(cases[:6] * 20, 8, True), 120, R1375)])
        running = t.is_alive() and not ended
    finally:
        GPUSortingSearch.cancelSort(0)
        t.join(30)
        config(0, 0, 120.0)
        config(1, 0, 120.0)
    assert got == want
    assert all(w == want[:6] * 20 for w in whole)
    assert running, ended  # the small searches did not wait for the long one


def test_two_default_searches_at_once(slots, oracle):
    from tdp1375_b200 import make_instances, search_batch
    cases = small_cases()[:6]
    want = verdicts(oracle, cases, [8] * 6)
    for slot in (0, 1):
        config(slot, 0, 4.0)
    results, errors = {0: [], 1: []}, []

    def worker(slot):
        try:
            for size in (1, 20, 1, 200, 1):
                res = search_batch(slot, make_instances(cases * size, 8, True), 6 * size, R1375)
                results[slot].append([r.status for r in res] == want * size)
        except RuntimeError as exc:
            errors.append(str(exc))

    threads = [threading.Thread(target=worker, args=(slot,)) for slot in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(60)
    for slot in (0, 1):
        config(slot, 0, 120.0)
    assert not errors
    assert results == {0: [True] * 5, 1: [True] * 5}
