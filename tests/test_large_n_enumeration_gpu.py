"""The restricted child enumerations on two symbol words per lane (n > 32): every enumeration mode
gives the oracle's verdict and sequences that replay, over cycle structures that reach each mode
(only odd cycles: triples; one even cycle: triples or pairs; several: dense; more same-cycle
triples than the list holds: pairs), on both sides of the 32-position boundary."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

R1375 = float(np.float32(2) / np.float32(1.375))


@pytest.fixture(scope="module")
def slots(native_lib):
    """Slots of this module alone: other modules destroy and create theirs."""
    from tdp1375_b200 import GPUSortingSearch
    GPUSortingSearch(1, 2, 256 << 20, 1 << 21)
    yield
    GPUSortingSearch.destroySlots()


def instance(rng, n, lengths, unoriented):
    """pi a random arrangement; cycles of the given lengths on random symbols, the rest fixed."""
    pi = rng.permutation(n)
    where = np.empty(n, np.int64)
    where[pi] = np.arange(n)
    spi = np.arange(n)
    q, at = rng.permutation(n), 0
    for size in lengths:
        cyc = q[at:at + size]
        if unoriented:
            cyc = cyc[np.argsort(-where[cyc])]
        spi[cyc] = np.roll(cyc, -1)
        at += size
    return pi, spi


SHAPES = [([3] * 11, 33, 3, False), ([3] * 12, 36, 3, False), ([5, 3, 3], 34, 6, True), ([3, 3], 63, 4, True),
          ([4, 4], 34, 5, True), ([4, 3, 2], 35, 5, True), ([2, 2, 3], 33, 4, True), ([7, 3], 40, 5, True),
          ([9], 33, 5, True), ([13], 45, 3, False), ([17, 3, 3], 38, 2, False), ([33], 33, 2, False),
          ([30, 10], 63, 2, False), ([2] * 16, 33, 2, False)]


@pytest.mark.parametrize("lengths,n,depth,full", SHAPES)
def test_enumeration_modes_match_oracle(slots, oracle, lengths, n, depth, full):
    from tdp1375_b200 import api, make_instances, native, search_batch
    rng = np.random.Generator(np.random.PCG64([n, depth, len(lengths)]))
    cases = []
    for k in range(6):
        pi, spi = instance(rng, n, lengths, k % 2 == 0)
        cases.append((pi, spi, oracle.count_even(spi)))
    want = [oracle.search_gpu_rule([int(x) for x in pi], [int(x) for x in spi], even, R1375, depth, full, dedup=True,
                                   tight=True)[0] for pi, spi, even in cases]
    base = api.engine_config(1)
    for sparse in (0, 1, 2):
        for tight in (0, 1):
            api.set_engine_config(1, native.EngineConfig(base.blocks_per_sm, base.poll_interval, tight,
                                                         base.task_capacity, base.time_limit_s, sparse))
            try:
                res = search_batch(1, make_instances(cases, depth, full), len(cases), R1375)
            finally:
                api.set_engine_config(1, base)
            assert [r.status for r in res] == want, (sparse, tight)
            for (pi, spi, even), r in zip(cases, res):
                if r.status == 1:
                    pos = [[r.positions[3 * d + t] for t in range(3)] for d in range(r.depth)]
                    ok, _ = oracle.replay_positions([int(x) for x in pi], [int(x) for x in spi], pos, even, R1375, full)
                    assert ok
