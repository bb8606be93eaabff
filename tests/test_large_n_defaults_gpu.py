"""The restricted enumerations on two symbol words per lane (n > 32) as they run by default: with the
reduction of commuting moves, recency replacement and unprobed leaves."""
import numpy as np
import pytest

from test_large_n_enumeration_gpu import SHAPES, instance

pytestmark = pytest.mark.gpu

R1375 = float(np.float32(2) / np.float32(1.375))


@pytest.fixture(scope="module")
def slots(native_lib):
    """Slots of this module alone: other modules destroy and create theirs."""
    from tdp1375_b200 import GPUSortingSearch
    GPUSortingSearch(1, 1, 256 << 20, 1 << 21)
    yield
    GPUSortingSearch.destroySlots()


@pytest.mark.parametrize("lengths,n,depth,full", SHAPES)
def test_default_modes_match_oracle(slots, oracle, lengths, n, depth, full):
    from tdp1375_b200 import api, make_instances, search_batch
    rng = np.random.Generator(np.random.PCG64([depth, n, len(lengths)]))
    cases = []
    for k in range(2 if depth == 5 else 6):
        pi, spi = instance(rng, n, lengths, k % 2 == 0)
        cases.append((pi, spi, oracle.count_even(spi)))
    want = [oracle.search_gpu_rule([int(x) for x in pi], [int(x) for x in spi], even, R1375, depth, full, dedup=True,
                                   tight=True)[0] for pi, spi, even in cases]
    cfg = api.engine_config(0)
    assert cfg.commute == 1 and cfg.table_replacement == 2 and cfg.probe_leaves == 0 and cfg.sparse_enumeration == 2
    for sparse in (2, 1, 0):
        cfg.sparse_enumeration = sparse
        api.set_engine_config(0, cfg)
        try:
            res = search_batch(0, make_instances(cases, depth, full), len(cases), R1375)
        finally:
            cfg.sparse_enumeration = 2
            api.set_engine_config(0, cfg)
        assert [r.status for r in res] == want, sparse
        for (pi, spi, even), r in zip(cases, res):
            if r.status == 1:
                pos = [[r.positions[3 * d + t] for t in range(3)] for d in range(r.depth)]
                ok, _ = oracle.replay_positions([int(x) for x in pi], [int(x) for x in spi], pos, even, R1375, full)
                assert ok
