"""Work sharing between warps at every density: a poll after every chunk (more donors than idle
warps), the default and none in practice, on one block per SM and on all, for one search (one warp
starts, all others wait) and for a batch.  Verdicts are the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

R1375 = float(np.float32(2) / np.float32(1.375))


@pytest.fixture(scope="module")
def slots(native_lib):
    """Slots of this module alone: other modules destroy and create theirs."""
    from tdp1375_b200 import GPUSortingSearch
    GPUSortingSearch(1, 1, 256 << 20, 1 << 21)
    yield
    GPUSortingSearch.destroySlots()


@pytest.mark.parametrize("poll", [1, 2, 8, 1 << 20])
@pytest.mark.parametrize("blocks", [0, 1])
def test_verdicts_at_every_sharing_rate(slots, oracle, poll, blocks):
    from tdp1375_b200 import api, make_instances, native, search_batch
    from tdp1375_b200.cases import three_permutation
    rng = np.random.Generator(np.random.PCG64(11))
    cases = [three_permutation(m, rng) for m in (3, 4, 5, 5, 5, 6, 6)]
    want = [oracle.search_gpu_rule(list(map(int, pi)), list(map(int, spi)), even, R1375, 8, True, dedup=True,
                                   tight=True)[0] for pi, spi, even in cases]
    base = api.engine_config(0)
    api.set_engine_config(0, native.EngineConfig(blocks, poll, base.tight_bound, base.task_capacity, base.time_limit_s,
                                                 base.sparse_enumeration))
    try:
        for _ in range(3):
            res = search_batch(0, make_instances(cases, 8, True), len(cases), R1375)
            assert [r.status for r in res] == want
        for case, status in zip(cases, want):
            assert search_batch(0, make_instances([case], 8, True), 1, R1375)[0].status == status
    finally:
        api.set_engine_config(0, base)
