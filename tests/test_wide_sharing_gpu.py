"""Launches of many searches that stop at their first sequence share work late: handing out pieces
of a search early widens its front and with it the nodes expanded before the sequence is met (3,000
searches of 8..10 3-cycles in a launch: 1,182 M nodes per 20,000 searches at 16 chunks per poll,
about 960 M by default)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

R1375 = float(np.float32(2) / np.float32(1.375))


@pytest.fixture(scope="module")
def slots(native_lib):
    """Slots of this module alone: other modules destroy and create theirs."""
    from tdp1375_b200 import GPUSortingSearch
    GPUSortingSearch(1, 1, 256 << 20, 1 << 26)
    yield
    GPUSortingSearch.destroySlots()


def test_wide_partial_batches_expand_fewer_nodes(slots):
    """Nodes of the default against those of a poll after 17 chunks (a value the launch takes as it
    is), the same batches in turn."""
    from tdp1375_b200 import api, learned_eval, make_instances, search_batch
    cases = learned_eval.eval_cases(9000)
    nodes = {16: 0, 17: 0}
    cfg = api.engine_config(0)
    assert cfg.poll_interval == 16
    for _ in range(3):
        for poll in nodes:
            cfg.poll_interval = poll
            api.set_engine_config(0, cfg)
            for at in range(0, 9000, 3000):
                part = cases[at:at + 3000]
                res = search_batch(0, make_instances(part, 11, False), len(part), R1375)
                assert all(r.status == 1 for r in res[:len(part)])
                nodes[poll] += api.last_stats(0).nodes
    assert nodes[16] < 0.93 * nodes[17]
