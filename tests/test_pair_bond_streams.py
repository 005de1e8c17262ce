"""GPU: the random streams of a block whose round ends because no event is left (a total rate of 0).

One pair-bond vacancy in its sector draws ahead in batches of 8.  At 107 K nearly all rates are below 2.2e-16 /s, and
round 7 of the first input ends after 24 selections and round 4 of the second after 7520, whole batches.  The streams then
stand where the last selection left them: every later hop, and a run continued from a snapshot, equals the oracle's.
"""
import numpy as np
import pytest

import pyoracle as po
from helpers import assert_same_events, oracle_job

pytestmark = pytest.mark.gpu

BOX = (24, 24, 24)
ALLOY = ((po.FE, 7000), (po.CU, 1500), (po.NI, 1000), (po.MN, 500))


@pytest.mark.parametrize("schedule", [0, 1])  # in one launch; round by round
@pytest.mark.parametrize("temperature,seed,last,selections", [(107.0, 26, 7, 24), (110.0, 32, 4, 7520)])
def test_streams_after_a_round_that_runs_out_of_events(temperature, seed, last, selections, schedule):
    import akmc_b200 as ak

    kw = dict(model=po.MODEL_PAIRBOND, seed=seed, temperature=temperature, window=1e18)
    o = oracle_job(box=BOX, alloy=ALLOY, n_vacancies=4, **kw)
    start = o.occupancy()
    o.run_rounds(16)
    want = o.events()
    assert (want["round"] == last).sum() == selections and np.all(want["n_act"][want["round"] == last] == 1)

    def same(eng, events):
        assert_same_events(eng.events(), events)
        assert np.array_equal(eng.occupancy(0), o.occupancy())
        evo, hops = eng.block_clocks(0)
        evo_o, hops_o = o.block_state()
        assert np.array_equal(hops, hops_o) and np.array_equal(evo.view(np.uint64), evo_o.view(np.uint64))

    def engine():
        eng = ak.Engine(event_log_capacity=1 << 14)
        cfg = ak.job_config(BOX, energy_model=ak.MODEL_PAIRBOND, seed=seed, temperature=temperature, window=1e18)
        eng.add_job(cfg, start)
        eng.prepare()
        eng.set_round_schedule(schedule)
        return eng

    with engine() as eng, engine() as other:
        eng.run_rounds(last + 1)
        eng.sync()
        other.restore_snapshot(0, eng.save_snapshot(0))
        for e in (eng, other):
            e.run_rounds(16 - (last + 1))
            e.sync()
        same(eng, want)
        same(other, want[want["round"] > last])
