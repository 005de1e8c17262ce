"""GPU: vacancies that change their block all the time, under the dependency-driven schedule.

Blocks of 8 cells (the smallest), about one vacancy in two blocks and some 20 hops a visit: most rounds are passed over as
empty while neighbours carry vacancies into their sectors, so a mark that came too late would lose hops.  Everything
equals the oracle's, bit for bit.
"""
import numpy as np
import pytest

import pyoracle as po
from helpers import QUATERNARY, assert_same_events, device_job, oracle_job

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("take", [0, 1])
@pytest.mark.parametrize("model,precision,hop_budget", [(po.MODEL_PAIRBOND, po.FP64, 0), (po.MODEL_PAIRBOND, po.FP64, 40000),
                                                        (po.MODEL_EAM, po.FP64, 0)])
def test_hand_overs_between_the_smallest_blocks(model, precision, hop_budget, take):
    import akmc_b200 as ak

    box, blocks = (64, 64, 56), (8, 8, 7)
    kw = dict(blocks=blocks, model=model, precision=precision, seed=11, temperature=800.0, window=1e-8)
    o = oracle_job(box=box, alloy=QUATERNARY, n_vacancies=220, **kw)
    with ak.Engine(event_log_capacity=1 << 20, flow_take=take) as eng:
        device_job(eng, o, box, hop_budget=hop_budget, **kw)
        eng.prepare()
        assert eng.round_schedule() == ak.SCHEDULE_FLOW
        for n in (1, 63, 192):
            eng.run_rounds(n)
        eng.sync()
        if hop_budget:
            o.run(hop_budget, 256)
        else:
            o.run_rounds(256)
        assert_same_events(eng.events(), o.events())
        assert np.array_equal(eng.occupancy(0), o.occupancy())
        evo, hops = eng.block_clocks(0)
        evo_o, hops_o = o.block_state()
        assert np.array_equal(hops, hops_o) and np.array_equal(evo.view(np.uint64), evo_o.view(np.uint64))
