"""GPU: the per-hop entry points on a job that has ended (its rounds or its hop budget).

A finished job has no events: its total rate is 0, nothing is selected, and its lattice, hops and clocks stay.
"""
import numpy as np
import pytest

import pyoracle as po
from helpers import device_job, oracle_job

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("end", [dict(max_rounds=8), dict(hop_budget=1)])
@pytest.mark.parametrize("model", [po.MODEL_PAIRBOND, po.MODEL_EAM])
def test_a_finished_job_has_no_events(model, end):
    import akmc_b200 as ak

    o = oracle_job(box=(16, 16, 16), model=model, n_vacancies=20, seed=3)
    with ak.Engine() as eng:
        device_job(eng, o, (16, 16, 16), model=model, seed=3, **end)
        eng.prepare()
        assert sum(eng.calculate(0, s) > 0 for s in range(8)) > 0
        eng.run_rounds(8)
        eng.sync()
        state, occ = eng.job_state(0), eng.occupancy(0)
        assert state["done"] and state["hops"] > 0
        for s in range(8):
            assert eng.calculate(0, s) == 0.0
            assert len(eng.calculated_rates()[0]) == 0
            ev = eng.select_and_perform(0, s, 0.5)
            assert ev.from_site == -1 and ev.total == 0.0
        assert eng.job_state(0) == state and np.array_equal(eng.occupancy(0), occ)
        eng.load_occupancy(0, o.occupancy())  # restarted: its events are back
        assert sum(eng.calculate(0, s) > 0 for s in range(8)) > 0
