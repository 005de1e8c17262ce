"""GPU: a context's only block, whose rounds run in one launch of the persistent kernel.

Vacancy counts around the slots a thread reads at once (64, one each; more than 224, two each), a sector that comes to
hold more than the 64 a block-round takes (380 vacancies: 73 by the ninth round), calls just below and at the number of rounds that takes this way, and a pair-bond vacancy that
stays in its sector for more hops than its path list holds (512).  Everything equals the oracle's, bit for bit.
"""
import numpy as np
import pytest

import pyoracle as po
from helpers import QUATERNARY, assert_same_events, device_job, oracle_job

pytestmark = pytest.mark.gpu


def _same(ak, calls, box, **kw):
    o = oracle_job(box=box, alloy=QUATERNARY, **kw)
    kw.pop("n_vacancies")
    with ak.Engine(event_log_capacity=1 << 20) as eng:
        device_job(eng, o, box, **kw)
        eng.prepare()
        for n in calls:
            eng.run_rounds(n)
        eng.sync()
        o.run_rounds(sum(calls))
        assert_same_events(eng.events(), o.events())
        assert np.array_equal(eng.occupancy(0), o.occupancy())
        evo_d, hops_d = eng.block_clocks(0)
        evo_o, hops_o = o.block_state()
        assert np.array_equal(hops_d, hops_o)
        assert np.array_equal(evo_d.view(np.uint64), evo_o.view(np.uint64))
        assert eng.job_state(0)["round"] == sum(calls) == eng.counters()["rounds"]
        return o.events()


@pytest.mark.parametrize("n_vacancies", [1, 64, 65, 230])
def test_rounds_of_the_only_block_equal_the_oracles(n_vacancies):
    import akmc_b200 as ak

    _same(ak, (3, 4, 1, 17), (24, 24, 24), model=po.MODEL_PAIRBOND, n_vacancies=n_vacancies, seed=5)


@pytest.mark.parametrize("schedule", [0, 1])  # in one launch; round by round
def test_a_sector_that_comes_to_hold_more_than_64_is_reported(schedule):
    import akmc_b200 as ak

    o = oracle_job(box=(24, 24, 24), model=po.MODEL_PAIRBOND, alloy=QUATERNARY, n_vacancies=380, seed=5)
    with ak.Engine() as eng:
        device_job(eng, o, (24, 24, 24), model=po.MODEL_PAIRBOND, seed=5)
        eng.prepare()
        eng.set_round_schedule(schedule)
        eng.run_rounds(25)
        with pytest.raises(ak.AkmcError) as e:
            eng.sync()
        assert e.value.status == -7


def test_a_vacancy_that_fills_its_path_list():
    import akmc_b200 as ak

    ev = _same(ak, (8,), (32, 32, 32), model=po.MODEL_PAIRBOND, n_vacancies=1, seed=29, temperature=420.0,
               window=1e-3)
    assert np.unique(ev["round"], return_counts=True)[1].max() > 512
