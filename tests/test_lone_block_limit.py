"""GPU: the sweep limit of the dependency-driven schedule is no limit for a context's only block.

Under the automatic schedule its rounds run in one launch of that schedule's kernel, but are reported as round by round,
which never gives up: with a limit of one sweep a call still runs all of its rounds.  Set to the dependency-driven
schedule, the limit holds.
"""
import numpy as np
import pytest

from helpers import device_job, oracle_job

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("room", [{}, dict(max_jobs=4, max_block_edge=16, max_blocks=300, max_vacancies=64)])
def test_a_lone_blocks_rounds_are_all_run(room):
    import akmc_b200 as ak

    o = oracle_job(box=(16, 16, 16), n_vacancies=8, seed=3)
    with ak.Engine(flow_sweep_limit=1, **room) as eng:
        device_job(eng, o, (16, 16, 16), seed=3)
        eng.prepare()
        o.run_rounds(16)
        assert eng.round_schedule() == ak.SCHEDULE_ROUNDS
        eng.run_rounds(16)
        eng.sync()
        assert np.array_equal(eng.occupancy(0), o.occupancy()) and eng.job_state(0)["round"] == 16
        eng.set_round_schedule(ak.SCHEDULE_FLOW)
        eng.run_rounds(16)
        with pytest.raises(ak.AkmcError) as e:
            eng.sync()
        assert e.value.status == -4
