"""GPU: the kernel timing mode times the kernels that run without it.

A context's only block runs four rounds or more in one launch under the automatic schedule, timed or not; below that,
and when the schedule is set, a launch a round.  The trajectory is the same.
"""
import numpy as np
import pytest

from helpers import device_job, oracle_job

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("schedule,rounds,launches", [(0, 16, 1), (0, 3, 3), (1, 16, 16), (2, 16, 1)])
def test_timed_launches_are_those_of_the_call(schedule, rounds, launches):
    import akmc_b200 as ak

    o = oracle_job(box=(16, 16, 16), n_vacancies=8, seed=3)
    with ak.Engine() as eng:
        device_job(eng, o, (16, 16, 16), seed=3)
        eng.prepare()
        o.run_rounds(2 * rounds)
        eng.set_round_schedule(schedule)
        eng.run_rounds(rounds)
        eng.set_kernel_timing(True)
        eng.run_rounds(rounds)
        eng.sync()
        ms, n = eng.kernel_timing()
        assert n == launches and ms > 0.0
        assert np.array_equal(eng.occupancy(0), o.occupancy())
