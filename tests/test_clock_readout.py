"""GPU: a job's sector clocks and hops, read from whole block records (up to 192 blocks) or packed on the device first."""
import time

import numpy as np
import pytest

import pyoracle as po
from helpers import QUATERNARY, device_job, oracle_job

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blocks", [(1, 1, 1), (8, 6, 4), (8, 5, 5), (7, 7, 7)])
def test_clocks_of_every_block_equal_the_oracles(blocks):
    import akmc_b200 as ak

    box = tuple(8 * b for b in blocks)
    kw = dict(blocks=blocks, model=po.MODEL_PAIRBOND, seed=4)
    o = oracle_job(box=box, alloy=QUATERNARY, n_vacancies=1 + int(np.prod(blocks)) // 2, **kw)
    with ak.Engine() as eng:
        device_job(eng, oracle_job(box=(8, 8, 8), n_vacancies=1), (8, 8, 8))  # a job before it
        job = device_job(eng, o, box, **kw)
        eng.prepare()
        eng.run_rounds(24)
        evo, hops = eng.block_clocks(job)
    o.run_rounds(24)
    evo_o, hops_o = o.block_state()
    assert np.array_equal(hops, hops_o) and np.array_equal(evo.view(np.uint64), evo_o.view(np.uint64))


def test_one_blocks_clocks_cost_one_copy():
    import akmc_b200 as ak

    def seconds(call):
        t = []
        for _ in range(200):
            t0 = time.perf_counter()
            call()
            t.append(time.perf_counter() - t0)
        return sorted(t)[60]

    o = oracle_job(box=(16, 16, 16), n_vacancies=4)
    with ak.Engine() as eng:
        device_job(eng, o, (16, 16, 16))
        eng.prepare()
        # a job's state is one copy of one record too: 16 us both; packed first, 33
        assert seconds(lambda: eng.block_clocks(0)) < 1.6 * seconds(lambda: eng.job_state(0))
