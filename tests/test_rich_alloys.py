"""GPU: jobs most of whose atoms are solutes, whose several vacancies are evaluated jump by jump, not by the terms of a
moving Fe atom.

The way is chosen by the first lattice; the results are the oracle's either way, also for a reloaded lattice of another
composition.  An evaluation costs more there (each jump's 76 sites are its own), but no more than jump by jump on all
warps: in a box of Cu at most 1.75 times that in a box of Fe (measured 1.33-1.59; 1.97-2.48 on half of the warps).
"""
import time

import numpy as np
import pytest

import pyoracle as po
from helpers import assert_same_events, device_job, oracle_job

pytestmark = pytest.mark.gpu

RICH = ((po.FE, 1500), (po.CU, 7000), (po.NI, 1000), (po.MN, 500))
POOR = ((po.FE, 7500), (po.CU, 2500))


@pytest.mark.parametrize("alloy,reload", [(RICH, RICH), (RICH, POOR), (POOR, RICH)])
@pytest.mark.parametrize("precision", [po.FP64, po.FP32C])
@pytest.mark.parametrize("warps", [8, 4])
def test_a_rich_alloys_runs_equal_the_oracles(warps, precision, alloy, reload):
    import akmc_b200 as ak

    kw = dict(box=(32, 18, 16), blocks=(2, 1, 1), precision=precision, seed=6, n_vacancies=40)
    first, o = oracle_job(alloy=alloy, **kw), oracle_job(alloy=reload, **kw)
    box = kw.pop("box")
    kw.pop("n_vacancies")
    with ak.Engine(event_log_capacity=1 << 18, eval_warps=warps) as eng:
        device_job(eng, first, box, **kw)
        eng.prepare()
        eng.load_occupancy(0, o.occupancy())
        eng.run_rounds(48)
        eng.sync()
        o.run_rounds(48)
        assert_same_events(eng.events(), o.events())
        assert np.array_equal(eng.occupancy(0), o.occupancy()) and np.array_equal(eng.rho(0), o.rho())


@pytest.mark.parametrize("precision", [po.FP64, po.FP32C])
def test_a_rich_alloys_rates_equal_the_oracles(precision):
    import akmc_b200 as ak

    o = oracle_job(box=(16, 16, 16), alloy=RICH, precision=precision, n_vacancies=40, seed=6)
    seen = 0
    with ak.Engine() as eng:
        device_job(eng, o, (16, 16, 16), precision=precision, seed=6)
        eng.prepare()
        for sector in range(8):
            eng.calculate(0, sector)
            for site, de, rates in zip(*eng.calculated_rates()):
                _, r, d = o.vacancy_rates(int(site))
                assert np.array_equal(rates, r) and np.array_equal(de[r > 0], d[r > 0])
                seen += 1
    assert seen == 40


@pytest.mark.parametrize("warps", [8, 4])
def test_a_box_of_copper_is_evaluated_by_all_warps(warps):
    import akmc_b200 as ak

    eam = ak.eam_johnson(42)

    def seconds_an_evaluation(code):
        occ = ak.create_lattice((20, 20, 20), ((code, 1),), 40, 7)
        with ak.Engine(eval_warps=warps) as eng:
            eng.add_job(ak.job_config((20, 20, 20), eam=eam, seed=3), occ)
            eng.prepare()
            best = 1.0
            for _ in range(5):
                eng.load_occupancy(0, occ)
                eng.sync()
                n = eng.counters()["evaluations"]
                t = time.perf_counter()
                eng.run_rounds(64)
                eng.sync()
                t = time.perf_counter() - t
                best = min(best, t / (eng.counters()["evaluations"] - n))
            return best

    assert seconds_an_evaluation(ak.CU) < 1.75 * seconds_an_evaluation(ak.FE)
