"""GPU: the two ways a lattice's densities are built, by its solutes and site by site.

A launch of fewer than 148 large tiles, and a job with more than a tenth of solutes, goes site by site; many small boxes in
one context, or one large box, by their solutes.  The densities are exact integers: they must equal the oracle's.
"""
import time

import numpy as np
import pytest

import pyoracle as po
from helpers import device_job, oracle_job

pytestmark = pytest.mark.gpu


def _alloy(cu):
    return ((po.FE, 10000 - cu), (po.CU, cu))


def test_many_ragged_boxes_of_both_sorts_in_one_context():
    import akmc_b200 as ak

    boxes = [(8, 8, 8), (9, 17, 10), (33, 16, 9), (40, 33, 8)] * 10
    jobs = [(b, oracle_job(box=b, blocks=tuple(max(1, e // 12) for e in b), alloy=_alloy(cu), n_vacancies=5, seed=s))
            for s, (b, cu) in enumerate([(b, cu) for b in boxes for cu in (134, 3000)])]
    with ak.Engine() as eng:
        for b, o in jobs:
            device_job(eng, o, b, blocks=tuple(max(1, e // 12) for e in b))
        eng.prepare()
        for turned in (False, True):  # as prepared; then each lattice with its axes reversed
            if turned:
                occ = [o.occupancy()[::-1].copy() for _, o in jobs]
                for (_, o), x in zip(jobs, occ):
                    o.set_occupancy(x)
                eng.load_occupancies(np.concatenate(occ))
                eng.sync()
            for k, (_, o) in enumerate(jobs):
                assert np.array_equal(eng.rho(k), o.rho()), k


@pytest.mark.parametrize("first,then", [(134, 134), (134, 3000), (3000, 134)])
def test_a_large_box_reloaded_with_another_composition(first, then):
    import akmc_b200 as ak

    kw = dict(box=(100, 99, 97), blocks=(7, 7, 7), n_vacancies=20)
    a, b = (oracle_job(alloy=_alloy(cu), seed=s, **kw) for cu, s in ((first, 1), (then, 2)))
    with ak.Engine() as eng:
        device_job(eng, a, kw["box"], blocks=kw["blocks"])
        eng.prepare()
        assert np.array_equal(eng.rho(0), a.rho())
        eng.load_occupancy(0, b.occupancy())
        eng.sync()
        assert np.array_equal(eng.rho(0), b.rho())


def test_a_small_boxs_load_does_not_depend_on_its_solutes():
    import akmc_b200 as ak

    def seconds(cu):
        occ = ak.create_lattice((20, 20, 20), _alloy(cu), 4, 7)
        with ak.Engine() as eng:
            eng.add_job(ak.job_config((20, 20, 20), eam=ak.eam_johnson(42), seed=3), occ)
            eng.prepare()
            best = 1.0
            for _ in range(30):
                t = time.perf_counter()
                eng.load_occupancy(0, occ)
                eng.sync()
                best = min(best, time.perf_counter() - t)
            return best

    assert seconds(5000) < 1.35 * seconds(134)  # 57 and 58 us; 110 and 65 by solutes
