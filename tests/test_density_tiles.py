"""GPU: a lattice laid out in the device rows and its density build, at the edges of their tiles.

Rows of 16 sites (the smallest box) and of sizes that are no multiple of 16 or 64, planes that end inside a
tile, and both ways a tile is summed: by its solutes (dilute) and site by site (more than 12% solutes).  The
densities are exact integers: they must equal the oracle's.
"""
import numpy as np
import pytest

import pyoracle as po
from helpers import device_job, oracle_job

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cu", [134, 3000])
@pytest.mark.parametrize("box", [(8, 8, 8), (9, 17, 10), (33, 16, 9), (40, 33, 8)])
def test_loaded_lattices_and_densities_equal_the_oracles(box, cu):
    import akmc_b200 as ak

    blocks = tuple(max(1, b // 12) for b in box)
    alloy = ((po.FE, 10000 - cu), (po.CU, cu))
    a, b = (oracle_job(box=box, blocks=blocks, alloy=alloy, n_vacancies=5, seed=s) for s in (3, 4))
    with ak.Engine() as eng:
        for o in (a, b):
            device_job(eng, o, box, blocks=blocks)
        eng.prepare()
        for j, o in enumerate((a, b)):
            assert np.array_equal(eng.rho(j), o.rho())
        # the other lattice into each job: one at a time, then all at once
        eng.load_occupancy(0, b.occupancy())
        eng.sync()
        assert np.array_equal(eng.occupancy(0), b.occupancy()) and np.array_equal(eng.rho(0), b.rho())
        whole = np.concatenate([b.occupancy(), a.occupancy()])
        eng.load_occupancies(whole)
        eng.sync()
        assert np.array_equal(eng.occupancies(), whole)
        assert np.array_equal(eng.rho(0), b.rho()) and np.array_equal(eng.rho(1), a.rho())
