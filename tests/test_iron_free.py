"""GPU: boxes without iron under potentials whose density function of iron is far larger than the other species'.

The terms shared by a vacancy's jumps are those of a moving Fe atom.  Where no Fe atom can move they lie off the density
table, which is no error: nothing may depend on iron's tables at all, so the run equals, bit for bit, the one under
tables with a small density function of iron.
"""
import numpy as np
import pytest

import pyoracle as po

pytestmark = pytest.mark.gpu

BOX = (16, 16, 16)


@pytest.mark.parametrize("vacancies", [1, 24])
@pytest.mark.parametrize("precision", [po.FP64, po.FP32C])
def test_irons_tables_do_not_matter_without_iron(precision, vacancies):
    import akmc_b200 as ak

    occ = ak.create_lattice(BOX, ((ak.CU, 9000), (ak.NI, 1000)), vacancies, 5)
    runs = []
    for iron in (0.05, 1.0):
        eam = ak.eam_johnson(42)
        for x in range(4):
            for i in range(5):
                eam.f_shell[x][i] *= iron if x == 0 else 0.05
        cfg = ak.job_config(BOX, energy_model=ak.MODEL_EAM, precision=precision, eam=eam, seed=9)
        with ak.Engine(event_log_capacity=1 << 16) as eng:
            eng.add_job(cfg, occ)
            eng.prepare()
            first = [(eng.calculate(0, s), eng.calculated_rates()) for s in range(8)]
            eng.run_rounds(64)
            eng.sync()  # raises when a density left the table
            runs.append((first, eng.events(), eng.occupancy(0), eng.rho(0), eng.block_clocks(0)))
    (f0, e0, o0, r0, c0), (f1, e1, o1, r1, c1) = runs
    assert len(e0) == len(e1) > 0
    for (t0, rates0), (t1, rates1) in zip(f0, f1):
        assert t0 == t1
        a, b = np.argsort(rates0[0]), np.argsort(rates1[0])
        assert all(np.array_equal(x[a], y[b]) for x, y in zip(rates0, rates1))
    k0, k1 = np.lexsort((e0["hop"], e0["round"])), np.lexsort((e1["hop"], e1["round"]))
    assert e0[k0].tobytes() == e1[k1].tobytes()
    assert np.array_equal(o0, o1) and np.array_equal(r0, r1)
    assert all(np.array_equal(x, y) for x, y in zip(c0, c1))
