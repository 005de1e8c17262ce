"""GPU: a reloaded lattice with sites that hold no atom's code (3, 5, 6 or 7), beside a vacancy.

Such a site never jumps: its rate is 0, and the run leaves it where it is.  With the pair-bond model it binds as a vacancy
does, so the other jumps' energies are those of the same lattice with a vacancy there.  Densities count it as none, up to
the largest code a byte holds, both ways they are built.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOX = (16, 16, 16)


@pytest.mark.parametrize("code", [3, 5, 6, 7])
@pytest.mark.parametrize("model,precision", [(0, 0), (1, 0), (1, 1)])
def test_a_site_without_an_atoms_code_never_jumps(model, precision, code):
    import akmc_b200 as ak

    eam = ak.eam_johnson(42) if model else None

    def engine(occ):
        eng = ak.Engine()
        eng.add_job(ak.job_config(BOX, energy_model=model, precision=precision, eam=eam, seed=2), occ)
        eng.prepare()
        return eng

    iron = np.full(2 * 16 ** 3, ak.FE, np.uint8)
    at = 2 * 3 + 32 * (3 + 16 * 3)   # a vacancy at an even site of the first sector ...
    odd = at + 1                     # ... and its first neighbour up in x, y and z (jump 7)
    one, two = iron.copy(), iron.copy()
    one[at] = two[at] = two[odd] = 0
    other = one.copy()
    other[odd] = code
    with engine(one) as eng, engine(two) as ref:
        eng.load_occupancy(0, other)
        assert eng.calculate(0, 0) > 0 and ref.calculate(0, 0) > 0
        sites, de, rates = eng.calculated_rates()
        assert list(sites) == [at] and rates[0, 7] == 0.0 and de[0, 7] == 0.0 and np.all(rates[0, :7] > 0)
        if model == 0:
            s2, de2, rates2 = ref.calculated_rates()
            k = int(np.nonzero(s2 == at)[0][0])
            assert np.array_equal(de[0], de2[k]) and np.array_equal(rates[0], rates2[k])
        eng.run_rounds(64)
        eng.sync()
        end = eng.occupancy(0)
        assert end[odd] == code and (end == 0).sum() == 1 and (end == ak.FE).sum() == len(iron) - 2


@pytest.mark.parametrize("edge,blocks", [(16, 1), (96, 4)])  # built site by site; by its solutes
def test_densities_do_not_count_other_codes(edge, blocks):
    import akmc_b200 as ak

    box, n = (edge,) * 3, 2 * edge ** 3
    with ak.Engine() as eng:
        one = np.full(n, ak.FE, np.uint8)
        one[0] = 0
        eng.add_job(ak.job_config(box, blocks=(blocks,) * 3, eam=ak.eam_johnson(42)), one)
        eng.prepare()
        codes = np.arange(256, dtype=np.int64)
        others = codes[(codes > 0) & ~np.isin(codes, [ak.FE, ak.CU, ak.NI, ak.MN])].astype(np.uint8)
        at = 1 + np.arange(len(others)) * (n // 300)
        other, vacant = one.copy(), one.copy()
        other[at], vacant[at] = others, 0
        eng.load_occupancy(0, other)
        eng.sync()
        rho = eng.rho(0)
        assert np.array_equal(eng.occupancy(0), other)
        eng.load_occupancy(0, vacant)
        with pytest.raises(ak.AkmcError):  # more vacancies than the job holds; its densities are built all the same
            eng.sync()
        assert np.array_equal(eng.rho(0), rho)
