"""GPU: what a lattice takes of device memory on its way in.

The memory a job is admitted against is its own: its lattice and density rows, with their halos.  An EAM lattice is staged
in the rows of its densities, a pair-bond one through at most 16 Mi sites of the context.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class Pool:
    """The device's default memory pool: the bytes in use, and the most since the last reset."""

    def __init__(self):
        import torch

        torch.zeros(1, device="cuda")
        self.cuda = C.CDLL("libcuda.so.1")
        self.pool = C.c_void_p()
        assert self.cuda.cuDeviceGetDefaultMemPool(C.byref(self.pool), 0) == 0

    def _get(self, attribute):
        v = C.c_uint64()
        assert self.cuda.cuMemPoolGetAttribute(self.pool, attribute, C.byref(v)) == 0
        return v.value

    def used(self):
        return self._get(7)

    def reset(self):
        assert self.cuda.cuMemPoolSetAttribute(self.pool, 8, C.byref(C.c_uint64(0))) == 0
        return self.used()

    def high(self):
        return self._get(8)


def test_an_admitted_job_takes_no_more_than_its_rows():
    import akmc_b200 as ak

    pool = Pool()
    eam = ak.eam_johnson(42)
    with ak.Engine(max_jobs=4, max_block_edge=24, max_blocks=512, max_vacancies=512) as eng:
        small = ak.create_lattice((16, 16, 16), ((ak.FE, 1),), 2, 1)
        eng.add_job(ak.job_config((16, 16, 16), eam=eam), small)
        eng.prepare()
        e, n = 96, 2 * 96 ** 3
        occ = ak.create_lattice((e, e, e), ((ak.FE, 98), (ak.CU, 2)), 30, 1)
        before = pool.reset()
        job = eng.admit_job(ak.job_config((e, e, e), blocks=(4, 4, 4), eam=eam), occ)
        rows = 5 * 240 * e * e  # 192 sites and 48 halo entries a row, a byte and a density each
        assert abs(pool.used() - before - rows) < 65536  # (small tables of the job set come and go)
        assert pool.high() - before < rows + n // 2
        eng.retire_job(job)
        assert pool.used() - before < n // 2


def test_a_pair_bond_lattice_of_more_than_one_portion():
    import akmc_b200 as ak

    box, blocks = (204, 203, 210), (9, 9, 9)
    first, then = (ak.create_lattice(box, ((ak.FE, 97), (ak.CU, 3)), 200, s) for s in (1, 2))
    cfg = ak.job_config(box, blocks=blocks, energy_model=ak.MODEL_PAIRBOND, seed=5)
    ends = []
    for lattice in (first, then):
        with ak.Engine() as eng:
            eng.add_job(cfg, lattice)
            eng.prepare()
            eng.load_occupancy(0, then)
            eng.sync()
            assert np.array_equal(eng.occupancy(0), then)
            eng.run_rounds(8)
            ends.append((eng.occupancy(0), eng.job_state(0)["hops"]))
    assert np.array_equal(ends[0][0], ends[1][0]) and ends[0][1] == ends[1][1] > 0
    with ak.Engine() as eng:
        eng.add_job(cfg, first)
        eng.prepare()
        then[np.nonzero(then == 0)[0][-1]] = ak.FE  # one vacancy short, in the last portion
        eng.load_occupancy(0, then)
        with pytest.raises(ak.AkmcError) as e:
            eng.sync()
        assert e.value.status == -1
