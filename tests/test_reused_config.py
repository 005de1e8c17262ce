"""GPU: one JobConfig structure filled anew for each job that is added or admitted.

The library copies it when the job is added: what is read back of a job is of the job, not of the structure's later
contents.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_block_clocks_of_jobs_added_from_one_structure():
    import akmc_b200 as ak

    cfg = ak.job_config((16, 16, 16), blocks=(1, 1, 1), energy_model=ak.MODEL_PAIRBOND)
    occ = ak.create_lattice((16, 16, 16), ((ak.FE, 1),), 3, 1)
    with ak.Engine(max_jobs=4, max_block_edge=16, max_blocks=64, max_vacancies=64) as eng:
        eng.add_job(cfg, occ)
        cfg.blocks[:] = [2, 1, 1]
        eng.add_job(cfg, occ)
        cfg.blocks[:] = [2, 2, 1]
        eng.prepare()
        third = eng.admit_job(cfg, occ)
        cfg.blocks[:] = [0, 0, 2]  # 0: one block
        fourth = eng.admit_job(cfg, occ)
        cfg.blocks[:] = [2, 2, 2]
        for job, n in ((0, 1), (1, 2), (third, 4), (fourth, 2)):
            evo, hops = eng.block_clocks(job)
            assert evo.shape == (n, 8) and hops.shape == (n,) and np.all(hops == 0)
            assert eng.job_state(job)["n_blocks"] == n
        eng.retire_job(third)
        with pytest.raises(ak.AkmcError) as e:
            eng.block_clocks(third)
        assert e.value.status == -9
        again = eng.admit_job(cfg, occ)
        assert eng.block_clocks(again)[0].shape == (8, 8)
