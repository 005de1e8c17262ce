"""GPU: what a context's first per-hop call and its end cost.

The answers of the per-hop calls and of the cluster statistics take no pinned memory, which is dear to get (milliseconds)
and waits for all work on the device when it is given back: a context's first call is no slower than a few of the
later ones, and a context ends while another stream is busy.
"""
import time

import pytest

from helpers import device_job, oracle_job

pytestmark = pytest.mark.gpu


def test_the_first_call_costs_what_later_ones_do_and_the_end_waits_for_nobody():
    import torch

    import akmc_b200 as ak

    o = oracle_job(box=(16, 16, 16), n_vacancies=8, seed=3)
    busy = torch.cuda.Stream()
    first, later, end, waited = [], [], [], []
    for k in range(6):
        eng = ak.Engine()
        device_job(eng, o, (16, 16, 16), seed=3)
        eng.prepare()
        t = [time.perf_counter()]
        for _ in range(4):
            eng.calculate(0, 0)
            eng.cluster_stats(0)
            t.append(time.perf_counter())
        if k:
            with torch.cuda.stream(busy):
                torch.cuda._sleep(100_000_000)  # some 50 ms
            t.append(time.perf_counter())
            eng.close()
            t.append(time.perf_counter())
            waited.append(busy.query())  # the sleep has ended: the context waited for it
            busy.synchronize()
            first.append(t[1] - t[0])
            later.append(min(b - a for a, b in zip(t[1:4], t[2:5])))
            end.append(t[-1] - t[-2])
        else:
            eng.close()
    assert sorted(first)[2] < 8 * sorted(later)[2], (first, later)
    assert sum(waited) < 3 and sorted(end)[2] < 0.01, (waited, end)
