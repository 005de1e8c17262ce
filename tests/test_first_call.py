"""GPU: what a context's first per-hop call and its end cost, and whose answers it gets.

Pinned memory is dear to get (milliseconds), and giving it back waits for all work on the device.  The records that the
per-hop calls and the cluster statistics answer in are pinned once for a device's contexts, 16 of them; a context
without one has its answers copied.  So a context's first call is no slower than a few of the later ones, a context ends
while another stream is busy, and more contexts than records get their own answers all the same.
"""
import threading
import time

import numpy as np
import pytest

import pyoracle as po
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


def _answers(eng):
    """Totals, rates and one event of every sector, and the cluster statistics."""
    out = []
    for sector in range(8):
        total = eng.calculate(0, sector)
        sites, de, rates = eng.calculated_rates()
        order = np.argsort(sites)
        ev = eng.select_and_perform(0, sector, 0.37) if total > 0 else None
        out.append((total, sites[order].tobytes(), de[order].tobytes(), rates[order].tobytes(),
                    (ev.from_site, ev.to_site, ev.species, ev.total) if ev else None))
    iso, hist = eng.cluster_stats(0)
    return out, iso, hist.tobytes()


def _context(seed):
    import akmc_b200 as ak

    o = oracle_job(box=(16, 16, 16), alloy=((po.FE, 90), (po.CU, 10)), n_vacancies=6, seed=seed)
    eng = ak.Engine()
    device_job(eng, o, (16, 16, 16), seed=seed)
    eng.prepare()
    return eng


def test_more_contexts_than_records():
    alone = []
    for seed in range(20):
        with _context(seed) as eng:
            assert len(eng.calculated_rates()[0]) == 0  # none before the first akmc_calculate
            alone.append(_answers(eng))
    for _ in range(2):  # the records come back
        engines = [_context(seed) for seed in range(20)]
        assert [_answers(e) for e in engines] == alone
        for e in engines[::2] + engines[1::2]:
            e.close()
    assert len({repr(a) for a in alone}) == 20  # they are different answers


def test_contexts_come_and_go_in_several_threads():
    want = []
    for seed in range(4):
        with _context(seed) as eng:
            want.append(_answers(eng))
    wrong = []

    def work(k):
        for n in range(10):
            seed = (k + n) % 4
            with _context(seed) as eng:
                if _answers(eng) != want[seed]:
                    wrong.append((k, n))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
