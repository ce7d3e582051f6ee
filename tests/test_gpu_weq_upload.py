"""Water-equivalence volumes of 1.7, 6.6 and 10 MB: from pageable memory they go up in pieces
through the page-locked slots (one piece, the slots' last one ragged, and more pieces than
the slots hold), which are made for the 32nd such volume, and by the driver's copy before;
from page-locked memory in one copy. The dose is the same bits, also for a
second volume that follows while the first beam may still run."""
import numpy as np
import pytest
import torch

from _parity import run_gpu
from subsecondpbs_b200 import phantoms

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ray_mm", [1.0, 0.5, 0.4])
def test_pageable_and_page_locked_volumes(ray_mm):
    case = phantoms.weq_case(ray_mm=ray_mm, n_layers=2)
    first = np.array(case["beam"]["water_equivalence"], np.float32)
    second = first.copy()
    second[9:] *= 0.9
    assert first.nbytes > 1 << 20
    doses = []
    for locked in (False, True):
        keep = [torch.from_numpy(v).pin_memory() if locked else torch.from_numpy(v.copy()) for v in (first, second)]
        beams = [dict(case["beam"], water_equivalence=k.numpy()) for k in keep]
        eng = run_gpu(case, beams=beams, keep_debug=False)
        doses.append(eng.read_dose())
        if not locked:
            prepared = [eng.prepare_beam(b) for b in beams]
            for _ in range(20):
                eng.reset_dose()
                for b in prepared:
                    eng.add_beam(b)
            doses.append(eng.read_dose())
        eng.close()
    assert doses[0].max() > 0.0
    assert np.array_equal(doses[0], doses[1]) and np.array_equal(doses[1], doses[2])


def test_slots_shared_by_two_contexts():
    case = phantoms.weq_case(ray_mm=0.5, n_layers=2)
    other = dict(case["beam"], water_equivalence=np.array(case["beam"]["water_equivalence"], np.float32))
    other["water_equivalence"][9:] *= 0.9
    engines = [run_gpu(case, beams=[b], keep_debug=False) for b in (case["beam"], other)]
    want = [e.read_dose() for e in engines]
    prepared = [e.prepare_beam(b) for e, b in zip(engines, (case["beam"], other))]
    for _ in range(25):
        for e, b in zip(engines, prepared):
            e.reset_dose()
            e.add_beam(b)
    got = [e.read_dose() for e in engines]
    for e in engines:
        e.close()
    assert np.array_equal(want[0], got[0]) and np.array_equal(want[1], got[1])
    assert not np.array_equal(want[0], want[1])


def test_slots_shared_by_threads():
    """Six contexts on six threads, more than there are slots to lend."""
    from concurrent.futures import ThreadPoolExecutor

    case = phantoms.weq_case(ray_mm=0.5, n_layers=2)
    base = np.array(case["beam"]["water_equivalence"], np.float32)

    def beam(k):
        v = base.copy()
        v[9:] *= np.float32(1.0 - 0.02 * k)
        return dict(case["beam"], water_equivalence=v)

    def work(k):
        eng = run_gpu(case, beams=[beam(k)], keep_debug=False)
        first = eng.read_dose()
        prepared = eng.prepare_beam(beam(k))
        for _ in range(15):
            eng.reset_dose()
            eng.add_beam(prepared)
        last = eng.read_dose()
        eng.close()
        return first, last

    alone = [work(k)[0] for k in range(6)]
    with ThreadPoolExecutor(6) as pool:
        got = list(pool.map(work, range(6)))
    for want, (first, last) in zip(alone, got):
        assert np.array_equal(want, first) and np.array_equal(want, last)
