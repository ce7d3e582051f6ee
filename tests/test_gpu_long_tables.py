"""A radiation-length table of 240 KB, longer than a block's shared memory: the IDD kernel
does not stage it, so the beam runs. The entries behind the proton table's own repeat its
last value and the dose is the same bits."""
import numpy as np
import pytest

from _parity import run_gpu
from subsecondpbs_b200 import phantoms

pytestmark = pytest.mark.gpu


def test_long_radiation_length_table(hetero_small_case):
    want = run_gpu(hetero_small_case, keep_debug=False).read_dose()
    e = dict(hetero_small_case["energy"])
    t = np.asarray(e["rrl_vector"], np.float32)
    e["rrl_vector"] = np.concatenate([t, np.full(60000 - t.size, t[-1], np.float32)])
    e["n_rrl_samples"] = 60000
    got = run_gpu(dict(hetero_small_case, energy=e), keep_debug=False).read_dose()
    assert want.max() > 0.0
    assert np.array_equal(got, want)
