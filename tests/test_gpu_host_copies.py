"""The one-shot wrapper's box copies through the page-locked slots: boxes of whole planes
per slot, of rows of one plane, and below the slots' smallest size give the dose of the
resident context, for a dose that holds values and for one that starts at zero."""
import ctypes as C

import numpy as np
import pytest

from subsecondpbs_b200 import _lib as L
from subsecondpbs_b200 import phantoms
from subsecondpbs_b200.cudaCalDoseRTD import _with_luts, raytracedicom_wrapper

from _parity import run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,res", [((48, 48, 40), 2.0), ((150, 131, 67), 1.0), ((1201, 901, 5), 0.1)])
def test_copies(dims, res):
    case = phantoms.heterogeneous_case(dims=(96, 96, 64), n_layers=2, target_radius_mm=10.0)
    case = dict(case, dose_dims=dims, dose_resolution=(res,) * 3, dose_corner=tuple(-0.5 * res * d for d in dims))
    want = run_gpu(case, keep_debug=False).read_dose()
    top = float(want.max())
    assert top > 0.0
    keys = ("ct", "ct_dims", "ct_resolution", "ct_corner", "dose_dims", "dose_resolution", "dose_corner", "beam", "energy")
    got = raytracedicom_wrapper(*(case[k] for k in keys))
    # The deterministic dose but for the legacy sums: bits of single precision.
    assert np.abs(got - want).max() <= 1e-6 * top
    # On top of a dose: single precision of the sum.
    d, keep = L.beam_desc(case["beam"])
    ed, ke = L.energy_desc(_with_luts(case["energy"], None))
    ct = np.ascontiguousarray(case["ct"], np.float32)
    dose = np.linspace(0.0, top, want.size, dtype=np.float32).reshape(want.shape)
    sum64 = dose.astype(np.float64) + want
    fp = C.POINTER(C.c_float)
    L.check(L.load().pbs_subsecond_wrapper(
        ct.ctypes.data_as(fp), L.int3(case["ct_dims"]), L.float3(case["ct_resolution"]), L.float3(case["ct_corner"]),
        dose.ctypes.data_as(fp), L.int3(dims), L.float3(case["dose_resolution"]), L.float3(case["dose_corner"]),
        C.byref(d), 1, C.byref(ed), 0, 0, 0))
    assert np.abs(dose - sum64).max() <= 1e-6 * top
    del keep, ke
