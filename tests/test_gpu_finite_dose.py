"""The one-shot call on a dose of zeros says whether the dose is finite, and the Python face
raises where it is not. Each beam, or each layer where the layers are transferred one by one
(the reference's depth convention), is within single precision and their sum is not."""
import ctypes as C
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from subsecondpbs_b200 import _lib as L
from subsecondpbs_b200 import phantoms
from subsecondpbs_b200.cudaCalDoseRTD import _with_luts, raytracedicom_wrapper

pytestmark = pytest.mark.gpu

KEYS = ("ct", "ct_dims", "ct_resolution", "ct_corner", "dose_dims", "dose_resolution", "dose_corner", "beam", "energy")


def case_of(scale):
    """Eight layers of one energy; tables in units of 1e-9, so that the weights are smaller
    than the dose and within single precision like it."""
    case = phantoms.heterogeneous_case(dims=(64, 48, 40), n_layers=8, e_range=(80.0, 80.0), target_radius_mm=8.0)
    case["energy"] = dict(case["energy"], cidd_matrix=np.asarray(case["energy"]["cidd_matrix"]) * np.float32(1e9))
    w = np.asarray(case["beam"]["spot_weights"], np.float64) * scale
    assert w.max() < 1e38
    case["beam"] = dict(case["beam"], spot_weights=w.astype(np.float32))
    return case


def _call(case, n_beams, finite):
    d, keep = L.beam_desc(case["beam"])
    ed, ke = L.energy_desc(_with_luts(case["energy"], None))
    beams = (type(d) * n_beams)(*[d] * n_beams)
    ct = np.ascontiguousarray(case["ct"], np.float32)
    dims = case["dose_dims"]
    dose = np.zeros(dims[::-1], np.float32)
    fp = C.POINTER(C.c_float)
    rc = L.load().pbs_subsecond_wrapper_zeroed(
        ct.ctypes.data_as(fp), L.int3(case["ct_dims"]), L.float3(case["ct_resolution"]), L.float3(case["ct_corner"]),
        dose.ctypes.data_as(fp), L.int3(dims), L.float3(case["dose_resolution"]), L.float3(case["dose_corner"]),
        beams, n_beams, C.byref(ed), 0, 0, 0, None if finite is None else C.byref(finite))
    del keep, ke
    return rc, dose


def test_sum_of_beams_beyond_single_precision():
    finite = C.c_int(-1)
    rc, dose = _call(case_of(1.0), 2, finite)
    assert rc == L.PBS_OK and finite.value == 1 and np.isfinite(dose).all()
    case = case_of(2.5e38 / (0.5 * float(dose.max())))
    for n_beams in (1, 2):
        finite = C.c_int(-1)
        rc, dose = _call(case, n_beams, finite)
        assert rc == L.PBS_OK and finite.value == (n_beams == 1) and np.isfinite(dose).all() == (n_beams == 1)
    assert _call(case, 1, None)[0] == L.PBS_ERR_INVALID_ARGUMENT


def test_python_face_raises():
    case = case_of(1.0)
    top = float(raytracedicom_wrapper(*(case[k] for k in KEYS)).max())
    code = ("import sys; sys.path[:0] = {path!r}; import test_gpu_finite_dose as t\n"
            "case = t.case_of({scale!r})\n"
            "try:\n    t.raytracedicom_wrapper(*(case[k] for k in t.KEYS))\n"
            "except RuntimeError as e:\n    print('raised', e)\nelse:\n    print('returned')\n")
    here = Path(__file__).resolve().parent
    for scale, want in ((1e37 / top, "returned"), (6e38 / top, "raised raytracedicom_wrapper produced non-finite")):
        r = subprocess.run([sys.executable, "-c", code.format(path=[str(here), str(here.parent)], scale=scale)],
                           capture_output=True, text=True, env=dict(os.environ, PBS_COMPAT_BEV_Z_SHIFT="1"), timeout=300)
        assert r.returncode == 0 and r.stdout.startswith(want), r.stdout + r.stderr
