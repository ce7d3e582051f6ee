"""The transfer's two patches (beams along x, and along y or oblique) on a dose grid whose
sizes fill neither: the dose against the oracle, and the influence rows' norms, summed in
one kernel, against the exported columns."""
import numpy as np
import pytest

from subsecondpbs_b200 import phantoms
from subsecondpbs_b200.cudaCalDoseRTD import DoseEngine
from subsecondpbs_b200.precision import max_rel_err

from _parity import oracle_run, run_gpu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def case():
    c = phantoms.heterogeneous_case(dims=(96, 96, 64), n_layers=3, target_radius_mm=14.0)
    return dict(c, dose_dims=(45, 37, 29), dose_resolution=(3.3, 2.7, 3.1), dose_corner=(-74.0, -50.0, -43.0))


@pytest.mark.parametrize("angle", [0.0, 20.0, 90.0, 255.0])
def test_dose_and_norms(case, angle):
    beam = phantoms.rotate_beam(case["beam"], angle)
    eng = run_gpu(case, beams=[beam], keep_debug=False)
    want = oracle_run(case, beams=[beam])["dose"]
    # The path's bound for FP32 arithmetic against the FP64 oracle.
    assert max_rel_err(eng.read_dose(), want) < 1e-4
    # Columns in single precision (6e-8 each, squared 1.2e-7), norms rounded once.
    a = eng.influence_csc(beam).astype(np.float64)
    rows = np.asarray(a.multiply(a).sum(axis=1)).ravel()
    got = eng.influence_row_norms(beam).ravel()
    assert rows.max() > 0
    assert np.abs(got - rows).max() <= 5e-7 * rows.max()
    assert np.all(np.abs(got - rows) <= 5e-7 * rows + 1e-37)
    eng.close()
