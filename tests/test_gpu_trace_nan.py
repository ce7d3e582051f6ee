"""Entry step of a CT with NaN voxels in the air before the body: a cumulative HU+1000 that
is not below 150 is the entry, so the first NaN sample is (bev_ray_tracing.cu:65-159). Step
counts are whole numbers and have to be the oracle's."""
import numpy as np
import pytest

from _parity import run_gpu
from oracle import oracle as O
from subsecondpbs_b200 import _lib as L
from subsecondpbs_b200 import phantoms

pytestmark = pytest.mark.gpu


# The beam comes in from +x; the NaN slab's distance from the grid's end decides where in
# its depth segment a ray meets it.
@pytest.mark.parametrize("slab", [(76, 77), (82, 83), (85, 90)])
def test_entry_step_of_nan_samples(slab):
    case = phantoms.heterogeneous_case(dims=(96, 48, 40), res=(2.1, 2.0, 2.0), target_radius_mm=10.0, e_range=(66.0, 90.0),
                                       n_layers=2)
    ct = np.full_like(case["ct"], -1000.0)
    ct[:, :, :60] = 0.0
    ct[20:, :, slab[0]:slab[1]] = np.nan
    case["ct"] = ct
    eng = run_gpu(case, keep_debug=True)
    cap = O.dose(case, capture=True)["capture"]
    pl = cap["plan"]
    first = eng.debug(L.PBS_DBG_FIRST_INSIDE, 0, (pl["ray_y"], pl["ray_x"]), np.int32)
    want = np.asarray(cap["first_inside"])
    assert len(np.unique(want)) > 1 and want.max() - want.min() > 8  # rays beside the slab enter at the body
    assert np.array_equal(first, want)
