"""LET rows of the biological maps that fit a block's shared memory and rows that do not,
with one and with several depth samples, against the oracle."""
import numpy as np
import pytest

from oracle import oracle as O
from subsecondpbs_b200 import phantoms
from subsecondpbs_b200.cudaCalDoseRTD import DoseEngine

from _parity import DOSE_TOL_FRAC_DMAX

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth_step,samples", [(0.5, 1), (0.5, 6), (320.0 / 12288, 5), (320.0 / 12289, 5), (0.02, 1)])
def test_let_rows(depth_step, samples):
    case = phantoms.heterogeneous_case(dims=(64, 64, 48), n_layers=3, target_radius_mm=14.0)
    bio = phantoms.bio_model("lq", depth_step_mm=depth_step)
    bio["let_samples"] = samples
    eng = DoseEngine(0)
    eng.set_energy(case["energy"])
    eng.set_ct(case["ct"], case["ct_dims"], case["ct_resolution"], case["ct_corner"])
    eng.set_dose_grid(case["dose_dims"], case["dose_resolution"], case["dose_corner"])
    eng.set_bio_model(bio)
    eng.reset_dose()
    eng.add_beam(case["beam"])
    r = O.dose(case, bio=bio)
    hot = r["dose"] > 0.1 * r["dose"].max()
    # The path's own tolerance: the dose's, as for the maps of the other models.
    for name in ("letd", "alpha", "rbe_dose"):
        got, want = eng.read_bio_map(name).astype(np.float64), O.bio_map(bio, r["bio_acc"], name)
        assert float((np.abs(got - want)[hot] / np.abs(want[hot])).max()) < DOSE_TOL_FRAC_DMAX, name
    eng.close()
