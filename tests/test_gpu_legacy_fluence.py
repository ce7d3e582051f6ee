"""Subspot fluence of the legacy path (one warp per subspot) against the oracle where a
subspot covers less than one group of 32 columns or rows, several of them, or one of
each."""
import numpy as np
import pytest

from subsecondpbs_b200 import phantoms

from _parity import oracle_run, run_gpu, stage_report

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sigma", [(1.0, 1.0), (9.0, 1.0), (1.0, 9.0), (12.0, 12.0)])
def test_ray_weights_match_the_oracle(sigma):
    case = phantoms.heterogeneous_case(dims=(64, 64, 48), n_layers=2, target_radius_mm=14.0)
    beam = phantoms.legacy_beam(case["beam"])
    sub = np.array(beam["subspot_data"])
    sub[..., 3:5] = sigma
    beam = dict(beam, subspot_data=sub)
    eng = run_gpu(case, beams=[beam])
    rep = stage_report(eng, oracle_run(case, beams=[beam], capture=True, capture_layers=True)["capture"])
    # A distance of up to 64 mm carries 4e-6 mm of rounding, which moves an erf by at most
    # 1.13 * 4e-6 / (1.41 * sigma); two ends, two axes, and cells of at least 0.38 of the
    # kernel's height: 3.4e-5, and 1e-5 for a sum of up to 100 single-precision terms.
    assert rep["ray_weight_rel"] < 1e-4
