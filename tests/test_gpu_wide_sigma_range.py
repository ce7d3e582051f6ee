"""Superposition and adjoint of items whose sources' rSigma spans 0.0005 to 0.02: two
layers on 0.1 mm rays whose sigmas come from a lateral profile, 70 mm in the layer that
carries the dose and 1.7 mm in one of a ten-thousandth of its weight. Both have the
overflow radius, so every item holds both, and the interpolation has to be exact relative
to the wide sources' own peaks, not the narrow ones'.

Tolerances: the forward's as in test_gpu_superpose_nodes (3e-6 of the largest BEV cell, to
which the wide layer gives most), the adjoint's as in test_gpu_adjoint_nodes (1e-5)."""
import numpy as np
import pytest

from _parity import run_gpu
from oracle import oracle as O
from subsecondpbs_b200 import _lib as L
from subsecondpbs_b200 import phantoms
from test_gpu_superpose_nodes import PAD, _superpose

pytestmark = pytest.mark.gpu

SIGMAS = (100.0, 2.4)  # mm; the profile model takes 1 / sqrt(2) of them


def _case():
    case = phantoms.heterogeneous_case(dims=(48, 48, 40), target_radius_mm=2.0, n_layers=2, e_range=(84.0, 88.0),
                                       ray_spacing=0.1, sigma_range=(2.0, 2.0))
    beam = phantoms.with_carbon_profile(case["beam"])
    prof = beam["profile_data"].reshape(2, -1, 5)
    prof[:, :, 0], prof[:, :, 1], prof[:, :, 4] = 1.0, 0.0, 1.0
    for row, sigma in enumerate(SIGMAS):
        prof[row, :, 2:4] = sigma
    beam["profile_data"] = prof.reshape(-1)
    beam["beam_para_data"] = np.zeros_like(beam["beam_para_data"])
    n = len(beam["spot_weights"]) // 2
    beam["spot_weights"] = (beam["spot_weights"] * np.repeat([1e3, 1e-1], n)).astype(np.float32)
    return case, beam, n


def test_superposition_of_wide_and_narrow_layers():
    case, beam, _ = _case()
    eng = run_gpu(case, beams=[beam], carbon_profile=1)
    st = eng.beam_stats()
    S, (X, Y) = st["tracer_steps"], st["superp_dims"]
    bev = np.zeros((S, Y + 2 * PAD, X + 2 * PAD))
    own = []
    lo = hi = None
    for layer in range(2):
        ls = eng.layer_stats(layer)
        batch = O.batch(np.array(ls["tile_rad_counts"], np.int32))[1]
        idd = eng.debug(L.PBS_DBG_IDD, layer, (S, Y, X))
        rs = eng.debug(L.PBS_DBG_RSIGMA, layer, (S, Y, X))
        codes = eng.debug(L.PBS_DBG_TILE_BINS, layer, (S, Y // 8 * (X // 32)), np.uint8)
        radii = _superpose(idd, rs, codes, batch, bev)[1]
        own.append(bev.max())
        assert radii == {32}
        used = rs[idd > 0]
        lo, hi = (used.min(), used.max()) if layer == 0 else (min(lo, used.min()), max(hi, used.max()))
    got = eng.debug(L.PBS_DBG_BEV_DOSE, 0, bev.shape).astype(np.float64)
    eng.close()
    top = bev.max()
    assert own[0] > 0.5 * top  # the wide layer's peak is that of the whole
    assert lo < 6e-4 and 0.015 < hi < 0.02, (lo, hi)
    assert np.abs(got - bev).max() <= 3e-6 * top, np.abs(got - bev).max() / top


def test_adjoint_of_wide_and_narrow_layers():
    case, beam, n = _case()
    # The wide layer's dose by itself: its range of rSigma is narrow.
    w = np.array(beam["spot_weights"])
    alone = dict(beam, spot_weights=np.where(np.arange(2 * n) < n, w, 0.0).astype(np.float32))
    eng = run_gpu(case, beams=[alone], keep_debug=False, carbon_profile=1)
    dose = eng.read_dose64()
    rng = np.random.Generator(np.random.PCG64(7))
    for axis in range(3):
        g = rng.lognormal(0.0, 0.5, dose.shape)
        g[tuple(slice(axis % 2, None, 2) if i == axis else slice(None) for i in range(3))] = 0.0
        want = float((g * dose).sum())
        assert want > 0.0
        got = float(w[:n].astype(np.float64) @ eng.adjoint_beam(beam, g)[:n].astype(np.float64))
        assert abs(got - want) <= 1e-5 * want, (axis, got / want - 1.0)
    eng.close()
