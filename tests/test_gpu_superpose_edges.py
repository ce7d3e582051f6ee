"""The superposition of one spot, the beam of an influence column, at the edges of the
sources' footprints, where the interpolation in rSigma leaves residues of either sign and a
cell that ends below zero is taken as zero.

Bound per cell, absolute: the interpolation misses each source that covers the cell by at
most 2.5e-7 of its own peak; the rest (node tables, node weights, single-precision sums) is
relative to what the widest node spreads there, 1.2e-6 of the cell's own value where that
is large and 1.2e-6 * 0.02 of the peaks at an edge (e^-4.5 of a peak and the nodes' spread
of one another). Together 3e-7 of the covering sources' peaks and 1.2e-6 of the cell."""
import numpy as np
import pytest

import test_gpu_superpose_nodes as nodes
from _parity import run_gpu
from oracle import oracle as O
from subsecondpbs_b200 import _lib as L
from subsecondpbs_b200 import phantoms
from test_gpu_superpose_nodes import PAD

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ray_spacing", [0.35, 1.0, 2.0])
def test_footprint_edges(ray_spacing, monkeypatch):
    case = phantoms.heterogeneous_case(dims=(48, 48, 40), res=(2.0, 2.0, 2.0), target_radius_mm=1.0, n_layers=1,
                                       e_range=(80.0, 80.0), ray_spacing=ray_spacing)
    assert len(case["beam"]["spot_weights"]) == 1
    eng = run_gpu(case)
    st, ls = eng.beam_stats(), eng.layer_stats(0)
    S, (X, Y) = st["tracer_steps"], st["superp_dims"]
    planes = [eng.debug(w, 0, (S, Y, X)) for w in (L.PBS_DBG_IDD, L.PBS_DBG_RSIGMA)]
    codes = eng.debug(L.PBS_DBG_TILE_BINS, 0, (S, Y // 8 * (X // 32)), np.uint8)
    batch = O.batch(np.array(ls["tile_rad_counts"], np.int32))[1]
    want, peaks = np.zeros((2, S, Y + 2 * PAD, X + 2 * PAD))
    nodes._superpose(*planes, codes, batch, want)
    weights = nodes._weights
    monkeypatch.setattr(nodes, "_weights", lambda r, R: np.repeat(weights(r, R)[:, :, :1], R + 1, axis=2))
    nodes._superpose(*planes, codes, batch, peaks)
    got = eng.debug(L.PBS_DBG_BEV_DOSE, 0, want.shape).astype(np.float64)
    eng.close()
    assert got.min() >= 0.0
    assert (np.abs(got - want) <= 3e-7 * peaks + 1.2e-6 * want).all(), (
        (np.abs(got - want) - 1.2e-6 * want) / np.maximum(peaks, 1e-300)).max()
    edge = (want > 0.0) & (want < 1e-6 * want.max())
    assert edge.any()
