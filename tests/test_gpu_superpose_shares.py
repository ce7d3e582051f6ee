"""How the warps of the tile superposition share the work items: fewer items than
multiprocessors, fewer than warps, and more than warps, against the definition in 64 bits
(tolerance of test_gpu_superpose_nodes: 3e-6 of the largest BEV cell; an item left out or
taken twice is at least a source's peak)."""
import numpy as np
import pytest

from _parity import run_gpu
from oracle import oracle as O
from subsecondpbs_b200 import _lib as L
from subsecondpbs_b200 import phantoms
from test_gpu_superpose_nodes import PAD, _superpose

pytestmark = pytest.mark.gpu


# One layer: every live tile is an item. 148 multiprocessors with 16 warps of the instance
# for radii up to 15.
@pytest.mark.parametrize("items,kw", [
    ((1, 147), dict(dims=(32, 32, 24), target_radius_mm=0.5, ray_spacing=3.0)),
    ((149, 2367), dict(dims=(48, 48, 40), target_radius_mm=10.0)),
    ((2369, 1 << 20), dict(dims=(128, 128, 96), target_radius_mm=40.0, e_range=(150.0, 150.0)))])
def test_every_item_once(items, kw):
    case = phantoms.heterogeneous_case(**dict(dict(res=(2.0, 2.0, 2.0), n_layers=1, e_range=(66.0, 66.0)), **kw))
    eng = run_gpu(case)
    st, ls = eng.beam_stats(), eng.layer_stats(0)
    S, (X, Y) = st["tracer_steps"], st["superp_dims"]
    bev = np.zeros((S, Y + 2 * PAD, X + 2 * PAD))
    codes = eng.debug(L.PBS_DBG_TILE_BINS, 0, (S, Y // 8 * (X // 32)), np.uint8)
    batch = O.batch(np.array(ls["tile_rad_counts"], np.int32))[1]
    _superpose(eng.debug(L.PBS_DBG_IDD, 0, (S, Y, X)), eng.debug(L.PBS_DBG_RSIGMA, 0, (S, Y, X)), codes, batch, bev)
    got = eng.debug(L.PBS_DBG_BEV_DOSE, 0, bev.shape).astype(np.float64)
    eng.close()
    live = codes[(codes & 0x80 != 0) & (codes != 0xFF)] & 0x3F
    narrow = sum(int((live == q).sum()) for q in range(len(batch)) if batch[q] <= 15)
    assert items[0] <= narrow <= items[1], narrow
    assert np.abs(got - bev).max() <= 3e-6 * bev.max(), np.abs(got - bev).max() / bev.max()
