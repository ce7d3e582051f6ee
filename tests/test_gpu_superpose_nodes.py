"""The tile superposition against its definition (complete_superposition.cu:264-335) in
64 bits, on the library's own IDD, rSigma and tile radii.

The cases reach the edges of the interpolation in rSigma: more than 32 layers of one
tile (two groups of the work list), radii above 15 and at the overflow bucket, radii
below 3 (erfc weights), and a density step along the field that spreads one tile's
rSigma over more than one node range.

Tolerance, relative to the largest BEV cell: the interpolation is within 2.5e-7 of a
source's peak, the two node table factors are each within 3e-7, and the node weights,
with a Lebesgue constant of about 2 and some ten roundings of 6e-8, within 1.2e-6; the
sum stays below 3e-6. The errors are not of one sign: the BEV total has to agree to 1e-6."""
import numpy as np
import pytest

from oracle import oracle as O
from subsecondpbs_b200 import _lib as L
from subsecondpbs_b200 import phantoms

pytestmark = pytest.mark.gpu

PAD = 32


def _case(name):
    kw = dict(dims=(48, 48, 40), res=(2.0, 2.0, 2.0), target_radius_mm=10.0, e_range=(66.0, 90.0), n_layers=3)
    kw.update({"one_layer": dict(n_layers=1, e_range=(80.0, 80.0)), "forty_layers": dict(n_layers=40),
               "fine_rays": dict(ray_spacing=0.35), "finest_rays": dict(ray_spacing=0.1, target_radius_mm=2.0, n_layers=1),
               "coarse_rays": dict(ray_spacing=3.0), "density_step": dict(), "density_step_across": dict(dims=(96, 48, 40))}[name])
    case = phantoms.heterogeneous_case(**kw)
    if name.startswith("density_step"):
        # The beam travels along -x: dense and thin halves side by side, along z (the
        # tiles' short side) or y (within the tiles' rows). A ray leaves the body at its
        # last step above HU -850, so the thin half of the first case is dead.
        if name == "density_step":
            ct = np.full_like(case["ct"], -850.0)
            ct[ct.shape[0] // 2:] = 1400.0
        else:
            ct = np.full_like(case["ct"], -600.0)
            ct[:, ct.shape[1] // 2:] = 2000.0
        case["ct"] = ct
    return case


def _weights(r, R):
    """e_r(0..R) of every source, [n][256][R + 1]."""
    special = pytest.importorskip("scipy.special")
    edge = special.erf(r[:, :, None] * (np.arange(R + 1) + 0.5))
    e = edge.copy()
    e[:, :, 1:] = 0.5 * (edge[:, :, 1:] - edge[:, :, :-1])
    return e


def _superpose(idd, rs, codes, batch, bev):
    """Adds one layer's live tiles to bev; idd, rs [S][Y][X], codes [S][tiles]. Returns the
    largest ratio of rSigma within a tile and the radii met."""
    S, Y, X = idd.shape
    ty, tx = Y // 8, X // 32
    tiles = lambda v: v.reshape(S, ty, 8, tx, 32).transpose(0, 1, 3, 2, 4).reshape(S * ty * tx, 256)  # noqa: E731
    i, r, c = tiles(idd), tiles(rs), codes.reshape(-1)
    # Steps past the layer's end have code 0xff.
    live = np.nonzero((c & 0x80).astype(bool) & (c != 0xFF))[0]
    radius = np.array([batch[q & 0x3F] for q in c[live]], int)
    sy, sx = np.divmod(np.arange(256), 32)
    ratio = 1.0
    for R in np.unique(radius):
        for n in np.array_split(live[radius == R], max(1, int((radius == R).sum()) // 64)):
            dose = np.where(i[n] > 0.0, i[n], 0.0).astype(np.float64)
            s = np.where(i[n] > 0.0, r[n], 1.0).astype(np.float64)
            ratio = max(ratio, float((np.where(dose > 0, s, 0).max(axis=1) / np.where(dose > 0, s, np.inf).min(axis=1)).max()))
            e = _weights(s, R)

            def spread(extent, at):
                d = np.abs(np.arange(extent)[None, :] - R - at[:, None])
                v = np.take_along_axis(e, np.broadcast_to(np.minimum(d, R)[None], (len(n),) + d.shape), axis=2)
                return np.where(d <= R, v, 0.0)

            f = np.einsum("nsy,nsx->nyx", spread(8 + 2 * R, sy), spread(32 + 2 * R, sx) * dose[:, :, None], optimize=True)
            for q, t in enumerate(n):
                k, tile = divmod(int(t), ty * tx)
                y0, x0 = tile // tx * 8 - R + PAD, tile % tx * 32 - R + PAD
                bev[k, y0:y0 + 8 + 2 * R, x0:x0 + 32 + 2 * R] += f[q]
    return ratio, set(np.unique(radius).tolist())


@pytest.mark.parametrize("name", ["one_layer", "forty_layers", "fine_rays", "finest_rays", "coarse_rays", "density_step",
                                  "density_step_across"])
def test_superposition_matches_its_definition(name):
    from _parity import run_gpu

    case = _case(name)
    eng = run_gpu(case)
    st = eng.beam_stats()
    S, (X, Y) = st["tracer_steps"], st["superp_dims"]
    bev = np.zeros((S, Y + 2 * PAD, X + 2 * PAD))
    ratio, radii = 1.0, set()
    for layer in range(st["num_layers"]):
        ls = eng.layer_stats(layer)
        batch = O.batch(np.array(ls["tile_rad_counts"], np.int32))[1]
        idd = eng.debug(L.PBS_DBG_IDD, layer, (S, Y, X))
        rs = eng.debug(L.PBS_DBG_RSIGMA, layer, (S, Y, X))
        codes = eng.debug(L.PBS_DBG_TILE_BINS, layer, (S, Y // 8 * (X // 32)), np.uint8)
        q, met = _superpose(idd, rs, codes, batch, bev)
        ratio, radii = max(ratio, q), radii | met
    got = eng.debug(L.PBS_DBG_BEV_DOSE, 0, bev.shape).astype(np.float64)
    top = bev.max()
    assert top > 0.0
    assert np.abs(got - bev).max() <= 3e-6 * top, np.abs(got - bev).max() / top
    assert abs(got.sum() - bev.sum()) <= 1e-6 * bev.sum(), got.sum() / bev.sum() - 1.0
    # The cases reach what they are for.
    if name == "forty_layers":
        assert st["num_layers"] > 32 and st["layer_chunks"] == 1
    if name == "fine_rays":
        assert max(radii) > 15
    if name == "finest_rays":
        assert 32 in radii
    if name == "coarse_rays":
        assert min(radii) <= 1
    if name == "density_step_across":
        assert ratio > 1.6
