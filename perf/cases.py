"""Performance cases of the dose library: what its users have it compute, through the
package's public entry points, from one layer in a small water box to a 20,000-spot
field on a 1 mm CT.

`call` says which entry point a case runs:
  dose      DoseEngine.reset_dose / add_beam / read_dose with CT, tables and grid resident
  gradient  autograd.plan_dose, an FP64 least-squares objective and its gradient with
            respect to every spot weight (one step of an inverse planner)
  norms     DoseEngine.influence_row_norms over a target (columns of the influence matrix)
  bio       DoseEngine.add_beam with an LQ model set, then the RBE-weighted dose map
  wrapper   raytracedicom_wrapper, the drop-in call: host arrays in, host dose out
`fluence` is how the beam gives its spots: lattice (spot lists), legacy (subspot table)
or weq (a CarbonPBS water-equivalence export).
"""
import math

import numpy as np
import torch

from subsecondpbs_b200 import phantoms
from subsecondpbs_b200.autograd import plan_dose
from subsecondpbs_b200.cudaCalDoseRTD import DoseEngine, plan_beam, raytracedicom_wrapper

PITCH_MM = 5.0  # spot pitch of every field, as in the benchmark

_BASE = dict(call="dose", fluence="lattice", ion="proton", halo=False, phantom="body", beams=1, gantry=90.0, sad=2000.0,
             ray=1.0, sigma_lo=3.0, sigma_hi=6.0, spots=0)


def _case(**kw):
    return dict(_BASE, **kw)


def listed():
    return [
        # One energy layer of 91 spots in a water box: the smallest plan there is (QA of a
        # single layer, a commissioning run). Launches and host planning dominate.
        _case(name="water_1_layer", phantom="water", nx=64, ny=64, nz=128, res=2.0, layers=1, e_lo=150.0, e_hi=150.0,
              radius=25.0, gantry=0.0, sad=10000.0, sigma_lo=4.0, sigma_hi=4.0),
        # A small oblique field on a small CT (the parity tests' mid size).
        _case(name="small_oblique", nx=96, ny=96, nz=64, res=2.0, layers=6, e_lo=70.0, e_hi=150.0, radius=20.0,
              gantry=30.0),
        # The benchmark's beam: 20 layers, 3020 spots on a 2 mm CT of 256 x 256 x 160.
        _case(name="headline", nx=256, ny=256, nz=160, res=2.0, layers=20, e_lo=70.0, e_hi=180.0, radius=32.0),
        # Odd grid sizes, spacing, ray pitch, layer count and angle, two beams.
        _case(name="odd_sizes", nx=187, ny=203, nz=91, res=2.3, layers=13, e_lo=83.0, e_hi=171.0, radius=27.0,
              gantry=217.0, beams=2, ray=1.3),
        # A large target on a 1 mm CT: the largest field of the serving stream (20,000 spots).
        _case(name="fine_20k_spots", nx=512, ny=512, nz=200, res=1.0, layers=40, e_lo=70.0, e_hi=180.0, radius=59.0),
        # Carbon ions with the nuclear halo, three fields of 40 layers on a 1 mm CT.
        _case(name="carbon_halo", ion="carbon", halo=True, nx=512, ny=512, nz=200, res=1.0, layers=40, e_lo=120.0,
              e_hi=400.0, radius=29.0, gantry=0.0, beams=3),
        # One iteration of an inverse planner: four beams of 36 layers, dose, objective, gradient.
        _case(name="plan_gradient", call="gradient", phantom="water", nx=64, ny=64, nz=128, res=2.0, layers=36,
              e_lo=66.0, e_hi=112.0, radius=39.0, gantry=0.0, beams=4, sad=10000.0, sigma_lo=4.0, sigma_hi=4.0),
        # Influence-matrix columns: the row norms over the target of 192 spots of the benchmark's beam.
        _case(name="influence_192", call="norms", nx=256, ny=256, nz=160, res=2.0, layers=20, e_lo=70.0, e_hi=180.0,
              radius=32.0, spots=192),
        # A CarbonPBS export: the transport comes in as water-equivalent depths.
        _case(name="weq_import", fluence="weq", nx=128, ny=128, nz=96, res=2.0, layers=10, e_lo=70.0, e_hi=130.0,
              radius=24.0),
        # Legacy beams without spot lists: the rays span the whole projected grid.
        _case(name="legacy_fluence", fluence="legacy", nx=96, ny=96, nz=64, res=2.0, layers=6, e_lo=70.0, e_hi=130.0,
              radius=24.0),
        # Biological optimisation: RBE-weighted dose of one field under an LQ model.
        _case(name="rbe_map", call="bio", nx=128, ny=128, nz=96, res=2.0, layers=12, e_lo=75.0, e_hi=150.0, radius=26.0),
        # The drop-in call of the reference's Python module, everything on the host.
        _case(name="wrapper_host", call="wrapper", nx=256, ny=256, nz=160, res=2.0, layers=20, e_lo=70.0, e_hi=180.0,
              radius=32.0),
    ]


def draw(rng):
    """A case of the ranges above. Its cost stays within the largest listed case's."""
    most = max(work(c)["flops"] for c in listed())

    def log(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    while True:
        kind = rng.choice(["dose", "dose", "dose", "multi", "halo", "gradient", "norms", "weq", "legacy", "bio",
                           "wrapper"])
        nx, ny, nz = int(round(log(56, 512))), int(round(log(56, 512))), int(round(log(48, 200)))
        res = round(rng.uniform(1.0, 3.0), 2)
        lateral = min(nx, ny, nz) * res
        thick = 0.9 * min(nx, ny) * res
        carbon = kind == "halo"
        # Ranges that end inside the body, within the tables' energies.
        r_hi = min(rng.uniform(0.45, 0.85) * thick, 265.0 if carbon else 290.0)
        r_lo = max(rng.uniform(0.4, 0.9) * r_hi, 36.0 if carbon else 33.0)
        if r_hi < 40.0 or nx * ny * nz > 512 * 512 * 200:
            continue
        a, p = (270.0 / 400.0 ** 1.675, 1.675) if carbon else (0.022, 1.77)
        radius = round(min(log(8.0, 60.0), 0.4 * lateral), 1)
        small = kind in ("gradient", "legacy", "bio", "weq")
        c = _case(call={"gradient": "gradient", "norms": "norms", "bio": "bio", "wrapper": "wrapper"}.get(kind, "dose"),
                  fluence=kind if kind in ("weq", "legacy") else "lattice", ion="carbon" if carbon else "proton",
                  halo=carbon, nx=nx, ny=ny, nz=nz, res=res, layers=int(round(log(1, 24 if small else 40))),
                  e_lo=round((r_lo / a) ** (1.0 / p), 1), e_hi=round((r_hi / a) ** (1.0 / p), 1), radius=radius,
                  gantry=round(rng.uniform(0.0, 360.0), 1), beams=rng.randint(2, 4) if kind in ("multi", "gradient") else 1,
                  ray=rng.choice([1.0, 1.0, 1.5, 2.0]), sad=rng.choice([2000.0, 10000.0]),
                  spots=rng.randint(16, 192) if kind == "norms" else 0)
        if small and nx * ny * nz > 160 ** 3:
            continue
        if kind == "legacy" and max(nx, ny, nz) * res > 260.0:
            continue  # the legacy ray grid spans the projected dose grid
        if kind == "gradient" and _rays(c) * c["layers"] * max(nx, ny) > 4e7:
            continue  # every layer of a gradient's beam has to fit the layer budget
        if kind == "norms" and len(phantoms.hex_spots(radius, PITCH_MM)) * c["layers"] < c["spots"]:
            continue
        if work(c)["flops"] <= most:
            return c


# ---- inputs -----------------------------------------------------------------------


def _rays(case):
    """Rays under the field: the spot disc with three sigma around it."""
    return (2.0 * (case["radius"] + 3.0 * case["sigma_hi"]) / case["ray"] + 1.0) ** 2


def _mean_depth(case):
    a, p = (270.0 / 400.0 ** 1.675, 1.675) if case["ion"] == "carbon" else (0.022, 1.77)
    return 0.5 * a * (case["e_lo"] ** p + case["e_hi"] ** p)


def work(case):
    """Bytes: the CT read and the dose written once (FP64 dose and its gradient in the
    planning step). FLOPs: per depth step, energy layer and ray under the field about 50
    for the depth dose and sigma, and 60 to spread it laterally (two passes of a 15-tap
    Gaussian); transposed once more for a gradient, per spot for influence columns, per
    channel for the biological map."""
    voxels = case["nx"] * case["ny"] * case["nz"]
    ray_steps = _rays(case) * _mean_depth(case) / case["res"]
    per_layer = ray_steps * 110.0
    n = case["layers"] * case["beams"]
    byts = 8.0 * voxels
    flops = per_layer * n
    if case["call"] == "gradient":
        byts += 16.0 * voxels
        flops *= 2.0
    elif case["call"] == "norms":
        # A spot lights three sigma around itself.
        spot = (6.0 * case["sigma_hi"] / case["ray"]) ** 2 * _mean_depth(case) / case["res"]
        flops = spot * 110.0 * case["spots"]
    elif case["call"] == "bio":
        flops += per_layer * n * 60.0 / 110.0 * 3.0
    return {"bytes": byts, "flops": flops}


def _ct(case, gen):
    """The package's heterogeneous phantom (body ellipsoid, lung slab, two bone
    cylinders; HU) or a water box (HU + 1000 = 1000), made on the GPU: [Z][Y][X]."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["phantom"] == "water":
        return torch.full((nz, ny, nx), 1000.0, device="cuda")
    z = torch.arange(nz, device="cuda").float()[:, None, None] - (nz - 1) / 2.0
    y = torch.arange(ny, device="cuda").float()[None, :, None] - (ny - 1) / 2.0
    x = torch.arange(nx, device="cuda").float()[None, None, :] - (nx - 1) / 2.0
    noise = torch.randn((nz, ny, nx), device="cuda", generator=gen)
    body = (x / (0.45 * nx)) ** 2 + (y / (0.45 * ny)) ** 2 + (z / (0.45 * nz)) ** 2 <= 1.0
    lung = (y > 0.10 * ny) & (y < 0.30 * ny) & (z.abs() < 0.30 * nz)
    r2 = (0.05 * min(nx, ny)) ** 2
    bone = ((x + 0.18 * nx) ** 2 + (y + 0.12 * ny) ** 2 <= r2) | ((x - 0.20 * nx) ** 2 + (y + 0.20 * ny) ** 2 <= r2)
    hu = torch.where(lung, -800.0 + 50.0 * noise, 20.0 * noise)
    hu = torch.where(bone, 950.0 + 120.0 * noise.clamp(-2.0, 2.0), hu)
    return torch.where(body, hu, torch.full_like(hu, -1000.0)).contiguous()


def _grid(case):
    dims = (case["nx"], case["ny"], case["nz"])
    res = (case["res"],) * 3
    return dims, res, tuple(-0.5 * (d - 1) * case["res"] for d in dims)


def _energy(case):
    return phantoms.carbon_tables() if case["ion"] == "carbon" else phantoms.proton_tables()


def _beams(case, rng):
    L = case["layers"]
    spots = phantoms.hex_spots(case["radius"], PITCH_MM)
    energies = np.linspace(case["e_lo"], case["e_hi"], L).astype(np.float32)
    sig = np.linspace(case["sigma_hi"], case["sigma_lo"], L).astype(np.float32)
    counts = np.full(L, len(spots), np.int32)
    base = {
        "energies": energies, "spot_sigmas": np.stack([sig, sig], axis=1), "ray_spacing": (case["ray"],) * 2, "steps": 0,
        "source_dist": (case["sad"],) * 2, "spot_offset": (0.0, 0.0, 0.0),
        "spot_delta": (PITCH_MM, PITCH_MM * math.sqrt(3.0) / 2.0, 0.0), "sad": case["sad"],
        "layer_spot_counts": counts, "spot_positions": np.tile(spots, (L, 1)).reshape(-1),
        "subspot_data": phantoms.subspot_lut(L, 7, sig, rng),
    }
    out = []
    for k in range(case["beams"]):
        b = phantoms.rotate_beam(base, case["gantry"] + 360.0 * k / case["beams"])
        b["spot_weights"] = rng.lognormal(0.0, 0.5, int(counts.sum())).astype(np.float32)
        if case["fluence"] == "legacy":
            b = phantoms.legacy_beam(b)
        elif case["fluence"] == "weq":
            b = _with_weq(case, b, rng)
        out.append(b)
    return out


def _with_weq(case, beam, rng):
    """The beam as a CarbonPBS export: depths per lateral texel and step behind the
    9-value header, spot positions as texel coordinates (phantoms.weq_case)."""
    dims, res, corner = _grid(case)
    st = plan_beam(beam, _energy(case), dims, res, corner, dims, res, corner)
    step, n_steps = abs(float(st["fan_delta"][2])), int(st["tracer_steps"])
    depth0 = 0.5 * sum(float(v) for v in st["source_dist"]) - float(st["fan_corner"][2])
    n_xy = 2 * int(math.ceil((case["radius"] + 3.0 * case["sigma_hi"] + 8.0) / case["ray"])) + 1
    weq, x0 = phantoms.weq_volume(n_xy, case["ray"], n_steps, step, rng)
    header = np.array([depth0, step, n_steps, x0, case["ray"], n_xy, x0, case["ray"], n_xy], np.float32)
    pos = beam["spot_positions"].reshape(-1, 2)
    return dict(beam, water_equivalence=np.concatenate([header, weq.reshape(-1)]), ray_weq_header=header,
                spot_positions=((pos - np.float32(x0)) / case["ray"] + 0.5).astype(np.float32).reshape(-1),
                spot_positions_are_indices=True)


def _target(case):
    """Linear indices of a target sphere at the isocentre and of a shell around it."""
    dims, res, corner = _grid(case)
    ax = [torch.arange(dims[i], device="cuda") * res[i] + corner[i] for i in (2, 1, 0)]
    r = (ax[0][:, None, None] ** 2 + ax[1][None, :, None] ** 2 + ax[2][None, None, :] ** 2).sqrt().reshape(-1)
    rt = min(25.0, 0.8 * case["radius"])
    return torch.nonzero(r <= rt).reshape(-1), torch.nonzero((r > rt) & (r <= rt + 20.0)).reshape(-1)


def _inputs(case, seed):
    gen = torch.Generator("cuda").manual_seed(seed)
    rng = np.random.Generator(np.random.PCG64(seed))
    return _ct(case, gen), _beams(case, rng)


def prepare(case, seed):
    ct, beams = _inputs(case, seed)
    grid = _grid(case)
    s = {"case": case, "energy": _energy(case), "grid": grid, "beams": beams}
    if case["call"] == "wrapper":
        s["ct"] = ct.cpu().numpy()
        return s
    e = DoseEngine(0)
    e.set_energy(s["energy"])
    e.set_ct(ct, *grid)
    e.set_dose_grid(*grid)
    e.synchronize()
    s["engine"] = e
    s["out"] = torch.empty((case["nz"], case["ny"], case["nx"]), device="cuda")
    if case["call"] == "gradient":
        w = np.concatenate([b["spot_weights"] for b in beams])
        s["weights"] = torch.from_numpy(w).cuda().requires_grad_()
        s["target"], s["shell"] = _target(case)
        return s
    s["prepared"] = [e.prepare_beam(b) for b in beams]
    if case["call"] == "norms":
        s["voxels"] = _target(case)[0].cpu().numpy()
        total = len(beams[0]["spot_weights"])
        s["begin"] = int(np.random.Generator(np.random.PCG64(seed + 1)).integers(total - case["spots"] + 1))
    elif case["call"] == "bio":
        e.set_bio_model(phantoms.bio_model("lq"))
    return s


PRESCRIPTION_GY = 2.0


def _objective(dose, target, shell):
    """FP64 least squares: the prescription in the target, nothing in the shell."""
    d = dose.reshape(-1)
    return ((d[target] - PRESCRIPTION_GY) ** 2).mean() + (d[shell] ** 2).mean()


def run(s):
    case = s["case"]
    if case["call"] == "wrapper":
        return raytracedicom_wrapper(s["ct"], *s["grid"], *s["grid"], s["beams"][0], s["energy"])
    e = s["engine"]
    if case["call"] == "gradient":
        loss = _objective(plan_dose(s["weights"], e, s["beams"]), s["target"], s["shell"])
        (grad,) = torch.autograd.grad(loss, s["weights"])
        return {"loss": loss.detach().float(), "grad": grad}
    if case["call"] == "norms":
        return e.influence_row_norms(s["prepared"][0], s["voxels"], s["begin"], case["spots"])
    e.reset_dose()
    for b in s["prepared"]:
        e.add_beam(b, nuclear_correction=case["halo"])
    if case["call"] == "bio":
        return e.read_bio_map("rbe_dose", s["out"])
    return e.read_dose(s["out"])


# ---- the same results in 64 bits ----------------------------------------------------
# The method restated in plain torch: coordinates and planning decisions in 32-bit
# floats, as the method defines them, everything that carries dose in 64 bits.

TILE_X, TILE_Y, PAD = 32, 8, 32
F = np.float32


def exact(case, seed):
    if case["fluence"] != "lattice" or case["call"] in ("norms", "bio"):
        return None
    ct, beams = _inputs(case, seed)
    hu = ct.double() if case["phantom"] == "water" else ct.double() + 1000.0
    plans = [_Plan(case, b, hu) for b in beams]
    dose = torch.zeros((case["nz"], case["ny"], case["nx"]), dtype=torch.float64, device="cuda")
    for p in plans:
        for bev, geo in p.bevs(case["halo"]):
            dose += p.transfer(bev, geo)
    if case["call"] != "gradient":
        return dose.cpu().numpy() if case["call"] == "wrapper" else dose
    dose.requires_grad_()
    loss = _objective(dose, *_target(case))
    (g,) = torch.autograd.grad(loss, dose)
    return {"loss": loss.detach(), "grad": torch.cat([p.gradient(g) for p in plans])}


def _dot(a, b):
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]


def _cross(a, b):
    return np.array([a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]], F)


def _unit(v):
    v = np.asarray(v, F)
    n = np.sqrt(_dot(v, v))
    return (v / n).astype(F) if n > 1e-8 else v


def _mul(m, v):
    return np.array([_dot(r, v) for r in m], F)


def _matmul(a, b):
    return np.array([[_dot(r, b[:, j]) for j in range(3)] for r in a], F)


def _inv(m):
    a, b, c = m
    det = (a[0] * (b[1] * c[2] - b[2] * c[1]) - a[1] * (b[0] * c[2] - b[2] * c[0])
           + a[2] * (b[0] * c[1] - b[1] * c[0]))
    adj = np.array([[b[1] * c[2] - b[2] * c[1], a[2] * c[1] - a[1] * c[2], a[1] * b[2] - a[2] * b[1]],
                    [b[2] * c[0] - b[0] * c[2], a[0] * c[2] - a[2] * c[0], a[2] * b[0] - a[0] * b[2]],
                    [b[0] * c[1] - b[1] * c[0], a[1] * c[0] - a[0] * c[1], a[0] * b[1] - a[1] * b[0]]], F)
    return _matmul(adj, np.diag(np.full(3, F(1) / det)))


def _axis(values):
    """Pitch, origin and count of the regular axis that holds the spot coordinates."""
    u = []
    for v in np.unique(np.asarray(values, F)):
        if not u or v - u[-1] > F(1e-4):
            u.append(v)
    step = min(np.diff(np.array(u, F)))
    return step, u[0], int(np.rint((u[-1] - u[0]) / step)) + 1


def _align(lo, hi, ref, step, multiple):
    first = int(np.ceil((lo - ref) / step - F(1e-4)))
    last = int(np.floor((hi - ref) / step + F(1e-4)))
    return F(ref + F(first) * step), -(-(last - first + 1) // multiple) * multiple


def _lerp(table, x):
    """Linear table value at fractional index x, clamped to the table (64 bits)."""
    x = torch.nan_to_num(x, nan=0.0).clamp(0.0, table.numel() - 1.0)
    i = x.floor().long().clamp(max=table.numel() - 2) if table.numel() > 1 else x.long()
    return table[i] + (table[(i + 1).clamp(max=table.numel() - 1)] - table[i]) * (x - i)


def _sample(vol, x, y, z):
    """Trilinear sample of [Z][Y][X] at texel coordinates, zero outside."""
    nz, ny, nx = vol.shape
    x, y, z = (v.double().clamp(-2.0, n + 1.0) for v, n in ((x, nx), (y, ny), (z, nz)))
    x0, y0, z0 = x.floor(), y.floor(), z.floor()
    flat, out = vol.reshape(-1), torch.zeros_like(x)
    for c in range(8):
        xi, yi, zi = x0 + (c & 1), y0 + ((c >> 1) & 1), z0 + (c >> 2)
        w = (1.0 - (x - xi).abs()) * (1.0 - (y - yi).abs()) * (1.0 - (z - zi).abs())
        ok = (xi >= 0) & (yi >= 0) & (zi >= 0) & (xi < nx) & (yi < ny) & (zi < nz)
        i = ((zi.clamp(0, nz - 1) * ny + yi.clamp(0, ny - 1)) * nx + xi.clamp(0, nx - 1)).long()
        out += torch.where(ok, w * flat[i], torch.zeros_like(w))
    return out


def _first_larger(v, value):
    """Index of the first entry above value (ascending v), the last one if none is."""
    i = int(np.searchsorted(v, value, side="right"))
    return min(i, len(v) - 1)


class _Plan:
    """One lattice beam: its ray grid, traced rays, and per-layer depth dose and sigma."""

    def __init__(self, case, beam, hu):
        self.case, self.beam, self.e = case, beam, _energy(case)
        dims, res, corner = _grid(case)
        res, corner = np.array(res, F), np.array(corner, F)
        z = _unit(_cross(_unit(beam["beam_xdir"]), _unit(beam["beam_ydir"])))
        if _dot(z, _unit(beam["beam_direction"])) < 0:
            z = -z
        x = _unit(beam["beam_xdir"])
        x = _unit(x - z * _dot(x, z))
        y = _unit(_cross(z, x))
        if _dot(y, _unit(beam["beam_ydir"])) < 0:
            y = -y
        x = _unit(_cross(y, z))
        sad = F(beam["sad"])
        iso = (np.asarray(beam["source_position"], F) + z * sad).astype(F)
        to_world = np.stack([x, -y, -z], axis=1)
        inv = _inv(to_world)
        scale = np.diag(F(1) / res)
        self.m = _matmul(scale, to_world)  # gantry -> index
        self.v = (_mul(scale, iso) + -corner / res).astype(F)
        shift = _mul(inv, -iso)
        ends = np.array([[F(i) * F(d - 1) * r + c for i in (0, 1)] for d, r, c in zip(dims, res, corner)], F)
        gz = [(_mul(inv, np.array([ends[0][i & 1], ends[1][(i >> 1) & 1], ends[2][i >> 2]], F)) + shift)[2]
              for i in range(8)]
        ray = F(case["ray"])
        pos = beam["spot_positions"].reshape(-1, 2)
        self.dx, self.ox, self.nx = _axis(pos[:, 0])
        self.dy, self.oy, self.ny = _axis(pos[:, 1])
        margin = F(3) * F(case["sigma_hi"]) + F(0.5) * ray
        cx, self.rx = _align(self.ox - margin, self.ox + F(self.nx - 1) * self.dx + margin, self.ox, ray, TILE_X)
        cy, self.ry = _align(self.oy - margin, self.oy + F(self.ny - 1) * self.dy + margin, self.oy, ray, TILE_Y)
        self.steps = int(np.ceil((max(gz) - min(gz)) / res[2])) + 1
        self.corner = np.array([cx, cy, max(gz)], F)
        self.delta = np.array([ray, ray, -res[2]], F)
        self.dist = F(case["sad"])
        ix = np.rint((pos[:, 0] - self.ox) / self.dx).astype(int)
        iy = np.rint((pos[:, 1] - self.oy) / self.dy).astype(int)
        layer = np.repeat(np.arange(case["layers"]), beam["layer_spot_counts"])
        self.cell = torch.from_numpy((layer * self.ny + iy) * self.nx + ix).cuda()
        w = torch.from_numpy(beam["spot_weights"]).cuda()
        self.lattice = torch.zeros(case["layers"] * self.ny * self.nx, device="cuda").index_add(0, self.cell, w)
        self.lattice = self.lattice.double().reshape(case["layers"], self.ny, self.nx)
        self._trace(hu)
        self._fluence()

    def _trace(self, hu):
        c, d, t = self.corner, self.delta, self.m.T
        i = torch.arange(self.rx, device="cuda").float()[None, :].expand(self.ry, self.rx)
        j = torch.arange(self.ry, device="cuda").float()[:, None].expand(self.ry, self.rx)
        one_z = float(F(1) - c[2] / self.dist)
        off = t[2] - t[0] * (c[0] / self.dist) - t[1] * (c[1] / self.dist)
        transl = self.v + t[2] * c[2] + t[0] * (c[0] * (F(1) - c[2] / self.dist)) + t[1] * (c[1] * (F(1) - c[2] / self.dist))
        ci, cj = t[0] * d[0], t[1] * d[1]
        inv_dist = float(self.dist)
        start = [float(ci[k]) * (i * one_z) + float(cj[k]) * (j * one_z) + float(transl[k]) + 0.5 for k in range(3)]
        inc = [(float(off[k]) - float(ci[k]) * (i / inv_dist) - float(cj[k]) * (j / inv_dist)) * float(d[2]) for k in range(3)]
        ux, uy = (float(c[0]) + i * float(d[0])) / inv_dist, (float(c[1]) + j * float(d[1])) / inv_dist
        length = (abs(float(d[2])) * (1.0 + ux * ux + uy * uy).sqrt()).double()
        tab = {k: torch.from_numpy(self.e[k + "_vector"]).cuda().double() for k in ("density", "sp", "rrl")}
        self.rrl = tab["rrl"]
        self.rho = torch.empty((self.steps, self.ry, self.rx), dtype=torch.float64, device="cuda")
        self.wepl = torch.empty_like(self.rho)
        cum_hu, cum = torch.zeros_like(length), torch.zeros_like(length)
        before, last = torch.zeros_like(i).long(), torch.zeros_like(i).long()
        outside = torch.ones_like(i).bool()
        for k in range(self.steps):
            h = _sample(hu, *(p - 0.5 for p in start))
            cum_hu += h
            self.rho[k] = _lerp(tab["density"], h * self.e["density_scale_fact"])
            cum += length * _lerp(tab["sp"], h * self.e["sp_scale_fact"])
            self.wepl[k] = cum
            outside &= cum_hu < 150.0
            before[outside] = k
            last[h > 150.0] = k
            start = [p + q for p, q in zip(start, inc)]
        self.fin, self.fout = before + 1, last + 1
        self.first = int(self.fin.min())
        self.wmin = self.wepl.reshape(self.steps, -1).min(dim=1).values.cpu().numpy()

    def _layer(self, l):
        """Energy index, depth scale and peak depth of layer l (32-bit table lookups)."""
        en, tab = F(self.beam["energies"][l]), self.e["energies_per_u"]
        k = int(np.clip(np.searchsorted(tab, en, side="left") - 1, 0, len(tab) - 2))
        t = F(np.clip((en - tab[k]) / (tab[k + 1] - tab[k]), F(0), F(1)))
        idx = F(k) + t
        k, t = int(idx), idx - F(int(idx))
        k1 = min(k + 1, len(tab) - 1)
        at = lambda v: F(v[k] + (v[k1] - v[k]) * t)  # noqa: E731
        return k, k1, float(t), at(self.e["scale_facts"]), at(self.e["peak_depths"])

    def _fluence(self):
        c, entry = self.case, F(self.first) * self.delta[2] + self.corner[2]
        mult = F(1) - entry / self.dist
        self.entry = entry
        L = c["layers"]
        sig = np.linspace(c["sigma_hi"], c["sigma_lo"], L).astype(F)
        self.conv = []
        for l in range(L):
            peak = self._layer(l)[4]
            base = F(0.00270) / (peak - F(4.5)) * entry * entry + F(-4.39) / (peak - F(3.86)) * entry
            s = np.sqrt(max(base + sig[l] * sig[l], F(0))) * (F(0.97) if c["halo"] else F(1))
            mats = []
            for n_out, n_in, d, o, corner in ((self.rx, self.nx, self.dx, self.ox, self.corner[0]),
                                              (self.ry, self.ny, self.dy, self.oy, self.corner[1])):
                pix = self.delta[0]
                se = s / (pix * mult)
                if not se > 0:  # no fluence where the air model narrows the spot to nothing
                    mats.append(torch.zeros((n_out, n_in), dtype=torch.float64, device="cuda"))
                    continue
                r, reach = 1.0 / (math.sqrt(2.0) * float(se)), F(3) * se + F(0.5)
                x, i = np.arange(n_out, dtype=F)[:, None], np.arange(n_in, dtype=F)[None, :]
                step, off = d / pix, (o - corner) / pix
                dist = (i * step + off - x).astype(F)
                ok = torch.from_numpy((dist < reach) & (i >= np.ceil((x - reach - off) / step))).cuda()
                dist = torch.from_numpy(dist).cuda().double()
                m = 0.5 * (torch.erf((dist + 0.5) * r) - torch.erf((dist - 0.5) * r))
                mats.append(torch.where(ok, m, torch.zeros_like(m)))
            self.conv.append(mats)

    def ray_weights(self, l, lattice):
        return self.conv[l][1] @ lattice @ self.conv[l][0].T

    def depth_dose(self, l, w, halo):
        """Depth dose per unit ray weight [S][Y][X] from the first step on, 1/(sqrt 2 sigma),
        and with the halo its own pair per unit lattice weight."""
        k0, k1, t, scale, peak = self._layer(l)
        scale, peak_f = float(scale), float(peak)
        nS = self.e["n_energy_samples"]
        row = lambda m: (torch.from_numpy(m.reshape(-1, nS)[[k0, k1]]).cuda().double().T  # noqa: E731
                         @ torch.tensor([1.0 - t, t], dtype=torch.float64, device="cuda"))
        f0, c, d, dist = self.first, self.corner, self.delta, float(self.dist)
        stop = min(_first_larger(self.wmin, F(1.05) * peak), self._passive())
        if stop <= f0:
            return None
        sp, rho = self.wepl[f0:stop], self.rho[f0:stop]
        k = torch.arange(f0, stop, dtype=torch.float64, device="cuda")[:, None, None]
        old = torch.cat([torch.zeros_like(sp[:1]), sp[:-1]])
        cd = _lerp(row(self.e["cidd_matrix"]), sp * scale)
        dcd = cd - torch.cat([torch.zeros_like(cd[:1]), cd[:-1]])
        eref, delta_s, dip = (169.0, 0.06, 0.0) if halo else (198.81, 0.21, 1.0)
        a, b = F(0.00270) / (peak - F(4.5)), F(-4.39) / (peak - F(3.86))
        quad = float(a * d[2] * d[2])
        lin = float(F(2) * a * d[2] * c[2] + b * d[2])
        before = sp < peak_f
        res_e = 8.639415 * (peak_f - 0.5 * (sp + old)).clamp(min=0.0) ** 0.5649718
        beta_p = res_e + 938.3 - 938.3 ** 2 / (res_e + 938.3)
        step = abs(float(d[2]))
        th2 = eref / beta_p ** 2 * step * rho * _lerp(self.rrl, rho * self.e["rrl_scale_fact"])
        zero = torch.zeros_like(sp)
        inc2 = torch.where(before, 2.0 * th2 * step * step, zero).cumsum(0)
        scat = torch.where(before, inc2, zero).cumsum(0)
        n_before = before.double().cumsum(0)
        div0 = lin + (2.0 * f0 - 1.0) * quad
        prev = lambda v: torch.cat([torch.zeros_like(v[:1]), v[:-1]])  # noqa: E731
        grow = prev(scat) + div0 + 2.0 * quad * prev(n_before)
        sig2 = -div0 + torch.where(before, grow, -1.5 * dip * grow * rho).cumsum(0)
        zk = float(c[2]) + k * float(d[2])
        width = float(d[0]) * (1.0 - zk / dist)
        rs = width / (math.sqrt(2.0) * (sig2.sqrt() + delta_s))
        dx, dz, cz = F(d[0]), F(d[2]), F(c[2])
        dist_f = self.dist
        vol = abs(dx * dx * dz)
        v0 = vol * (F(1) - cz / dist_f - cz / dist_f + (cz * cz + dz * dz / F(12)) / (dist_f * dist_f))
        v1 = vol * dz * (F(-1) / dist_f - F(1) / dist_f + F(2) * cz / (dist_f * dist_f))
        v2 = vol * dz * dz / (dist_f * dist_f)
        mass = rho * (float(v0) + k * float(v1) + k * k * float(v2))
        al = self.fout.clamp(max=stop)
        alive = (sp <= float(F(1.05) * peak)) & (k < al) & (al >= f0) & (w >= 1e-6)
        alive &= k >= self.fin - 1
        inf = torch.full_like(sp, math.inf)
        unit = torch.where(alive & (mass > 1e-2), dcd / mass, zero)
        rs = torch.where(alive, rs, inf)
        if not halo:
            return unit, rs, None, None
        mid = 0.5 * (sp + old) * scale
        nw = _lerp(row(self.e["nuc_weight_matrix"]), mid)
        s2 = _lerp(row(self.e["nuc_sq_sigma_matrix"]), mid)
        spacing = F(PITCH_MM) if PITCH_MM > 1.5 * self.case["ray"] else self.dx
        spot = float(F(abs(spacing / d[0])))
        sg = np.linspace(self.case["sigma_hi"], self.case["sigma_lo"], self.case["layers"]).astype(F)[l]
        entry_sq = float(a * self.entry * self.entry + b * self.entry + sg * sg)
        n_rs = 0.5 * spot * 2.0 * width / (math.sqrt(2.0) * (sig2 + s2 + entry_sq).sqrt())
        return unit * (1.0 - nw), rs, unit * nw / spot ** 2, torch.where(alive, n_rs, inf)

    def _passive(self):
        top = max(float(self._layer(l)[4]) for l in range(self.case["layers"]))
        return min(_first_larger(self.wmin, F(1.05) * F(top)), int(self.fout.max()))

    @staticmethod
    def superpose(idd, rs, bev):
        """Adds a layer's tiles to bev [S][Y + 2 PAD][X + 2 PAD]: each 32 x 8 tile spreads its
        sources over the radius of its widest one, sparse radii joined with the next wider."""
        S, Y, X = idd.shape
        ty, tx = Y // TILE_Y, X // TILE_X
        tiles = lambda v: v.reshape(S, ty, TILE_Y, tx, TILE_X).permute(0, 1, 3, 2, 4).reshape(S * ty * tx, -1)  # noqa: E731
        i, r = tiles(idd), tiles(rs)
        low = torch.where(r == r, r, torch.full_like(r, math.inf)).min(dim=1).values.float()
        rad = (3.0 / (1.41421354 * low) + 0.5).clamp(max=33.0).int().cpu().numpy()
        hist = np.bincount(rad, minlength=34)
        hist[32] += hist[33]
        to = np.arange(34)
        top = max([q for q in range(33) if hist[q] > 0], default=0)
        rec, have = top, np.zeros(33, int)
        for q in range(top, 0, -1):
            to[q] = rec
            have[rec] += hist[q]
            if have[rec] >= 16:
                rec = q - 1
        to[33] = to[32]
        live = ((i > 0.0).any(dim=1)).cpu().numpy()
        rad = to[rad]
        flat = bev.reshape(-1)
        BY, BX = bev.shape[1:]
        sy = (torch.arange(256, device="cuda") // TILE_X)[None, :, None]
        sx = (torch.arange(256, device="cuda") % TILE_X)[None, :, None]
        for R in np.unique(rad[live]):
            R = int(R)
            ids = torch.from_numpy(np.nonzero(live & (rad == R))[0]).cuda()
            H, W = TILE_Y + 2 * R, TILE_X + 2 * R
            oy, ox = torch.arange(H, device="cuda"), torch.arange(W, device="cuda")
            at = max(1, int(3e8 / (256 * (H + W) * 8)))
            for n0 in range(0, len(ids), at):
                n = ids[n0:n0 + at]
                ss = r[n]
                edge = torch.erf(ss[:, :, None] * (torch.arange(R + 1, device="cuda") + 0.5))
                e = 0.5 * (edge - torch.cat([-edge[:, :, :1], edge[:, :, :-1]], dim=2))
                e = torch.where((i[n] > 0.0)[:, :, None], e, torch.zeros_like(e))

                def spread(o, s):
                    d = (o[None, None, :] - R - s).abs().expand(len(n), -1, -1)
                    v = e.gather(2, d.clamp(max=R))
                    return torch.where(d <= R, v, torch.zeros_like(v))

                f = spread(oy, sy).transpose(1, 2) @ (spread(ox, sx) * i[n][:, :, None])
                k, t = n // (ty * tx), n % (ty * tx)
                y0, x0 = (t // tx) * TILE_Y - R + PAD, (t % tx) * TILE_X - R + PAD
                idx = (k[:, None, None] * BY + y0[:, None, None] + oy[None, :, None]) * BX + x0[:, None, None] + ox
                flat = flat.index_add(0, idx.reshape(-1), f.reshape(-1))
        return flat.reshape(bev.shape)

    def bevs(self, halo):
        """The beam's BEV dose (and the halo's), with the lateral grid each lies on."""
        new = lambda y, x: torch.zeros((self.steps, y + 2 * PAD, x + 2 * PAD), dtype=torch.float64, device="cuda")  # noqa: E731
        ny, nx = -(-self.ny // TILE_Y) * TILE_Y, -(-self.nx // TILE_X) * TILE_X
        main, side = new(self.ry, self.rx), new(ny, nx)
        f0 = self.first
        if halo:
            gy = np.floor((self.oy + np.arange(self.ny, dtype=F) * self.dy - self.corner[1]) / self.delta[1] + F(0.5)).astype(int)
            gx = np.floor((self.ox + np.arange(self.nx, dtype=F) * self.dx - self.corner[0]) / self.delta[0] + F(0.5)).astype(int)
            gy, gx = torch.from_numpy(gy).cuda()[:, None], torch.from_numpy(gx).cuda()[None, :]
        for l in range(self.case["layers"]):
            w = self.ray_weights(l, self.lattice[l])
            got = self.depth_dose(l, w, halo)
            if got is None:
                continue
            unit, rs, n_unit, n_rs = got
            n = unit.shape[0]
            main[f0:f0 + n] = self.superpose(unit * w, rs, main[f0:f0 + n])
            if halo:
                i = torch.zeros((n, ny, nx), dtype=torch.float64, device="cuda")
                r = torch.full_like(i, math.inf)
                i[:, :self.ny, :self.nx] = n_unit[:, gy, gx] * self.lattice[l]
                r[:, :self.ny, :self.nx] = n_rs[:, gy, gx]
                side[f0:f0 + n] = self.superpose(i, r, side[f0:f0 + n])
        out = [(main, (self.delta, self.corner))]
        if halo:
            out.append((side, (np.array([self.dx, self.dy, self.delta[2]], F),
                               np.array([self.ox, self.oy, self.corner[2]], F))))
        return out

    def _fan(self, geo, z):
        """BEV texel coordinates of the dose voxels of slice z (32 bits)."""
        delta, corner = geo
        mi = _inv(self.m)
        v = _mul(mi, -self.v)
        inv = F(1) / delta
        off = (-corner * inv + np.array([PAD, PAD, 0], F)).astype(F)
        off[2] = -corner[2] * inv[2] + -F(self.first)
        x = torch.arange(self.case["nx"], device="cuda").float()[None, :]
        y = torch.arange(self.case["ny"], device="cuda").float()[:, None]
        c = mi.T * inv
        p = [x * float(c[0][k]) + y * float(c[1][k]) + float((v * inv)[k]) + float(F(z) * c[2][k]) for k in range(3)]
        norm = float(inv[2] * self.dist)
        for k in (0, 1):
            p[k] = p[k] * (1.0 + p[2] / (norm - p[2]))
        return [p[k] + float(off[k]) for k in range(3)]

    def transfer(self, bev, geo):
        out = []
        for z in range(self.case["nz"]):
            f = self._fan(geo, z)
            ok = (f[0] >= -0.5) & (f[1] >= -0.5) & (f[2] >= -0.5)
            out.append(torch.where(ok, _sample(bev[self.first:], f[0], f[1], f[2]), torch.zeros_like(f[0]).double()))
        return torch.stack(out).clamp(min=0.0)

    def gradient(self, g):
        """Gradient with respect to the spot weights for the dose gradient g."""
        shape = (self.steps, self.ry + 2 * PAD, self.rx + 2 * PAD)
        bev = torch.zeros(shape, dtype=torch.float64, device="cuda", requires_grad=True)
        g_bev = torch.zeros_like(bev)
        geo = (self.delta, self.corner)
        for z in range(self.case["nz"]):
            f = self._fan(geo, z)
            ok = (f[0] >= -0.5) & (f[1] >= -0.5) & (f[2] >= -0.5)
            v = _sample(bev[self.first:], f[0], f[1], f[2])
            g_bev += torch.autograd.grad((v * torch.where(ok, g[z], torch.zeros_like(g[z]))).sum(), bev)[0]
        f0, parts = self.first, []
        for l in range(self.case["layers"]):
            lat = self.lattice[l].clone().requires_grad_()
            w = self.ray_weights(l, lat)
            got = self.depth_dose(l, w.detach(), False)
            if got is None:
                parts.append(torch.zeros_like(lat))
                continue
            n = got[0].shape[0]
            b = self.superpose(got[0] * w, got[1], torch.zeros_like(g_bev[f0:f0 + n]))
            parts.append(torch.autograd.grad((b * g_bev[f0:f0 + n]).sum(), lat)[0])
        return torch.stack(parts).reshape(-1)[self.cell]
