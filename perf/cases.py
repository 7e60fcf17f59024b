"""The work that a user of the projector pair has it do, as timed cases: projections, reconstruction steps and gradients
through the public Python entry points, from the 8-ring scanner whose calls last tens of microseconds to the clinical
scanner's 72.6 million lines of response.

A case names a scanner (`geom`), an operation (`op`) and its options.  Data are synthetic: an ellipse with hot spheres,
and Poisson counts around the ellipse's analytic line integrals (so that the inputs depend on the seed alone, not on
the projector under test).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from stir_b200 import _abi
from stir_b200 import geometry as G
from stir_b200.autograd import PoissonLogLikelihood, Prior
from stir_b200.listmode import PoissonLogLikelihoodWithLinearModelForMeanAndListModeDataWithProjMatrixByBin as ListMode
from stir_b200.listmode import pack_events
from stir_b200.osmaposl import OSMAPOSLReconstruction, QuadraticPrior, RelativeDifferencePrior
from stir_b200.projectors import RayTracingProjector
from stir_b200.subsets import basic_views_in_subset, related_views, views_in_subset

DEV = "cuda:0"

# rings, detectors per ring, ring spacing (mm), radius (mm), span, largest ring difference, tangential positions,
# timing bins (1: none), image (nz, ny, nx), voxel size (z, xy) in mm, tangential rays per bin
SMALL = dict(rings=8, dets=288, spacing=4.0, radius=300.0, span=1, delta=7, tang=64, tof=1, nz=15, ny=64, nx=64,
             vz=2.0, vxy=4.0, rays=1)
CLINICAL = dict(rings=64, dets=504, spacing=4.06, radius=328.0, span=11, delta=60, tang=344, tof=1, nz=127, ny=344,
                nx=344, vz=2.03, vxy=2.09, rays=1)
HALF = dict(CLINICAL, ny=172, nx=172, vxy=4.18)  # the clinical scanner at half the transaxial resolution
TOF = dict(SMALL, tof=33)
# a brain-size scanner with an odd image that is not square, and two rays per bin
RAGGED = dict(rings=13, dets=196, spacing=5.2, radius=210.0, span=3, delta=9, tang=57, tof=1, nz=25, ny=61, nx=75,
              vz=2.6, vxy=5.1, rays=2)
# a whole-body scanner with half the clinical one's rings, odd sizes
MEDIUM = dict(rings=32, dets=392, spacing=4.4, radius=405.0, span=7, delta=24, tang=211, tof=1, nz=63, ny=171, nx=171,
              vz=2.2, vxy=4.0, rays=1)


def listed():
    return [
        # set-up checks, phantoms and small animal scanners: a projection and its adjoint, tens of microseconds each,
        # so launches count
        dict(name="pair_small", op="pair", subsets=1, **SMALL),
        # the same scanner's reconstruction step, 6 subsets: the smallest call of all
        dict(name="osem_small", op="osem", subsets=6, **SMALL),
        # odd sizes, a rectangular image, two tangential rays per bin
        dict(name="pair_ragged", op="pair", subsets=1, **RAGGED),
        # a mid-size scanner, odd sizes
        dict(name="pair_medium", op="pair", subsets=1, **MEDIUM),
        # the headline: every line of the clinical scanner, forward (attenuation factors, simulation, a full gradient)
        dict(name="forward_clinical", op="forward", subsets=1, **CLINICAL),
        # and back (sensitivities, a full gradient)
        dict(name="back_clinical", op="back", subsets=1, mode=_abi.BACKPROJECT_ATOMIC, **CLINICAL),
        # back projection that repeats bit for bit, one of 7 subsets
        dict(name="back_deterministic", op="back", subsets=7, mode=_abi.BACKPROJECT_DETERMINISTIC, **CLINICAL),
        # clinical reconstruction: one OSEM sub-iteration of 21 subsets
        dict(name="osem_clinical", op="osem", subsets=21, **CLINICAL),
        # a training or variational step: Poisson log-likelihood and its gradient for a batch of 8 images, with a
        # Relative Difference penalty, value and gradient through torch.autograd
        dict(name="gradient_batch", op="gradient", subsets=1, batch=8, **HALF),
        # list mode: the sub-gradient of 2 million events on one of 21 subsets
        dict(name="listmode_clinical", op="listmode", subsets=21, events=2_000_000, **CLINICAL),
        # time of flight: a projection of all 33 timing bins and its adjoint
        dict(name="pair_tof", op="pair", subsets=1, **TOF),
        # time-of-flight reconstruction with a quadratic prior: one sub-iteration of 21 subsets
        dict(name="osem_tof_prior", op="osem", subsets=21, beta=0.05, **TOF),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["pair", "pair", "forward", "back", "back", "osem", "osem", "gradient", "listmode"])
    tof = rng.choice([1, 1, 1, rng.randrange(5, 34)]) if op in ("pair", "osem") else 1
    for _ in range(100):
        rings = log_int(4, 8) if tof > 1 else log_int(4, 64)
        dets = 4 * log_int(24, 72 if tof > 1 else 126)
        span = 1 if tof > 1 else rng.choice([s for s in (1, 3, 5, 7, 9, 11, 11) if s <= rings and (s > 1 or rings <= 16)])
        delta = rng.randrange((span - 1) // 2, rings)
        tang = rng.randrange(dets // 5, int(0.68 * dets))
        g = dict(rings=rings, dets=dets, spacing=round(rng.uniform(3.2, 6.4), 2), radius=round(rng.uniform(0.55, 1.05) * dets, 1),
                 span=span, delta=delta, tang=tang, tof=tof, rays=rng.choice([1, 1, 1, 2]) if tof == 1 else 1)
        pdi = _projdata(g)
        if pdi.size <= 4e7:
            break
    fov = 2 * g["radius"] * math.sin(math.pi * (tang / 2) / dets)
    ny = log_int(33, 80 if tof > 1 else 344)
    nx = ny if rng.random() < 0.7 else max(33, min(344, int(ny * rng.uniform(0.8, 1.25))))
    g.update(nz=2 * rings - 1, ny=ny, nx=nx, vz=g["spacing"] / 2, vxy=round(rng.uniform(0.75, 1.1) * fov / max(nx, ny), 3))
    case = dict(op=op, subsets=rng.choice([1, 1, 7, 14, 21]), **g)
    if op == "osem":
        case["subsets"] = rng.choice([4, 6, 7, 14, 21])
        if rng.random() < 0.4:
            case["beta"] = 0.05
    if op == "back":
        case["mode"] = rng.choice([_abi.BACKPROJECT_ATOMIC, _abi.BACKPROJECT_DETERMINISTIC])
    if op == "gradient":
        case["batch"] = rng.randrange(1, 5)
    if op == "listmode":
        case["events"] = log_int(20_000, 2_000_000)
    return case


# ---- the scanner, its projector (kept between calls, as a program that meets new data keeps it) -------------------

_GEOM = ("rings", "dets", "spacing", "radius", "span", "delta", "tang", "tof", "nz", "ny", "nx", "vz", "vxy", "rays")
_projectors = {}


def _projdata(c):
    sc = G.Scanner(c["rings"], c["dets"], c["radius"], 0.0, c["spacing"],
                   float(np.float32(math.pi * c["radius"] / c["dets"])), 0.0)
    if c["tof"] > 1:
        sc.timing_resolution, sc.size_of_timing_pos, sc.max_num_timing_poss = 550.0, 50.0, c["tof"]
    return G.ProjDataInfoCTI(sc, c["span"], c["delta"], c["dets"] // 2, c["tang"],
                             tof_mash_factor=1 if c["tof"] > 1 else 0)


def _projector(c):
    key = tuple(c[k] for k in _GEOM)
    if key not in _projectors:
        while len(_projectors) >= 3:
            _projectors.pop(next(iter(_projectors)))
        img = G.ImageGeometry(c["nz"], c["ny"], c["nx"], (c["vz"], c["vxy"], c["vxy"]))
        _projectors[key] = RayTracingProjector(_projdata(c), img, num_tangential_LORs=c["rays"], device=0)
    return _projectors[key]


# ---- inputs ------------------------------------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _phantom(c, seed):
    """An elliptical body of activity 1 with hot spheres at seeded places, and a smooth texture of a few per cent:
    device layout [y][x][z]."""
    ny, nx, nz, v = c["ny"], c["nx"], c["nz"], c["vxy"]
    y = ((torch.arange(ny, device=DEV) - ny // 2) * v).view(-1, 1, 1)
    x = ((torch.arange(nx, device=DEV) - nx // 2) * v).view(1, -1, 1)
    z = ((torch.arange(nz, device=DEV) - nz / 2) * c["vz"]).view(1, 1, -1)
    ax, ay = 0.40 * min(nx, ny) * v, 0.30 * min(nx, ny) * v
    img = (((x / ax) ** 2 + (y / ay) ** 2) <= 1.0).float().expand(ny, nx, nz).clone()
    r = np.random.default_rng(seed)
    for _ in range(6):
        rad = r.uniform(0.03, 0.08) * min(nx, ny) * v
        cx, cy, cz = r.uniform(-0.5, 0.5) * ax, r.uniform(-0.5, 0.5) * ay, r.uniform(-0.4, 0.4) * nz * c["vz"]
        img[((x - cx) ** 2 + (y - cy) ** 2 + (z - cz) ** 2) <= rad ** 2] = 4.0
    img *= 1.0 + 0.05 * torch.rand(img.shape, generator=_gen(seed), device=DEV)
    return img + 0.02


def _chords(c, pdi):
    """The ellipse's chord length (mm) per (view, tangential position)."""
    n, v = min(c["nx"], c["ny"]), c["vxy"]
    ax, ay = 0.40 * n * v, 0.30 * n * v
    phi = torch.arange(pdi.num_views, device=DEV, dtype=torch.float64).view(-1, 1) * (math.pi / pdi.num_views)
    t = torch.arange(c["tang"], device=DEV, dtype=torch.float64).view(1, -1) - c["tang"] // 2
    s = c["radius"] * torch.sin(t * (math.pi / c["dets"]))
    q = (ax * torch.cos(phi)) ** 2 + (ay * torch.sin(phi)) ** 2
    return 2 * ax * ay * torch.sqrt(torch.clamp(q - s * s, min=0.0)) / q


def _spread(pdi, view_tang, tof=None):
    """Device-layout projection data ([timing bin][segment][view][tangential][axial]) constant along the axis."""
    parts = []
    for k in range(tof if tof is not None else max(1, pdi.num_tof_bins)):
        for seg in range(-pdi.max_segment_num, pdi.max_segment_num + 1):
            parts.append(view_tang.float()[:, :, None].expand(-1, -1, pdi.get_num_axial_poss(seg)).reshape(-1))
    return torch.cat(parts)


def _data(c, pdi, seed):
    """Counts in the model's units (y, additive a, multiplicative m): mean m (chord + a), about 4 events per bin
    through the middle without TOF."""
    g = _gen(seed + 1)
    chord = _chords(c, pdi)
    ntof = max(1, pdi.num_tof_bins)
    att = torch.exp(-0.0096 * chord)
    m_nt = _spread(pdi, att, tof=1)
    m_nt *= 0.8 + 0.4 * torch.rand(m_nt.shape, generator=g, device=DEV)
    mean = _spread(pdi, chord / ntof, tof=1)
    add = torch.full_like(mean, float(0.3 * chord.mean() / ntof))
    scale = 4.0 / float((chord * att).max()) * ntof
    y = torch.poisson(((mean + add) * m_nt * scale).repeat(ntof), generator=g) / scale
    return y, add.repeat(ntof), m_nt.repeat(ntof)


def prepare(case, seed):
    c = dict(case)
    proj = _projector(c)
    pdi = proj.proj_data_info
    s = dict(case=c, proj=proj)
    op = c["op"]
    if op in ("pair", "forward"):
        s["x"] = _phantom(c, seed)
        s["out"] = proj.empty_projdata()
    if op == "pair":
        s["back"] = proj.empty_image()
    if op == "back":
        s["y"] = _data(c, pdi, seed)[0]
        s["out"] = proj.empty_image()
    if op == "osem":
        y, add, m = _data(c, pdi, seed)
        prior = QuadraticPrior(c["beta"]) if c.get("beta") else None
        r = OSMAPOSLReconstruction(proj, y, additive=add, mult=m, num_subsets=c["subsets"], num_subiterations=2,
                                   prior=prior, use_tofsens=True)
        r.set_up()
        r.subiteration_num = c["subsets"] + 1  # the second full iteration's first subset
        s.update(recon=r, x0=_phantom(c, seed), x=proj.empty_image())
    if op == "gradient":
        data = [_data(c, pdi, seed + 7 * b) for b in range(c["batch"])]
        y = torch.stack([d[0] for d in data])
        add, m = data[0][1], data[0][2]
        del data
        s["x"] = torch.stack([_phantom(c, seed + 7 * b) for b in range(c["batch"])]).requires_grad_()
        s["loglik"] = PoissonLogLikelihood(proj, y, additive=add, mult=m, subset_num=0, num_subsets=c["subsets"])
        s["penalty"] = Prior(proj, RelativeDifferencePrior(0.1))
    if op == "listmode":
        r = np.random.default_rng(seed)
        n = c["events"]
        views = np.array(views_in_subset(proj.geometry, 0, c["subsets"], proj.info.symmetries_used))
        bins = np.zeros((n, 5), np.int32)
        seg = r.integers(-pdi.max_segment_num, pdi.max_segment_num + 1, n)
        nax = np.array([pdi.get_num_axial_poss(int(k)) for k in range(-pdi.max_segment_num, pdi.max_segment_num + 1)])
        half = max(1, c["tang"] // 3)
        bins[:, 0] = seg
        bins[:, 1] = views[r.integers(0, len(views), n)]
        bins[:, 2] = (r.random(n) * nax[seg + pdi.max_segment_num]).astype(np.int32)
        bins[:, 3] = r.integers(-half, half + 1, n)
        s["obj"] = ListMode(proj, pack_events(bins, corr=np.full(n, 20.0, np.float32)), num_subsets=c["subsets"], has_add=True)
        s["bins"] = bins
        s["x"] = _phantom(c, seed)
        s["out"] = proj.empty_image()
    return s


def run(s):
    c, proj = s["case"], s["proj"]
    op, n = c["op"], c["subsets"]
    if op == "forward":
        return proj.forward_dev(s["x"], out=s["out"], num_subsets=n)
    if op == "back":
        return proj.back_dev(s["y"], out=s["out"], num_subsets=n, mode=c["mode"])
    if op == "pair":
        proj.forward_dev(s["x"], out=s["out"], num_subsets=n)
        proj.back_dev(s["out"], out=s["back"], num_subsets=n)
        return s["out"], s["back"]
    if op == "osem":
        s["x"].copy_(s["x0"])  # every pass starts from the same estimate
        return s["recon"].update_estimate(s["x"])
    if op == "gradient":
        loss = s["penalty"](s["x"]) - s["loglik"](s["x"])
        grad, = torch.autograd.grad(loss, s["x"])
        return loss.detach(), grad
    if op == "listmode":
        return s["obj"].compute_sub_gradient_without_penalty(s["x"], 0, out=s["out"])
    raise ValueError(op)


# ---- sizes, tolerances -------------------------------------------------------------------------------------------

def _lines(c):
    """(lines of response in the call, row elements per line): the elements by the average path of a line through
    the cylinder (4 / pi voxels per voxel length), twice as many where an axial position spans two planes."""
    pdi = _projdata(c)
    nv = c["dets"] // 2
    bits = (3 if nv % 4 == 0 else 2) if c["nx"] == c["ny"] else 2
    views = sum(len(related_views(v, nv, bits)) for v in basic_views_in_subset(nv, bits, 0, c["subsets"]))
    t = np.arange(c["tang"]) - c["tang"] // 2
    s = c["radius"] * np.sin(t * math.pi / c["dets"])
    rad = 0.5 * min(c["nx"], c["ny"]) * c["vxy"]
    chord = float(2 * np.sqrt(np.maximum(rad * rad - s * s, 0)).mean())
    per = chord / c["vxy"] * 4 / math.pi * (2 if c["span"] == 1 else 1) * c["rays"] ** 0.5
    return pdi.size * views / nv, per


def work(case):
    c = case
    lines, per = _lines(c)
    img = 4.0 * c["nz"] * c["ny"] * c["nx"]
    one = 2.0 * lines * per  # multiply-adds of one projection
    bytes_, flops = {
        "forward": (img + 4 * lines, one),
        "back": (img + 4 * lines, one),
        "pair": (2 * (img + 4 * lines), 2 * one),
        "osem": (3 * img + 4 * 2 * lines, 2 * one),
        "gradient": (c.get("batch", 1) * (2 * img + 4 * lines) + 8 * lines, c.get("batch", 1) * 2 * one),
        "listmode": (2 * img + 28.0 * c.get("events", 0), 4.0 * per * c.get("events", 0)),
    }[c["op"]]
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    """32-bit sums of a few hundred products, in any order: up to 2.2e-7 against 64 bits and 7e-7 (largest value) between
    two orders; four times that, and room for single values, whose sums differ more than the whole.  The batch's gradient
    is a difference of two back projections of about the same size."""
    if case["op"] == "gradient":
        return {"rel": 3e-6, "max": 5e-5}
    return {"rel": 1e-6, "max": 2e-5}


# ---- 64 bits -----------------------------------------------------------------------------------------------------

class _Rows:
    """The matrix of a subset's lines as padded (column, plane, value) rows per segment.  The rows themselves are the
    problem's data (STIR defines them by a 32-bit ray tracer), listed by the matrix through get_row at the first axial
    position; the sums over them are torch's in 64 bits."""

    def __init__(self, c, proj, subset, subsets):
        pdi = proj.proj_data_info
        self.c, self.pdi = c, pdi
        self.views = views_in_subset(proj.geometry, subset, subsets, proj.info.symmetries_used)
        self.nz = c["nz"]
        oy, ox = proj.geometry.min_y, proj.geometry.min_x
        t0 = pdi.min_tangential_pos_num
        self.ntof = max(1, pdi.num_tof_bins)
        k0 = -(self.ntof // 2)
        self.blocks = []
        off = 0
        tof_stride = pdi.size // self.ntof
        for seg in range(-pdi.max_segment_num, pdi.max_segment_num + 1):
            nax = pdi.get_num_axial_poss(seg)
            npa = 1
            rows, bins = [], []
            for k in range(self.ntof):
                for v in self.views:
                    for t in range(c["tang"]):
                        coords, vals = proj.get_row(seg, v, 0, t0 + t, k0 + k)
                        if len(vals) == 0:
                            continue
                        rows.append((coords, vals))
                        bins.append(k * tof_stride + off + (v * c["tang"] + t) * nax)
            if nax > 1 and rows:  # planes per axial position
                for v in self.views:
                    a, _ = proj.get_row(seg, v, 0, 0)
                    b, _ = proj.get_row(seg, v, 1, 0)
                    if len(a) and len(b):
                        npa = int(b[:, 0].min() - a[:, 0].min())
                        break
            off += nax * pdi.num_views * c["tang"]
            for i in range(0, len(rows), 4096):
                part = rows[i:i + 4096]
                L = max(len(v) for _, v in part)
                col = np.zeros((len(part), L), np.int64)
                z = np.zeros((len(part), L), np.int64)
                w = np.zeros((len(part), L), np.float64)
                for j, (q, v) in enumerate(part):
                    col[j, :len(v)] = ((q[:, 1] - oy).astype(np.int64) * c["nx"] + (q[:, 2] - ox)) * c["nz"]
                    z[j, :len(v)] = q[:, 0] - proj.geometry.min_z
                    w[j, :len(v)] = v
                self.blocks.append((nax, npa, *(torch.from_numpy(a).to(DEV) for a in (col, z, w)),
                                    torch.tensor(bins[i:i + 4096], device=DEV)))

    def _parts(self):
        for nax, npa, col, z, w, bins in self.blocks:
            step = max(1, int(2e7 // (nax * col.shape[1])))
            a = torch.arange(nax, device=DEV).view(1, 1, -1)
            for i in range(0, col.shape[0], step):
                zz = z[i:i + step, :, None] + npa * a
                inside = (zz >= 0) & (zz < self.nz)
                yield (col[i:i + step, :, None] + zz.clamp(0, self.nz - 1), inside * w[i:i + step, :, None],
                       bins[i:i + step, None] + a[0])

    def forward(self, x):
        x = x.double().reshape(-1)
        out = torch.zeros(self.pdi.size, dtype=torch.float64, device=DEV)
        for idx, w, bins in self._parts():
            out[bins] = (x[idx] * w).sum(1)
        return out

    def back(self, y):
        y = y.double()
        out = torch.zeros(self.c["ny"] * self.c["nx"] * self.c["nz"], dtype=torch.float64, device=DEV)
        for idx, w, bins in self._parts():
            out.index_add_(0, idx.reshape(-1), (w * y[bins][:, None, :]).reshape(-1))
        return out.view(self.c["ny"], self.c["nx"], self.c["nz"])


def exact(case, seed):
    c = dict(case)
    pdi = _projdata(c)
    op = c["op"]
    lines, per = _lines(c)
    rows = lines / pdi.size * pdi.num_views * c["tang"] * (2 * pdi.max_segment_num + 1) * c["tof"]
    if rows > 250_000 or lines * per > 1.5e10 or op == "gradient":
        return None
    s = prepare(case, seed)
    proj = s["proj"]
    A = _Rows(c, proj, 0, c["subsets"])
    if op == "forward":
        return A.forward(s["x"])
    if op == "back":
        return A.back(s["y"])
    if op == "pair":
        f = A.forward(s["x"])
        return f, A.back(f)
    if op == "listmode":
        f = A.forward(s["x"])
        b = torch.from_numpy(s["bins"].astype(np.int64)).to(DEV)
        S = pdi.max_segment_num
        nax = torch.tensor([pdi.get_num_axial_poss(k) for k in range(-S, S + 1)], device=DEV)
        first = torch.cumsum(nax, 0) - nax
        i = first[b[:, 0] + S] * (pdi.num_views * c["tang"]) + \
            (b[:, 1] * c["tang"] + b[:, 3] - pdi.min_tangential_pos_num) * nax[b[:, 0] + S] + b[:, 2]
        h = torch.zeros_like(f).index_add_(0, i, 1.0 / (f[i] + 20.0))
        return A.back(h)
    if op == "osem":
        r, x = s["recon"], s["x0"].double()
        y = r.y.double()
        f = A.forward(s["x0"]) + r.additive.double()
        # as STIR's divide_and_truncate: bins of at most a millionth of their viewgram's largest count give 0, ratios
        # are cut at 1e4
        ratio = torch.where(y > 0, torch.clamp(y / f, max=1e4), torch.zeros_like(y))
        u = A.back(ratio)
        # the sensitivity is an input of the step (32 bits, prepared once)
        den = r.sensitivities[0].double()
        if r.prior is not None:
            den = den * torch.clamp(1 + _quadratic_gradient(c, x) * r.prior.penalisation_factor, 0.1, 10.0)
        small = 0.0 if r.prior is None else 1e-6 * float(u.max())
        q = torch.where((den.abs() <= small) & (u.abs() <= small), torch.zeros_like(u), u / den)
        return x * torch.clamp(q, min=0.0, max=3.4028234663852886e38)
    return None


def _quadratic_gradient(c, x):
    """sum over the 26 neighbours of (x - neighbour) times voxel size x / distance."""
    g = torch.zeros_like(x)
    n = x.shape
    for dy in (-1, 0, 1):
        for dx in (-1, 0, 1):
            for dz in (-1, 0, 1):
                if (dy, dx, dz) == (0, 0, 0):
                    continue
                w = c["vxy"] / math.sqrt((dx * c["vxy"]) ** 2 + (dy * c["vxy"]) ** 2 + (dz * c["vz"]) ** 2)
                a = tuple(slice(max(0, -d), n[k] - max(0, d)) for k, d in enumerate((dy, dx, dz)))
                b = tuple(slice(max(0, d), n[k] - max(0, -d)) for k, d in enumerate((dy, dx, dz)))
                g[a] += w * (x[a] - x[b])
    return g
