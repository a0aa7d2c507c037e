"""What the framework is timed on: the passes, projections and whole
reconstructions that its users run, from a 2D slice to the 256x256x81 job.

Every input is made from the seed with torch alone: a water disc with hot
spheres, closed-form line integrals through it, Poisson counts, and a positive
current estimate.  ``exact`` restates the Siddon walk in torch: lengths,
sums, ratios and updates in 64 bits (which voxel a ray enters and leaves by is
decided in the float arithmetic that defines the walk)."""
import math

import numpy as np
import torch

import apirl_b200 as ap
from apirl_b200 import _lib
from apirl_b200.batch import Batch, Job
from apirl_b200.geometry import ImageGeom, Sino2DGeom, Sino3DGeom

DEV = "cuda:0"
MU = 0.0096  # water, per mm


def _big(**kw):
    """The 256x256x81 image and the 1261-sinogram span-1 scanner (336 x 336 per sinogram)."""
    return dict(n=256, nz=81, dxy=2.08, dz=2.03, n_r=336, n_proj=336, rings=41, pitch=4.054, max_rd=20, span=1,
                rfov=266.24, r_scanner=443.0, scanner="cylindrical", disc=100.0, **kw)


def _job(n, nz, **kw):
    """A reconstruction job's geometry: round(1.3 n) radial bins and angles at the voxel pitch, (nz + 1) / 2 rings."""
    nr = int(round(1.3 * n))
    return dict(n=n, nz=nz, dxy=2.08, dz=2.03, n_r=nr, n_proj=nr, rings=(nz + 1) // 2, pitch=4.06, max_rd=nz // 4,
                span=1, rfov=nr * 2.08 / 2.0, r_scanner=443.0, scanner="cylindrical", disc=0.38 * n * 2.08, **kw)


def listed():
    return [
        # One iteration of 2D MLEM on one slice: the smallest pass, where latency counts.
        dict(name="mlem_2d_pass", kind="em2d", n=128, n_r=192, n_proj=192, dxy=2.08, rfov=199.68, r_scanner=443.0,
             disc=100.0, total=1.0e6),
        # The whole 2D reconstruction as a program calls it, host arrays in and out.
        dict(name="mlem_2d_job", kind="job2d", n=128, n_r=192, n_proj=192, dxy=2.08, rfov=199.68, r_scanner=443.0,
             disc=100.0, total=1.0e6, iters=60),
        # An OSEM sub-iteration over every bin of the subset: the form for data with an additive or no geometry image.
        dict(name="osem_full_256", kind="em", subset=0, nsub=21, counts="uint32", total=5.0e8, add=False, **_big()),
        # The same over the bins with counts (geometry image): how a long job's sub-iterations run.
        dict(name="osem_listed_256", kind="listed", subset=0, nsub=21, counts="uint32", total=5.0e8, add=False,
             **_big()),
        # A small short scan: low counts in 16 bits, most bins empty, a few tens of microseconds of work.
        dict(name="osem_listed_64", kind="listed", subset=3, nsub=9, counts="uint16", total=3.0e5, add=False,
             **_job(64, 41)),
        # 3D MLEM (all angles) of corrected float data with scatter and randoms added to the estimate.
        dict(name="mlem_additive_100", kind="em", subset=-1, nsub=1, counts="float32", total=2.0e7, add=True,
             **_job(100, 41)),
        # Forward projection of one subset: simulation, residuals, other algorithms than EM.
        dict(name="project_256", kind="project", subset=0, nsub=21, **_big()),
        # Its adjoint: corrections, sensitivities.
        dict(name="backproject_256", kind="backproject", subset=0, nsub=21, **_big()),
        # Ratio and backprojection given an estimate: a user's own EM loop.
        dict(name="divide_back_128", kind="divide", subset=2, nsub=7, total=3.0e7, **_job(128, 41)),
        # Attenuation factors of a mu map on the Siemens mMR geometry, 12 of its 252 angles (span 11).
        dict(name="acf_mmr", kind="acf", n=172, nz=127, dxy=4.17252, dz=2.03125, n_r=344, n_proj=252, rings=64,
             pitch=4.0625, max_rd=60, span=11, rfov=297.0, r_scanner=328.0, scanner="mmr", disc=140.0, subset=0,
             nsub=21),
        # Several rays per bin (detector width modelled): every bin walks 6 rays.
        dict(name="osem_sampled_64", kind="sampled", subset=1, nsub=8, counts="float32", total=3.0e6, add=False, ns=3,
             nas=2, **_job(64, 21)),
        # A queue of mixed jobs through one batch engine that is kept, host arrays in and out.
        dict(name="batch_mixed", kind="batch", jobs=10, iters=2, budget=6 << 30),
    ]


def draw(rng):
    kind = rng.choice(["em2d", "em", "em", "listed", "listed", "project", "backproject", "divide", "acf", "sampled"])
    n = int(round(math.exp(rng.uniform(math.log(32), math.log(256)))))
    if kind == "em2d":
        nr = int(round(1.5 * n))
        return dict(kind=kind, n=n, n_r=nr, n_proj=rng.randint(nr // 2, nr), dxy=2.08, rfov=0.75 * n * 2.08,
                    r_scanner=443.0, disc=0.38 * n * 2.08, total=float(10 ** rng.uniform(4.5, 7)))
    if kind == "sampled":
        n = min(n, 80)
    nz = rng.choice([1, rng.randint(2, 20), rng.randint(21, 81), rng.randint(21, 81)])
    if kind == "acf":
        nz = max(2, nz)
        rings = max(2, nz // 2)
        rd = max(1, rings - 1 - rng.randint(0, rings // 4))
        c = dict(kind=kind, n=n, nz=nz, dxy=594.0 / n, dz=260.0 / nz, n_r=rng.choice([172, 344]),
                 n_proj=rng.randint(90, 252), rings=rings, pitch=260.0 / rings, max_rd=rd, span=rng.choice([1, 3, 5]),
                 rfov=297.0, r_scanner=328.0, scanner="mmr", disc=140.0)
    else:
        c = dict(kind=kind, **_job(n, nz))
        if rng.random() < 0.3:
            c.update(span=3, max_rd=max(1, c["max_rd"]))
    c["nsub"] = min(rng.randint(1, 21), c["n_proj"])
    limit = 1.5e9 / (6 if kind == "sampled" else 1)
    while _segments(dict(c, subset=0)) > limit and c["nsub"] < c["n_proj"]:
        c["nsub"] = min(c["n_proj"], c["nsub"] * 2)
    if _segments(dict(c, subset=0)) > limit:
        c["n_proj"] = c["nsub"] = 48
    c["subset"] = -1 if c["nsub"] == 1 else rng.randrange(c["nsub"])
    bins = _sinos(c) * c["n_proj"] * c["n_r"]
    if kind in ("em", "listed", "divide", "sampled"):
        c["total"] = float(bins * 10 ** rng.uniform(-1.3, 0.7))
    if kind in ("em", "listed", "sampled"):
        c["counts"] = rng.choice(["uint32", "uint16", "float32"])
        c["add"] = rng.random() < 0.3
    if kind == "sampled":
        c["ns"], c["nas"] = rng.choice([(2, 1), (3, 2), (1, 2)])
    return c


# ---- geometry ---------------------------------------------------------------
def _geoms(c):
    if c["kind"] in ("em2d", "job2d"):
        return ImageGeom(c["n"], c["n"], 1, c["dxy"], c["dxy"], 1.0), Sino2DGeom(c["n_proj"], c["n_r"], c["rfov"],
                                                                                c["r_scanner"])
    ig = ImageGeom(c["n"], c["n"], c["nz"], c["dxy"], c["dxy"], c["dz"])
    if c["scanner"] == "mmr":
        return ig, Sino3DGeom.mmr(c["n_proj"], c["n_r"], c["rings"], c["span"], c["max_rd"])
    make = Sino3DGeom.span1 if c["span"] == 1 else Sino3DGeom.span
    head = (c["n_proj"], c["n_r"], c["rings"], c["rfov"], c["rings"] * c["pitch"], c["r_scanner"])
    return ig, make(*head, c["max_rd"]) if c["span"] == 1 else make(*head, c["span"], c["max_rd"])


def _sinos(c):
    return 1 if c["kind"] in ("em2d", "job2d") else _geoms(c)[1].n_sinos


def _angles(c):
    s, k = c.get("subset", -1), c.get("nsub", 1)
    return list(range(c["n_proj"])) if s < 0 else list(range(s, c["n_proj"], k))


def _lor(c, angles, samples=1):
    """End points of the LORs in the plane, float32 [angle, r, sample, 4] (the scanner's own float expressions)."""
    f = np.float32
    n_r = c["n_r"]
    inc_a = f(180) / f(c["n_proj"])
    ang = np.array(angles, f) * inc_a
    if c.get("scanner") == "mmr":
        radius, doi = f(328.0), f(9.6)
        b = f(4.0891) / f(2)
        b = b if n_r == 344 else b * f(344) / f(n_r)
        lr = b / f(2) + b * (np.arange(n_r, dtype=f) - f(n_r // 2))
        r = ((radius + doi * np.cos(lr / radius)) * np.sin(lr / radius))[:, None]
        phi = ang[:, None] - (np.arange(n_r) % 2).astype(f)[None] * inc_a / f(2)
        reff = radius + doi
    else:
        rinc = (f(2) * f(c["rfov"])) / f(n_r)
        r = (rinc / f(2) + np.arange(n_r, dtype=f) * rinc - f(c["rfov"]))[:, None]
        phi = np.repeat(ang[:, None], n_r, 1)
        reff = f(c["r_scanner"])
        if samples > 1:
            o = np.arange(samples, dtype=f)[None]
            r = r - rinc / f(2) + rinc / f(samples) * o + rinc / f(2 * samples)
    phi = (phi * f(0.01745329251994329576)).astype(f)
    co, si = np.cos(phi)[:, :, None], np.sin(phi)[:, :, None]
    aux = np.sqrt(reff * reff - r * r).astype(f)[None]
    r = r[None]
    return np.stack([r * co + si * aux, r * si - co * aux, r * co - si * aux, r * si + co * aux], -1).astype(f)


def _ends(c, samples=1):
    """Axial end points of every sinogram, float32 [sinogram, sample, 2]."""
    f = np.float32
    _, sg = _geoms(c)
    afov = f(260.0) if c.get("scanner") == "mmr" else f(sg.axial_fov)
    zinc = afov / f(sg.n_rings)
    ring = zinc / f(2) + np.arange(sg.n_rings, dtype=f) * zinc
    dz = zinc / f(samples)
    out = []
    for mn, mx in zip(sg.min_rd, sg.max_rd):
        for s in range(2 * sg.n_rings):
            pairs = [(s - b, b) for b in range(sg.n_rings) if mn <= s - 2 * b <= mx and 0 <= s - b < sg.n_rings]
            if pairs:
                m = [(ring[pairs[0][k]] + ring[pairs[-1][k]]) / f(2) for k in (0, 1)]
                out.append([[v - zinc / f(2) + dz / f(2) + f(q) * dz for v in m] for q in range(samples)])
    return np.array(out, f)


def _segments(c):
    """About how many voxels one pass walks through (one direction)."""
    half = 0.5 * c["n"] * c["dxy"]
    r = np.abs(np.linspace(-c["rfov"], c["rfov"], c["n_r"]))
    chord = np.where(r < half, 2 * np.sqrt(np.maximum(half * half - r * r, 0)), 0) * 1.15
    return float(_sinos(c) * len(_angles(c)) * chord.sum() / c["dxy"] * 1.27)


# ---- inputs -----------------------------------------------------------------
def _phantom(c, seed):
    """Disc radius and hot spheres (x, y, z, radius), and the voxel centres."""
    rng = np.random.default_rng([seed, 7])
    afov = c.get("nz", 1) * c.get("dz", 1.0)
    rad = c["disc"] * rng.uniform(0.9, 1.0)
    balls = []
    for _ in range(4):
        d, th = 0.8 * rad * math.sqrt(rng.random()), 2 * math.pi * rng.random()
        balls.append((d * math.cos(th), d * math.sin(th), afov * rng.random(), rad * rng.uniform(0.06, 0.15)))
    return rad, balls


def _image(c, seed, gen):
    """A positive current estimate: the phantom with noise on it, a low background around it."""
    rad, balls = _phantom(c, seed)
    nz = c.get("nz", 1)
    x = (torch.arange(c["n"], device=DEV) + 0.5 - 0.5 * c["n"]) * c["dxy"]
    z = (torch.arange(nz, device=DEV) + 1.0) * c.get("dz", 1.0)
    img = ((x[None, :, None] ** 2 + x[None, None, :] ** 2) < rad * rad).float().expand(nz, -1, -1).clone()
    for bx, by, bz, br in balls:
        dz2 = (z[:, None, None] - bz) ** 2 if nz > 1 else torch.zeros(1, 1, 1, device=DEV)
        img[((x[None, None, :] - bx) ** 2 + (x[None, :, None] - by) ** 2 + dz2) < br * br] = 4.0
    noise = torch.rand(img.shape, generator=gen, device=DEV)
    return (img * (0.5 + noise) + 0.02 * (0.2 + noise)).reshape(-1).contiguous()


def _expected(c, seed, angles):
    """Attenuated line integrals through the phantom for the listed angles, float32 [sinogram, angle, r]."""
    rad, balls = _phantom(c, seed)
    lor = torch.from_numpy(_lor(c, angles)[:, :, 0].astype(np.float64)).to(DEV)
    p, d = lor[..., :2], lor[..., 2:] - lor[..., :2]
    dxy = (d * d).sum(-1).sqrt()
    off = (p[..., 0] * d[..., 1] - p[..., 1] * d[..., 0]).abs() / dxy
    disc = (2.0 * (rad * rad - off * off).clamp(min=0).sqrt()).float()
    flat = c["kind"] in ("em2d", "job2d")
    z = np.zeros((1, 2)) if flat else _ends(c)[:, 0].astype(np.float64)
    out = torch.empty((len(z),) + tuple(disc.shape), device=DEV)
    d, p, dxy2 = d.float(), p.float(), (dxy * dxy).float()
    step = max(1, (1 << 24) // max(1, disc.numel()))
    for s in range(0, len(z), step):
        za = torch.from_numpy(z[s:s + step]).to(DEV).float()
        dz = (za[:, 1] - za[:, 0])[:, None, None]
        len2 = dxy2[None] + dz * dz
        stretch = (len2 / dxy2[None]).sqrt()
        act = disc[None] * stretch
        for bx, by, bz, br in balls:
            wx, wy, wz = p[..., 0] - bx, p[..., 1] - by, 0.0 if flat else (za[:, 0] - bz)[:, None, None]
            wd = (wx * d[..., 0] + wy * d[..., 1])[None] + (0.0 if flat else wz * dz)
            w2 = (wx * wx + wy * wy)[None] + (0.0 if flat else wz * wz)
            act = act + 3.0 * 2.0 * (br * br - (w2 - wd * wd / len2)).clamp(min=0).sqrt()
        out[s:s + step] = act * torch.exp(-MU * disc[None] * stretch)
    return out


def _make_counts(c, seed, gen):
    """Counts of the whole sinogram, [sinogram, angle, r] flattened, in the case's type."""
    lam = _expected(c, seed, list(range(c["n_proj"])))
    lam *= c["total"] / float(lam.double().sum())
    m = torch.poisson(lam, generator=gen).reshape(-1)
    if c.get("counts", "float32") == "uint32":
        return m.to(torch.int32).view(torch.uint32)
    return m.to(torch.int16).view(torch.uint16) if c.get("counts") == "uint16" else m


def _inputs(c, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    d = {"x": _image(c, seed, gen)}
    k = c["kind"]
    if k in ("em2d", "job2d", "em", "listed", "sampled"):
        d["m"] = _make_counts(c, seed, gen)
        if c.get("add"):
            mean = c["total"] / d["m"].numel()
            d["add"] = 0.05 + mean * (0.1 + 0.1 * torch.rand(d["m"].numel(), generator=gen, device=DEV))
    if k in ("backproject", "divide"):
        nb = _sinos(c) * len(_angles(c)) * c["n_r"]
        if k == "backproject":
            d["v"] = 0.25 + torch.rand(nb, generator=gen, device=DEV)
        else:
            lam = _expected(c, seed, _angles(c)).reshape(-1)
            lam *= c["total"] / c["nsub"] / float(lam.double().sum())
            d["m"] = torch.poisson(lam, generator=gen)
            d["e"] = lam * (0.7 + 0.6 * torch.rand(nb, generator=gen, device=DEV))
    if k == "acf":
        d["x"] = (d["x"] * MU * 0.5).contiguous()
    return d


def _batch_specs(c, seed):
    """Mixed jobs: geometries, subsets and count levels of a served queue (the same geometries for every seed)."""
    shape = np.random.default_rng(4)
    out = []
    for i in range(c["jobs"]):
        n, nz = int(shape.choice([64, 96, 128])), int(shape.choice([1, 21, 41]))
        j = dict(kind="batch", counts=str(shape.choice(["float32", "uint32", "uint16"])),
                 total=float(10 ** shape.uniform(5, 7.3)), **_job(n, nz))
        out.append((j, int(shape.integers(7, 15)), seed * 100 + i))
    return out


# ---- what a program holds, and one pass --------------------------------------
def prepare(case, seed):
    c, k = case, case["kind"]
    if k == "batch":
        jobs = []
        for j, nsub, s in _batch_specs(c, seed):
            m = _make_counts(j, s, torch.Generator(device=DEV).manual_seed(s))
            m = m.view(torch.int32 if m.dtype == torch.uint32 else torch.int16 if m.dtype == torch.uint16 else m.dtype)
            h = m.cpu().numpy().view(np.dtype(j["counts"]))
            jobs.append(Job(*_geoms(j), h, c["iters"], nsub, update_positive_sens=True))
        return {"kind": k, "batch": Batch(0, c["budget"]), "jobs": jobs}
    ig, sg = _geoms(c)
    d = _inputs(c, seed)
    if k == "job2d":
        return {"kind": k, "ig": ig, "sg": sg, "m": d["m"].cpu().numpy(), "iters": c["iters"],
                "x0": np.ones(ig.n_voxels, np.float32)}
    P = ap.SiddonProjector(ig, sg)
    s = {"kind": k, "P": P, "sel": (c.get("subset", -1), c.get("nsub", 1)), **d}
    if k == "sampled":
        P.set_sampling(c["ns"], c["nas"])
    if k in ("em2d", "em", "listed", "sampled"):
        s["bp"] = torch.zeros(ig.n_voxels, device=DEV)
        s["sens"] = torch.zeros(ig.n_voxels, device=DEV)
        s["lik"] = torch.zeros(1, dtype=torch.float64, device=DEV)
        if k == "em2d":
            P.backproject(torch.ones(P.num_bins(), device=DEV), s["sens"])
        else:
            P.backproject_ones(s["sens"], *s["sel"])
        s.setdefault("add", None)
    if k == "listed":  # without factors the sensitivity is the geometry image
        P.set_option(_lib.APIRL_OPT_SPARSE_IMAGE, _lib.APIRL_SPARSE_GEOMETRY)
        s["zero_add"] = None
        if s["add"] is not None:
            a = s["add"].view(_sinos(c), c["n_proj"], c["n_r"])[:, _angles(c)]
            s["zero_add"] = a.double().sum().reshape(1)
    if k in ("project", "acf"):
        s["out"] = torch.zeros(P.num_bins(*s["sel"]), device=DEV)
    if k in ("backproject", "divide"):
        s["out"] = torch.zeros(ig.n_voxels, device=DEV)
    return s


def run(state):
    s, k = state, state["kind"]
    if k == "batch":
        return s["batch"].run_all(s["jobs"])
    if k == "job2d":
        return ap.mlem_2d(s["ig"], s["sg"], s["m"], s["x0"], s["iters"])
    P, sel = s["P"], s["sel"]
    if k in ("em2d", "em", "sampled"):
        P.em_pass(s["m"], s["x"], s["bp"], s["sens"], *sel, add=s["add"], ge=False, lik=s["lik"])
        return [s["x"], s["lik"]]
    if k == "listed":
        P.em_pass_sparse(s["m"], s["x"], s["bp"], s["sens"], s["sens"], *sel, add=s["add"], zero_add=s["zero_add"],
                         ge=False, lik=s["lik"])
        return [s["x"], s["lik"]]
    if k == "project":
        return P.project(s["x"], s["out"], *sel)
    if k == "acf":
        return P.generate_acf(s["x"], s["out"], *sel)
    if k == "backproject":
        return P.backproject(s["v"], s["out"].zero_(), *sel)
    return P.divide_and_backproject(s["m"], s["e"], s["out"].zero_(), *sel)


def work(case):
    """Each input read once, each output written once; four operations for a segment and direction."""
    c, k = case, case["kind"]
    if k == "batch":
        b = f = 0.0
        for j, nsub, _ in _batch_specs(c, 0):
            nv, nb = j["n"] ** 2 * j["nz"], _sinos(j) * j["n_proj"] * j["n_r"]
            b += nb * (2 if j["counts"] == "uint16" else 4) + 8 * nv + 16.0 * nv * c["iters"] * nsub
            f += 4.0 * _segments(j) * (c["iters"] + 1)
        return {"bytes": b, "flops": f}
    nv = c["n"] ** 2 * c.get("nz", 1)
    nb = _sinos(c) * len(_angles(c)) * c["n_r"]
    seg = _segments(c) * c.get("ns", 1) * c.get("nas", 1)
    hit = min(1.0, c["disc"] / c["rfov"])  # bins through the object: those with counts
    if k == "job2d":
        return {"bytes": 4.0 * nb + 8.0 * nv, "flops": 4.0 * seg * (1 + hit) * c["iters"]}
    if k in ("em2d", "em", "listed", "sampled"):
        size = 2 if c.get("counts") == "uint16" else 4
        return {"bytes": nb * (size + (4.0 if c.get("add") else 0)) + 12.0 * nv,
                "flops": 4.0 * seg * (2 * hit if k == "listed" else 1 + hit)}
    return {"bytes": 4.0 * nv + 4.0 * nb * (2 if k == "divide" else 1), "flops": 4.0 * seg}


# ---- the same in 64 bits -----------------------------------------------------
def _walk(c, visit):
    """Calls visit(voxel index, length) for every step of the walks of all rays of the case's subset, rays in bin
    order with a bin's samples innermost; length is 0 where a ray is outside the image or has ended."""
    f32 = torch.float32
    ig, _ = _geoms(c)
    flat = c["kind"] in ("em2d", "job2d")
    lor = torch.from_numpy(_lor(c, _angles(c), c.get("ns", 1))).to(DEV).reshape(-1, c.get("ns", 1), 4)
    if flat:
        p = lor.reshape(-1, 4)
        z0 = vz = torch.zeros(p.shape[0], device=DEV)
    else:
        ends = torch.from_numpy(_ends(c, c.get("nas", 1))).to(DEV)
        ns, nas = lor.shape[1], ends.shape[1]
        shape = (ends.shape[0], lor.shape[0], ns, nas)
        p = lor[None, :, :, None, :].expand(*shape, 4).reshape(-1, 4)
        e = ends[:, None, None, :, :].expand(*shape, 2).reshape(-1, 2)
        z0, vz = e[:, 0].clone(), e[:, 1] - e[:, 0]
    px, py = p[:, 0].clone(), p[:, 1].clone()
    vx, vy = p[:, 2] - px, p[:, 3] - py
    del p, lor
    d = [np.float32(v) for v in (ig.dx, ig.dy, ig.dz)]
    rf, oz = (d[0] * np.float32(ig.nx)) / np.float32(2), d[2] / np.float32(2)
    low, high = torch.tensor(-rf, device=DEV), torch.tensor(rf, device=DEV)
    ax1, ax2, ay1, ay2 = (low - px) / vx, (high - px) / vx, (low - py) / vy, (high - py) / vy
    big = torch.finfo(f32).max
    amin = torch.maximum(torch.where(vx == 0, -big, torch.minimum(ax1, ax2)),
                         torch.where(vy == 0, -big, torch.minimum(ay1, ay2)))
    amax = torch.minimum(torch.where(vx == 0, big, torch.maximum(ax1, ax2)),
                         torch.where(vy == 0, big, torch.maximum(ay1, ay2)))
    amin = torch.where((amin < 0) | (amin > 1), 0.0, amin)
    amax = torch.where((amax < 0) | (amax > 1), 1.0, amax)
    del ax1, ax2, ay1, ay2

    def index(p0, v, a, o, w):  # the voxel at a, in the walk's float arithmetic
        return torch.floor(((p0 + v * a) - torch.tensor(o, device=DEV)) / torch.tensor(w, device=DEV)).int()

    axes = [(px, vx, -rf, d[0]), (py, vy, -rf, d[1])] + ([] if flat else [(z0, vz, oz, d[2])])
    at = [index(p0, v, amin, o, w) for p0, v, o, w in axes]
    to = [index(p0, v, amax, o, w) for p0, v, o, w in axes]
    n = sum((b - a).abs() for a, b in zip(at, to))
    dims = [ig.nx, ig.ny, ig.nz]
    if flat:
        miss = torch.zeros_like(n, dtype=torch.bool)
        for a, b, m in zip(at, to, dims):
            miss |= ((a < 0) & (b < 0)) | ((a >= m) & (b >= m))
        n[miss] = 0
    length = sum(v.double() ** 2 for _, v, _, _ in axes).sqrt()
    inc = [torch.sign(v).int() for _, v, _, _ in axes]
    ac = amin.double()
    nxt, gap = [], []
    for i, (p0, v, o, w) in enumerate(axes):
        t = (float(o) + (at[i] + (v > 0)).double() * float(w) - p0.double()) / v.double()
        t = torch.where(v == 0, math.inf, t)
        nxt.append(torch.where(t < 0, ac, t) if flat else t)
        gap.append(torch.where(v == 0, 0.0, (float(w) / v.double()).abs()))
    del px, py, vx, vy, z0, vz, axes, amin, amax, to
    stride = [1, ig.nx, ig.nx * ig.ny]
    spare = torch.arange(n.numel(), device=DEV) % ig.n_voxels  # where a length of 0 goes
    for m in range(int(n.max())):
        an = nxt[0]
        for t in nxt[1:]:
            an = torch.minimum(an, t)
        ok = n > m
        idx = torch.zeros_like(spare)
        for a, k, s in zip(at, dims, stride):
            ok &= (a >= 0) & (a < k)
            idx += a * s
        visit(torch.where(ok, idx, spare), torch.where(ok, (an - ac) * length, 0.0))
        ac = an
        free = torch.ones_like(ok)
        for i in range(len(at)):
            hit = free & (nxt[i] == an)
            free &= ~hit
            at[i] += inc[i] * hit
            nxt[i] = torch.where(hit, nxt[i] + gap[i], nxt[i])


def _bins(c):
    return _sinos(c) * len(_angles(c)) * c["n_r"]


def _forward(c, x):
    rays = c.get("ns", 1) * c.get("nas", 1)
    acc = torch.zeros(_bins(c) * rays, dtype=torch.float64, device=DEV)
    x = x.double()

    def visit(idx, seg):
        acc.add_(seg * x[idx])

    _walk(c, visit)
    return acc.view(-1, rays).sum(1)


def _back(c, *vs):
    rays = c.get("ns", 1) * c.get("nas", 1)
    nv = c["n"] ** 2 * c.get("nz", 1)
    out = [torch.zeros(nv, dtype=torch.float64, device=DEV) for _ in vs]
    vs = [v.double().repeat_interleave(rays) if rays > 1 else v.double() for v in vs]

    def visit(idx, seg):
        for o, v in zip(out, vs):
            o.index_add_(0, idx, seg * v)

    _walk(c, visit)
    return out


def _em(c, d, x):
    """(backprojected ratio, likelihood, (counts, ratio)) of one EM pass."""
    pick = lambda a: a.view(_sinos(c), c["n_proj"], c["n_r"])[:, _angles(c)].reshape(-1).double()
    m = d["m"]
    if m.dtype in (torch.uint16, torch.uint32):
        m = m.view(torch.int16 if m.dtype == torch.uint16 else torch.int32)
    m, e = pick(m), _forward(c, x)
    if d.get("add") is not None:
        e = e + pick(d["add"])
    r = torch.where((m != 0) & (e != 0), m / e, 0.0)
    lik = torch.where(e > 0, m * torch.log(e.clamp(min=1e-300)) - e, 0.0).sum().reshape(1)
    bp, = _back(c, r)
    return bp, lik, (m, r)


def exact(case, seed):
    c, k = case, case["kind"]
    if k == "batch":  # some hundred passes over ten geometries: minutes
        return None
    d = _inputs(c, seed)
    if k == "project":
        return _forward(c, d["x"])
    if k == "acf":
        a = _forward(c, d["x"])
        return torch.where(a != 0, torch.exp(a), 1.0)
    if k == "backproject":
        return _back(c, d["v"])[0]
    if k == "divide":
        m, e = d["m"].double(), d["e"].double()
        return _back(c, torch.where(e != 0, m / e, m))[0]
    sens = _back(c, torch.ones(_bins(c), dtype=torch.float64, device=DEV))[0]
    if k != "job2d":
        x = d["x"].double()
        bp, lik, _ = _em(c, d, x)
        return [torch.where(sens > 0, x * bp / sens.clamp(min=1e-300), 0.0), lik]
    low = sens[sens != 0].min()
    thr = low + (sens.max() - low) * 1e-4
    x, liks = torch.ones_like(sens), []
    for _ in range(c["iters"]):
        bp, lik, (m, r) = _em(c, d, x)
        liks.append(lik)
        x = torch.where(sens > thr, x * bp / sens.clamp(min=1e-300), 0.0)
    last = torch.where(r > 0, m * torch.log(r.clamp(min=1e-300)) - r, 0.0).sum().reshape(1)
    return [x.cpu().numpy(), torch.cat(liks + [last]).cpu().numpy(), sens.cpu().numpy()]
