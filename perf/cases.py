"""The work whose speed is followed: whole reconstruction calls from host tracks
and iterations of a prepared reconstruction, from the smallest scan (12^3 voxels,
thousands of muons, where a call is mostly launches and allocations) to the
256 x 256 x 128 grid with 20 million muons, in both precisions and every update.

A case is a dict of plain values; its "kind" says which entry point it goes through:

  call      MutoMLSD / MutoMAP / MutoPoCA / MutoPoCut / MutoSLR / MutoSLRIter (config).reconstruct(tracks)
  iterate   set_image, iterate(n), image of a handle prepared once (a program that
            restarts a scan from an image and looks at the result every n iterations)
  batch     Batch.reconstruct_all: many uneven scans in one handle
  gradient  nll_grad of a prepared handle (one evaluation of a gradient solver)
  fit       fit_tracks: raw detector records to tracks

The mixed form holds lambda, its lists and its sums in 32 bits, so its images are
kept as float32 arrays (the image file's default precision); the FP64 form's and
the one-shot methods' images stay float64.

Tracks are made here with torch: cos^2 zenith angles below 60 degrees, log-uniform
momenta of 1 to 10 GeV/c, entry points uniform over the grid's top, Gaussian
scattering per layer through a phantom of iron, lead, aluminium and concrete blocks
in air, three detector planes 500 mm apart on either side with 1 mm hits, and
least-squares lines through them.
"""
import math

import numpy as np
import torch

import muontomography_gb300 as M

X0_MM = {"air": 303900.0, "iron": 17.57, "lead": 5.612, "aluminium": 88.97, "concrete": 115.0}
START = 1.0e-7  # the initial lambda of every case, rad^2 / mm
GAP, PLANES, HIT_MM = 500.0, 3, 1.0
THETA_MAX = math.pi / 3


def listed():
    return [
        # a few thousand muons on a coarse grid, as in a quick look at a scan: the call's fixed costs
        {"name": "call_median_12", "kind": "call", "method": "mlsd", "update": "median", "precision": "mixed",
         "nx": 12, "ny": 12, "nz": 12, "mm": 50.0, "muons": 4000, "iterations": 5},
        # the 1 m cube of 50 mm voxels with 100 k muons, in full and in FP64
        {"name": "call_median_20_fp64", "kind": "call", "method": "mlsd", "update": "median", "precision": "fp64",
         "nx": 20, "ny": 20, "nz": 20, "mm": 50.0, "muons": 100_000, "iterations": 20},
        # a day's scan on the full grid, from pinned host tracks to the image
        {"name": "call_mean_256", "kind": "call", "method": "mlsd", "update": "mean", "precision": "mixed",
         "nx": 256, "ny": 256, "nz": 128, "mm": 10.0, "muons": 2_000_000, "iterations": 30},
        # the PoCA image that most scans start from
        {"name": "call_poca_256", "kind": "call", "method": "poca", "update": "none", "precision": "fp64",
         "nx": 256, "ny": 256, "nz": 128, "mm": 10.0, "muons": 4_000_000, "iterations": 0},
        # the in-place iterative straight-line image on the 1 m cube, an odd number of muons
        {"name": "call_slr_iter_20", "kind": "call", "method": "slr_iter", "update": "none", "precision": "fp64",
         "nx": 20, "ny": 20, "nz": 20, "mm": 50.0, "muons": 30_011, "iterations": 3},
        # the 2 m cube of 20 mm voxels, the reference's default (median) update
        {"name": "iterate_median_100", "kind": "iterate", "method": "mlsd", "update": "median", "precision": "mixed",
         "nx": 100, "ny": 100, "nz": 100, "mm": 20.0, "muons": 5_000_000, "iterations": 10},
        # the same update with the 26-neighbour prior (p = 2: with p = 1 the choice among a cubic's
        # roots turns on rounding, so two runs cannot be compared)
        {"name": "iterate_map_128", "kind": "iterate", "method": "map", "update": "median", "precision": "mixed",
         "nx": 128, "ny": 128, "nz": 64, "mm": 15.0, "muons": 5_000_000, "iterations": 5},
        # the full grid's iterations over resident lists
        {"name": "iterate_mean_256", "kind": "iterate", "method": "mlsd", "update": "mean", "precision": "mixed",
         "nx": 256, "ny": 256, "nz": 128, "mm": 10.0, "muons": 20_000_000, "iterations": 10},
        # the FP64 form on a ragged grid (the form that the mixed one is checked against)
        {"name": "iterate_mean_odd_fp64", "kind": "iterate", "method": "mlsd", "update": "mean", "precision": "fp64",
         "nx": 91, "ny": 77, "nz": 53, "mm": 17.0, "muons": 1_500_000, "iterations": 10},
        # many uneven scans at once
        {"name": "batch_24", "kind": "batch", "method": "mlsd", "update": "mean", "precision": "mixed",
         "scans": 24, "muons": 20_000, "muons_max": 400_000, "iterations": 20},
        # one evaluation of the MAP objective's gradient
        {"name": "gradient_map_96", "kind": "gradient", "method": "map", "update": "mean", "precision": "mixed",
         "nx": 96, "ny": 96, "nz": 48, "mm": 20.0, "muons": 2_000_000, "iterations": 0},
        # raw detector records to tracks, one percent of them broken
        {"name": "fit_600k", "kind": "fit", "method": "fit", "update": "none", "precision": "mixed",
         "records": 600_011, "layers": 8, "middle": 4},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["call", "call", "call", "iterate", "iterate", "iterate", "oneshot", "oneshot", "batch",
                       "gradient", "fit"])
    if kind == "fit":
        layers = rng.randint(4, 12)
        return {"kind": "fit", "method": "fit", "update": "none", "precision": rng.choice(["mixed", "fp64"]),
                "records": _log_int(rng, 1000, 600_000), "layers": layers, "middle": rng.randint(2, layers - 2)}
    if kind == "batch":
        lo = _log_int(rng, 2000, 20_000)
        return {"kind": "batch", "method": "mlsd", "update": "mean", "precision": "mixed",
                "scans": rng.randint(3, 24), "muons": lo, "muons_max": _log_int(rng, lo, 400_000),
                "iterations": rng.randint(5, 20)}
    side = _log_int(rng, 10, 200)
    nx, ny, nz = (max(6, int(round(side * rng.uniform(0.7, 1.25)))) for _ in range(3))
    nz = min(nz, 128)
    mm = 2000.0 / max(nx, ny) * rng.uniform(0.8, 1.25)
    case = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "mm": round(mm, 3)}
    if kind == "oneshot":
        method = rng.choice(["poca", "poca", "pocut", "slr", "slr_iter"])
        if method == "slr_iter":  # its passes are one after another: the sizes of the 1 m cube
            nx, ny, nz = (rng.randint(8, 20) for _ in range(3))
            case.update(nx=nx, ny=ny, nz=nz, mm=50.0, muons=_log_int(rng, 1000, 30_000))
        else:
            case["muons"] = _log_int(rng, 4000, 4_000_000)
        case.update(kind="call", method=method, update="none", precision="fp64",
                    iterations=rng.randint(1, 3) if method == "slr_iter" else 0,
                    length_weighted=rng.random() < 0.7)
        return case
    update = rng.choice(["mean", "mean", "median", "median", "percentile"])
    method = "map" if rng.random() < 0.25 else "mlsd"
    # muons so that the pairs stay below the listed cases' (about nz per kept muon)
    most = {"call": 2_000_000, "iterate": 6_000_000, "gradient": 2_000_000}[kind]
    case.update(method=method, update=update, precision=rng.choice(["mixed", "mixed", "fp64"]),
                muons=_log_int(rng, 4000, most), iterations=rng.randint(3, 10),
                straight=rng.random() < 0.15, energy=rng.random() < 0.8)
    if kind == "gradient":
        case["iterations"] = 0
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _generator(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(seed)
    return g


def _grid(c):
    h = c["mm"]
    return M.Grid(c["nx"], c["ny"], c["nz"], -c["nx"] * h / 2, -c["ny"] * h / 2, -c["nz"] * h / 2, h, h, h)


def _lambda_of(material):
    return (13.6 / 3000.0) ** 2 / X0_MM[material]


def _phantom(c, seed):
    """lambda of an (nz, ny, nx) phantom: 3 to 12 blocks of 0.05 to 0.2 of the grid's width."""
    rng = np.random.default_rng(seed)
    shape = np.array([c["nx"], c["ny"], c["nz"]])
    lam = np.full((c["nz"], c["ny"], c["nx"]), _lambda_of("air"), np.float32)
    for k in range(int(rng.integers(3, 13))):
        edge = np.maximum(rng.uniform(0.05, 0.2, 3) * shape.max(), 1.0)
        lo = rng.uniform(0.0, np.maximum(shape - edge, 0.0) + 1e-9)
        a, b = lo.astype(int), np.minimum(np.ceil(lo + edge).astype(int), shape)
        lam[a[2]:b[2], a[1]:b[1], a[0]:b[0]] = _lambda_of(("iron", "lead", "aluminium", "concrete")[k % 4])
    return torch.from_numpy(lam).to(_device())


def _line(z, h):
    """Least-squares line through hits h (n, planes) at heights z: value at z = 0 and slope."""
    z = torch.tensor(z, dtype=torch.float64, device=h.device)
    zc = z - z.mean()
    b = (h * zc).sum(1) / (zc * zc).sum()
    return h.mean(1) - b * z.mean(), b


def _tracks(c, seed, n=None):
    """(n, 14) float64 tracks on the device."""
    n = c["muons"] if n is None else n
    lam, gen, dev = _phantom(c, seed), _generator(seed), _device()
    out = torch.empty((n, 14), dtype=torch.float64, device=dev)
    for k in range(0, n, 4_000_000):
        _tracks_into(out[k:k + 4_000_000], c, lam, gen)
    return out


def _tracks_into(out, c, lam, gen):
    n, dev = out.shape[0], out.device
    nx, ny, nz, h = c["nx"], c["ny"], c["nz"], c["mm"]

    def uniform():
        return torch.rand(n, generator=gen, device=dev, dtype=torch.float64)

    c3 = math.cos(THETA_MAX) ** 3
    ct = (c3 + uniform() * (1.0 - c3)) ** (1.0 / 3.0)
    phi = 2 * math.pi * uniform()
    tan = (1.0 / (ct * ct) - 1.0).clamp_min(0.0).sqrt()
    slope = torch.stack([tan * torch.cos(phi), tan * torch.sin(phi)])  # per unit of depth
    p = 10.0 ** uniform()
    pos = torch.stack([(uniform() - 0.5) * nx * h, (uniform() - 0.5) * ny * h])
    top, bottom = nz * h / 2, -nz * h / 2

    def fitted(pos, slope, z0, planes):  # the line seen by planes at heights `planes`
        depth = torch.tensor([z0 - z for z in planes], dtype=torch.float64, device=dev)
        res = []
        for a in range(2):
            hits = pos[a][:, None] + slope[a][:, None] * depth
            hits += HIT_MM * torch.randn(hits.shape, generator=gen, device=dev, dtype=torch.float64)
            res.append(_line(planes, hits))
        norm = (res[0][1] ** 2 + res[1][1] ** 2 + 1.0).sqrt()
        at = torch.stack([res[0][0] + res[0][1] * z0, res[1][0] + res[1][1] * z0, torch.full_like(norm, z0)], 1)
        return at, torch.stack([res[0][1] / norm, res[1][1] / norm, 1.0 / norm], 1)

    pin, din = fitted(pos, slope, top, [top + k * GAP for k in range(PLANES)])
    # transport in 32 bits, a layer at a time: correlated (angle, displacement) kicks
    pos, slope, k2 = pos.float(), slope.float(), ((3.0 / p) ** 2).float()
    for z in reversed(range(nz)):
        mid = pos + slope * (0.5 * h)
        ix, iy = torch.floor(mid[0] / h + nx / 2).long(), torch.floor(mid[1] / h + ny / 2).long()
        inside = (ix >= 0) & (ix < nx) & (iy >= 0) & (iy < ny)
        lv = lam[z].reshape(-1)[(iy.clamp(0, ny - 1) * nx + ix.clamp(0, nx - 1))] * inside
        length = h * (slope[0] ** 2 + slope[1] ** 2 + 1.0).sqrt()
        s = (lv * k2 * length).sqrt()
        k = torch.randn((4, n), generator=gen, device=dev, dtype=torch.float32)
        pos = pos + slope * h + s * length * (0.5 * k[0:2] + 0.28867513 * k[2:4])
        slope = torch.tan(torch.atan(slope) + s * k[0:2])
    pout, dout = fitted(pos.double(), slope.double(), bottom, [bottom - k * GAP for k in range(PLANES)])
    out[:, 0], out[:, 1] = p, p
    out[:, 2:5], out[:, 5:8], out[:, 8:11], out[:, 11:14] = pin, pout, din, dout


def _config(c, **more):
    cfg = {"has_energy": c.get("energy", True), "straight_line": c.get("straight", False), "precision": c["precision"],
           "initialize_method": 2, "initialize_value": START, "num_iteration": c.get("iterations", 0),
           "update_with_mean": c["update"] in ("mean", "percentile"),
           "mean_percentile": 80 if c["update"] == "percentile" else 100, "early_stop": False, "eps": 1.0e-8}
    if c["kind"] != "batch":
        cfg["grid"] = _grid(c).json()
    if c["method"] == "map":
        cfg.update(beta=0.01, p=2.0, delta=0.1 * START * 1.0e7, all_neighbours=True)
    if c["method"] in ("poca", "pocut", "slr", "slr_iter"):
        cfg.update(length_weighted=c.get("length_weighted", True), angle_unit_mag=1000.0, has_energy=False)
    if c["method"] == "pocut":
        cfg["cut_percentile"] = 0.9
    cfg.update(more)
    return cfg


METHODS = {"mlsd": "MutoMLSD", "map": "MutoMAP", "poca": "MutoPoCA", "pocut": "MutoPoCut", "slr": "MutoSLR",
           "slr_iter": "MutoSLRIter"}


def _host(t):
    """A device tensor in host memory, pinned where a program would pin it (large track sets)."""
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=t.is_cuda and t.numel() > 1_000_000)
    h.copy_(t)
    return h


def _batch_scans(c):
    """The cases of a batch's scans: cubes of 16, 24, 32 or 48 voxels of 20 mm, muons log-uniform."""
    rng = np.random.default_rng(c["scans"])  # a site's scanners keep their sizes; the tracks are new each time
    out = []
    for _ in range(c["scans"]):
        n = int(rng.choice([16, 24, 32, 48]))
        m = int(math.exp(rng.uniform(math.log(c["muons"]), math.log(max(c["muons_max"], c["muons"] + 1)))))
        out.append({**c, "nx": n, "ny": n, "nz": n, "mm": 20.0, "muons": m})
    return out


def _records(c, seed):
    """(records, 2 layers + 2) hits of straight lines with 1 mm smearing above and below, 1 % NaN."""
    gen, dev, n, nz = _generator(seed), _device(), c["records"], c["layers"]
    z = _layers(c)
    xy = (torch.rand((n, 1, 2), generator=gen, device=dev, dtype=torch.float64) - 0.5) * 2000.0
    s = 0.5 * torch.randn((n, 1, 2), generator=gen, device=dev, dtype=torch.float64)
    kink = 0.01 * torch.randn((n, 1, 2), generator=gen, device=dev, dtype=torch.float64)
    zt = torch.from_numpy(z).to(dev)[None, :, None]
    hits = xy + s * zt + kink * zt.clamp_max(0.0)
    hits += HIT_MM * torch.randn(hits.shape, generator=gen, device=dev, dtype=torch.float64)
    rec = torch.empty((n, 2 * nz + 2), dtype=torch.float64, device=dev)
    rec[:, 0] = rec[:, -1] = 10.0 ** torch.rand(n, generator=gen, device=dev, dtype=torch.float64)
    rec[:, 1:-1] = hits.reshape(n, -1)
    rec[torch.randperm(n, generator=gen, device=dev)[:n // 100], 1] = float("nan")
    return rec.to(torch.float32 if c["precision"] == "mixed" else torch.float64).cpu().numpy()


def _layers(c):
    up, low = c["middle"], c["layers"] - c["middle"]
    return np.concatenate([1000.0 + GAP * np.arange(up)[::-1], -1000.0 - GAP * np.arange(low)])


def _log_image(c, seed):
    """log lambda of a gradient evaluation: the start image with a smooth seeded variation."""
    rng = np.random.default_rng(seed)
    n = c["nx"] * c["ny"] * c["nz"]
    return np.log(START) + 0.3 * np.sin(np.arange(n) * 1e-3 + rng.uniform(0, 6.28)) + 0.05 * rng.standard_normal(n)


def prepare(case, seed):
    c = case
    if c["kind"] == "fit":
        return {"case": c, "records": _records(c, seed), "layers": _layers(c)}
    if c["kind"] == "batch":
        scans = _batch_scans(c)
        return {"case": c, "rays": [_host(_tracks(s, seed * 64 + k)).numpy() for k, s in enumerate(scans)],
                "batch": M.Batch(_config(c), [_grid(s) for s in scans])}
    rays = _tracks(c, seed)
    if c["kind"] == "call":
        h = _host(rays)
        return {"case": c, "config": _config(c), "hold": h, "rays": h.numpy()}
    rec = getattr(M, METHODS[c["method"]])(_config(c))
    if rays.is_cuda:
        torch.cuda.synchronize()
    rec.load_tracks(None, rays.data_ptr(), rays.shape[0])
    rec.prepare()
    state = {"case": c, "rec": rec}
    if c["kind"] == "gradient":
        state["log"] = _log_image(c, seed)
    else:
        state["start"] = np.full((c["nx"], c["ny"], c["nz"]), START, order="F")
    return state


def _kept(c, image):
    return image if c["precision"] == "fp64" else image.astype(np.float32)


def run(state):
    c = state["case"]
    if c["kind"] == "fit":
        return M.fit_tracks(state["records"], state["layers"], c["middle"])
    if c["kind"] == "batch":
        return [_kept(c, image) for image in state["batch"].reconstruct_all(state["rays"])]
    if c["kind"] == "call":
        with getattr(M, METHODS[c["method"]])(state["config"]) as rec:
            return _kept(c, rec.reconstruct(state["rays"]))
    if c["kind"] == "gradient":
        value, grad = state["rec"].nll_grad(state["log"])
        return {"value": _kept(c, np.float64(value)), "grad": _kept(c, grad)}
    state["rec"].set_image(state["start"])
    state["rec"].iterate(c["iterations"])
    return _kept(c, state["rec"].image())


# ---------------------------------------------------------------------------
# the least work of one pass
# ---------------------------------------------------------------------------
def _pairs(c):
    """(kept muons, pairs) expected: straight lines from the tracks' distribution through the grid, the
    fraction whose closest approach lies inside taken as 0.45."""
    g = torch.Generator().manual_seed(1)
    n = 20_000
    u = torch.rand((4, n), generator=g, dtype=torch.float64)
    c3 = math.cos(THETA_MAX) ** 3
    ct = (c3 + u[0] * (1.0 - c3)) ** (1.0 / 3.0)
    tan = (1.0 / (ct * ct) - 1.0).clamp_min(0.0).sqrt()
    sx, sy = (tan * torch.cos(2 * math.pi * u[1])).abs(), (tan * torch.sin(2 * math.pi * u[1])).abs()
    # depth until a side or the bottom, in voxels
    depth = torch.minimum(torch.minimum(u[2] * c["nx"] / sx.clamp_min(1e-9), u[3] * c["ny"] / sy.clamp_min(1e-9)),
                          torch.full_like(ct, float(c["nz"])))
    voxels = float((1.0 + depth * (1.0 + sx + sy)).mean())
    kept = 0.45 * c["muons"]
    return kept, kept * voxels


def work(case):
    c = case
    if c["kind"] == "fit":
        item = 4 if c["precision"] == "mixed" else 8
        row = (2 * c["layers"] + 2) * item
        return {"bytes": c["records"] * (row + 112.0), "flops": c["records"] * (20.0 * c["layers"] + 400.0)}
    if c["kind"] == "batch":
        each = [work({**s, "kind": "call"}) for s in _batch_scans(c)]
        return {"bytes": sum(w["bytes"] for w in each), "flops": sum(w["flops"] for w in each)}
    voxels = c["nx"] * c["ny"] * c["nz"]
    kept, pairs = _pairs(c)
    real = 8 if c["precision"] == "fp64" else 4
    # an iteration reads every pair's voxel, length and tail once, the muons' data and the image
    once = {"bytes": pairs * (4 + 2 * real) + kept * 7 * real + 2.0 * voxels * real, "flops": 30.0 * pairs}
    image = 2.0 * voxels * real
    if c["kind"] == "iterate":
        return {"bytes": c["iterations"] * once["bytes"] + image, "flops": c["iterations"] * once["flops"]}
    if c["kind"] == "gradient":
        return {"bytes": once["bytes"] + 3.0 * voxels * 8, "flops": once["flops"] + 26 * 10.0 * voxels}
    rays = c["muons"] * 112.0
    if c["method"] in ("poca", "pocut", "slr"):
        return {"bytes": rays + voxels * 8.0, "flops": 10.0 * pairs}
    if c["method"] == "slr_iter":
        walk = pairs / 0.45
        return {"bytes": rays + voxels * 8.0 + (c["iterations"] - 1) * walk * 20.0,
                "flops": (10.0 + 6.0 * (c["iterations"] - 1)) * walk}
    return {"bytes": rays + image + pairs * (4 + 2 * real) + c["iterations"] * once["bytes"],
            "flops": 20.0 * pairs + c["iterations"] * once["flops"]}


# ---------------------------------------------------------------------------
# the same results in 64 bits, in plain torch and numpy
# ---------------------------------------------------------------------------
def exact(case, seed):
    c = case
    if c["kind"] == "fit":
        return _exact_fit(c, seed)
    if c["kind"] == "batch":
        if sum(_pairs(s)[1] for s in _batch_scans(c)) * c["iterations"] > 4e9:
            return None
        return [_exact_em(s, _tracks(s, seed * 64 + k)) for k, s in enumerate(_batch_scans(c))]
    if c["method"] == "slr_iter":
        return _exact_slr_iter(c, _tracks(c, seed))
    pairs = _pairs(c)[1]
    if c["method"] in ("poca", "pocut", "slr"):
        return _exact_one_shot(c, _tracks(c, seed)) if pairs < 4e8 else None
    sorts = 4 if c["update"] in ("median", "percentile") else 1
    if pairs > 2.5e8 or pairs * max(c["iterations"], 1) * sorts > 8e9:
        return None
    if c["kind"] == "gradient":
        return _exact_gradient(c, _tracks(c, seed), _log_image(c, seed))
    return _exact_em(c, _tracks(c, seed))


def _corner(c):
    h = c["mm"]
    return [-c["nx"] * h / 2, -c["ny"] * h / 2, -c["nz"] * h / 2], [c["nx"], c["ny"], c["nz"]], h


def _walk(c, p1, p2):
    """Voxels and lengths along the segments p1 -> p2 (n, 3): lists over the steps of (segment, voxel, length)."""
    lo, num, h = _corner(c)
    eps = 1.0e-6
    d = p2 - p1
    seg = (d[:, 0] ** 2 + d[:, 1] ** 2 + d[:, 2] ** 2).sqrt()
    first, last, ok = [], [], torch.ones_like(seg, dtype=torch.bool)
    for k in range(3):
        moving = d[:, k].abs() > eps
        safe = torch.where(moving, d[:, k], torch.ones_like(seg))
        a0 = torch.where(moving, (lo[k] - p1[:, k]) / safe, torch.full_like(seg, -0.1))
        an = torch.where(moving, (lo[k] + h * num[k] - p1[:, k]) / safe, torch.full_like(seg, 1.1))
        ok &= moving | ((p1[:, k] >= lo[k]) & (p1[:, k] < lo[k] + h * num[k]))
        first.append(torch.minimum(a0, an))
        last.append(torch.maximum(a0, an))
    amin = torch.maximum(torch.maximum(first[0], first[1]), first[2]).clamp_min(0.0)
    amax = torch.minimum(torch.minimum(last[0], last[1]), last[2]).clamp_max(1.0)
    ok &= amin < amax
    live = ok.nonzero()[:, 0]
    d, p1, seg, amin, amax = d[live], p1[live], seg[live], amin[live], amax[live]
    idx, step, da, an = [], [], [], []
    for k in range(3):
        dk = d[:, k]
        moving = dk.abs() > eps
        safe = torch.where(moving, dk, torch.ones_like(dk))
        nudge = torch.where(dk <= 0, -eps, eps)
        i = ((amin * dk + p1[:, k] - lo[k]) / h + nudge).trunc()
        s = torch.where(moving, torch.sign(dk), torch.zeros_like(dk))
        a = torch.where(moving, h / safe.abs(), torch.zeros_like(dk))
        nxt = (i * h + lo[k] - p1[:, k]) / safe + torch.where(s > 0, a, torch.zeros_like(a))
        nxt = torch.where(moving, nxt, torch.full_like(nxt, 1.1))
        nxt = torch.where((amin - first[k][live]).abs() < eps, amin + a, nxt)
        idx.append(i.long()); step.append(s.long()); da.append(a); an.append(nxt)
    alpha, since = amin.clone(), amin.clone()
    out = []
    for _ in range(num[0] + num[1] + num[2] + 8):
        on = alpha < amax
        if not bool(on.any()):
            break
        if int(on.sum()) * 2 < on.numel():  # the walks that have ended are dropped
            keep = on.nonzero()[:, 0]
            live, seg, amax, alpha, since = live[keep], seg[keep], amax[keep], alpha[keep], since[keep]
            idx, step, da, an = ([v[keep] for v in q] for q in (idx, step, da, an))
            on = on[keep]
        v = idx[0] + num[0] * (idx[1] + num[1] * idx[2])
        t0 = (an[0] < an[1]) & (an[0] < an[2])
        axis = [t0, ~t0 & (an[1] < an[2])]
        axis.append(~(axis[0] | axis[1]))
        now = torch.where(axis[0], an[0], torch.where(axis[1], an[1], an[2]))
        alpha = torch.where(on, now, alpha)
        for k in range(3):
            m = axis[k] & on
            an[k] = torch.where(m, an[k] + da[k], an[k])
            idx[k] = idx[k] + step[k] * m
        part = torch.minimum(alpha, amax) - since
        put = on & (part > eps)
        at = put.nonzero()[:, 0]
        out.append((live[at], v[at], part[at] * seg[at]))
        since = torch.where(put, alpha, since)
    return out


def _dot(a, b):
    return (a * b).sum(1)


def _closest(rays, eps):
    pin, pout, din, dout = rays[:, 2:5], rays[:, 5:8], rays[:, 8:11], rays[:, 11:14]
    w = pin - pout
    a, b, cc, d, e = _dot(din, din), _dot(din, dout), _dot(dout, dout), _dot(din, w), _dot(dout, w)
    den = a * cc - b * b
    flat = den.abs() < eps
    safe = torch.where(flat, torch.ones_like(den), den)
    ti, to = (b * e - cc * d) / safe, (a * e - b * d) / safe
    p = 0.5 * (pin + ti[:, None] * din + pout + to[:, None] * dout)
    return torch.where(flat[:, None], 0.5 * (pin + pout), p)


def _paths(c, rays, ps):
    """The merged paths of kept muons: (muon, voxel, length, tail) over all pairs."""
    n = rays.shape[0]
    dev = rays.device
    if c.get("straight", False):
        steps = _walk(c, rays[:, 2:5], rays[:, 5:8])
    else:
        inner, outer = _walk(c, rays[:, 2:5], ps), _walk(c, ps, rays[:, 5:8])
        count = torch.zeros(n, dtype=torch.long, device=dev)
        seen = torch.zeros(n, dtype=torch.bool, device=dev)
        for m, _, _ in inner:
            count[m] += 1
        first = torch.zeros(n, dtype=torch.float64, device=dev)  # length of the first outer voxel
        rest = []
        for m, v, l in outer:
            new = ~seen[m]
            first[m[new]] = l[new]
            seen[m] = True
            rest.append((m[~new], v[~new], l[~new]))
        at = torch.zeros(n, dtype=torch.long, device=dev)
        steps = []
        for m, v, l in inner:  # the outer half's first voxel is the inner half's last
            at[m] += 1
            steps.append((m, v, torch.where(at[m] == count[m], l + first[m], l)))
        steps += rest
    run_len = torch.zeros(n, dtype=torch.float64, device=dev)
    muon, vox, length, upto = [], [], [], []
    for m, v, l in steps:
        run_len[m] += l
        muon.append(m.int()); vox.append(v.int()); length.append(l); upto.append(run_len[m])
    muon, vox, length, upto = torch.cat(muon), torch.cat(vox), torch.cat(length), torch.cat(upto)
    return muon, vox, length, run_len[muon.long()] - upto


def _angles(rays):
    din, dout = rays[:, 8:11], rays[:, 11:14]
    return [torch.atan2(din[:, k], din[:, 2]) - torch.atan2(dout[:, k], dout[:, 2]) for k in range(2)]


class _Em:
    """The EM model of one scan in 64 bits: kept muons, their paths and the iteration's sums."""

    def __init__(self, c, rays):
        lo, num, h = _corner(c)
        eps = 1.0e-8
        ps = _closest(rays, eps)
        keep = torch.ones(rays.shape[0], dtype=torch.bool, device=rays.device)
        for k in range(3):
            keep &= (ps[:, k] >= lo[k] + eps) & (ps[:, k] <= lo[k] + h * num[k] - eps)
        keep &= (ps[:, 2] >= rays[0, 7] + eps) & (ps[:, 2] < rays[0, 4] - eps)
        rays, ps = rays[keep], ps[keep]
        self.c, self.V, self.N = c, num[0] * num[1] * num[2], rays.shape[0]
        self.muon, self.vox, self.L, self.T = _paths(c, rays, ps)
        self.mult = torch.bincount(self.vox, minlength=self.V)
        din, dout, pin, pout = rays[:, 8:11], rays[:, 11:14], rays[:, 2:5], rays[:, 5:8]
        self.S = _angles(rays)
        si, so = (lo[2] - pin[:, 2]) / din[:, 2], (lo[2] - pout[:, 2]) / dout[:, 2]
        tilt = (1.0 + (din[:, 0] / din[:, 2]) ** 2 + (din[:, 1] / din[:, 2]) ** 2).sqrt()
        self.D = []
        for k in range(2):
            ai, ao = torch.atan2(din[:, k], din[:, 2]), torch.atan2(dout[:, k], dout[:, 2])
            shift = (pout[:, k] + so * dout[:, k]) - (pin[:, k] + si * din[:, k])
            self.D.append(shift * torch.cos(ai) * tilt * torch.cos(ao) / torch.cos(ao - ai))
        self.pr2 = (3.0 / rays[:, 0]) ** 2 if c.get("energy", True) else torch.ones_like(rays[:, 0])
        self.E = (4.0 / 1.0e6, 2.0 / 1000.0, 6.0)  # hit errors of 1 mm, planes 1000 mm apart and away

    def _sum(self, index, values, n):
        out = torch.zeros(n, dtype=torch.float64, device=values.device)
        for k in range(0, values.numel(), 1 << 27):
            out.index_add_(0, index[k:k + (1 << 27)], values[k:k + (1 << 27)])
        return out

    def pair_terms(self, lam):
        """g of every pair and the cost of every muon at the image lam."""
        L, T = self.L, self.T
        l = lam[self.vox.long()]
        w11 = L * L * L / 3.0 + (L + T) * L * T
        w01 = L * T + 0.5 * L * L
        s00, s01, s11 = (self.pr2 * self._sum(self.muon, l * w, self.N) + e for w, e in zip((L, w01, w11), self.E))
        det = s00 * s11 - s01 * s01
        ok = det.abs() > 1e-12
        r = torch.where(ok, 1.0 / torch.where(ok, det, torch.ones_like(det)), torch.zeros_like(det))
        i00, i01, i11 = s11 * r, -s01 * r, s00 * r
        k0, k1, k2 = -i00, -2.0 * i01, -i11
        quad = torch.zeros_like(det)
        for S, D in zip(self.S, self.D):
            u0, u1 = i00 * S + i01 * D, i01 * S + i11 * D
            k0, k1, k2 = k0 + 0.5 * u0 * u0, k1 + u0 * u1, k2 + 0.5 * u1 * u1
            quad = quad + S * u0 + D * u1
        cost = torch.where(ok & (det > 0), torch.log(det.clamp_min(1e-300)) + 0.5 * quad, torch.zeros_like(det))
        m = self.muon.long()
        g = (self.pr2 * k0)[m] * L + (self.pr2 * k1)[m] * w01 + (self.pr2 * k2)[m] * w11
        return g, cost

    def ml_step(self, lam):
        c = self.c
        g, _ = self.pair_terms(lam)
        M_, zero = self.mult.double(), torch.zeros_like(lam)
        if c["update"] == "mean":
            return torch.where(self.mult > 0, lam + lam * lam * self._sum(self.vox, g, self.V) / (2.0 * M_.clamp_min(1.0)),
                               zero)
        # g in voxel order, ascending within a voxel
        order = torch.argsort(g)
        order = order[torch.argsort(self.vox[order], stable=True)]
        g = g[order]
        start = torch.cumsum(self.mult, 0) - self.mult
        some = self.mult > 0
        if c["update"] == "median":
            hi = g[(start + self.mult // 2).clamp_max(g.numel() - 1)]
            low = g[(start + (self.mult - 1) // 2).clamp_max(g.numel() - 1)]
            return torch.where(some, lam + lam * lam * (hi + low) * 0.25, zero)
        jm = torch.minimum((0.8 * M_).long().clamp_min(1), self.mult)
        vox = self.vox[order].long()
        rank = torch.arange(g.numel(), device=g.device) - start[vox]
        low = rank < jm[vox]
        total = self._sum(vox[low].int(), g[low], self.V)
        return torch.where(some, lam + 0.5 * lam * lam * total / jm.clamp_min(1).double(), zero)


def _stencil(c, dev):
    """Neighbour index (V, 26) with clamped edges, faces first, then edges, then corners; and their weights."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    j = torch.arange(nx * ny * nz, device=dev)
    x, y, z = j % nx, (j // nx) % ny, j // (nx * ny)
    cols, w = [], []
    for order in (1, 2, 3):
        for o in range(27):
            ox, oy, oz = o % 3 - 1, (o // 3) % 3 - 1, o // 9 - 1
            if abs(ox) + abs(oy) + abs(oz) != order:
                continue
            cols.append((x + ox).clamp(0, nx - 1) + nx * ((y + oy).clamp(0, ny - 1) + ny * (z + oz).clamp(0, nz - 1)))
            w.append(1.0 / math.sqrt(order))
    return cols, w


def _map_step(c, last, ml, mult):
    """The MAP update with p = 2: the best of the cubic's roots and the ML value."""
    beta, unit = 0.01, 1.0e7
    some = mult > 0
    Mj = mult.double().clamp_min(1.0)
    lj, lm = last * unit, ml * unit
    cols, w = _stencil(c, last.device)
    s0, s1, s2 = (torch.zeros_like(lj) for _ in range(3))
    for j, wk in zip(cols, w):
        a = lj + lj[j]
        s0, s1, s2 = s0 + wk, s1 + wk * a, s2 + wk * a * a
    p2, p3 = -beta / Mj * 4.0 * s1, beta / Mj * 8.0 * s0
    ca, cb, cc = p2 / p3, 1.0 / p3, -lm / p3
    x = -ca / 3.0
    r = 1.0 + torch.maximum(torch.maximum(ca.abs(), cb.abs()), cc.abs())
    x = torch.where(((x + ca) * x + cb) * x + cc > 0, -r, r)
    more = torch.ones_like(some)
    for _ in range(200):
        xn = x - (((x + ca) * x + cb) * x + cc) / ((3.0 * x + 2.0 * ca) * x + cb)
        xn = torch.where(more, xn, x)
        more = more & ((xn - x).abs() > 1e-8 * x.abs())
        x = xn
        if not bool(more.any()):
            break
    D = x + ca
    E = D * x + cb
    disc = D * D - 4.0 * E
    q = -0.5 * (D + torch.where(D >= 0, 1.0, -1.0) * disc.clamp_min(0.0).sqrt())
    other = torch.where(q.abs() > 1e-8, E / torch.where(q == 0, torch.ones_like(q), q), q)
    best, value = None, None
    for cand, allowed in ((x, some), (q, disc >= 0), (other, disc >= 0), (lm, some)):
        pos = cand.clamp_min(1e-300)
        v = torch.where(cand > 0, Mj * (torch.log(pos) + lm / pos), torch.zeros_like(cand))
        v = v + beta * (4.0 * cand * cand * s0 - 4.0 * cand * s1 + s2)
        v = torch.where((cand < 0) | ~allowed, torch.full_like(v, 1.7976931348623157e308), v)
        if best is None:
            best, value = cand, v
        else:
            best, value = torch.where(v < value, cand, best), torch.minimum(v, value)
    return torch.where(some, best / unit, torch.zeros_like(best))


def _image_of(c, flat):
    return flat.cpu().numpy().reshape((c["nx"], c["ny"], c["nz"]), order="F")


def _exact_em(c, rays):
    em = _Em(c, rays)
    lam = torch.full((em.V,), START, dtype=torch.float64, device=rays.device)
    if c["precision"] == "mixed":
        lam = lam.float().double()
    for _ in range(c["iterations"]):
        ml = em.ml_step(lam)
        lam = _map_step(c, lam, ml, em.mult) if c["method"] == "map" else ml
    return _image_of(c, lam)


def _exact_gradient(c, rays, log):
    em = _Em(c, rays)
    x = torch.from_numpy(log).to(rays.device)
    lam = torch.where(em.mult > 0, torch.exp(x), torch.zeros_like(x))
    g, cost = em.pair_terms(lam)
    value = float(cost.sum())
    grad = -lam * em._sum(em.vox, g, em.V)
    if c["method"] == "map":
        beta, delta, l = 0.01, 0.1 * START * 1.0e7, lam * 1.0e7
        dl = torch.zeros_like(l)
        for j, wk in zip(*_stencil(c, l.device)):
            t = l - l[j]
            value += float((2.0 * beta * wk * (t * t + delta * delta)).sum())
            slope = 2.0 * beta * wk * 2.0 * t
            dl += slope
            dl.index_add_(0, j, -slope)
        grad = grad + torch.where(em.mult > 0, l * dl, torch.zeros_like(l))
    return {"value": np.float64(value), "grad": grad.cpu().numpy()}


def _exact_one_shot(c, rays):
    lo, num, h = _corner(c)
    V = num[0] * num[1] * num[2]
    dev = rays.device
    img, weight = torch.zeros(V, dtype=torch.float64, device=dev), torch.zeros(V, dtype=torch.float64, device=dev)
    weighted = c.get("length_weighted", True)
    ax, ay = (1000.0 * a for a in _angles(rays))
    if c["method"] == "slr":
        p1, p2 = _slr_ends(c, rays)
        total = (p1 - p2).square().sum(1).sqrt()
        steps = _walk(c, p1, p2)
        a2, count = ax * ax + ay * ay, torch.zeros(rays.shape[0], dtype=torch.float64, device=dev)
        for m, _, _ in steps:
            count[m] += 1.0
        for m, v, l in steps:
            if weighted:
                weight.index_add_(0, v, l / h)
                img.index_add_(0, v, 0.5 * a2[m] * (l / total[m]) ** 2)
            else:
                weight.index_add_(0, v, torch.ones_like(l))
                img.index_add_(0, v, 0.5 * a2[m] / count[m] ** 2)
    else:
        ps = _closest(rays, 1.0e-8)
        i = torch.stack([((ps[:, k] - lo[k]) / h).trunc() for k in range(3)], 1)
        keep = (ps[:, 2] >= rays[0, 7]) & (ps[:, 2] <= rays[0, 4])
        for k in range(3):
            keep &= (i[:, k] >= 0) & (i[:, k] < num[k])
        rays, ps, i = rays[keep], ps[keep], i[keep].long()
        at = i[:, 0] + num[0] * (i[:, 1] + num[1] * i[:, 2])
        value = (ax[keep] ** 2 + ay[keep] ** 2) / 2.0
        if c["method"] == "pocut":  # the lowest 90 % of a voxel's values
            order = torch.argsort(value)
            order = order[torch.argsort(at[order], stable=True)]
            mult = torch.bincount(at, minlength=V)
            start = torch.cumsum(mult, 0) - mult
            rank = torch.arange(order.numel(), device=dev) - start[at[order]]
            low = order[rank < (mult.double() * 0.9).long()[at[order]]]
            img.index_add_(0, at[low], value[low])
        else:
            img.index_add_(0, at, value)
        for half, (a, b) in enumerate(((rays[:, 2:5], ps), (ps, rays[:, 5:8]))):
            for m, v, l in _walk(c, a, b):
                if weighted:
                    weight.index_add_(0, v, l)
                else:
                    put = v if half == 0 else v[v != at[m]]
                    weight.index_add_(0, put, torch.full((put.numel(),), h, dtype=torch.float64, device=dev))
    low = weight < 1.0e-8
    return _image_of(c, torch.where(low, torch.zeros_like(img), img / torch.where(low, torch.ones_like(weight), weight)))


def _slr_ends(c, rays):
    lo, num, h = _corner(c)
    pin, pout, din, dout = rays[:, 2:5], rays[:, 5:8], rays[:, 8:11], rays[:, 11:14]
    t1, t2 = (lo[2] + h * num[2] - pin[:, 2]) / din[:, 2], (lo[2] - pout[:, 2]) / dout[:, 2]
    return pin + t1[:, None] * din, pout + t2[:, None] * dout


def _exact_slr_iter(c, rays):
    lo, num, h = _corner(c)
    V, n = num[0] * num[1] * num[2], rays.shape[0]
    p1, p2 = _slr_ends(c, rays)
    total = (p1 - p2).square().sum(1).sqrt()
    ax, ay = (1000.0 * a for a in _angles(rays))
    steps = _walk(c, p1, p2)
    m, v, l = (torch.cat([s[k] for s in steps]) for k in range(3))
    order = torch.argsort(m, stable=True)
    m, v, l = m[order], v[order], l[order]
    count = torch.bincount(m, minlength=n)
    a2 = 0.5 * (ax * ax + ay * ay)
    if c.get("length_weighted", True):
        w, iv = l / h, a2[m] * (l / total[m]) ** 2
    else:
        w, iv = torch.ones_like(l), a2[m] / count[m].double() ** 2
    off = np.concatenate([[0], np.cumsum(count.cpu().numpy())])
    v, w, iv = v.cpu().numpy(), w.cpu().numpy(), iv.cpu().numpy()
    img, weight = np.bincount(v, iv, V), np.bincount(v, w, V)
    for _ in range(c["iterations"] - 1):
        for k in range(n):
            a, b = off[k], off[k + 1]
            if a == b:
                continue
            at = v[a:b]
            now = img[at]
            weight[at] += w[a:b]
            img[at] = now + iv[a:b] * (now / now.sum())
    out = np.where(weight < 1.0e-8, 0.0, img / np.where(weight < 1.0e-8, 1.0, weight))
    return out.reshape((c["nx"], c["ny"], c["nz"]), order="F")


def _exact_fit(c, seed):
    rec = _records(c, seed).astype(np.float64)
    rec = rec[~np.isnan(rec).any(1)]
    z, mid = _layers(c), c["middle"]
    out = np.empty((rec.shape[0], 14))
    out[:, 0], out[:, 1] = rec[:, 0], rec[:, -1]
    for (a, b), zt, where, direction in (((0, mid), z[mid - 1], 2, 8), ((mid, z.size), z[mid], 5, 11)):
        hits = np.stack([rec[:, 1 + 2 * a:1 + 2 * b:2], rec[:, 2 + 2 * a:2 + 2 * b:2],
                         np.broadcast_to(z[a:b], (rec.shape[0], b - a))], 2)
        centre = hits.mean(1)
        r = hits - centre[:, None]
        d = np.linalg.eigh(np.einsum("nki,nkj->nij", r, r))[1][:, :, 2]
        d = d * np.where(d[:, 2:3] < 0, -1.0, 1.0)
        t = (zt - centre[:, 2]) / d[:, 2]
        out[:, where:where + 3] = centre + t[:, None] * d
        out[:, where + 2] = zt
        out[:, direction:direction + 3] = d
    return out
