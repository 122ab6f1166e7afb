"""The work that users of this framework have it do, as cases whose time can be measured.

Each case goes through the public entry points of `mgpukde_tiled_b200`: whole studies from host arrays
(`kde_raster`), the same path step by step on device-resident inputs, several tiles in one launch, the two
fixed-bandwidth selections, the adaptive search, and the out-of-core raster.  Inputs are made on the GPU from a
seed: points of a Gaussian mixture (or uniform ones), lognormal weights, and star-shaped study areas, as in the
repository's own synthetic workloads (`synth.py`).

listed() names the cases, draw() gives more of the same ranges, prepare() makes a case's inputs, run() is one pass,
work() what a pass cannot do without, and exact() the results in 64 bits, written here in plain torch.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import mgpukde_tiled_b200 as mk

NODATA = -9999.0
TWO_PI = float(np.float32(2.0 * math.pi))  # the kernel's normalisation is defined with the float constant
FLOOR = float(np.float32(1e-14))  # the leave-one-out density's floor


# ---------------------------------------------------------------- the cases --
def _study(name, op, n, ncols, nrows, h, *, cs=1.0, org=0.0, clusters=20, edge=4, mask=True, weights=True, varh=False,
           pinned=False, nodata=0.0):
    """A density raster: n points, ncols x nrows cells of side cs with the corner at (org, org), bandwidth h (in
    coordinates), edge correction on a mask of cells `edge` times as large (0: none), `nodata` outside the study area."""
    return {"name": name, "op": op, "n": n, "ncols": ncols, "nrows": nrows, "h": h, "cs": cs, "org": org,
            "clusters": clusters, "edge": edge, "mask": mask, "weights": weights, "varh": varh, "pinned": pinned,
            "nodata": nodata}


def listed():
    return [
        # the smallest study: the size of the redwood sample (62 seedlings in the unit square, 128 x 128 cells)
        _study("study-plot", "study", 62, 128, 128, 0.12, cs=1.0 / 128.0, clusters=0, edge=1, weights=False,
               nodata=NODATA),
        # an ordinary study from ordinary (pageable) arrays: ragged raster, large coordinates, a bandwidth of 9 cells
        _study("study-county", "study", 60_000, 2311, 1873, 9.0, org=9870.0),
        # per-point bandwidths out of a file, no edge correction, no mask
        _study("study-varh", "study", 8_000, 1500, 1101, 20.0, edge=0, mask=False, varh=True),
        # a large study from page-locked arrays: the single-large workload
        _study("study-region", "study", 1_000_000, 10_000, 10_000, 50.0, clusters=50, pinned=True),
        # the same path on inputs that stay on the GPU, step by step
        _study("resident-region", "resident", 1_000_000, 10_000, 10_000, 50.0, clusters=50),
        # a fine bandwidth (4 cells) on a large ragged raster: many small discs
        _study("resident-fine", "resident", 800_000, 6001, 5003, 4.0, clusters=50, org=39_620.0),
        # the tiles of several requests in one launch, as the serving loop's ticks submit them
        {"name": "tiles-mixed", "op": "tiles", "jobs": 8, "n_lo": 1_000, "n_hi": 200_000, "side_lo": 256,
         "side_hi": 2048, "h_lo": 5.0, "h_hi": 60.0},
        # bandwidth selection on a pilot sample, and on the bandwidth-selection workload
        {"name": "select-pilot", "op": "select", "n": 2_000, "side": 500.0, "nh": 16, "h_lo": 5.0, "h_hi": 100.0,
         "edge": True, "clusters": 20},
        {"name": "select-region", "op": "select", "n": 200_000, "side": 5000.0, "nh": 64, "h_lo": 5.0, "h_hi": 500.0,
         "edge": True, "clusters": 20},
        # the golden-section search from the rule of thumb (h_option 1)
        {"name": "golden-county", "op": "golden", "n": 20_000, "side": 2000.0, "edge": True, "clusters": 20},
        # the adaptive search over (h, alpha) (h_option 2)
        {"name": "adaptive-county", "op": "adaptive", "n": 50_000, "side": 2500.0, "edge": True, "clusters": 20},
        # the raster that goes to host memory tile by tile, a background and many small clusters
        {"name": "stream-country", "op": "stream", "n": 3_000_000, "side": 16_000, "tile": 4096, "h": 30.0,
         "clusters": 500},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    op = rng.choice(["study", "study", "resident", "resident", "tiles", "select", "select", "golden", "adaptive", "stream"])
    if op in ("study", "resident"):
        side = _log(rng, 100, 5000) if op == "study" else _log(rng, 400, 9000)
        ncols, nrows = max(16, int(side * rng.uniform(0.6, 1.3))), max(16, int(side * rng.uniform(0.6, 1.3)))
        hc = min(_log(rng, 2.0, 80.0), 0.1 * min(ncols, nrows))  # in cells
        pairs = _log(rng, 2e6, 3e10)  # (point, cell) pairs inside the cutoff
        n = int(min(1_000_000, max(60, min(pairs / (28.3 * hc * hc), ncols * nrows / 4.0))))
        cs = rng.choice([1.0, 1.0, 0.5, 4.0])
        return {k: v for k, v in _study("", op, n, ncols, nrows, round(hc * cs, 3), cs=cs,
                                        org=rng.choice([0.0, 0.0, 9870.0, 39_620.0]), clusters=rng.choice([0, 20, 50]),
                                        edge=rng.choice([0, 2, 4]), mask=rng.random() < 0.7, weights=rng.random() < 0.7,
                                        varh=rng.random() < 0.25, pinned=rng.random() < 0.5,
                                        nodata=rng.choice([0.0, 0.0, NODATA])).items() if k != "name"}
    if op == "tiles":
        lo = int(_log(rng, 200, 600))
        return {"op": op, "jobs": rng.randint(2, 12), "n_lo": int(_log(rng, 500, 5000)), "n_hi": int(_log(rng, 2e4, 3e5)),
                "side_lo": lo, "side_hi": rng.randint(lo + 100, 2048), "h_lo": 5.0, "h_hi": round(rng.uniform(20.0, 80.0), 2)}
    if op == "stream":
        side = rng.randint(3000, 14_000)
        return {"op": op, "n": int(side * side * _log(rng, 1e-4, 1.2e-2)), "side": side,
                "tile": rng.choice([1024, 2048, 4096, 4096]), "h": round(_log(rng, 5.0, 60.0), 2),
                "clusters": rng.choice([50, 500])}
    n = int(_log(rng, 300, {"select": 80_000, "golden": 50_000, "adaptive": 50_000}[op]))
    case = {"op": op, "n": n, "side": round(11.2 * math.sqrt(n) * rng.uniform(0.8, 1.6), 1), "edge": rng.random() < 0.75,
            "clusters": rng.choice([0, 10, 20])}
    if op == "select":
        h_lo = rng.uniform(3.0, 8.0)
        case |= {"nh": rng.randint(4, 40), "h_lo": round(h_lo, 3), "h_hi": round(max(2 * h_lo, case["side"] * rng.uniform(0.03, 0.12)), 3)}
    return case


# --------------------------------------------------------------- the inputs --
@functools.lru_cache(None)
def _context():
    return mk.Context(0)  # one per process, as a program keeps it


def _gen(seed):
    return torch.Generator("cuda").manual_seed(int(seed))


def _points(n, x0, y0, width, height, clusters, g, background=0.0, spread=0.04):
    """n points of a mixture of `clusters` Gaussians (0: uniform) in the rectangle; draws outside are redrawn."""
    u = torch.rand(n, 2, generator=g, device="cuda", dtype=torch.float64)
    if clusters:
        c = torch.rand(clusters, 2, generator=g, device="cuda", dtype=torch.float64)
        s = (0.125 + 0.875 * torch.rand(clusters, generator=g, device="cuda", dtype=torch.float64)) * spread
        k = torch.randint(clusters, (n,), generator=g, device="cuda")
        todo = torch.arange(round(n * background), n, device="cuda")
        while len(todo):
            kk = k[todo]
            z = torch.randn(len(todo), 2, generator=g, device="cuda", dtype=torch.float64)
            u[todo] = c[kk] + s[kk, None] * z
            todo = todo[((u[todo] < 0) | (u[todo] > 1)).any(1)]
    xy = u * torch.tensor([width, height], device="cuda", dtype=torch.float64)
    return (xy[:, 0] + x0).float().contiguous(), (xy[:, 1] + y0).float().contiguous()


def _centres(grid):
    """Cell centres (x by column, y by row, row 0 on top): rounded to float, as doubles."""
    xll, yll, cs = (float(np.float32(v)) for v in (grid.xll, grid.yll, grid.cs))
    c = torch.arange(grid.ncols, device="cuda", dtype=torch.float64)
    r = torch.arange(grid.nrows, device="cuda", dtype=torch.float64)
    return (xll + (c + 0.5) * cs).float().double(), (yll + (grid.nrows - 0.5 - r) * cs).float().double()


def _star(seed, x0, y0, width, height):
    """A star-shaped polygon of 32 vertices in the rectangle."""
    r = np.random.default_rng(int(seed))
    a, q = np.sort(r.uniform(0.0, 2.0 * np.pi, 32)), r.uniform(0.35, 0.5, 32)
    return np.stack([x0 + width * (0.5 + q * np.cos(a)), y0 + height * (0.5 + q * np.sin(a))], 1)


def _mask(poly, grid):
    """1 inside the polygon, the grid's NoData value outside (even-odd, by cell centre)."""
    cx, cy = _centres(grid)
    out = torch.empty(grid.nrows, grid.ncols, device="cuda")
    step = max(1, (1 << 26) // grid.ncols)
    for r0 in range(0, grid.nrows, step):
        y = cy[r0:r0 + step]
        odd = torch.zeros(len(y), grid.ncols, device="cuda", dtype=torch.bool)
        for (ax, ay), (bx, by) in zip(poly, np.roll(poly, -1, 0)):
            cross = (y >= ay) != (y >= by)
            odd ^= cross[:, None] & (cx[None, :] < (ax + (y - ay) / (by - ay) * (bx - ax))[:, None])
        out[r0:r0 + step] = torch.where(odd, 1.0, grid.nodata)
    return out


def _weights(n, g):
    return torch.exp(0.5 * torch.randn(n, generator=g, device="cuda"))


def _host(t, pinned=False):
    return t.cpu().pin_memory().numpy() if pinned else t.cpu().numpy()


def _study_inputs(case, seed):
    g = _gen(seed)
    n, cs, org = case["n"], case["cs"], case["org"]
    dg = mk.Grid(case["ncols"], case["nrows"], org, org, cs, case["nodata"])
    width, height = dg.ncols * cs, dg.nrows * cs
    x, y = _points(n, org, org, width, height, case["clusters"], g)
    s = {"dg": dg, "x": x, "y": y, "w": _weights(n, g) if case["weights"] else None, "h_pp": None, "eg": None, "emask": None,
         "dmask": None, "h": case["h"]}
    if case["varh"]:
        s["h_pp"] = case["h"] * torch.exp(0.3 * torch.randn(n, generator=g, device="cuda")).clamp(0.4, 2.5)
    poly = _star(seed, org, org, width, height)
    if case["mask"]:
        s["dmask"] = _mask(poly, dg)
    if case["edge"]:
        k = case["edge"]
        s["eg"] = mk.Grid(-(-dg.ncols // k), -(-dg.nrows // k), org, org, cs * k, NODATA)
        s["emask"] = _mask(poly, s["eg"])
    return s


def _tile_inputs(case, seed):
    """One request per job: sizes spread over the case's ranges, small to large, bandwidths crosswise."""
    out, k = [], case["jobs"]
    for j in range(k):
        t = j / max(1, k - 1)
        n = round(case["n_lo"] * (case["n_hi"] / case["n_lo"]) ** t)
        side = round(case["side_lo"] * (case["side_hi"] / case["side_lo"]) ** ((j * 5 % k) / max(1, k - 1)))
        h = case["h_lo"] + (case["h_hi"] - case["h_lo"]) * ((j * 3 % k) / max(1, k - 1))
        g = _gen(seed * 1000 + j)
        x, y = _points(n, 0.0, 0.0, side, side, 10, g, spread=0.125)
        out.append({"x": x, "y": y, "w": _weights(n, g), "h": float(np.float32(h)), "dg": mk.Grid(side, side, 0.0, 0.0, 1.0, NODATA)})
    return out


def _sample_inputs(case, seed):
    """Points with unit weights and, with edge correction, a study area at cell 4."""
    g, side = _gen(seed), case["side"]
    x, y = _points(case["n"], 0.0, 0.0, side, side, case["clusters"], g, spread=0.08)
    eg = mk.Grid(math.ceil(side / 4.0), math.ceil(side / 4.0), 0.0, 0.0, 4.0, NODATA) if case["edge"] else None
    return {"x": x, "y": y, "w": torch.ones_like(x), "eg": eg, "emask": _mask(_star(seed, 0.0, 0.0, side, side), eg) if eg else None}


def _h_grid(case):
    k = np.arange(case["nh"])
    return (case["h_lo"] * (case["h_hi"] / case["h_lo"]) ** (k / (case["nh"] - 1))).astype(np.float32)


def prepare(case, seed):
    ctx, op = _context(), case["op"]
    if op == "study":
        s = _study_inputs(case, seed)
        for k in ("x", "y", "w", "h_pp", "dmask", "emask"):
            s[k] = None if s[k] is None else _host(s[k], case["pinned"])
        s["out"] = torch.empty(s["dg"].nrows, s["dg"].ncols, pin_memory=case["pinned"]).numpy()
    elif op == "resident":
        s = _study_inputs(case, seed)
        torch.cuda.synchronize()
        s["pts"] = mk.Points.wrap(ctx, s["x"], s["y"], s["w"], s["h_pp"])
        s["em"] = mk.Raster.wrap(ctx, s["eg"], s["emask"]) if s["eg"] else None
        hmax = float(s["h_pp"].max()) if case["varh"] else case["h"]
        s["reach"] = 3.0 * hmax * (1.0 + 1e-6)
        s["out"] = torch.empty(s["dg"].nrows, s["dg"].ncols, device="cuda")
    elif op == "tiles":
        s = {"jobs": [], "keep": []}
        for q in _tile_inputs(case, seed):
            torch.cuda.synchronize()
            pts = mk.Points.wrap(ctx, q["x"], q["y"], q["w"])
            idx = mk.Index(ctx, pts, q["h"])
            out = torch.empty(q["dg"].nrows, q["dg"].ncols, device="cuda")
            s["jobs"].append((idx, q["dg"], 0, 0, q["dg"].nrows, q["dg"].ncols, None, out))
            s["keep"].append((pts, q))
    elif op == "stream":
        g, side = _gen(seed), case["side"]
        dg = mk.Grid(side, side, 0.0, 0.0, 1.0, NODATA)
        eg = mk.Grid(-(-side // 5), -(-side // 5), 0.0, 0.0, 5.0, NODATA)
        x, y = _points(case["n"], 0.0, 0.0, side, side, case["clusters"], g, background=0.3, spread=0.005)
        s = {"dg": dg, "eg": eg, "x": x, "y": y, "w": _weights(case["n"], g), "emask": _mask(_star(seed, 0.0, 0.0, side, side), eg)}
        torch.cuda.synchronize()
        s["pts"] = mk.Points.wrap(ctx, s["x"], s["y"], s["w"])
        s["em"] = mk.Raster.wrap(ctx, eg, s["emask"])
        s["out"] = torch.empty(side, side, pin_memory=True).numpy()
    else:
        s = _sample_inputs(case, seed)
        torch.cuda.synchronize()
        s["pts"] = mk.Points.wrap(ctx, s["x"], s["y"], s["w"])
        s["em"] = mk.Raster.wrap(ctx, s["eg"], s["emask"]) if case["edge"] else None
        if op == "select":
            s["hgrid"] = _h_grid(case)
        else:
            s["h0"] = mk.rule_of_thumb(_host(s["x"]), _host(s["y"]), _host(s["w"]))
    s["case"] = dict(case)
    torch.cuda.synchronize()
    return s


# ------------------------------------------------------------------ one pass --
def run(s):
    ctx, case = _context(), s["case"]
    op = case["op"]
    if op == "study":
        den, ew, _ = mk.kde_raster(ctx, s["x"], s["y"], s["w"], s["h"], s["dg"], s["dmask"], s["eg"], s["emask"],
                                   h_pp=s["h_pp"], out=s["out"], return_ew=not case["pinned"])
        return {"density": den, "edge_weights": ew}
    if op == "tiles":
        mk.density_tiles(ctx, s["jobs"])
        return [j[-1] for j in s["jobs"]]
    pts, em = s["pts"], s["em"]
    if em is not None:
        mk.mark_boundary(ctx, em)
    if op == "resident":
        h = 0.0 if case["varh"] else s["h"]
        if em is not None:
            mk.calc_dist2_boundary(ctx, pts, em, reach=s["reach"])
            mk.edge_correction_weights(ctx, pts, em, h)
        else:
            mk.unit_edge_weights(ctx, pts)
        idx = mk.Index(ctx, pts, h)
        mk.density_tile(ctx, idx, s["dg"], 0, 0, s["dg"].nrows, s["dg"].ncols, s["dmask"], s["out"])
        idx.close()
        return s["out"]
    if op == "stream":
        mk.calc_dist2_boundary(ctx, pts, em, reach=3.0 * case["h"] * (1.0 + 1e-6))
        mk.edge_correction_weights(ctx, pts, em, case["h"])
        idx = mk.Index(ctx, pts, case["h"])
        mk.density_stream(ctx, idx, s["dg"], case["tile"], s["out"])
        idx.close()
        return s["out"]
    if op == "select":
        if em is not None:
            mk.calc_dist2_boundary(ctx, pts, em, reach=3.0 * float(s["hgrid"].max()) * (1.0 + 1e-6))
        logl, best = mk.log_likelihood_batch(ctx, pts, em, s["hgrid"])
        return {"logl": logl, "best": best}
    if em is not None:
        mk.calc_dist2_boundary(ctx, pts, em)
    if op == "golden":
        h, iterations = mk.mle_fixed_bandwidth(ctx, pts, em, s["h0"])
        return {"h": h, "iterations": iterations}
    h, alpha, lmax, iterations, hs = mk.adaptive_bandwidths(ctx, pts, em, s["h0"])
    return {"h": h, "alpha": alpha, "logl": lmax, "iterations": iterations, "hs": hs}


# -------------------------------------------------- what cannot be done without --
def work(case):
    """Bytes: each input read once, each output written once.  Operations: a multiply-add for each pair of a point
    and a cell inside the cutoff; 8 for each pair of points (distance, exponent, exponential, multiply-add).  The
    pairs are those of uniform points (clusters raise them, study areas lower them)."""
    op = case["op"]
    if op in ("study", "resident", "stream"):
        if op == "stream":
            cells = case["side"] * case["side"]
            area, io, cs = cells / 25.0 * 4, 12 * case["n"] + 4 * cells, 1.0
        else:
            cells, cs = case["ncols"] * case["nrows"], case["cs"]
            area = 4 * cells / case["edge"] ** 2 if case["edge"] else 0
            io = (8 + 4 * case["weights"] + 4 * case["varh"]) * case["n"] + 4 * cells * (1 + case["mask"])
        disc = math.pi * (3.0 * case["h"] / cs) ** 2
        return {"bytes": io + area, "flops": 2.0 * case["n"] * min(disc, cells) * (0.6 if case.get("mask") else 1.0)}
    if op == "tiles":
        b = f = 0.0
        k = case["jobs"]
        for j in range(k):
            n = case["n_lo"] * (case["n_hi"] / case["n_lo"]) ** (j / max(1, k - 1))
            side = case["side_lo"] * (case["side_hi"] / case["side_lo"]) ** ((j * 5 % k) / max(1, k - 1))
            h = case["h_lo"] + (case["h_hi"] - case["h_lo"]) * ((j * 3 % k) / max(1, k - 1))
            b += 32 * n + 4 * side * side
            f += 2.0 * n * min(math.pi * 9 * h * h, side * side)
        return {"bytes": b, "flops": f}
    n, area = case["n"], case["side"] ** 2
    hs = _h_grid(case) if op == "select" else [0.17 * case["side"] * n ** -0.25] * (34 if op == "golden" else 70)
    cells = area / 16.0 if case["edge"] else 0.0
    pairs = sum(n * n * min(1.0, 9.0 * math.pi * float(h) ** 2 / area) for h in hs)
    return {"bytes": 12.0 * n + 4 * cells, "flops": 8.0 * pairs}


# ------------------------------------------------------------------- in 64 bits --
# The definitions in plain torch: every pair by itself, distances and exponentials in double, no binning, no factors.
_CHUNK = 1 << 26


def _h2(h):
    return (h * h).double() if torch.is_tensor(h) else float(np.float32(h) * np.float32(h))


def _boundary_d2(x, y, emask, grid):
    """Squared distance of each point to the nearest boundary cell (valid, on the outer ring or next to NoData)."""
    valid = emask != NODATA
    inner = torch.nn.functional.pad(valid, (1, 1, 1, 1))
    full = torch.ones_like(valid)
    for dr in range(3):
        for dc in range(3):
            full &= inner[dr:dr + grid.nrows, dc:dc + grid.ncols]
    r, c = torch.nonzero(valid & ~full, as_tuple=True)
    cx, cy = _centres(grid)
    bx, by = cx[c], cy[r]
    d2 = torch.full((len(x),), math.inf, device="cuda", dtype=torch.float64)
    for p in range(0, len(x) if len(bx) else 0, max(1, _CHUNK // max(1, len(bx)))):
        q = slice(p, p + max(1, _CHUNK // len(bx)))
        dx, dy = bx[None, :] - x[q].double()[:, None], by[None, :] - y[q].double()[:, None]
        d2[q] = (dx * dx + dy * dy).min(1).values
    return d2


def _disc(cx, cy, x, y, h2):
    """exp(-d^2 / 2 h^2) of every (point, row, column), 0 outside the cutoff d^2 < 9 h^2."""
    dx2, dy2 = (cx[None, :] - x[:, None]) ** 2, (cy[None, :] - y[:, None]) ** 2
    d2 = dx2[:, None, :] + dy2[:, :, None]
    hh = h2[:, None, None] if torch.is_tensor(h2) else h2
    return torch.exp(d2 / (-2.0 * hh)).masked_fill_(d2 >= 9.0 * hh, 0.0)


def _edge64(x, y, h, d2b, emask, grid):
    """Edge-correction weights: 1 / (kernel mass on the valid cells), 1 for points 3h or more from the boundary."""
    e = torch.ones(len(x), device="cuda", dtype=torch.float64)
    h2 = _h2(h)
    near = torch.nonzero(d2b < 9.0 * h2)[:, 0]
    cx, cy = _centres(grid)
    v = (emask != NODATA).double()
    area = float(np.float32(grid.cs) * np.float32(grid.cs))
    step = max(1, _CHUNK // v.numel())
    for p in range(0, len(near), step):
        i = near[p:p + step]
        hh = h2[i] if torch.is_tensor(h2) else h2
        mass = (_disc(cx, cy, x[i].double(), y[i].double(), hh) * v).sum((1, 2))
        e[i] = 1.0 / (mass / (hh * TWO_PI) * area)
    return e


def _density64(x, y, wk, h, grid, mask):
    """wk: weight times edge weight of each point."""
    cx, cy = _centres(grid)
    h2 = _h2(h)
    k = wk / (h2 * TWO_PI)
    reach = 3.0 * float(torch.as_tensor(h).max()) * (1 + 1e-6)
    out = torch.zeros(grid.nrows, grid.ncols, device="cuda", dtype=torch.float64)
    rows = 16
    step = max(1, _CHUNK // (rows * grid.ncols))
    for r in range(0, grid.nrows, rows):
        yy = cy[r:r + rows]
        sel = torch.nonzero((y.double() >= yy[-1] - reach) & (y.double() <= yy[0] + reach))[:, 0]
        for p in range(0, len(sel), step):
            i = sel[p:p + step]
            f = _disc(cx, yy, x[i].double(), y[i].double(), h2[i] if torch.is_tensor(h2) else h2)
            out[r:r + rows] += (k[i][None, :] @ f.flatten(1)).view(len(yy), -1)
    return out if mask is None else torch.where(mask != grid.nodata, out, grid.nodata)


def _points64(x, y, wk, h, self_term):
    """The density at every point (its own term left out unless self_term); h by source point or one for all."""
    n, h2 = len(x), _h2(h)
    k = wk / (h2 * TWO_PI)
    xd, yd = x.double(), y.double()
    out = torch.empty(n, device="cuda", dtype=torch.float64)
    step = max(1, _CHUNK // n)
    for p in range(0, n, step):
        i = torch.arange(p, min(n, p + step), device="cuda")
        d2 = (xd[None, :] - xd[i, None]) ** 2 + (yd[None, :] - yd[i, None]) ** 2
        f = torch.exp(d2 / (-2.0 * h2)).masked_fill_(d2 >= 9.0 * h2, 0.0)
        if not self_term:
            f[i - p, i] = 0.0
        out[i] = f @ k
    return out


def _logl64(s, d2b, h):
    e = _edge64(s["x"], s["y"], h, d2b, s["emask"], s["eg"]) if s["eg"] else 1.0
    return float(torch.log(_points64(s["x"], s["y"], s["w"].double() * e, h, False).clamp_min(FLOOR)).sum())


def _adaptive_hs(s, d2b, h, alpha):
    e = _edge64(s["x"], s["y"], h, d2b, s["emask"], s["eg"]) if s["eg"] else 1.0
    den = _points64(s["x"], s["y"], s["w"].double() * e, h, True)
    return (float(np.float32(h)) * (den / torch.exp(torch.log(den).mean())) ** float(np.float32(alpha))).float()


def _adaptive64(s, d2b, h):
    """Hooke-Jeeves over (h, alpha) from (h, -0.5): float steps, likelihoods compared as floats, at most 31 moves."""
    f = np.float32
    seen = {}

    def ll(hh, aa):
        if (hh, aa) not in seen:
            seen[hh, aa] = f(_logl64(s, d2b, _adaptive_hs(s, d2b, hh, aa)))
        return seen[hh, aa]

    h, a = f(h), f(-0.5)
    sh, sa = f(h / f(10)), f(0.1)
    ends = f(sh / f(10)), f(sa / f(10))
    L = [ll(h, a), ll(f(h - sh), a), ll(f(h + sh), a), ll(h, f(a + sa)), ll(h, f(a - sa))]
    best, moves = L[0], 0
    while (sh > ends[0] or sa > ends[1]) and h - sh > 0 and moves <= 30:
        to = 0
        for i in range(5):
            if L[i] > best:
                best, to = L[i], i
        if to == 0:
            sh, sa = f(sh / f(2)), f(sa / f(2))
        elif to == 1:
            h, L[2], L[0] = f(h - sh), L[0], L[1]
        elif to == 2:
            h, L[1], L[0] = f(h + sh), L[0], L[2]
        else:  # both moves of alpha keep the likelihoods in the same places
            a = f(a + sa) if to == 3 else f(a - sa)
            L[3], L[0] = L[0], L[4]
        if to != 2:
            L[1] = ll(f(h - sh), a)
        if to != 1:
            L[2] = ll(f(h + sh), a)
        if to != 4:
            L[3] = ll(h, f(a + sa))
        if to != 3:
            L[4] = ll(h, f(a - sa))
        moves += 1
    return {"h": float(h), "alpha": float(a), "logl": float(best), "iterations": None, "hs": _adaptive_hs(s, d2b, h, a).double()}


def exact(case, seed):
    op = case["op"]
    if op == "stream":
        return None
    if op == "tiles":
        qs = _tile_inputs(case, seed)
        if sum(len(q["x"]) * (6 * q["h"] + 16) * q["dg"].ncols for q in qs) > 4e11:
            return None
        return [_density64(q["x"], q["y"], q["w"].double(), q["h"], q["dg"], None) for q in qs]
    if op in ("study", "resident"):
        hmax = 2.5 * case["h"] if case["varh"] else case["h"]
        rows = min(case["nrows"], 6 * hmax / case["cs"] + 16)
        cells = case["ncols"] * case["nrows"] / case["edge"] ** 2 if case["edge"] else 0
        if case["n"] * (rows * case["ncols"] + 0.1 * cells) > 4e11:
            return None
        s = _study_inputs(case, seed)
        h = s["h_pp"] if case["varh"] else case["h"]
        e = torch.ones(case["n"], device="cuda", dtype=torch.float64)
        if s["eg"]:
            e = _edge64(s["x"], s["y"], h, _boundary_d2(s["x"], s["y"], s["emask"], s["eg"]), s["emask"], s["eg"])
        den = _density64(s["x"], s["y"], e if s["w"] is None else s["w"].double() * e, h, s["dg"], s["dmask"])
        return {"density": den, "edge_weights": None if case["pinned"] else e} if op == "study" else den
    cells = (case["side"] / 4.0) ** 2 if case["edge"] else 0.0
    evaluations = {"select": case.get("nh", 0), "golden": 34, "adaptive": 150}[op]
    if evaluations * case["n"] * (case["n"] + 0.5 * cells) > 4e11:
        return None
    s = _sample_inputs(case, seed)
    d2b = _boundary_d2(s["x"], s["y"], s["emask"], s["eg"]) if s["eg"] else None
    if op == "select":
        return {"logl": np.array([_logl64(s, d2b, h) for h in _h_grid(case)]), "best": None}
    h0 = np.float32(mk.rule_of_thumb(_host(s["x"]), _host(s["y"]), _host(s["w"])))
    if op == "adaptive":
        return _adaptive64(s, d2b, h0)
    f = np.float32
    lo, hi = f(h0 / f(20)), f(f(2) * h0)
    width, factor = f(hi - lo), f(f(1) + np.sqrt(f(5)))
    end, moves = f(width / f(100)), 0
    while width > end and moves < 30:
        b, c = f(lo + f(width / factor)), f(hi - f(width / factor))
        if _logl64(s, d2b, b) > _logl64(s, d2b, c):
            hi = c
        else:
            lo = b
        width, moves = f(hi - lo), moves + 1
    return {"h": float(f(f(lo + hi) / f(2))), "iterations": None}
