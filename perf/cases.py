"""Cases by which the framework's speed is measured.

Each case is work that a program has the framework do through its public
entry points: the whole D8 pipeline on one DEM (small, ordinary, largest,
weighted, with nodata), many small DEMs under deferred status, the functions
called one by one, the drop-in host form, the two adjoints, the edge-list
functions, graphflood's single-flow graph and the batched form.  Sizes and
terrain follow libtopotoolbox_gb300/dems.py (its workloads) and the tests;
the terrain is made on the GPU from the seed alone.

Grids are column-major: a (nrows, ncols) grid is a contiguous tensor of shape
(ncols, nrows).
"""
import math
import random

import numpy as np
import torch
import torch.nn.functional as F

from libtopotoolbox_gb300 import api, autograd
from libtopotoolbox_gb300.api import dev
from libtopotoolbox_gb300.batch import Batch

AZIMUTH, ALTITUDE, CELLSIZE = 3.9269908, 1.0471976, 30.0

# Kinds of terrain (see `_terrain`): (Hurst exponent, relief in m).
TERRAIN = {"noise": (0.7, 200.0), "rounded": (0.8, 1000.0), "nodata": (0.75, 2000.0),
           "smooth": (0.7, 800.0)}


def listed():
    return [
        # The smallest everyday DEM: launches and host round trips count.
        {"name": "pipeline_512", "kind": "pipeline", "rows": 512, "cols": 512,
         "terrain": "noise", "weights": False, "hillshade": False},
        # An integer-metre DEM, a third of it flat, with its hillshade.
        {"name": "pipeline_4096", "kind": "pipeline", "rows": 4096, "cols": 4096,
         "terrain": "rounded", "weights": False, "hillshade": True},
        # A mosaic of DEM sheets with nodata outlets, the largest grid in use.
        {"name": "pipeline_16384", "kind": "pipeline", "rows": 16384, "cols": 16384,
         "terrain": "nodata", "weights": False, "hillshade": False},
        # A clipped catchment of odd size, accumulating runoff weights.
        {"name": "pipeline_weighted", "kind": "pipeline", "rows": 3001, "cols": 5003,
         "terrain": "nodata", "weights": True, "hillshade": False},
        # A stream of small DEMs whose statuses are read once at the end.
        {"name": "deferred_tiles", "kind": "deferred", "count": 8, "low": 128, "high": 768},
        # The reference's call sequence, one call per function, every output.
        {"name": "functions", "kind": "functions", "rows": 2999, "cols": 4001,
         "terrain": "rounded"},
        # A caller of the reference's C functions: host arrays in and out.
        {"name": "host_pipeline", "kind": "host", "rows": 2048, "cols": 1500,
         "terrain": "rounded"},
        # A training step through weighted accumulation.
        {"name": "accumulate_grad", "kind": "accumulate_grad", "rows": 8192, "cols": 8192},
        # A training step through the hillshade.
        {"name": "hillshade_grad", "kind": "hillshade_grad", "rows": 8192, "cols": 8192},
        # Edge list, drainage basins and sweeps over a catchment's network.
        {"name": "edges", "kind": "edges", "rows": 2001, "cols": 3003},
        # Graphflood's single-flow graph and drainage area (host arrays).
        {"name": "sfgraph", "kind": "sfgraph", "rows": 900, "cols": 1201, "d8": True},
        # Many independent DEMs in one batch.
        {"name": "batch", "kind": "batch", "count": 64, "low": 128, "high": 1024},
    ]


def _shape(rng, low, high):
    """Sides around a log-uniform geometric mean in [low, high], aspect ratio
    in [1/2, 2], rows * cols at most high^2."""
    side = math.exp(rng.uniform(math.log(low), math.log(high)))
    aspect = math.exp(rng.uniform(-math.log(2.0), math.log(2.0)) / 2)
    return max(3, int(side * aspect)), max(3, int(side / aspect))


def draw(rng):
    kind = rng.choice(["pipeline", "pipeline", "pipeline", "deferred", "functions", "host",
                       "accumulate_grad", "hillshade_grad", "edges", "sfgraph", "batch"])
    if kind == "deferred":
        low = rng.randrange(64, 256)
        return {"kind": kind, "count": rng.randrange(2, 13), "low": low,
                "high": low * rng.randrange(2, 5)}
    if kind == "batch":
        low = rng.randrange(64, 256)
        return {"kind": kind, "count": rng.randrange(8, 129), "low": low,
                "high": low * rng.randrange(2, 9)}
    high = {"pipeline": 16384, "functions": 6000, "host": 3000, "accumulate_grad": 8192,
            "hillshade_grad": 8192, "edges": 4096, "sfgraph": 1500}[kind]
    case = {"kind": kind, "rows": 0, "cols": 0}
    if kind in ("pipeline", "functions", "host"):
        case["terrain"] = rng.choice(["noise", "rounded", "nodata"])
    if kind == "pipeline":
        case["weights"] = rng.random() < 0.3
        case["hillshade"] = rng.random() < 0.3
        if case["weights"] or case["hillshade"] or case["terrain"] != "nodata":
            high = 10000  # the largest grids come plain and with nodata
    case["rows"], case["cols"] = _shape(rng, 96 if kind == "pipeline" else 256, high)
    if kind == "sfgraph":
        case["d8"] = rng.random() < 0.75
    return case


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

def _fractal(cols, rows, hurst, relief, gen):
    """Spectral-synthesis surface spanning [0, relief], shape (cols, rows)."""
    # synthesised on a padded grid, so that any side has a fast transform
    pc, pr = -(-cols // 64) * 64, -(-rows // 64) * 64
    ky = torch.fft.fftfreq(pc, device="cuda")[:, None]
    kx = torch.fft.rfftfreq(pr, device="cuda")[None, :]
    k2 = ky * ky + kx * kx
    k2[0, 0] = 1.0
    amp = k2.pow_(-(hurst + 1.0) / 2.0)
    amp[0, 0] = 0.0
    spec = torch.randn((pc, pr // 2 + 1), dtype=torch.complex64, device="cuda", generator=gen)
    spec *= amp
    z = torch.fft.irfft2(spec, s=(pc, pr))[:cols, :rows]
    lo, hi = torch.aminmax(z)
    return ((z - lo) * (relief / (hi - lo))).contiguous()


def _pits(z, count, depths, sigmas, rnd):
    cols, rows = z.shape
    for _ in range(count):
        ci, cj = rnd.uniform(0, rows), rnd.uniform(0, cols)
        depth, sigma = rnd.uniform(*depths), rnd.uniform(*sigmas)
        r = int(math.ceil(4 * sigma))
        i0, i1 = max(0, int(ci) - r), min(rows, int(ci) + r + 1)
        j0, j1 = max(0, int(cj) - r), min(cols, int(cj) + r + 1)
        gi = torch.exp(-(torch.arange(i0, i1, device="cuda") - ci) ** 2 / (2 * sigma * sigma))
        gj = torch.exp(-(torch.arange(j0, j1, device="cuda") - cj) ** 2 / (2 * sigma * sigma))
        z[j0:j1, i0:i1] -= depth * gj[:, None] * gi[None, :]


def _disks(shape, share, radii, rnd):
    """A mask of disks that cover about `share` of the grid."""
    cols, rows = shape
    mask = torch.zeros(shape, dtype=torch.bool, device="cuda")
    left = share * rows * cols
    while left > 0:
        ci, cj, r = rnd.uniform(0, rows), rnd.uniform(0, cols), rnd.uniform(*radii)
        i0, i1 = max(0, int(ci - r)), min(rows, int(ci + r) + 1)
        j0, j1 = max(0, int(cj - r)), min(cols, int(cj + r) + 1)
        ii = torch.arange(i0, i1, device="cuda") - ci
        jj = torch.arange(j0, j1, device="cuda") - cj
        mask[j0:j1, i0:i1] |= jj[:, None] ** 2 + ii[None, :] ** 2 <= r * r
        left -= math.pi * r * r
    return mask


def _terrain(kind, rows, cols, seed):
    """(dem, bc) on the GPU.

    noise    fractal plus U[0, 0.5) m of noise: small pits everywhere
    rounded  fractal with inverted Gaussian pits, rounded to 1 m: wide flats
    nodata   fractal with closed depressions and 5 % nodata disks, which the
             callers of the pipeline pass as -INF outlets (bc = 1)
    smooth   fractal alone
    """
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed * 7 + 1)
    rnd = random.Random(seed * 7 + 2)
    hurst, relief = TERRAIN[kind]
    z = _fractal(cols, rows, hurst, relief, gen)
    bc = torch.zeros((cols, rows), dtype=torch.uint8, device="cuda")
    bc[0, :] = bc[-1, :] = 1
    bc[:, 0] = bc[:, -1] = 1
    side = math.sqrt(rows * cols)
    if kind == "noise":
        z += 0.5 * torch.rand(z.shape, device="cuda", generator=gen)
    elif kind == "rounded":
        scale = side / 4096.0
        _pits(z, 100, (5.0, 50.0), (10.0 * scale, 200.0 * scale), rnd)
        z = z.round()
    elif kind == "nodata":
        scale = side / 16384.0
        _pits(z, 250, (1.0, 100.0), (5.0 * scale + 2, 60.0 * scale + 3), rnd)
        mask = _disks(z.shape, 0.05, (max(2.0, 20.0 * scale), max(3.0, 400.0 * scale)), rnd)
        z[mask] = -math.inf
        bc[mask] = 1
    return z.contiguous(), bc


def _weights(shape, seed):
    """Lognormal(0, 0.5) runoff weights."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed * 7 + 3)
    return torch.exp(0.5 * torch.randn(shape, device="cuda", generator=gen))


def _directions(dem, bc):
    """The direction grid a program has from its routing step, and a node
    order that is the same in every run: ascending accumulation (a receiver
    accumulates more than any of its donors)."""
    o = dev.d8_pipeline(dem, bc)
    return o["direction"], torch.sort(o["acc"].reshape(-1), stable=True)[1].contiguous()


def _tile_shapes(case):
    """Sides log-uniform in [low, high], aspect ratio in [1/2, 2]: the sizes
    are the case's, the terrain on them the seed's."""
    rng = random.Random(case["count"] * 1000003 + case["low"] * 1009 + case["high"])
    shapes = []
    for _ in range(case["count"]):
        side = math.exp(rng.uniform(math.log(case["low"]), math.log(case["high"])))
        aspect = math.sqrt(rng.uniform(0.5, 2.0))
        shapes.append((max(8, round(side * aspect)), max(8, round(side / aspect))))
    return shapes


def _tiles(case, seed):
    rnd = random.Random(seed * 7 + 4)
    tiles = []
    for rows, cols in _tile_shapes(case):
        gen = torch.Generator(device="cuda")
        gen.manual_seed(rnd.randrange(1 << 40))
        z = _fractal(cols, rows, rnd.uniform(0.6, 0.9), rnd.uniform(50.0, 1500.0), gen)
        z = (torch.round(z * 10.0) / 10.0).contiguous()  # decimetres
        bc = torch.zeros((cols, rows), dtype=torch.uint8, device="cuda")
        bc[0, :] = bc[-1, :] = 1
        bc[:, 0] = bc[:, -1] = 1
        tiles.append((z, bc))
    return tiles


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("deferred", "batch"):
        tiles = _tiles(case, seed)
        s["dems"], s["bcs"] = [t[0] for t in tiles], [t[1] for t in tiles]
        if kind == "batch":  # the plan, and results that lie one after another
            s["batch"] = Batch([(d.shape[1], d.shape[0]) for d in s["dems"]])
            total = sum(d.numel() for d in s["dems"])
            types = {"filled": torch.float32, "flats": torch.int32, "dist": torch.float32,
                     "direction": torch.uint8, "acc": torch.float32}
            s["flat"] = {k: torch.empty(total, dtype=t, device="cuda") for k, t in types.items()}
            s["outputs"] = {k: [] for k in types}
            at = 0
            for d in s["dems"]:
                for k in types:
                    s["outputs"][k].append(s["flat"][k][at:at + d.numel()].view(d.shape))
                at += d.numel()
        return s
    rows, cols = case["rows"], case["cols"]
    if kind in ("pipeline", "functions"):
        s["dem"], s["bc"] = _terrain(case["terrain"], rows, cols, seed)
        if case.get("weights"):
            s["w"] = _weights(s["dem"].shape, seed)
    elif kind == "host":
        dem, bc = _terrain(case["terrain"], rows, cols, seed)
        s["dem"], s["bc"] = dem.cpu().numpy().T, bc.cpu().numpy().T  # Fortran order
    elif kind == "accumulate_grad":
        dem, bc = _terrain("smooth", rows, cols, seed)
        s["direction"] = _directions(dem, bc)[0]
        s["w"] = _weights(dem.shape, seed).requires_grad_()
        s["g"] = torch.rand(dem.shape, device="cuda",
                            generator=torch.Generator(device="cuda").manual_seed(seed))
    elif kind == "hillshade_grad":
        s["dem"] = _terrain("smooth", rows, cols, seed)[0].requires_grad_()
        s["g"] = 2 * torch.rand((cols, rows), device="cuda",
                                generator=torch.Generator(device="cuda").manual_seed(seed)) - 1
    elif kind == "edges":
        dem, bc = _terrain("rounded", rows, cols, seed)
        s["direction"], s["node"] = _directions(dem, bc)
        s["node"] = s["node"].view(dem.shape)
        s["w"] = _weights(dem.shape, seed)
        n = int((s["direction"] != 0).sum())
        s["one"] = torch.ones(n, device="cuda")
        # the share of the water that each link passes on
        s["pass"] = 0.9 + 0.1 * torch.rand(
            n, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed))
    elif kind == "sfgraph":
        dem, _ = _terrain("noise", cols, rows, seed)  # (rows, cols), row-major
        s["topo"] = dem.double().cpu().numpy()
        s["bcs"] = np.ones((rows, cols), np.uint8)  # flow may leave at the edge
        s["bcs"][0, :] = s["bcs"][-1, :] = s["bcs"][:, 0] = s["bcs"][:, -1] = 3
    return s


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------

def _without_node(o):
    # Any order with donors before receivers is a right `node`, and two runs
    # give two of them: it is computed but cannot be compared by value.
    return {k: v for k, v in o.items() if k != "node"}


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "pipeline":
        angles = (AZIMUTH, ALTITUDE) if case["hillshade"] else None
        return _without_node(dev.d8_pipeline(s["dem"], s["bc"], weights=s.get("w"),
                                             hillshade_angles=angles, cellsize=CELLSIZE))
    if kind == "deferred":
        with dev.deferred():
            out = [dev.d8_pipeline(d, b) for d, b in zip(s["dems"], s["bcs"])]
        return [_without_node(o) for o in out]
    if kind == "functions":
        filled = dev.fillsinks(s["dem"], s["bc"])
        flats = dev.identifyflats(filled)
        costs, labels = dev.gwdt_computecosts(flats, s["dem"], filled)
        prev = torch.empty(costs.shape, dtype=torch.int64, device="cuda")
        dist = dev.gwdt(costs, flats, prev=prev)
        node, direction = dev.flow_routing_d8_carve(filled, dist, flats)
        acc = dev.flow_accumulation(direction)
        return {"filled": filled, "flats": flats, "costs": costs, "labels": labels,
                "dist": dist, "prev": prev, "direction": direction, "acc": acc}
    if kind == "host":
        return _without_node(api.d8_pipeline(s["dem"], s["bc"]))
    if kind == "accumulate_grad":
        acc = autograd.flow_accumulation(s["w"], s["direction"])
        grad, = torch.autograd.grad(acc, s["w"], s["g"])
        return {"acc": acc, "grad": grad}
    if kind == "hillshade_grad":
        shade = autograd.hillshade(s["dem"], AZIMUTH, ALTITUDE, CELLSIZE)
        grad, = torch.autograd.grad(shade, s["dem"], s["g"])
        return {"shade": shade, "grad": grad}
    if kind == "edges":
        source, target = dev.flow_routing_d8_edgelist(s["node"], s["direction"])
        basins = dev.drainagebasins(source, target, s["direction"])
        acc = dev.flow_accumulation_edgelist(source, target, s["one"], s["direction"])
        flow = dev.traverse_down_f32_add_mul(s["w"].reshape(-1).clone(), s["pass"], source,
                                             target)
        # the list's length is the terrain's; all of it is read by the three calls
        return {"basins": basins, "acc": acc, "flow": flow}
    if kind == "sfgraph":
        rcv, dist, donors, ndonors, stack = api.compute_sfgraph(s["topo"], s["bcs"], CELLSIZE,
                                                                case["d8"])
        area = api.compute_drainage_area_single_flow(rcv, s["topo"].shape, CELLSIZE, stack)
        return {"rcv": rcv.view(np.int64), "dist": dist, "donors": donors.view(np.int64),
                "ndonors": ndonors, "stack": stack.view(np.int64), "area": area}
    if kind == "batch":
        s["batch"].run(s["dems"], s["bcs"], outputs=s["outputs"])
        return s["flat"]
    raise ValueError(kind)


def work(case):
    kind = case["kind"]
    if kind in ("deferred", "batch"):
        n = sum(rows * cols for rows, cols in _tile_shapes(case))
    else:
        n = case["rows"] * case["cols"]
    # bytes of a pixel: each input read once, each output written once
    per = {
        # dem 4, bc 1 | filled 4, flats 4, dist 4, node 8, direction 1, acc 4
        "pipeline": 30 + (4 if case.get("weights") else 0) + (4 if case.get("hillshade") else 0),
        "deferred": 30,
        "host": 30,
        "batch": 22,  # as the pipeline, without node
        # fill 9, flats 8, costs 24, gwdt 20, routing 21, accumulation 5
        "functions": 87,
        # direction 1, weights 4, acc 4 | direction 1, gradient 4, result 4
        "accumulate_grad": 18,
        # dem 4, shade 4 | dem 4, gradient 4, result 4
        "hillshade_grad": 20,
        # list: node 8, direction 1, edges 16 | basins: edges 16, labels 8 |
        # sums: edges 20, acc 4 | sweep: edges 20, values 8
        "edges": 101,
        # topo 8, bc 1, receivers 8, distance 8, stack 8, donor slots, counts 1
        # | receivers 8, area 8
        "sfgraph": 50 + (64 if case.get("d8") else 32),
    }[kind]
    # comparisons and additions of the stencils and sums, about one per
    # neighbour and stage: far below the bytes' time
    flops = {"pipeline": 60, "deferred": 60, "host": 60, "batch": 60, "functions": 60,
             "accumulate_grad": 2, "hillshade_grad": 60, "edges": 4, "sfgraph": 30}[kind]
    return {"bytes": per * n, "flops": flops * n}


# ---------------------------------------------------------------------------
# The same outputs in 64 bits, by plain torch
# ---------------------------------------------------------------------------

def _receivers(direction):
    """Linear index of every pixel's receiver, -1 without one."""
    cols, rows = direction.shape
    d = direction.reshape(-1)
    r = torch.full((d.numel(),), -1, dtype=torch.int64, device=d.device)
    at = torch.arange(d.numel(), device=d.device)
    for k, (di, dj) in enumerate([(0, 1), (1, 1), (1, 0), (1, -1), (0, -1), (-1, -1), (-1, 0),
                                  (-1, 1)]):
        r = torch.where(d == 1 << k, at + dj * rows + di, r)
    return r


def _down(receivers, values, share=None):
    """values summed along the flow: path doubling, each round adding the
    sums of the pixels 2^k steps upstream."""
    total, to = values.clone(), receivers.clone()
    part = torch.ones_like(total) if share is None else share.clone()
    while True:
        on = torch.nonzero(to >= 0).reshape(-1)
        if not on.numel():
            return total
        dest = to[on]
        add = total[on] * part[on]
        total = total.index_add(0, dest, add)
        part[on] = part[on] * part[dest]
        to[on] = to[dest]


def _up(receivers, values):
    """values summed along every pixel's path to its outlet, itself included."""
    total, to = values.clone(), receivers.clone()
    while True:
        on = torch.nonzero(to >= 0).reshape(-1)
        if not on.numel():
            return total
        dest = to[on]
        add, nxt = total[dest], to[dest]
        total[on] += add
        to[on] = nxt


def _axis(z, dim, h):
    def at(k):
        return z.select(dim, k)

    inner = (z.narrow(dim, 2, z.shape[dim] - 2) - z.narrow(dim, 0, z.shape[dim] - 2)) / (2 * h)
    first = ((-at(2) + 4 * at(1) - 3 * at(0)) / (2 * h)).unsqueeze(dim)
    last = ((at(-3) - 4 * at(-2) + 3 * at(-1)) / (2 * h)).unsqueeze(dim)
    return torch.cat([first, inner, last], dim)


def _shade(z):
    """Hillshade in 64 bits of a grid stored (cols, rows): x along the rows'
    axis, which is the last."""
    az, alt = float(np.float32(AZIMUTH)), float(np.float32(ALTITUDE))
    zen = math.pi / 2 - alt
    sx, sy, sz = math.sin(zen) * math.cos(az), math.sin(zen) * math.sin(az), math.cos(zen)
    dx, dy = _axis(z, 1, CELLSIZE), _axis(z, 0, CELLSIZE)
    return (-dx * sx - dy * sy + sz) / torch.sqrt(dx * dx + dy * dy + 1)


def _pool(x):
    return F.max_pool2d(x[None, None], 3, 1, 1)[0, 0]


def _fixpoint(step, x, most):
    """step applied until nothing changes; None when that takes too long."""
    for _ in range(most):
        y = x
        for _ in range(32):
            y = step(y)
        if torch.equal(x, y):
            return y
        x = y
    return None


def _routing_surfaces(dem, bc, terrain):
    """(filled, costs, dist) by plain iteration, or Nones."""
    seed = bc == 1
    top = torch.where(seed, dem, torch.full_like(dem, math.inf))
    filled = _fixpoint(lambda f: torch.where(seed, dem, torch.maximum(dem, -_pool(-f))), top, 400)
    if filled is None or terrain == "nodata":  # depths of -INF in -INF: no costs there
        return filled, None, None
    flat = -_pool(-filled) >= filled
    flat[0, :] = flat[-1, :] = False
    flat[:, 0] = flat[:, -1] = False
    # presill: a flat with a neighbour of its elevation that is no flat
    cols, rows = dem.shape
    steps = [(a, b) for a in (-1, 0, 1) for b in (-1, 0, 1) if a or b]

    def near(x, a, b, fill):
        return F.pad(x, (1, 1, 1, 1), value=fill)[1 + a:1 + a + cols, 1 + b:1 + b + rows]

    presill = torch.zeros_like(flat)
    for a, b in steps:
        presill |= (near(filled, a, b, math.nan) == filled) & ~near(flat, a, b, True)
    presill &= flat
    # the deepest point of each flat, spread over it
    low = torch.full_like(dem, -math.inf)
    depth = torch.where(flat, filled - dem, low)
    deepest = _fixpoint(lambda d: torch.where(flat, _pool(d), low), depth, 400)
    if deepest is None:
        return filled, None, None
    costs = torch.where(flat, (deepest - depth).double() + 0.1, 0.0)
    c = torch.where(flat, costs, math.inf)
    edge = [(a, b, (near(c, a, b, math.inf) + c) * (math.sqrt(2.0) if a and b else 1.0) / 2)
            for a, b in steps]
    d0 = torch.where(presill, 1.0, math.inf).double()

    def relax(d):
        for a, b, w in edge:
            d = torch.minimum(d, near(d, a, b, math.inf) + w)
        return d

    dist = _fixpoint(relax, d0, 60)
    return filled, costs, None if dist is None else torch.where(flat, dist, 0.0)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("deferred", "batch", "sfgraph"):
        # deferred, batch: as the pipeline; sfgraph is computed in 64 bits
        return None
    s = prepare(case, seed)
    if kind in ("pipeline", "functions", "host"):
        dem, bc = s["dem"], s["bc"]
        if kind == "host":
            dem, bc = (torch.from_numpy(np.ascontiguousarray(x.T)).cuda() for x in (dem, bc))
        names = ["filled", "flats", "dist", "direction", "acc"]
        if kind == "functions":
            names += ["costs", "labels", "prev"]
        out = dict.fromkeys(names)
        if case.get("hillshade"):
            out["hillshade"] = _shade(dem.double()) if bool(torch.isfinite(dem).all()) and \
                dem.numel() < 100_000_000 else None
        if dem.numel() < 20_000_000:
            out["filled"], costs, out["dist"] = _routing_surfaces(dem, bc, case["terrain"])
            if kind == "functions":
                out["costs"] = costs
        if kind == "host":
            out = {k: v if v is None else v.cpu().numpy().T for k, v in out.items()}
        return None if all(v is None for v in out.values()) else out
    if kind == "hillshade_grad":
        z = s["dem"].detach().double().requires_grad_()
        shade = _shade(z)
        grad, = torch.autograd.grad(shade, z, s["g"].double())
        return {"shade": shade.detach(), "grad": grad}
    r = _receivers(s["direction"])
    if kind == "accumulate_grad":
        shape = s["direction"].shape
        return {"acc": _down(r, s["w"].detach().double().reshape(-1)).view(shape),
                "grad": _up(r, s["g"].double().reshape(-1)).view(shape)}
    # edges: the share of a pixel is that of its place in the list
    source = s["node"].reshape(-1)
    source = source[s["direction"].reshape(-1)[source] != 0]
    share = torch.zeros(r.numel(), dtype=torch.float64, device="cuda")
    share[source] = s["pass"].double()
    w = s["w"].double().reshape(-1)
    return {"basins": None,
            "acc": _down(r, torch.ones_like(w)).view(s["direction"].shape),
            "flow": _down(r, w, share)}
