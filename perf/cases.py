"""Timed cases of the max-flow / min-cut framework.

Every case takes one solve through a public entry point, from capacities to
the exact flow and both cut sets:

  device   GridGraph with device-resident capacities: setters, max_flow, masks
  host     GridGraph with host arrays: setters, max_flow, masks read back
  replay   Batch bound to device buffers, its CUDA graph replayed
  noalloc  the allocation-free entry point for small grids
  segment  image and markers -> mask (the segmentation front-end)
  layered  GenericGraph on the layered graph of tests/graphs.py
  random   GenericGraph on a random edge list

Grids are synthetic segmentation volumes like cugip_b200.volume's (blurred
balls or tubes on a noisy background, likelihood t-links, contrast n-links),
made on the GPU from the seed.  Schedules are the library's default or, where
"pulses" is set, one the autotuner picks for that kind of workload.
"""
import ctypes as C
import math
import random

import numpy as np
import torch

from cugip_b200 import _lib
from cugip_b200.graph_cut import SINK, SOURCE, Batch, GenericGraph, GridGraph, Policy
from cugip_b200.segment import segment

LARGEST_VOXELS = 405 * 377 * 362


def _grid(name, kind, x, y, z, objects, rmin, rmax, noise, shape="balls", back=False, pulses=0, regions=0,
          pairs=0, ctas=0, warp_bfs=0, instances=1):
    return dict(name=name, kind=kind, x=x, y=y, z=z, objects=objects, rmin=rmin, rmax=rmax, noise=noise, shape=shape,
                back=back, pulses=pulses, regions=regions, pairs=pairs, ctas=ctas, warp_bfs=warp_bfs,
                instances=instances)


def listed():
    return [
        # the smallest calls: latency and launches (a region of interest, directed n-links)
        _grid("small_24x20x12", "device", 24, 20, 12, 2, 3.0, 5.0, 0.08, back=True),
        # a 2-D image
        _grid("image_640x480", "device", 640, 480, 1, 24, 8.0, 60.0, 0.08),
        # the largest grid of the allocation-free entry point: a real-time loop
        _grid("noalloc_64", "noalloc", 64, 64, 64, 2, 12.0, 16.0, 0.05),
        # an ordinary volume with the defaults
        _grid("grid_128", "device", 128, 128, 128, 6, 8.0, 24.0, 0.05),
        # host arrays of an odd-sized volume with directed n-links, masks read back
        _grid("host_225x190x170", "host", 225, 190, 170, 16, 8.0, 36.0, 0.08, back=True),
        # the benchmark's volume on its production path
        _grid("grid_256_replay", "replay", 256, 256, 256, 40, 8.0, 40.0, 0.08, pulses=4, regions=2, pairs=8, ctas=3),
        # thin structures: many short augmenting paths everywhere
        _grid("tubes_512x512x128", "device", 512, 512, 128, 200, 2.0, 6.0, 0.1, shape="tubes", pulses=4, regions=4,
              pairs=8, ctas=4, warp_bfs=8),
        # a large scan, every extent odd or ragged, defaults
        _grid("large_405x377x362", "device", 405, 377, 362, 120, 8.0, 48.0, 0.08),
        # many instances of uneven sizes (extents 32..160) in one launch
        _grid("batch_48_replay", "replay", 160, 160, 160, 12, 4.0, 24.0, 0.05, pulses=2, regions=4, pairs=4, ctas=4,
              warp_bfs=8, instances=48),
        # the front-end: image and markers in, mask out (creates and frees its grid)
        _grid("segment_150x140x96", "segment", 150, 140, 96, 8, 8.0, 30.0, 0.08),
        # non-grid graphs: deep and narrow (the reference's unit-test graph), and flat and random
        dict(name="layered_100x1024", kind="layered", layers=100, width=1024, fan=8),
        dict(name="random_200k", kind="random", vertices=200003, edges=800011),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["device", "device", "device", "host", "replay", "batch", "noalloc", "segment", "layered",
                       "random"])
    if kind == "layered":
        width = int(_log_uniform(rng, 100, 3000))
        return dict(kind=kind, layers=int(_log_uniform(rng, 10, 150)), width=width, fan=rng.randint(3, 10))
    if kind == "random":
        n = int(_log_uniform(rng, 1000, 500000))
        return dict(kind=kind, vertices=n, edges=int(n * rng.uniform(2.0, 6.0)))
    if kind == "noalloc":
        x, y, z = (rng.randint(9, 64) for _ in range(3))
    elif kind == "batch":
        x, y, z = (rng.randint(64, 160) for _ in range(3))
    else:
        n = _log_uniform(rng, 5000, {"device": 4e7, "host": 8e6, "replay": 2.5e7, "segment": 6e6}[kind])
        flat = kind == "device" and n < 2e6 and rng.random() < 0.3
        side = n ** (1 / 2 if flat else 1 / 3)
        x = max(9, int(side * rng.uniform(0.7, 1.4)))
        y = max(9, int(side * rng.uniform(0.7, 1.4)))
        z = 1 if flat else max(5, int(n / (x * y)))
    tubes = kind == "device" and z > 32 and rng.random() < 0.3
    small = min(x, y, z) if z > 1 else min(x, y)
    tuned = rng.choice([(0, 0, 0, 0, 0), (4, 2, 8, 3, 0), (4, 4, 8, 4, 8), (2, 4, 4, 4, 8)])
    if kind in ("noalloc", "segment"):
        tuned = (0, 0, 0, 0, 0)
    c = _grid("", "replay" if kind == "batch" else kind, x, y, z,
              max(2, int(x * y * z / 170000.0)) if tubes else rng.randint(2, 40),
              2.0 if tubes else max(2.0, small / 32.0), 6.0 if tubes else max(3.0, small / rng.uniform(4.0, 8.0)),
              round(rng.uniform(0.04, 0.1), 3), "tubes" if tubes else "balls",
              kind in ("device", "host") and rng.random() < 0.4, *tuned,
              instances=int(_log_uniform(rng, 3, 40)) if kind == "batch" else 1)
    c.pop("name")
    return c


# ---------------------------------------------------------------- volumes
def _paint_balls(img, case, rnd, background):
    Z, Y, X = img.shape
    dev = img.device
    for _ in range(case["objects"]):
        r = min(rnd.uniform(case["rmin"], case["rmax"]), 0.5 * max(X, Y, Z))
        cen = [rnd.uniform(min(r, (n - 1) / 2), max(n - 1 - r, (n - 1) / 2)) for n in (X, Y, Z)]
        value = rnd.uniform(0.5, 0.9)
        R = r + 7.5
        lo = [max(0, int(c - R)) for c in cen]
        hi = [min(n, int(c + R) + 2) for c, n in zip(cen, (X, Y, Z))]
        ax = [(torch.arange(lo[i], hi[i], device=dev, dtype=torch.float32) - cen[i]) ** 2 for i in range(3)]
        d = torch.sqrt(ax[2][:, None, None] + ax[1][None, :, None] + ax[0][None, None, :])
        v = background + (value - background) * 0.5 * torch.erfc((d - r) / (math.sqrt(2.0) * 1.5))
        box = img[lo[2]:hi[2], lo[1]:hi[1], lo[0]:hi[0]]
        torch.maximum(box, v, out=box)


def _paint_tubes(img, case, rnd, value):
    Z, Y, X = img.shape
    dev = img.device
    for _ in range(case["objects"]):
        n = rnd.randint(4, 6)
        r = rnd.uniform(case["rmin"], case["rmax"])
        p = np.array([[rnd.uniform(0, X - 1), rnd.uniform(0, Y - 1), rnd.uniform(0, Z - 1)] for _ in range(n)])
        pts = []
        for i in range(n - 1):  # uniform Catmull-Rom, steps of half a voxel
            p0, p1, p2, p3 = p[max(i - 1, 0)], p[i], p[i + 1], p[min(i + 2, n - 1)]
            steps = max(1, int(math.ceil(np.linalg.norm(p2 - p1) / 0.5)))
            t = np.linspace(0.0, 1.0, steps + 1)[:, None]
            pts.append(0.5 * (2 * p1 + (p2 - p0) * t + (2 * p0 - 5 * p1 + 4 * p2 - p3) * t ** 2
                              + (3 * p1 - p0 - 3 * p2 + p3) * t ** 3))
        c = torch.from_numpy(np.rint(np.concatenate(pts)).astype(np.int64)).to(dev)
        k = int(r)
        o = torch.arange(-k, k + 1, device=dev)
        off = torch.stack(torch.meshgrid(o, o, o, indexing="ij"), -1).reshape(-1, 3)
        off = off[(off * off).sum(1) <= r * r]
        q = (c[:, None, :] + off[None, :, :]).reshape(-1, 3)
        ok = ((q >= 0) & (q < torch.tensor([X, Y, Z], device=dev))).all(1)
        q = q[ok]
        img.view(-1)[q[:, 0] + X * (q[:, 1] + Y * q[:, 2])] = value


def _image(case, x, y, z, seed, dev):
    tubes = case["shape"] == "tubes"
    bg, fg = (0.3, 0.7) if tubes else (0.2, 0.8)
    rnd = random.Random(seed)
    img = torch.full((z, y, x), bg, dtype=torch.float32, device=dev)
    if tubes:
        _paint_tubes(img, case, rnd, fg)
    else:
        _paint_balls(img, case, rnd, bg)
    gen = torch.Generator(device=dev).manual_seed(seed)
    clean = img.clone()
    img += case["noise"] * torch.randn(img.shape, generator=gen, device=dev)
    return img, clean, gen, bg, fg


def _capacities(case, x, y, z, seed, dev):
    """capS, capT, forward x/y/z and (directed n-links) backward x/y/z, int32, flat."""
    img, _, gen, bg, fg = _image(case, x, y, z, seed, dev)
    a = ((img - fg) ** 2 - (img - bg) ** 2) / (2 * 0.1 * 0.1)
    pfg = torch.sigmoid(-a).clamp(1e-6, 1.0)
    pbg = (1.0 - pfg).clamp(1e-6, 1.0)
    caps = [torch.round(-10.0 * torch.log(pbg)).to(torch.int32), torch.round(-10.0 * torch.log(pfg)).to(torch.int32)]
    del a, pfg, pbg
    for dim in (2, 1, 0):
        f = torch.zeros(img.shape, dtype=torch.int32, device=dev)
        n = img.shape[dim] - 1
        if n > 0:
            d = img.narrow(dim, 1, n) - img.narrow(dim, 0, n)
            f.narrow(dim, 0, n).copy_(torch.round(50.0 * torch.exp(-d * d / (2 * 0.1 * 0.1))).to(torch.int32))
        caps.append(f)
    if case["back"]:  # directed n-links: cheaper in one direction
        for f in caps[2:5]:
            w = torch.randint(0, 3, f.shape, generator=gen, device=dev, dtype=torch.int32)
            caps.append(f // (1 + w))
    return [c.reshape(-1).contiguous() for c in caps]


def _policy(case):
    if not case["pulses"]:
        return None
    return Policy(local_pulses=case["pulses"], region_relabels=case["regions"], sweeps_per_relabel=case["pairs"],
                  ctas_per_sm=case["ctas"], bfs_warp_min=case["warp_bfs"])


def _extents(case):
    """Extents of the instances (one for all seeds of a case, as in a program that keeps its batch)."""
    if case["instances"] == 1:
        return [(case["x"], case["y"], case["z"])]
    rnd = random.Random(case["instances"])
    return [tuple(rnd.randint(32, case[a]) for a in "xyz") for _ in range(case["instances"])]


def _layered_edges(layers, width, fan):
    i = np.arange(width)
    a, b, f = [], [], []
    for layer in range(1, layers):
        for j in range(fan):
            a.append((layer - 1) * width + i)
            b.append(layer * width + (i + j) % width)
            f.append(np.full(width, 1 if layer == layers // 2 else 20))
    return np.concatenate(a), np.concatenate(b), np.concatenate(f)


# ---------------------------------------------------------------- cases
def prepare(case, seed):
    _lib.check(_lib.load().cgc_init(0))
    dev = torch.device("cuda", 0)
    kind = case["kind"]
    if kind == "layered":
        a, b, f = _layered_edges(case["layers"], case["width"], case["fan"])
        rng = np.random.default_rng(seed)
        f = np.where(f == 1, rng.integers(1, 4, f.size), rng.integers(15, 25, f.size))
        n = case["layers"] * case["width"]
        src, snk = np.zeros(n, np.int32), np.zeros(n, np.int32)
        src[:case["width"]] = rng.integers(50000, 100000, case["width"])
        snk[-case["width"]:] = 100000
        return dict(kind=kind, g=GenericGraph(n, a, b, f, 2 * f), src=src, snk=snk)
    if kind == "random":
        rng = np.random.default_rng(seed)
        n, m = case["vertices"], case["edges"]
        cap = [rng.integers(0, 50, m) * (rng.random(m) >= 0.2) for _ in range(2)]
        term = [(rng.integers(0, 80, n) * (rng.random(n) >= 0.5)).astype(np.int32) for _ in range(2)]
        g = GenericGraph(n, rng.integers(0, n, m), rng.integers(0, n, m), *cap)
        return dict(kind=kind, g=g, src=term[0], snk=term[1])
    x, y, z = case["x"], case["y"], case["z"]
    if kind == "segment":
        img, clean, gen, bg, fg = _image(case, x, y, z, seed, dev)
        mk = torch.zeros(img.shape, dtype=torch.uint8, device=dev)
        pick = torch.rand(img.shape, generator=gen, device=dev) < 0.02
        mk[(clean > 0.45) & pick] = 255
        mk[(clean < bg + 0.02) & pick] = 128
        return dict(kind=kind, image=img, markers=mk)
    pol = _policy(case)
    if kind == "replay":
        ext = _extents(case)
        b = Batch(ext)
        at, total = [], 0
        for e in ext:
            at.append(total)
            total += -(-e[0] * e[1] * e[2] // 16) * 16
        source = torch.zeros(total, dtype=torch.uint8, device=dev)
        sink = torch.zeros(total, dtype=torch.uint8, device=dev)
        flows = torch.zeros(len(ext), dtype=torch.int64, device=dev)
        caps = []
        for i, e in enumerate(ext):
            c = _capacities(case, *e, seed * 1000 + i, dev)
            caps.append(c)
            b.bind_inputs(i, c[0].data_ptr(), c[1].data_ptr(), [t.data_ptr() for t in c[2:5]])
            b.bind_outputs(i, source.data_ptr() + at[i], sink.data_ptr() + at[i])
        b.graph_create(pol, flows.data_ptr())
        return dict(kind=kind, b=b, caps=caps, flows=flows, source=source, sink=sink)
    caps = _capacities(case, x, y, z, seed, dev)
    n = x * y * z
    if kind == "host":
        host = [torch.empty(n, dtype=torch.int32, pin_memory=True).copy_(c).numpy() for c in caps]
        masks = [torch.empty(n, dtype=torch.uint8, pin_memory=True).numpy() for _ in range(2)]
        return dict(kind=kind, g=GridGraph(x, y, z), caps=host, masks=masks, policy=pol)
    masks = [torch.zeros(n, dtype=torch.uint8, device=dev) for _ in range(2)]
    if kind == "noalloc":
        planes = (C.c_void_p * 3)(*[t.data_ptr() for t in caps[2:5]])
        return dict(kind=kind, dims=(x, y, z), caps=caps, planes=planes, masks=masks)
    return dict(kind=kind, g=GridGraph(x, y, z), caps=caps, masks=masks, policy=pol)


def run(state):
    kind = state["kind"]
    if kind == "device":
        g, c = state["g"], state["caps"]
        g.set_tweights_device(c[0].data_ptr(), c[1].data_ptr())
        for ax in range(3):
            g.set_nweights_device(ax, c[2 + ax].data_ptr(), c[5 + ax].data_ptr() if len(c) > 5 else None)
        flow = g.max_flow(state["policy"])
        g.fill_segments_device(state["masks"][0].data_ptr(), 1, 0, SOURCE)
        g.fill_segments_device(state["masks"][1].data_ptr(), 255, 0, SINK)
        return flow, state["masks"]
    if kind == "host":
        g, c = state["g"], state["caps"]
        g.set_tweights(c[0], c[1])
        for ax in range(3):
            g.set_nweights(ax, c[2 + ax], c[5 + ax] if len(c) > 5 else None)
        flow = g.max_flow(state["policy"])
        g.fill_segments(state["masks"][0], 1, 0, SOURCE)
        g.fill_segments(state["masks"][1], 255, 0, SINK)
        return flow, state["masks"]
    if kind == "replay":
        state["b"].graph_launch()
        return state["flows"], state["source"], state["sink"]
    if kind == "noalloc":
        c, p = state["caps"], state["planes"]
        flow = C.c_int64()
        _lib.check(_lib.load().cgc_grid_maxflow_noalloc(
            *state["dims"], c[0].data_ptr(), c[1].data_ptr(), p, p, None, None, C.byref(flow),
            state["masks"][0].data_ptr(), state["masks"][1].data_ptr()))
        return int(flow.value), state["masks"]
    if kind == "segment":
        mask, flow = segment(state["image"], state["markers"], sigma=0.1, gaussian=True)
        return flow, mask
    g = state["g"]
    g.set_tweights(state["src"], state["snk"])
    flow = g.max_flow()
    return flow, g.fill_segments(mask=1, which=SOURCE), g.fill_segments(mask=1, which=SINK)


def work(case):
    """Each capacity read once, each mask and flow written once; the solver's operations are integer ones."""
    kind = case["kind"]
    if kind in ("layered", "random"):
        n = case["layers"] * case["width"] if kind == "layered" else case["vertices"]
        m = (case["layers"] - 1) * case["width"] * case["fan"] if kind == "layered" else case["edges"]
        return {"bytes": 8 * n + 16 * m + 2 * n + 8, "flops": 0}
    n = sum(a * b * c for a, b, c in _extents(case))
    if kind == "segment":
        return {"bytes": n * (4 + 1 + 1) + 8, "flops": 0}
    return {"bytes": n * (4 * (8 if case["back"] else 5) + 2) + 8 * case["instances"], "flops": 0}


def exact(case, seed):
    """Every output is a whole number (a flow) or a byte mask, unique for its inputs: there is nothing to round."""
    return None
