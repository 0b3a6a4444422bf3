"""The work whose speed is measured: what a user of gahhg_b200 has it do.

Every case goes through the package's public entry points (Polygon, Grid,
Batch, Server), over the range from one small call to the largest
configuration.  A case is a dict of plain values:

  kind      query   points on the device against one polygon's index
            host    the same from and to host arrays (Grid.query)
            batch   many polygons, their points in one call
            serve   a burst of requests to a server with resident polygons
            build   a new polygon: its index, then labels for its points
            build_batch  many new polygons, then labels for all their points
            build_ref    the drop-in path of the reference's program: build,
                         classify and query in reference semantics
  shape     star (a jittered star ring with one round hole, the small
            configuration), fractal (midpoint displacement with round holes,
            the large one), mixed (the batch configuration's polygons)
  edges     vertices of the outer ring (mixed: the largest outer ring)
  points    query points (batch kinds: the most per polygon)
  near      points: uniform by area, or half of them within 10^U[-15,-3] rad
            of an edge, in that order or shuffled
  precision fp32 / fp64 (exact labels through that filter), reference

Outputs are the labels of all points (one byte each: 1 outside, 2 inside).
They are classes, not computed values, so there is no 64-bit value for them
to be near to: they are equal to another version's or wrong.
"""
import math

import numpy as np
import torch

import gahhg_b200 as G
from gahhg_b200 import synth

PRECISION = {"fp32": G.QUERY_FP32_FILTER, "fp64": G.QUERY_FP64_FILTER, "reference": G.QUERY_REFERENCE_FP64}


def listed():
    return [
        # one small request of an interactive caller: latency and launches
        {"name": "query_1k", "kind": "query", "shape": "star", "edges": 1000, "points": 1000, "near": "no",
         "precision": "fp32"},
        # the first configuration: a 1,000-gon with a hole, a million points
        {"name": "query_1m", "kind": "query", "shape": "star", "edges": 1000, "points": 1_000_000, "near": "no",
         "precision": "fp32"},
        # the headline: a polygon of a million edges, points all over the sphere
        {"name": "query_100m", "kind": "query", "shape": "fractal", "edges": 1_000_000, "points": 100_000_000,
         "near": "no", "precision": "fp32"},
        # the precision configuration: half of the points next to an edge
        {"name": "near_20m", "kind": "query", "shape": "fractal", "edges": 1_000_000, "points": 20_000_000,
         "near": "half", "precision": "fp32"},
        # the same kind of points in the order a feed would bring them, by the FP64 filter
        {"name": "near_shuffled_fp64", "kind": "query", "shape": "fractal", "edges": 300_000, "points": 5_000_001,
         "near": "shuffled", "precision": "fp64"},
        # the reference's own semantics, as its users have it: a million points
        {"name": "reference_1m", "kind": "query", "shape": "star", "edges": 1000, "points": 1_000_000, "near": "no",
         "precision": "reference"},
        # points that live in host memory (a file that was loaded), labels back in host memory
        {"name": "host_3m", "kind": "host", "shape": "fractal", "edges": 100_000, "points": 3_000_017, "near": "no",
         "precision": "fp32"},
        # the batch configuration, a part of it: many polygons of very different sizes in one call
        {"name": "batch_160", "kind": "batch", "shape": "mixed", "edges": 200_000, "polygons": 160,
         "points": 1_000_000, "near": "no", "precision": "fp32"},
        # the serving configuration: a burst of requests of 1 to 1,000,000 points
        {"name": "serve_96", "kind": "serve", "shape": "mixed", "edges": 20_000, "polygons": 32, "requests": 96,
         "points": 1_000_000, "near": "no", "precision": "fp32"},
        # a new large polygon comes in and is asked at once
        {"name": "build_1m", "kind": "build", "shape": "fractal", "edges": 1_000_000, "points": 1_000_000,
         "near": "no", "precision": "fp32"},
        # a set of new polygons comes in and is asked at once
        {"name": "build_batch_96", "kind": "build_batch", "shape": "mixed", "edges": 100_000, "polygons": 96,
         "points": 50_000, "near": "no", "precision": "fp32"},
        # what the reference's program does per invocation, on a coastline of 10,000 vertices
        {"name": "build_ref_10k", "kind": "build_ref", "shape": "fractal", "edges": 10_000, "points": 100_000,
         "near": "no", "precision": "reference"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["query", "query", "query", "query", "host", "batch", "batch", "serve", "build", "build_batch",
                       "build_ref"])
    if kind == "query":
        precision = rng.choice(["fp32", "fp32", "fp64", "reference"])
        shape = rng.choice(["star", "fractal"])
        edges = _log(rng, 50, 4000) if shape == "star" else _log(rng, 1000, 50_000 if precision == "reference" else
                                                                 1_000_000)
        near = rng.choice(["no", "half", "shuffled"])
        most = 5_000_000 if precision == "reference" else 100_000_000 if near == "no" else 20_000_000
        return {"kind": kind, "shape": shape, "edges": edges, "points": _log(rng, 300, most), "near": near,
                "precision": precision}
    if kind == "host":
        return {"kind": kind, "shape": "fractal", "edges": _log(rng, 1000, 300_000),
                "points": _log(rng, 1000, 10_000_000), "near": "no", "precision": rng.choice(["fp32", "fp64"])}
    if kind == "batch":
        return {"kind": kind, "shape": "mixed", "edges": _log(rng, 1000, 200_000), "polygons": _log(rng, 4, 160),
                "points": _log(rng, 2000, 1_000_000), "near": "no", "precision": rng.choice(["fp32", "fp32", "fp64"])}
    if kind == "serve":
        return {"kind": kind, "shape": "mixed", "edges": _log(rng, 1000, 20_000), "polygons": _log(rng, 2, 32),
                "requests": _log(rng, 4, 96), "points": _log(rng, 1000, 1_000_000), "near": "no", "precision": "fp32"}
    if kind == "build":
        return {"kind": kind, "shape": "fractal", "edges": _log(rng, 1000, 1_000_000),
                "points": _log(rng, 10_000, 1_000_000), "near": rng.choice(["no", "half"]), "precision": "fp32"}
    if kind == "build_batch":
        return {"kind": kind, "shape": "mixed", "edges": _log(rng, 1000, 100_000), "polygons": _log(rng, 4, 96),
                "points": _log(rng, 2000, 50_000), "near": "no", "precision": "fp32"}
    return {"kind": kind, "shape": "fractal", "edges": _log(rng, 500, 30_000), "points": _log(rng, 1000, 300_000),
            "near": "no", "precision": "reference"}


# ------------------------------------------------------------------ inputs --

def _rings(case, seed):
    """One polygon of the case's shape; its place, jitter and displacements from the seed."""
    rng = np.random.default_rng(seed)
    lon, lat = float(rng.uniform(-180.0, 180.0)), float(rng.uniform(-70.0, 70.0))
    n = case["edges"]
    if case["shape"] == "star":
        outer = synth.star_ring(lon, lat, n, 30.0, 0.2, rng)
        return [outer, synth.star_ring(lon, lat, max(4, n // 10), 5.0, 0.0, rng)]
    if n >= 200_000:  # the large configuration's polygon: ten holes of a hundredth of its vertices
        return synth.c1_polygon(seed=seed, n_outer=n, hole_n=max(4, n // 100))
    outer, _ = synth.displaced_ring(lon, lat, n, 40.0, base=64, amp_deg=4.0, rng=rng)
    return [outer, synth.star_ring(lon, lat, max(4, n // 20), 4.0, 0.0, rng)]


def _device_points(case, rings, seed):
    if case["near"] == "no":
        return synth.device_points(case["points"], seed, "cuda")
    n = case["points"]
    pts = synth.device_c2_points(rings, n + n % 2, seed, "cuda")[:n]
    if case["near"] == "shuffled":
        g = torch.Generator(device="cuda")
        g.manual_seed(seed)
        pts = pts[torch.randperm(case["points"], generator=g, device="cuda")].contiguous()
    return pts


def _mixed(case, seed):
    """Polygons of the batch configuration and log-uniform point counts in
    their caps (the counts are the case's, the same for every seed)."""
    polys = synth.c3_polygons(case["polygons"], seed=seed, vmax=case["edges"])
    most = case["points"]
    rng = np.random.default_rng(most)
    counts = [_log_np(rng, min(1000, most), most) for _ in polys]
    return polys, counts


def _log_np(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cap_points(polys, counts, seed):
    return synth.device_cap_points([c[0] for _r, c, _d in polys], [c[1] for _r, c, _d in polys],
                                   [d for _r, _c, d in polys], counts, seed, "cuda")


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "precision": PRECISION[case["precision"]]}
    if kind in ("query", "host", "build", "build_ref"):
        rings = _rings(case, seed)
        s["polygon"] = G.Polygon.from_rings(rings)
        if kind in ("query", "host"):
            semantics = G.SEMANTICS_REFERENCE if case["precision"] == "reference" else G.SEMANTICS_EXACT
            s["grid"] = G.Grid(s["polygon"], semantics=semantics).classify()
        if kind in ("query", "build"):
            s["points"] = _device_points(case, rings, seed)
            s["labels"] = torch.empty(case["points"], dtype=torch.uint8, device="cuda")
        else:
            s["points"] = synth.uniform_points(case["points"], np.random.default_rng(seed))
    elif kind in ("batch", "build_batch"):
        polys, counts = _mixed(case, seed)
        s["polygons"] = [G.Polygon.from_rings(r) for r, _c, _d in polys]
        s["offsets"] = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
        s["points"] = _cap_points(polys, counts, seed)
        s["labels"] = torch.empty(int(s["offsets"][-1]), dtype=torch.uint8, device="cuda")
        if kind == "batch":
            s["batch"] = G.Batch(s["polygons"])
    else:
        polys = synth.c3_polygons(case["polygons"], seed=seed, vmax=case["edges"])
        which = np.random.default_rng(seed + 1).integers(0, len(polys), case["requests"])
        rng = np.random.default_rng(case["points"])
        sizes = [_log_np(rng, 1, case["points"]) for _ in which]  # the case's, the same for every seed
        rng = np.random.default_rng(seed + 2)
        flat = [synth.cap_points(polys[p][1][0], polys[p][1][1], 1.8 * polys[p][2], n, rng)
                for p, n in zip(which, sizes)]
        s["offsets"] = np.concatenate([[0], np.cumsum(sizes)])
        s["points"] = np.concatenate(flat)
        s["labels"] = np.zeros(len(s["points"]), dtype=np.uint8)
        server = G.Server(hbm_budget=4 << 30)
        ids = []
        for rings, _c, _d in polys:
            pid, ticket = server.build(G.Polygon.from_rings(rings))
            server.wait(ticket)
            ids.append(pid)
        s["server"] = server
        s["requests"] = [ids[p] for p in which]
    return s


# -------------------------------------------------------------------- pass --

def run(s):
    kind = s["case"]["kind"]
    if kind == "query":
        s["grid"].query_device(s["points"].data_ptr(), len(s["points"]), s["labels"].data_ptr(), s["precision"],
                               stream=torch.cuda.current_stream().cuda_stream)
        return s["labels"]
    if kind == "host":
        return s["grid"].query(s["points"], s["precision"])
    if kind == "batch":
        s["batch"].query_device(s["points"].data_ptr(), s["offsets"], s["labels"].data_ptr(), s["precision"],
                                stream=torch.cuda.current_stream().cuda_stream, graph=True)
        return s["labels"]
    if kind == "serve":
        server, off = s["server"], s["offsets"]
        for k, pid in enumerate(s["requests"]):
            server.query(pid, s["points"][off[k]:off[k + 1]], labels=s["labels"][off[k]:off[k + 1]], detached=True)
        server.drain()
        return s["labels"]
    if kind == "build":
        grid = G.Grid(s["polygon"]).classify()
        grid.query_device(s["points"].data_ptr(), len(s["points"]), s["labels"].data_ptr(), s["precision"],
                          stream=torch.cuda.current_stream().cuda_stream, sync=True)
        return s["labels"]
    if kind == "build_batch":
        batch = G.Batch(s["polygons"])
        batch.query_device(s["points"].data_ptr(), s["offsets"], s["labels"].data_ptr(), s["precision"],
                           stream=torch.cuda.current_stream().cuda_stream, sync=True)
        return s["labels"]
    grid = G.Grid(s["polygon"], semantics=G.SEMANTICS_REFERENCE).classify()
    return grid.query(s["points"], s["precision"])


def work(case):
    """16 bytes of lon/lat in and a label out per point, 16 bytes per polygon
    vertex where vertices are inputs; per point a cell's two multiply-adds
    and, per point next to an edge, one crossing test (three determinants)."""
    n, e = case["points"], case["edges"]
    if case["shape"] == "mixed":
        mean = (n - min(1000, n)) / math.log(n / min(1000, n)) if n > 1000 else n
        if case["kind"] == "serve":
            mean = (n - 1) / math.log(n)
        n = mean * (case["requests"] if case["kind"] == "serve" else case["polygons"])
        e = (e - 16) / math.log(e / 16) * 1.2 * case["polygons"]
    bytes_ = 17 * n
    if case["kind"].startswith("build"):
        bytes_ += 16 * 1.1 * e
    flops = 4 * n + (27 * n if case["near"] != "no" else 0)
    return {"bytes": bytes_, "flops": flops}
