"""Timed cases of the matcher: one pass each through its public entry points.

The cases follow one matching iteration of a stereo pair, on the sizes of this
repository's workloads (a 4096^2 pair with a 1024^2 grid, candidates 8 to 512
per node at 0.5 m over a noisy TIN) and their neighbours:

  planes   image pyramid, Sobel magnitude and orientation of one image
  match    VerticalLineLocus on resident data (7x7 or 11x11 window), level 0
  refine   VerticalLineLocus at a coarse level's even iteration (the next
           finer level's windows and the orthoimage NCC take part)
  host     VerticalLineLocus on host buffers, as a program linking the drop-in
           calls it
  voxel    InitializeVoxel, VerticalLineLocus and AWNCC with semi-global
           aggregation
  seeddem  VerticalLineLocus_seeddem
  blunder  VerticalLineLocus_blunder
  tin      TINCreate_list of the matched points
  points   SelectMPs, blunder_detection_TIN and SetHeightRange
  search   Ortho_blunder (the TIN triangles' height search)

Image sizes are those of tiles cut from a scene, so most are no multiple of
anything; grids are `rows` x `nodes`.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from setsm_b200 import abi, level, synth, vll

GSD = 0.5
_ctx = None
_stream = None


def _context():
    """The program's matcher context, on a stream of its own."""
    global _ctx, _stream
    if _ctx is None:
        _ctx = vll.Context(0)
        _stream = torch.cuda.Stream()
        _ctx.set_stream(_stream.cuda_stream)
    return _ctx


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # one small tile: launches and host work count
        {"name": "match tile", "kind": "match", "size": 403, "nodes": 100, "rows": 90,
         "template": 11, "k_min": 16, "k_max": 64},
        # the ordinary level-0 pass, 7x7 window
        {"name": "match 7x7", "kind": "match", "size": 4096, "nodes": 1024, "rows": 1024,
         "template": 11, "k_min": 8, "k_max": 512},
        # the wide window on a large tile of odd width
        {"name": "match 11x11 ragged", "kind": "match", "size": 5003, "nodes": 1249, "rows": 1201,
         "template": 15, "k_min": 8, "k_max": 512},
        # level 2, second iteration
        {"name": "refine level 2", "kind": "refine", "size": 3276, "nodes": 205, "rows": 199,
         "level": 2, "template": 11, "k_min": 32, "k_max": 64},
        # a drop-in call on host buffers
        {"name": "host call", "kind": "host", "size": 1501, "nodes": 375, "rows": 360,
         "template": 11, "k_min": 16, "k_max": 128},
        # level 0 with semi-global aggregation
        {"name": "voxel iteration", "kind": "voxel", "size": 2050, "nodes": 512, "rows": 509,
         "template": 11, "k_min": 8, "k_max": 256},
        # a whole pyramid's planes
        {"name": "planes", "kind": "planes", "size": 6001, "rows": 5000, "levels": 5},
        {"name": "seed DEM", "kind": "seeddem", "size": 4096, "nodes": 1024, "rows": 1024},
        {"name": "blunder", "kind": "blunder", "size": 2998, "nodes": 749, "rows": 700},
        # half of a grid's nodes matched
        {"name": "tin", "kind": "tin", "nodes": 700, "rows": 640, "fraction": 0.5},
        {"name": "points", "kind": "points", "size": 2400, "nodes": 600, "rows": 600},
        {"name": "search", "kind": "search", "size": 2801, "nodes": 700, "rows": 690,
         "fraction": 0.02},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["planes", "match", "match", "refine", "host", "voxel", "seeddem",
                       "blunder", "tin", "points", "search"])
    if kind == "planes":
        size = _log(rng, 300, 6000)
        return {"kind": kind, "size": size, "rows": max(200, int(size * rng.uniform(0.5, 1.0))),
                "levels": rng.randint(1, 5)}
    if kind == "tin":
        nodes = _log(rng, 60, 700)
        return {"kind": kind, "nodes": nodes, "rows": max(40, int(nodes * rng.uniform(0.5, 0.9))),
                "fraction": round(rng.uniform(0.02, 0.6), 3)}
    top = {"match": 1200, "refine": 200, "host": 400, "voxel": 500, "seeddem": 1000,
           "blunder": 800, "points": 600, "search": 700}[kind]
    nodes = _log(rng, 64 if kind != "search" else 150, top)
    c = {"kind": kind, "size": 4 * nodes + rng.randint(0, 7), "nodes": nodes,
         "rows": max(48, int(nodes * rng.uniform(0.5, 1.0)))}
    if kind in ("match", "host", "voxel"):
        c["template"] = 15 if kind == "match" and rng.random() < 0.5 else 11
        c["k_min"] = rng.choice([8, 16, 32])
        c["k_max"] = {"match": 512, "host": 128, "voxel": 256}[kind] // rng.choice([1, 2])
    if kind == "refine":
        c["level"] = rng.choice([2, 3])
        c["size"] = 16 * nodes + rng.randint(0, 15) if c["level"] == 2 else 24 * nodes
        c["template"] = 11
        c["k_min"], c["k_max"] = 16, rng.choice([48, 64])
    if kind == "search":
        c["fraction"] = round(rng.uniform(0.01, 0.03), 4)
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _scene(size, seed):
    return synth.make_scene(synth.SceneSpec(seed=seed, image_size=size, iterations=5),
                            device="cuda", rows_per_chunk=2048)


def _grid(scene, nodes, rows):
    """`rows` x `nodes` grid nodes over the scene (its first rows)."""
    g = synth.make_grid(scene, nodes, scene.spec.image_size * GSD / nodes, device="cuda")
    n = nodes * rows
    b = g.boundary.copy()
    b[3] = b[1] + rows * g.resolution
    return synth.Grid(b, g.resolution, nodes, rows, g.pts[:n], g.wgs[:n], g.truth[:n])


def _ranges(grid, k_min, k_max, step, noise, seed):
    """Height ranges around a prior that is off the truth smoothly (a coarse
    TIN's error): log-uniform candidate counts, whole metres."""
    rng = np.random.default_rng(seed)
    n = grid.width * grid.height
    side = 24
    err = torch.from_numpy(rng.normal(0.0, noise, (1, 1, side, side)))
    err = torch.nn.functional.interpolate(err, size=(grid.height, grid.width), mode="bilinear",
                                          align_corners=True).reshape(-1).numpy()
    prior = grid.truth + err
    k = np.exp(rng.uniform(math.log(k_min), math.log(k_max), n))
    span = np.maximum(1, np.round(k * step)).astype(np.int64)
    lo = np.floor(prior - span / 2).astype(np.int64)
    return lo, lo + span, prior


def _planes(ctx, img):
    h, w = img.shape
    mag = torch.empty_like(img)
    ori = torch.empty((h, w), dtype=torch.uint8, device=img.device)
    ctx.preprocess_device(img.data_ptr(), w, h, mag.data_ptr(), ori.data_ptr())
    return img, mag, ori


def _pyramid(ctx, img, levels):
    out = [img]
    for _ in range(levels):
        h, w = out[-1].shape
        d = torch.empty((h // 2, w // 2), dtype=img.dtype, device=img.device)
        ctx.pyramid_down_device(out[-1].data_ptr(), w, h, d.data_ptr())
        out.append(d)
    return out


def _bytes(a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).copy()).cuda()


def _desc(scene, grid, gp3, planes, **kw):
    """Level descriptor whose planes and grid arrays are on the device;
    returns it with what has to stay alive."""
    tiny = [level.ImageLevel(image=np.zeros((2, 2), np.uint16), mag=np.zeros((2, 2), np.uint16),
                             ori=np.zeros((2, 2), np.uint8), rpc=scene.rpcs[ci])
            for ci in range(2)]
    li = level.LevelInputs(tiny, grid.pts, grid.wgs, grid.width, grid.height, grid.boundary, gp3,
                           check_matching_rate=kw.pop("cmr", True),
                           grid_resolution=grid.resolution, resolution=GSD, dem_resolution=2.0,
                           minmax_height=(-500.0, 3000.0), param=scene.param, **kw)
    d = li.desc()
    keep = [torch.from_numpy(grid.pts).cuda(), torch.from_numpy(grid.wgs).cuda(), planes]
    d.grid_pts, d.grid_wgs = keep[0].data_ptr(), keep[1].data_ptr()
    for ci in range(2):
        e = d.images[ci]
        img, mag, ori = planes[ci][0]
        e.image, e.mag, e.ori = img.data_ptr(), mag.data_ptr(), ori.data_ptr()
        e.height, e.width = img.shape
        if "next" in planes[ci]:
            img, mag, ori = planes[ci]["next"]
            e.image_next, e.mag_next, e.ori_next = img.data_ptr(), mag.data_ptr(), ori.data_ptr()
            e.height_next, e.width_next = img.shape
        if "b" in planes[ci]:
            img, mag = planes[ci]["b"][:2]
            e.image_b, e.mag_b = img.data_ptr(), mag.data_ptr()
            e.height_b, e.width_b = img.shape
    return d, keep


def _step(lev):
    """The height step of a level: half its pixel, at most 3 m."""
    return min(math.floor(GSD * (1 << lev) / 2.0 * 1000.0 + 0.1) / 1000.0, 3.0)


def _match_state(ctx, case, seed, cmr=True, sgm=0):
    scene = _scene(case["size"], seed)
    grid = _grid(scene, case["nodes"], case["rows"])
    lo, hi, prior = _ranges(grid, case.get("k_min", 8), case.get("k_max", 128), 0.5, 3.0, seed + 1)
    gp3 = level.make_gridpt3(lo, hi, prior)
    planes = [{0: _planes(ctx, scene.images[ci])} for ci in range(2)]
    d, keep = _desc(scene, grid, gp3, planes, height_step=0.5, cmr=cmr, sgm_py=sgm,
                    template_size=case.get("template", 11))
    n = grid.width * grid.height
    return {"desc": d, "keep": keep, "grid": grid, "scene": scene, "gp3_host": gp3, "n": n,
            "gp3": _bytes(gp3), "ncc": torch.zeros(n * 24, dtype=torch.uint8, device="cuda")}


def _prep_match(ctx, case, seed):
    return _match_state(ctx, case, seed)


def _prep_refine(ctx, case, seed):
    lev = case["level"]
    scene = _scene(case["size"], seed)
    grid = _grid(scene, case["nodes"], case["rows"])
    step = _step(lev)
    lo, hi, prior = _ranges(grid, case["k_min"], case["k_max"], step, 3.0, seed + 1)
    rng = np.random.default_rng(seed + 2)
    # the previous iteration's orthoimage NCC per node
    on = np.where(rng.random(lo.shape) < 0.6, 800, 100)
    gp3 = level.make_gridpt3(lo, hi, prior, ortho_ncc=on)
    planes = []
    for ci in range(2):
        pyr = _pyramid(ctx, scene.images[ci], lev)
        planes.append({0: _planes(ctx, pyr[lev]), "next": _planes(ctx, pyr[lev - 1])})
    d, keep = _desc(scene, grid, gp3, planes, pyramid_step=lev, iteration=2, height_step=step,
                    template_size=case["template"], sgm_py=0)
    n = grid.width * grid.height
    return {"desc": d, "keep": keep, "gp3": _bytes(gp3), "n": n,
            "ncc": torch.zeros(n * 24, dtype=torch.uint8, device="cuda")}


def _prep_host(ctx, case, seed):
    scene = _scene(case["size"], seed)
    grid = _grid(scene, case["nodes"], case["rows"])
    lo, hi, prior = _ranges(grid, case["k_min"], case["k_max"], 0.5, 3.0, seed + 1)
    images = []
    for ci in range(2):
        img, mag, ori = _planes(ctx, scene.images[ci])
        images.append(level.ImageLevel(image=img.cpu().numpy().view(np.uint16),
                                       mag=mag.cpu().numpy().view(np.uint16),
                                       ori=ori.cpu().numpy(), rpc=scene.rpcs[ci]))
    inp = level.LevelInputs(images, grid.pts, grid.wgs, grid.width, grid.height, grid.boundary,
                            level.make_gridpt3(lo, hi, prior), template_size=case["template"],
                            height_step=0.5, grid_resolution=grid.resolution, resolution=GSD,
                            param=scene.param)
    return {"inputs": inp, "ncc": inp.new_nccresult()}


def _prep_voxel(ctx, case, seed):
    s = _match_state(ctx, case, seed, cmr=False, sgm=1)
    # room for the widest range at every node, as a program reserves it
    s["cap"] = cap = s["n"] * (case["k_max"] + 16)
    s["vox"] = torch.zeros(cap * 4, dtype=torch.uint8, device="cuda")
    s["off"] = torch.empty(s["n"] + 1, dtype=torch.int64, device="cuda")
    s["gp3_work"] = torch.empty_like(s["gp3"])
    return s


def _prep_planes(ctx, case, seed):
    img = _scene(case["size"], seed).images[0][:case["rows"]].contiguous()
    pyr = [img]
    for _ in range(case["levels"] - 1):
        pyr.append(torch.empty((pyr[-1].shape[0] // 2, pyr[-1].shape[1] // 2), dtype=img.dtype,
                               device="cuda"))
    return {"pyr": pyr, "mag": [torch.empty_like(p) for p in pyr],
            "ori": [torch.empty(p.shape, dtype=torch.uint8, device="cuda") for p in pyr]}


def _heights_off(gp3, grid, rng):
    """Node heights of an unfinished grid: most near the truth, some off by up
    to 40 m, some unmatched."""
    n = len(gp3)
    h = grid.truth + rng.normal(0.0, 1.0, n)
    h = np.where(rng.random(n) < 0.15, h + rng.uniform(-40.0, 40.0, n), h)
    gp3["Height"] = np.where(rng.random(n) < 0.05, -1000.0, h).astype(np.float32)


def _prep_seeddem(ctx, case, seed):
    s = _match_state(ctx, case, seed)
    g = s["gp3_host"]
    _heights_off(g, s["grid"], np.random.default_rng(seed + 5))
    s["gp3"] = _bytes(g)
    s["gp3_work"] = torch.empty_like(s["gp3"])
    return s


def _prep_blunder(ctx, case, seed):
    scene = _scene(case["size"], seed)
    grid = _grid(scene, case["nodes"], case["rows"])
    lo, hi, prior = _ranges(grid, 8, 128, 0.5, 3.0, seed + 1)
    gp3 = level.make_gridpt3(lo, hi, prior)
    _heights_off(gp3, grid, np.random.default_rng(seed + 5))
    planes = []
    for ci in range(2):
        pyr = _pyramid(ctx, scene.images[ci], 1)
        planes.append({0: _planes(ctx, pyr[0]), "b": _planes(ctx, pyr[1])})
    d, keep = _desc(scene, grid, gp3, planes, height_step=0.5, template_size=11)
    d.blunder_level = 1
    g = _bytes(gp3)
    return {"desc": d, "keep": keep, "gp3": g, "gp3_work": torch.empty_like(g), "grid": grid,
            "scene": scene, "gp3_host": gp3, "b": [planes[ci]["b"] for ci in range(2)],
            "out": torch.empty(len(gp3), dtype=torch.float32, device="cuda")}


def _node_points(nodes, rows, res, fraction, rng):
    n = nodes * rows
    sel = np.sort(rng.choice(n, size=max(16, int(fraction * n)), replace=False))
    pts = np.zeros(len(sel), dtype=abi.POINT3_DTYPE)
    pts["x"] = 1000.0 + (sel % nodes) * res
    pts["y"] = -2000.0 + (sel // nodes) * res
    pts["flag"] = 1
    return sel, pts


def _prep_tin(ctx, case, seed):
    rng = np.random.default_rng(seed)
    nodes, rows, res = case["nodes"], case["rows"], 2.0
    _, pts = _node_points(nodes, rows, res, case["fraction"], rng)
    pts["z"] = rng.uniform(0.0, 300.0, len(pts))
    cap = 2 * len(pts) + 16
    return {"pts": _bytes(pts), "n": len(pts), "res": res, "cap": cap,
            "bound": np.array([1000.0, -2000.0, 1000.0 + nodes * res, -2000.0 + rows * res]),
            "tris": torch.zeros(cap * 12, dtype=torch.uint8, device="cuda")}


def _triangles(ctx, d_pts, n, boundary, res):
    cap = 2 * n + 16
    tris = torch.empty(cap * 12, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    m = ctx.tin_create_device(d_pts.data_ptr(), n, boundary, res, tris.data_ptr(), cap)
    return tris[:m * 12].clone(), m


_SELECT = (0.6, 0.2, 0.8, 0.7, 1, 1.5, 1, 10.0)


def _prep_points(ctx, case, seed):
    """The records of a matched level, its matched points and their TIN."""
    s = _match_state(ctx, case, seed)
    n = s["n"]
    torch.cuda.synchronize()
    ctx.vertical_line_locus_device(s["desc"], s["gp3"].data_ptr(), s["ncc"].data_ptr())
    g = s["gp3"].clone()
    pts = torch.zeros(n * 32, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    m = ctx.select_mps_device(s["desc"], s["ncc"].data_ptr(), g.data_ptr(), pts.data_ptr(), n,
                              *_SELECT)
    rng = np.random.default_rng(seed + 3)
    host = pts[:m * 32].cpu().numpy().view(abi.POINT3_DTYPE).copy()
    host["flag"] = np.where(rng.random(m) < 0.1, 1, 0)
    host["z"] += np.where(rng.random(m) < 0.03, rng.uniform(-40.0, 40.0, m), 0.0)
    s["m"] = m
    s["mpts"] = torch.zeros(n * 32, dtype=torch.uint8, device="cuda")
    s["mpts"][:m * 32] = _bytes(host)
    s["tris"], s["n_tris"] = _triangles(ctx, s["mpts"], m, s["grid"].boundary,
                                        s["grid"].resolution)
    oncc = np.where(rng.random(n) < 0.2, rng.uniform(-1.0, 0.3, n), rng.uniform(0.3, 1.0, n))
    s["oncc"] = torch.from_numpy(oncc.astype(np.float32)).cuda()
    s["gp3_work"] = torch.empty_like(s["gp3"])
    s["sel"] = torch.zeros(n * 32, dtype=torch.uint8, device="cuda")
    s["mpts_work"] = torch.empty_like(s["mpts"])
    s["det"] = torch.zeros(n, dtype=torch.uint8, device="cuda")
    s["result"] = torch.zeros(n * 20, dtype=torch.uint8, device="cuda")
    return s


def _prep_search(ctx, case, seed):
    s = _match_state(ctx, case, seed)
    grid, g = s["grid"], s["gp3_host"]
    rng = np.random.default_rng(seed + 5)
    sel, pts = _node_points(grid.width, grid.height, grid.resolution, case["fraction"], rng)
    truth = grid.truth[sel]
    anchor = rng.random(len(sel)) < 0.6
    pts["x"], pts["y"] = grid.pts[sel, 0], grid.pts[sel, 1]
    pts["z"] = np.where(anchor, truth, truth + rng.uniform(-25.0, 25.0, len(sel)))
    g["anchor_flag"][sel] = np.where(anchor, 1, 2)
    g["minHeight"][sel] = np.floor(truth - 40.0).astype(np.int16)
    g["maxHeight"][sel] = np.ceil(truth + 40.0).astype(np.int16)
    s["gp3"], s["pts"], s["m"] = _bytes(g), _bytes(pts), len(sel)
    s["tris"], s["n_tris"] = _triangles(ctx, s["pts"], len(sel), grid.boundary, grid.resolution)
    s["gp3_work"], s["pts_work"] = torch.empty_like(s["gp3"]), torch.empty_like(s["pts"])
    return s


_PREP = {"match": _prep_match, "refine": _prep_refine, "host": _prep_host, "voxel": _prep_voxel,
         "planes": _prep_planes, "seeddem": _prep_seeddem, "blunder": _prep_blunder,
         "tin": _prep_tin, "points": _prep_points, "search": _prep_search}


def prepare(case, seed):
    ctx = _context()
    s = _PREP[case["kind"]](ctx, case, int(seed))
    s["kind"] = case["kind"]
    torch.cuda.synchronize()
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _ugrid(t):
    return t.view(-1, 20)[:, :18]      # without the record's padding


def _points(t):
    return {"xyz": t.view(torch.float64).view(-1, 4)[:, :3], "flag": t.view(-1, 32)[:, 24]}


def _run_match(ctx, s):
    ctx.vertical_line_locus_device(s["desc"], s["gp3"].data_ptr(), s["ncc"].data_ptr())
    return s["ncc"]


def _run_host(ctx, s):
    ncc = s["ncc"]
    ncc.fill(0)
    st = ctx.vertical_line_locus(s["inputs"], ncc)
    return {"ncc": ncc.view(np.uint8), "count": int(st.accessable_grid)}


def _run_voxel(ctx, s):
    g, ncc = s["gp3_work"], s["ncc"]
    g.copy_(s["gp3"])
    ncc.zero_()
    n = ctx.initialize_voxel_device(s["desc"], g.data_ptr(), ncc.data_ptr(), None,
                                    s["vox"].data_ptr(), s["cap"], s["off"].data_ptr())
    ctx.vertical_line_locus_device(s["desc"], g.data_ptr(), ncc.data_ptr(), s["vox"].data_ptr(),
                                   s["off"].data_ptr())
    ctx.awncc_device(s["desc"], g.data_ptr(), ncc.data_ptr(), s["vox"].data_ptr(),
                     s["off"].data_ptr())
    v = s["vox"].view(-1, 4)
    return {"ncc": ncc, "ugrid": _ugrid(g), "voxels": n, "flag": v[:, 0], "incc": v[:, 2:]}


def _run_planes(ctx, s):
    for i, img in enumerate(s["pyr"]):
        h, w = img.shape
        ctx.preprocess_device(img.data_ptr(), w, h, s["mag"][i].data_ptr(), s["ori"][i].data_ptr())
        if i + 1 < len(s["pyr"]):
            ctx.pyramid_down_device(img.data_ptr(), w, h, s["pyr"][i + 1].data_ptr())
    return {"pyramid": s["pyr"][1:], "mag": s["mag"], "ori": s["ori"]}


def _run_seeddem(ctx, s):
    g = s["gp3_work"]
    g.copy_(s["gp3"])
    ctx.seeddem_device(s["desc"], g.data_ptr())
    return _ugrid(g)


def _run_blunder(ctx, s):
    g = s["gp3_work"]
    g.copy_(s["gp3"])
    ctx.blunder_device(s["desc"], g.data_ptr(), 1, False, s["out"].data_ptr())
    return {"ncc": s["out"], "ugrid": _ugrid(g)}


def _run_tin(ctx, s):
    n = ctx.tin_create_device(s["pts"].data_ptr(), s["n"], s["bound"], s["res"],
                              s["tris"].data_ptr(), s["cap"])
    return {"triangles": s["tris"].view(torch.int32), "count": n}


def _run_points(ctx, s):
    d, g, pts = s["desc"], s["gp3_work"], s["mpts_work"]
    g.copy_(s["gp3"])
    pts.copy_(s["mpts"])
    s["det"].zero_()
    n = ctx.select_mps_device(d, s["ncc"].data_ptr(), g.data_ptr(), s["sel"].data_ptr(), s["n"],
                              *_SELECT)
    counts, zext = np.zeros(2, np.int64), np.array([1e5, -1e5])
    ctx.blunder_detection_tin_device(d, 1, s["oncc"].data_ptr(), True, 1, 60.0, pts.data_ptr(),
                                     s["det"].data_ptr(), s["m"], s["tris"].data_ptr(),
                                     s["n_tris"], g.data_ptr(), counts, zext)
    ext = ctx.set_height_range_device(d, pts.data_ptr(), s["m"], s["tris"].data_ptr(),
                                      s["n_tris"], g.data_ptr(), s["result"].data_ptr(), 2, 1.5,
                                      False)
    return {"selected": _points(s["sel"]), "count": n, "flags": _points(pts)["flag"],
            "detected": s["det"], "ugrid": _ugrid(g), "ranges": _ugrid(s["result"]),
            "counts": counts, "zext": zext, "extent": list(ext)}


def _run_search(ctx, s):
    g, pts = s["gp3_work"], s["pts_work"]
    g.copy_(s["gp3"])
    pts.copy_(s["pts"])
    rounds = ctx.ortho_blunder_device(s["desc"], 1.5, pts.data_ptr(), s["m"],
                                      s["tris"].data_ptr(), s["n_tris"], g.data_ptr())
    return {"points": _points(pts), "ugrid": _ugrid(g), "rounds": rounds}


_RUN = {"match": _run_match, "refine": _run_match, "host": _run_host, "voxel": _run_voxel,
        "planes": _run_planes, "seeddem": _run_seeddem, "blunder": _run_blunder, "tin": _run_tin,
        "points": _run_points, "search": _run_search}


def run(state):
    with torch.cuda.stream(_stream):
        return _RUN[state["kind"]](_ctx, state)


# ---------------------------------------------------------------------------
# the work a pass cannot do without
# ---------------------------------------------------------------------------
def _mean_k(case):
    lo, hi = case["k_min"], case["k_max"]
    return (hi - lo) / math.log(hi / lo) if hi > lo else float(lo)


_SAMPLE = 60.0       # operations of one window sample in both images and planes
_PROJECT = 200.0     # operations of one RPC projection


def work(case):
    kind = case["kind"]
    if kind == "planes":
        px = sum((case["size"] >> i) * (case["rows"] >> i) for i in range(case["levels"]))
        down = sum((case["size"] >> i) * (case["rows"] >> i) for i in range(1, case["levels"]))
        # image read, magnitude, orientation and the next level written
        return {"bytes": px * 5.0 + down * 2.0, "flops": px * (20 + 2 * 107.0) + down * 162.0}
    n = case["nodes"] * case["rows"]
    if kind == "tin":
        m = case["fraction"] * n
        return {"bytes": m * (32 + 24.0), "flops": m * math.log2(m) * 40}
    share = case["rows"] / case["nodes"]
    planes = 2 * 5.0 * case["size"] ** 2 * share       # image, magnitude, orientation, two images
    rec = n * (16 + 20 + 24.0)                          # lon/lat, UGRID, NCCresult
    if kind in ("match", "host", "voxel"):
        samples = {11: 45, 15: 109}[case["template"]]
        k = n * _mean_k(case)
        b, f = planes + rec + n * 24.0, k * (samples * _SAMPLE + 2 * _PROJECT)
        if kind == "voxel":
            b, f = b + n * 84.0 + k * 4, f + k * 8 * 6
        return {"bytes": b, "flops": f}
    if kind == "refine":
        lev = case["level"]
        samples = 45 if lev == 2 else 69
        k = n * _mean_k(case)
        return {"bytes": planes * 1.25 / 4 ** (lev - 1) / 4 + rec + n * 24.0,
                "flops": k * (2 * samples * _SAMPLE + 2 * _PROJECT) + n * 2 * samples * _SAMPLE}
    if kind == "seeddem":
        return {"bytes": planes * 0.8 + n * 56.0,
                "flops": n * 16 * (2 * _PROJECT + 100) + n * 109 * _SAMPLE}
    if kind == "blunder":
        return {"bytes": planes * 0.2 + n * 60.0,
                "flops": n * 4 * (2 * _PROJECT + 100) + n * 49 * _SAMPLE}
    if kind == "points":
        m = 0.9 * n
        return {"bytes": n * (24 + 20 + 16 + 32 + 4 + 3 * 20.0) + m * (64 + 24 * 2),
                "flops": m * 1000.0}
    m = case["fraction"] * n
    # five rounds over about two triangles per candidate point, 80 m of heights
    return {"bytes": planes * 0.8 + n * 40.0 + m * 88,
            "flops": n * 60 * (2 * _PROJECT + 4 * _SAMPLE)}


# ---------------------------------------------------------------------------
# the blunder pass's NCC in 64 bits, in plain torch
# ---------------------------------------------------------------------------
def _lonlat(p, x, y):
    """Inverse polar stereographic projection."""
    e2 = p["e"] ** 2
    e4, e6, e8 = e2 ** 2, e2 ** 3, e2 ** 4
    rho = torch.sqrt(x * x + y * y)
    chi = math.pi / 2 - 2 * torch.atan(rho * p["t_c"] / (p["a"] * p["m_c"]))
    phi = (chi + (e2 / 2 + 5 * e4 / 24 + e6 / 12 + 13 * e8 / 360) * torch.sin(2 * chi)
           + (7 * e4 / 48 + 29 * e6 / 240 + 811 * e8 / 11520) * torch.sin(4 * chi)
           + (7 * e6 / 120 + 81 * e8 / 1120) * torch.sin(6 * chi)
           + (4279 * e8 / 161280) * torch.sin(8 * chi))
    lam = p["lambda_0"] + torch.atan2(x, -y)
    lam = torch.where(lam < -math.pi, lam + 2 * math.pi, lam)
    return lam * (180 / math.pi), phi * (180 / math.pi)


def _rpc(r, lon, lat, h):
    """Sample and line of an RPC00B model."""
    L, P, H = (lon - r[2]) / r[7], (lat - r[3]) / r[8], (h - r[4]) / r[9]
    t = [torch.ones_like(L), L, P, H, L * P, L * H, P * H, L * L, P * P, H * H, P * L * H,
         L ** 3, L * P * P, L * H * H, L * L * P, P ** 3, P * H * H, L * L * H, P * P * H, H ** 3]
    c = [sum(float(r[10 + 20 * j + i]) * t[i] for i in range(20)) for j in range(4)]
    return c[2] / c[3] * r[6] + r[1], c[0] / c[1] * r[5] + r[0]


def exact(case, seed):
    if case["kind"] != "blunder":
        return None      # records, planes, points and triangles: whole values
    s = prepare(case, seed)
    grid, scene, dev = s["grid"], s["scene"], "cuda"
    res, b, W, Hn = 2 * GSD, grid.boundary, grid.width, grid.height
    ow, oh = int((b[2] - b[0]) / res) + 1, int((b[3] - b[1]) / res) + 1
    ax = lambda o, m, step: o + torch.arange(m, dtype=torch.float64, device=dev) * step  # noqa: E731
    tx, ty = ax(b[0], ow, res), ax(b[1], oh, res)
    # (divided by tensors: torch multiplies by a scalar's reciprocal)
    by, bg = (torch.tensor(v, dtype=torch.float64, device=dev) for v in (res, grid.resolution))
    col, row = ((tx - b[0]) / bg).long(), ((ty - b[1]) / bg).long()
    height = torch.from_numpy(s["gp3_host"]["Height"].astype(np.float64)).to(dev).view(Hn, W)
    ok = ((row < Hn)[:, None] & (col < W)[None, :])
    z = height[row.clamp(max=Hn - 1)][:, col.clamp(max=W - 1)]
    ok &= z != -1000
    X, Y = tx[None, :].expand(oh, ow), ty[:, None].expand(oh, ow)
    lon, lat = _lonlat(scene.param, X, Y)
    coords = []
    for ci in range(2):
        x, y = _rpc(scene.rpcs[ci], lon, lat, z)
        r = scene.rpcs[ci]
        x, y = x.clamp(0, r[1] + r[6] * 1.2), y.clamp(0, r[0] + r[5] * 1.2)
        coords.append([torch.where(ok, x / 2, 0.0), torch.where(ok, y / 2, 0.0)])
    gx = torch.from_numpy(grid.pts[:, 0].copy()).to(dev)
    gy = torch.from_numpy(grid.pts[:, 1].copy()).to(dev)
    half, offs = 5, []
    for dr in range(-half, half + 1):
        for dc in range(-half, half + 1):
            if dr * dr + dc * dc <= (half - 1) ** 2:
                offs.append((dr, dc))
    s1 = half // 2
    s2 = s1 + int(s1 / 2.0 + 0.5)
    vals, use, depth = [], [], []
    for dr, dc in offs:
        px, py = gx + dc * res, gy + dr * res
        ic, ir = ((px - b[0]) / by).trunc().long(), ((py - b[1]) / by).trunc().long()
        nc, nr = ((px - b[0]) / bg).trunc().long(), ((py - b[1]) / bg).trunc().long()
        u = ((ic >= 0) & (ic < ow) & (ir >= 0) & (ir < oh) & (nc >= 0) & (nc < W) & (nr >= 0)
             & (nr < Hn))
        u &= height[nr.clamp(0, Hn - 1), nc.clamp(0, W - 1)] != -1000
        v = []
        for ci in range(2):
            x = coords[ci][0][ir.clamp(0, oh - 1), ic.clamp(0, ow - 1)]
            y = coords[ci][1][ir.clamp(0, oh - 1), ic.clamp(0, ow - 1)]
            img, mag = s["b"][ci][:2]
            h, w = img.shape
            u &= (x >= 0) & (y >= 0) & (x + 1 < w) & (y + 1 < h)
            x, y = x.clamp(0, w - 1 - 1e-9), y.clamp(0, h - 1 - 1e-9)
            xi, yi = x.floor().long(), y.floor().long()
            fx, fy = x - xi, y - yi
            for plane in (img, mag):
                t = plane.long().bitwise_and(0xFFFF).double()
                v.append(t[yi, xi] * (1 - fx) * (1 - fy) + t[yi, xi + 1] * fx * (1 - fy)
                         + t[yi + 1, xi] * (1 - fx) * fy + t[yi + 1, xi + 1] * fx * fy)
        use.append(u & (v[0] > 0) & (v[2] > 0))
        vals.append(torch.stack(v))
        r2 = dr * dr + dc * dc
        d = 0
        for k, sub in ((1, s1), (2, s2)):
            if r2 <= (half - sub + 1) ** 2 and max(abs(dr), abs(dc)) <= half - sub:
                d = k
        depth.append(d)
    vals, use = torch.stack(vals), torch.stack(use)
    depth = torch.tensor(depth, device=dev)
    total = torch.zeros(len(gx), dtype=torch.float64, device=dev)
    count, full = torch.zeros_like(total), torch.ones_like(use[0])
    for win in range(3):
        m = (use & (depth >= win)[:, None]).double()
        n = m.sum(0)
        full &= n > 0
        for p in (0, 1):
            a, c = vals[:, p], vals[:, p + 2]
            da = (a - (a * m).sum(0) / n.clamp(min=1)) * m
            dc = (c - (c * m).sum(0) / n.clamp(min=1)) * m
            va, vc = (da * da).sum(0), (dc * dc).sum(0)
            fine = (va > 1e-8) & (vc > 1e-8)
            total += torch.where(fine, (da * dc).sum(0) / torch.sqrt(va * vc), 0.0)
            count += fine
    ncc = torch.where(full & (count > 0), total / count.clamp(min=1), 0.0)
    return {"ncc": ncc, "ugrid": None}
