"""Calls whose time depends on the inputs' kind and not only on their size:
each against a call of the same sizes in the same process.  The factors leave
room for half as much again as measured."""
import time

import numpy as np
import pytest

from tests import cases

pytestmark = pytest.mark.gpu


def median_time(call, prepare, n=9):
    import torch
    t = []
    for _ in range(n + 2):
        args = prepare()
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        call(*args)
        torch.cuda.synchronize()
        t.append(time.perf_counter() - t0)
    return float(np.median(t[2:]))


def on_device(inp):
    import torch
    io, keep = cases.device_level(torch, inp, inp.new_nccresult())
    return io[0], keep["gp3"], keep


def test_blunder_over_constant_areas(gpu_ctx):
    """Two fifths of both images constant: at most twice the scene's time
    (1.1 times as measured; 4.0 when every node there was evaluated exactly)."""
    import torch
    times = {}
    for flat in (False, True):
        inp = cases.make_variant_case(seed=14, size=768, nodes=360, res=1.0, blunder_level=0)
        if flat:
            for im in inp.images:
                y, x = np.ogrid[:768, :768]
                m = ((y // 61 * 7 + x // 61 * 13) % 5) < 2
                im.image_b, im.mag_b = np.where(m, 500, im.image_b).astype(np.uint16), im.mag_b.copy()
                im.mag_b[m] = 0
        d, gp3, keep = on_device(inp)
        out = torch.empty(inp.n, dtype=torch.float32, device="cuda")
        first = gp3.clone()
        times[flat] = median_time(
            lambda g: gpu_ctx.blunder_device(d, g.data_ptr(), 1, False, out.data_ptr()),
            lambda: (first.clone(),))
    assert times[True] < 2.0 * times[False], times


def test_blunder_beside_empty_areas(gpu_ctx):
    """Images with empty squares: at most 1.7 times the scene's time (1.1 as
    measured; 4.3 when a node whose own pixel is empty was evaluated exactly)."""
    import torch
    times = {}
    for empty in (False, True):
        inp = cases.make_variant_case(seed=14, size=768, nodes=360, res=1.0, blunder_level=0)
        if empty:
            for im in inp.images:
                y, x = np.ogrid[:768, :768]
                im.image_b = np.where(((y // 31 * 7 + x // 31 * 13) % 5) < 2, 0,
                                      im.image_b).astype(np.uint16)
        d, gp3, keep = on_device(inp)
        out = torch.empty(inp.n, dtype=torch.float32, device="cuda")
        first = gp3.clone()
        times[empty] = median_time(
            lambda g: gpu_ctx.blunder_device(d, g.data_ptr(), 1, False, out.data_ptr()),
            lambda: (first.clone(),))
    assert times[True] < 1.7 * times[False], times


def test_search_of_few_heights(gpu_ctx):
    """Three heights per triangle against 41 on the same triangles: at most
    0.65 of the time (0.48 as measured; 0.76 when three were screened too)."""
    import torch
    times = {}
    for half in (1, 20):
        inp, pts, tris = cases.make_tin_case(seed=9, size=1024, nodes=240, res=2.0, point_frac=0.2)
        inp.resolution = 1.0    # of the heights' step
        g = inp.gridpt3
        mid = (g["minHeight"].astype(int) + g["maxHeight"]) // 2
        g["minHeight"], g["maxHeight"] = mid - half, mid + half
        d, gp3, keep = on_device(inp)
        dev = lambda a: torch.from_numpy(a.view(np.uint8).copy()).cuda()
        p0, t = dev(pts), dev(tris)
        times[half] = median_time(
            lambda g, p: gpu_ctx.ortho_blunder_device(d, 1.0, p.data_ptr(), len(pts), t.data_ptr(),
                                                      len(tris), g.data_ptr()),
            lambda: (gp3.clone(), p0.clone()))
    assert times[1] < 0.65 * times[20], times


def test_height_range_of_few_triangles(gpu_ctx):
    """Some 130 triangles over a grid against 9 k: at most 2.5 times the time
    (1.2 as measured; 4.0 with eight lanes per triangle)."""
    import torch
    times = {}
    for frac in (0.0003, 0.02):
        inp, pts, tris = cases.make_range_case(seed=9, size=1024, nodes=480, res=1.0, point_frac=frac)
        d, gp3, keep = on_device(inp)
        p, t = (torch.from_numpy(a.view(np.uint8).copy()).cuda() for a in (pts, tris))
        out = torch.zeros(inp.n * 20, dtype=torch.uint8, device="cuda")
        times[frac] = median_time(
            lambda g: gpu_ctx.set_height_range_device(d, p.data_ptr(), len(pts), t.data_ptr(),
                                                      len(tris), g.data_ptr(), out.data_ptr(), 2, 1.5,
                                                      False),
            lambda: (gp3.clone(),))
    assert times[0.0003] < 2.5 * times[0.02], times
