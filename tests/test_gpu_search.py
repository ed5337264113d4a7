"""The screened height search (Ortho_blunder) against single searches that
cannot skip a height: where the screen ends (more heights than one pass of the
block, more inside cells than the list holds), where it does not decide
(constant and empty image areas, cells projecting outside the images) and with
three images.  Each single-height search gives the exact value of one height;
the search over the whole range keeps the first of their largest."""
import copy

import numpy as np
import pytest

from tests import cases
from tests.test_gpu_ortho_tin import searchable

pytestmark = pytest.mark.gpu

CASES = {
    "heights": dict(seed=38, size=512, nodes=64, res=3.0, point_frac=0.05, range_m=120.0),
    "cells": dict(seed=37, size=512, nodes=96, res=2.0, point_frac=0.002, range_m=20.0),
    "outside": dict(seed=40, size=512, nodes=30, res=20.0, point_frac=0.3, range_m=30.0),
    "images": dict(seed=35, size=512, nodes=32, res=8.0, n_images=3, anchor_frac=0.4, range_m=30.0),
}


@pytest.mark.parametrize("flat", [False, True])
@pytest.mark.parametrize("name", sorted(CASES))
def test_search_keeps_the_first_largest_height(gpu_ctx, name, flat):
    inp, pts, tris = cases.make_tin_case(**CASES[name])
    if flat:
        for im in inp.images:
            im.image, im.mag = im.image.copy(), im.mag.copy()
            h, w = im.image.shape
            im.image[: h // 2, : w // 2] = 500
            im.mag[: h // 2, : w // 2] = 0
    jobs = searchable(inp, pts, tris)
    step, found = 1.0 * inp.resolution, 0
    for three, node in jobs[:: max(1, len(jobs) // 6)][:6]:
        got = gpu_ctx.vertical_line_locus_ortho(inp, 1.0, three, node)
        lo, hi = int(inp.gridpt3["minHeight"][node]), int(inp.gridpt3["maxHeight"][node])
        best = (0, -9999.0, float("nan"))
        one = copy.copy(inp)
        for k in range(int((hi - lo) / step) + 1):
            h = float(np.float32(lo + k * step))
            if h != int(h):
                continue
            # a range without extent holds one height
            one.gridpt3 = inp.gridpt3.copy()
            one.gridpt3["minHeight"][node] = one.gridpt3["maxHeight"][node] = int(h)
            r = gpu_ctx.vertical_line_locus_ortho(one, 1.0, three, node)
            if r[1] != -9999.0 and (best[1] == -9999.0 or r[2] > best[2]):
                best = r
        # the whole-metre heights are among the searched ones
        if best[1] != -9999.0:
            found += 1
            assert got[2] >= best[2]
            if got[1] == int(got[1]) and got[2] == best[2]:
                assert got == best
        else:
            assert got[1] == -9999.0 or got[1] != int(got[1])
    assert found > 0 or flat
