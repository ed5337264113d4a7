"""SetHeightRange and blunder_detection_TIN choose the lanes per triangle and
per point by how many there are.  A list of triangles repeated gives the same
result (a node takes its smallest triangle), and points that are flagged
already take no part, so both calls are made at every choice with the same
triangles and points."""
import copy

import numpy as np
import pytest

from tests import cases

pytestmark = pytest.mark.gpu

CASES = {
    "dense": dict(seed=21, size=512, nodes=60, res=4.0, point_frac=0.5),
    "sparse": dict(seed=22, size=512, nodes=96, res=2.0, point_frac=0.004),
    "two": dict(seed=23, size=512, nodes=96, res=2.0, point_frac=0.0004),
}


def fields(a):
    return {f: a[f].tobytes() for f in a.dtype.names}


@pytest.mark.parametrize("name", sorted(CASES))
def test_height_range_of_repeated_triangles(gpu_ctx, name):
    inp, pts, tris = cases.make_range_case(**CASES[name])
    want = None
    for n in (1, 6200, 6400, 9400, 9600, 37000, 39000, 75000, 77000, 160000):
        i = copy.copy(inp)
        i.gridpt3 = inp.gridpt3.copy()
        t = np.tile(tris, -(-n // len(tris)))
        out, ext = gpu_ctx.set_height_range(i, pts, t, 2, 1.5, False)
        got = ([fields(out), fields(i.gridpt3)], ext)
        want = want or got
        assert got == want, len(t)


@pytest.mark.parametrize("name", sorted(CASES))
def test_tin_blunder_among_flagged_points(gpu_ctx, name):
    inp, pts, tris, oncc = cases.make_tin_blunder_case(**CASES[name])
    # points of 9 to 40 triangles: extra ones at the first points
    rng = np.random.default_rng(4)
    extra = np.zeros(60, tris.dtype)
    extra["a"] = np.arange(60) % 3
    extra["b"], extra["c"] = rng.integers(0, len(pts), (2, 60))
    tris = np.concatenate([tris, extra])
    want = None
    for more in (0, 9000, 9600, 40000):
        i = copy.copy(inp)
        i.gridpt3 = inp.gridpt3.copy()
        p = np.zeros(len(pts) + more, pts.dtype)
        p[: len(pts)] = pts
        for f in "xyz":
            p[f][len(pts):] = pts[f][0]
        p["flag"][len(pts):] = 1
        det, cnt, z = np.zeros(len(p), np.uint8), np.zeros(2, np.int64), np.array([1e5, -1e5])
        gpu_ctx.blunder_detection_tin(i, 1, oncc, True, 1, 60.0, p, det, tris, cnt, z)
        n = len(pts)
        got = (fields(p[:n]), det[:n].tobytes(), i.gridpt3["anchor_flag"].tobytes())
        want = want or got
        assert got == want, more
