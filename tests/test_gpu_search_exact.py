"""The screened height search against one that screens nothing (the numpy
restatement in ortho_oracle.py): the whole result of single searches over
scenes -- fractional winners, correlations near their thresholds, steep
planes, triangles of few and of more than 256 cells, one height to several
hundred --, and searches whose two best heights differ by less than the
screen's band while one of them rests on a sample that a coordinate error of
1e-8 pixel moves by more."""
import numpy as np
import pytest

from setsm_b200 import abi
from tests import cases, ortho_oracle as oo
from tests.test_gpu_ortho_tin import searchable

pytestmark = pytest.mark.gpu

# the map projection's last bit on rare cells (see test_gpu_ortho_tin.py)
RHO_TOL = 1e-9


def same(got, want):
    return (got[0] == want[0] and got[1] == want[1]
            and (np.isnan(want[2]) if np.isnan(got[2]) else abs(got[2] - want[2]) <= RHO_TOL))


CASES = {
    "cells25": dict(seed=38, size=512, nodes=64, res=3.0, point_frac=0.05, range_m=12.0),
    "cells3": dict(seed=41, size=512, nodes=64, res=3.0, point_frac=0.35, range_m=20.0),
    "cells400": dict(seed=37, size=512, nodes=128, res=1.5, point_frac=0.0006, range_m=6.0),
    "heights": dict(seed=39, size=512, nodes=48, res=4.0, point_frac=0.08, range_m=70.0),
    "level2": dict(seed=42, size=512, nodes=24, res=8.0, L=2, template=15, range_m=30.0),
    "images": dict(seed=35, size=512, nodes=32, res=6.0, n_images=3, anchor_frac=0.4, range_m=10.0),
    "one": dict(seed=38, size=512, nodes=64, res=3.0, point_frac=0.05, range_m=0.2),
    "few": dict(seed=38, size=512, nodes=64, res=3.0, point_frac=0.05, range_m=2.0),
    "seven": dict(seed=38, size=512, nodes=64, res=3.0, point_frac=0.05, range_m=1.0),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_single_searches(gpu_ctx, name):
    inp, pts, tris = cases.make_tin_case(**CASES[name])
    jobs = searchable(inp, pts, tris)
    found = 0
    for three, node in jobs[:: max(1, len(jobs) // 8)][:8]:
        want = oo.search(inp, 1.0, three, node)
        assert same(gpu_ctx.vertical_line_locus_ortho(inp, 1.0, three, node), want)
        found += want[1] != -9999.0
    assert found > 0


MPP = 3.0   # of the searches below


def near_tie(seed):
    """A steep triangle over constant images of which single texels deviate,
    so that two heights' correlations differ by at most 3e-7: the larger one's
    rests on a sample whose coordinate lies 1e-5 to 6e-5 pixel past a texel."""
    rng = np.random.default_rng(seed)
    inp, pts, _ = cases.make_tin_case(seed=38, size=512, nodes=64, res=3.0, point_frac=0.05)
    inp.resolution = 4.0   # heights 12 m apart: their cells' texels lie apart too
    for im in inp.images:
        im.image, im.mag = np.full_like(im.image, 700), np.zeros_like(im.mag)
    g = inp.grid_pts.reshape(64, 64, 2)
    while True:
        i, j = rng.integers(24, 34, 2)
        three = np.zeros(3, abi.POINT3_DTYPE)
        for k, (a, b) in enumerate(((i, j), (i, j + 6), (i + 6, j + 1))):
            three["x"][k], three["y"][k] = g[a, b]
        z0, dz = float(rng.integers(90, 140)), float(rng.integers(150, 170))
        three["z"] = z0, z0 + dz, z0 - dz
        node = int((i + 6) * 64 + j + 1)
        inp.gridpt3["minHeight"][node], inp.gridpt3["maxHeight"][node] = z0 - dz - 108, z0 - dz + 108
        hs = oo.heights(inp, MPP, node)
        t = oo.Triangle(inp, three)
        xy = np.stack([t.coords(h)[0] for h in hs])        # height, image, cell, axis
        if len(t.cx) < 12 or xy.min() < 8 or xy.max() > 500:
            continue
        frac = xy - np.floor(xy)
        at = np.argwhere((frac > 1e-5) & (frac < 6e-5))
        if not len(at):
            continue
        h1, im1, p, axis = at[0]
        h2 = (h1 + 9) % len(hs)
        lo = np.floor(xy).astype(int)
        # the texel blocks of all heights' cells must be apart from the used ones
        move = np.abs(xy[1, 0] - xy[0, 0]).max(axis=1)
        cells = [p] + [c for c in np.argsort(-move) if c != p][:2]
        if move[cells].min() < 2.5:
            continue
        images = [im.image for im in inp.images]

        def block(h, im, c, v, far=None):
            x, y = lo[h, im, c]
            if far is None:
                images[im][y:y + 2, x:x + 2] = v
            elif far == 0:
                images[im][y:y + 2, x + 1] = v
            else:
                images[im][y + 1, x:x + 2] = v

        dev = float(frac[h1, im1, p, axis]) * (65535 - 700)
        a1 = np.array([dev, *rng.choice([-1, 1]) * rng.integers(1, 5, 2)], float)
        b1 = np.array([rng.integers(4, 30), *rng.integers(-30, 30, 2)], float)
        n = len(t.cx)

        def corr(a, b):
            sa, sb = a.sum(0) / n, b.sum(0) / n
            return (((a * b).sum(0) - n * sa * sb)
                    / np.sqrt(((a * a).sum(0) - n * sa * sa) * ((b * b).sum(0) - n * sb * sb)))

        r1 = float(corr(a1, b1))
        if not 0.6 < r1 < 0.92:
            continue
        # the second height's blocks: whole numbers for a correlation just below
        a2 = rng.integers(2000, 60000, 3).astype(float)
        u = rng.integers(2000, 60000, (3, 1500000)).astype(float)
        r2 = corr(np.broadcast_to(a2[:, None], u.shape), u)
        d = r1 - r2
        ok = np.flatnonzero((d > 3e-8) & (d < 3e-7))
        if not len(ok):
            continue
        b2 = u[:, ok[0]]
        for k, c in enumerate(cells):
            block(h1, im1, c, int(700 + a1[k]) if k else 65535, None if k else axis)
            block(h1, 1 - im1, c, int(700 + b1[k]))
            block(h2, im1, c, int(700 + a2[k]))
            block(h2, 1 - im1, c, int(700 + b2[k]))
        e = [t.evaluate(h) for h in hs]
        rho = np.array([x[0] if x and x[2] >= 10 else -2.0 for x in e])
        o = np.argsort(-rho)
        if o[0] == h1 and o[1] == h2 and 2e-8 < rho[h1] - rho[h2] < 4e-7 and rho[h2] - rho[o[2]] > 1e-3:
            return inp, three, node
        for im in images:
            im[:] = 700


@pytest.mark.parametrize("seed", [0, 3, 5, 6, 9, 10, 11])
def test_near_tie(gpu_ctx, seed):
    inp, three, node = near_tie(seed)
    want = oo.search(inp, MPP, three, node)
    assert want[0] >= 10
    assert same(gpu_ctx.vertical_line_locus_ortho(inp, MPP, three, node), want)


WHOLE = {
    # few heights at small triangles, at triangles of more than 512 box cells
    # and more than 256 inside ones; several images; narrow and wide ranges
    "small": (dict(seed=38, size=512, nodes=48, res=4.0, point_frac=0.08), 2),
    "large": (dict(seed=37, size=512, nodes=128, res=1.5, point_frac=0.001), 1),
    "images": (dict(seed=35, size=512, nodes=24, res=8.0, n_images=3, anchor_frac=0.4), 3),
    "mixed": (dict(seed=31, size=512, nodes=40, res=5.0, point_frac=0.1), None),
}


@pytest.mark.parametrize("name", sorted(WHOLE))
def test_whole_calls(gpu_ctx, name):
    kw, span = WHOLE[name]
    inp, pts, tris = cases.make_tin_case(**kw)
    g = inp.gridpt3
    on = g["anchor_flag"] > 0
    mid = (g["minHeight"][on].astype(int) + g["maxHeight"][on]) // 2
    rng = np.random.default_rng(5)
    half = span if span else rng.choice([0, 1, 2, 3, 4, 12], len(mid))
    g["minHeight"][on], g["maxHeight"][on] = mid - half, mid + half
    got_g, got_p = g.copy(), pts.copy()
    oo.ortho_blunder(inp, 1.0, pts, tris)
    want = inp.gridpt3
    inp.gridpt3 = got_g
    gpu_ctx.ortho_blunder(inp, 1.0, got_p, tris)
    assert all(np.array_equal(got_p[f], pts[f]) for f in ("x", "y", "z", "flag"))
    assert np.array_equal(got_g["anchor_flag"], want["anchor_flag"])
    assert (want["anchor_flag"] == 3).any()
