"""blunder_detection_TIN and SetHeightRange on TINs whose points have few,
eight, more than eight and more than 32 triangles (hubs ringed by points) and
whose triangles' boxes lie either side of the size a lane sweeps by itself,
against stored digests (made with the implementation that the tests against
the reference build had compared)."""
import copy
import hashlib

import numpy as np
import pytest

from tests import cases

pytestmark = pytest.mark.gpu

CASES = {   # name: (spokes per hub, case) -> digest
    "few": (5, dict(seed=33, size=512, nodes=60, res=4.0, point_frac=0.5), "29affa1cedf4537f"),
    "eight": (8, dict(seed=34, size=512, nodes=60, res=4.0, point_frac=0.1), "d58b82d87e84211c"),
    "nine": (9, dict(seed=35, size=512, nodes=60, res=4.0, point_frac=0.02, L=1), "c279036eba842b4d"),
    "forty": (40, dict(seed=36, size=512, nodes=90, res=2.5, point_frac=0.01, L=2), "694f7e1093594237"),
}


def inputs(name):
    """A TIN case with two of its triangles' fans multiplied: hubs 0 and 1 in
    `spokes` extra triangles each with pairs of the other points."""
    spokes, kw, _ = CASES[name]
    inp, pts, tris = cases.make_tin_case(**kw)
    rng = np.random.default_rng(spokes)
    extra = np.zeros(2 * spokes, dtype=tris.dtype)
    for i in range(2 * spokes):
        extra["a"][i] = i % 2
        extra["b"][i], extra["c"][i] = 2 + rng.choice(len(pts) - 2, 2, replace=False)
    tris = np.concatenate([tris, extra])
    pts["flag"] = rng.random(len(pts)) < 0.1
    pts["z"] += np.where(rng.random(len(pts)) < 0.1, rng.uniform(-40, 40, len(pts)), 0)
    return inp, pts, tris, rng.uniform(-1, 1, inp.n).astype(np.float32)


def digest(ctx, name):
    inp, pts, tris, oncc = inputs(name)
    h = hashlib.sha256()
    fields = lambda a: [h.update(np.ascontiguousarray(a[f]).tobytes()) for f in a.dtype.names]
    for flag_blunder in (False, True):
        i, p = copy.copy(inp), pts.copy()
        i.gridpt3 = inp.gridpt3.copy()
        det, cnt, z = np.zeros(len(p), np.uint8), np.zeros(2, np.int64), np.array([1e5, -1e5])
        ctx.blunder_detection_tin(i, 1, oncc, flag_blunder, 1, 60.0, p, det, tris, cnt, z)
        fields(p), fields(i.gridpt3)
        h.update(det.tobytes() + cnt.tobytes() + z.tobytes())
    i = copy.copy(inp)
    i.gridpt3 = inp.gridpt3.copy()
    out, ext = ctx.set_height_range(i, pts, tris, 2, 1.5, False)
    fields(out), fields(i.gridpt3)
    h.update(np.array(ext).tobytes())
    return h.hexdigest()[:16]


@pytest.mark.parametrize("name", sorted(CASES))
def test_point_passes_digest(gpu_ctx, name):
    assert digest(gpu_ctx, name) == CASES[name][2]
