"""The triangulation's orders made by counting (up to 8192 points) and by
sorting, against digests of the sorting implementation's lists; and
SetHeightRange's cover pass at both sides of the triangle counts where it
changes the lanes per triangle: a list repeated to any length (the first of
equal triangles wins) gives the result of the list itself."""
import copy
import hashlib

import numpy as np
import pytest

from setsm_b200 import abi
from tests import cases

pytestmark = pytest.mark.gpu

RES, X0, Y0, W, H = 2.0, 1000.0, 5000.0, 140, 100
LISTS = {31: "53:e03e3658359b90b8", 32: "51:7b9d6487a7234d21", 33: "55:a7f32ad06331ae92",
         1023: "2010:1d4378d97061dfb5", 8191: "16106:5809f4fae720a50f",
         8192: "16103:17ad04f71e085b14", 8193: "16108:78151e2900073e0b"}


@pytest.mark.parametrize("n", sorted(LISTS))
def test_list_digest(gpu_ctx, n):
    rng = np.random.default_rng(sum(map(ord, f"n{n}")))
    cells = rng.permutation(W * H)[:n]
    p = np.zeros(n, dtype=abi.POINT3_DTYPE)
    j = (rng.random((n, 2)) - 0.5) * 0.8 * RES
    p["x"] = X0 + (cells % W) * RES + j[:, 0]
    p["y"] = Y0 + (cells // W) * RES + j[:, 1]
    t = gpu_ctx.tin_create(p, [X0, Y0, X0 + (W - 1) * RES, Y0 + (H - 1) * RES], RES)
    assert f"{len(t)}:" + hashlib.sha256(t.tobytes()).hexdigest()[:16] == LISTS[n]


@pytest.mark.parametrize("n_tris", [37888, 37889, 75776, 75777])
def test_cover_lanes(gpu_ctx, n_tris):
    inp, pts, tris = cases.make_tin_case(seed=33, size=512, nodes=60, res=4.0, point_frac=0.1)
    results = []
    for t in (tris, np.resize(tris, n_tris)):
        i = copy.copy(inp)
        i.gridpt3 = inp.gridpt3.copy()
        out, ext = gpu_ctx.set_height_range(i, pts, t, 2, 1.5, False)
        results.append((out, i.gridpt3, ext))
    a, b = results
    assert cases.field_mismatch(a[0], b[0]) == {}
    assert cases.field_mismatch(a[1], b[1]) == {}
    assert a[2] == b[2]
