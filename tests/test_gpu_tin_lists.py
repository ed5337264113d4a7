"""TINCreate_list's triangle lists, in order, against stored digests: full and
partly filled integer grids (co-circular points everywhere), subtree sizes
either side of the 100-point cut and of the block's 1024 points, lines, strips
and points beyond the extent.  The digests were stored from the implementation
whose lists the tests against the reference build had compared."""
import hashlib

import numpy as np
import pytest

from setsm_b200 import abi

pytestmark = pytest.mark.gpu

RES, X0, Y0 = 2.0, 1000.0, 5000.0

# (width, height, kept fraction or number of points, first row) -> digest
SETS = {
    "n3": (80, 80, 3, 0, "2:be3389a2442b014a"),
    "n4": (80, 80, 4, 0, "4:6c7215db59c11bfb"),
    "n7": (80, 80, 7, 0, "7:ed546835edefe874"),
    "n99": (80, 80, 99, 0, "180:973ca04e6cc593cd"),
    "n100": (80, 80, 100, 0, "184:40cbb3d7fc485a40"),
    "n199": (80, 80, 199, 0, "377:82f4e709286cfd51"),
    "n401": (80, 80, 401, 0, "771:d8a82e14cb65266e"),
    "n1024": (80, 80, 1024, 0, "1988:60acd3d59eda1502"),
    "n1025": (80, 80, 1025, 0, "1994:9e08d0cc0b355432"),
    "n2049": (80, 80, 2049, 0, "3989:e2a24dabc990f789"),
    "full": (64, 41, 1.0, 0, "5040:eb92c74164d68eab"),
    "row": (300, 1, 1.0, 0, "0:e3b0c44298fc1c14"),
    "column": (1, 300, 1.0, 0, "0:e3b0c44298fc1c14"),
    "strip": (900, 20, 0.5, 0, "17074:8f5b3a1406059fc7"),
    "half": (211, 190, 0.5, 0, "39665:f57b0deeaebf32aa"),
    "beyond": (30, 30, 600, 20, "1107:11e0ee3cf4e7a373"),
}


def points(name):
    w, h, keep, row0, _ = SETS[name]
    rng = np.random.default_rng(sum(map(ord, name)))
    n = keep if isinstance(keep, int) else int(keep * w * h)
    cells = rng.permutation(w * h)[:n]
    p = np.zeros(n, dtype=abi.POINT3_DTYPE)
    j = (rng.random((n, 2)) - 0.5) * 0.8 * RES
    p["x"] = X0 + (cells % w) * RES + j[:, 0]
    p["y"] = Y0 + (cells // w + row0) * RES + j[:, 1]
    return p, [X0, Y0, X0 + (w - 1) * RES, Y0 + (h - 1) * RES]


@pytest.mark.parametrize("name", sorted(SETS))
def test_triangle_list_digest(gpu_ctx, name):
    p, extent = points(name)
    tris = gpu_ctx.tin_create(p, extent, RES)
    digest = f"{len(tris)}:" + hashlib.sha256(tris.tobytes()).hexdigest()[:16]
    assert digest == SETS[name][4]
