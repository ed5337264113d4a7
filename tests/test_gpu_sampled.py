"""The sampled-raster node passes (seed DEM, blunder) against the per-node
kernels: window half-sizes either side of each compiled column count, grids
that do not fill a block, scenes whose pixels leave the images, empty and
constant image areas, unmatched nodes.  The digests are of the per-node
kernels' outputs, stored from the implementation that ran them at every size
(the reference's fixtures cover both)."""
import copy
import hashlib

import numpy as np
import pytest

from tests import cases

pytestmark = pytest.mark.gpu

CASES = {   # name: (case, flatten) -> digest of the UGRIDs and the NCC to 5 decimals
    "h5": (dict(seed=30, size=512, nodes=67, res=3.0), False, "d063a659e28e81ec"),
    "h7": (dict(seed=31, size=500, nodes=61, res=4.0, template=15), True, "91f8a84efdb6f0cb"),
    "h10": (dict(seed=32, size=500, nodes=20, res=25.0, template=21), False, "060487e81b8245ab"),
    "h15": (dict(seed=33, size=600, nodes=33, res=9.0, template=31), False, "b1c238fa959c3a0d"),
    "h16": (dict(seed=33, size=600, nodes=33, res=9.0, template=33), False, "24d9f4671d9a008e"),
    "tag": (dict(seed=22, size=512, nodes=40, res=6.0, L=1, template=15, matchtag=True,
                 blunder_level=1), True, "9d0a992917ff16ae"),
    "images": (dict(seed=28, size=512, nodes=32, res=8.0, n_images=3), False, "71df94ea351a5cb9"),
    "rough": (dict(seed=34, size=512, nodes=64, res=6.0, off_frac=0.9, off_m=200.0), True, "98fb54e07d4426eb"),
}


def digest(ctx, name):
    kw, flatten, _ = CASES[name]
    inp = cases.make_variant_case(**kw)
    if flatten:
        for im in inp.images:
            for f in ("image", "mag", "image_b", "mag_b"):
                a = getattr(im, f).copy()
                h, w = a.shape
                a[: h // 3, : w // 2] = 0
                a[h // 2:, w // 2:] = 700 if f.startswith("image") else 0
                setattr(im, f, a)
    h = hashlib.sha256()
    for call in ("seeddem", (1, False), (3, True)):
        i = copy.copy(inp)
        i.gridpt3 = inp.gridpt3.copy()
        if call == "seeddem":
            ctx.seeddem(i)
        else:
            ncc = ctx.blunder(i, *call)
            h.update(np.round(ncc.astype(np.float64), 5).tobytes())
        for f in i.gridpt3.dtype.names:
            h.update(np.ascontiguousarray(i.gridpt3[f]).tobytes())
    return h.hexdigest()[:16]


@pytest.mark.parametrize("name", sorted(CASES))
def test_sampled_passes_digest(gpu_ctx, name):
    assert digest(gpu_ctx, name) == CASES[name][2]
