"""The orthoimage window passes with three and five images: every target
image's NCC equals the pair's, the rasters take one sample of 16 bytes per
pixel and image, and the launches are counted as they are made."""
import copy

import numpy as np
import pytest

from setsm_b200 import vll
from tests import cases

pytestmark = pytest.mark.gpu

PASSES = {"seeddem": lambda c, i: c.seeddem(i), "blunder": lambda c, i: c.blunder(i, 1, False)}


def fresh(inp, images, **kw):
    i = copy.copy(inp)
    i.images, i.gridpt3 = list(images), inp.gridpt3.copy()
    for k, v in kw.items():
        setattr(i, k, v)
    return i


@pytest.mark.parametrize("name", sorted(PASSES))
@pytest.mark.parametrize("ref", [0, 2])
def test_each_target_is_its_pair(gpu_ctx, name, ref):
    """UGRID.ortho_ncc has two entries; the third image's NCC lands on the
    record's next field, so the triple's second target shows there."""
    inp = cases.make_variant_case(seed=28, size=512, nodes=32, res=8.0, n_images=3, minmax=(-9000, 9000))
    run = PASSES[name]
    triple = fresh(inp, inp.images, reference_id=ref)
    run(gpu_ctx, triple)
    # the first target's NCC alone: images {reference, target} as a pair
    order = [inp.images[ref], inp.images[1]]
    pair = fresh(inp, order)
    run(gpu_ctx, pair)
    assert np.array_equal(triple.gridpt3["ortho_ncc"][:, 1], pair.gridpt3["ortho_ncc"][:, 1])


@pytest.mark.parametrize("name", sorted(PASSES))
@pytest.mark.parametrize("images,launches", [(2, 4), (3, 5), (5, 7)])
def test_launches(gpu_ctx, name, images, launches):
    """A raster launch for the reference and the first target, one for each
    further target, the flags, the nodes and the listed nodes."""
    inp = cases.make_variant_case(seed=28, size=512, nodes=32, res=8.0, n_images=3)
    ims = [inp.images[k] for k in (0, 1, 2, 1, 2)][:images]
    before = gpu_ctx.launch_count()
    PASSES[name](gpu_ctx, fresh(inp, ims))
    assert gpu_ctx.launch_count() - before == launches


def test_raster_bytes():
    """Three images of a 2049 x 2049 raster: 3 x 16 bytes per pixel (and less
    than a quarter of one image's for all else)."""
    import torch
    inp = cases.make_variant_case(seed=28, size=1024, nodes=32, res=16.0, n_images=3)
    pixels = (int((inp.boundary[2] - inp.boundary[0]) / 0.25) + 1) ** 2
    assert pixels > 4.1e6
    ctx = vll.Context(0)
    try:
        # the images' buffers, over a raster of a few pixels
        ctx.blunder(fresh(inp, inp.images, resolution=16.0), 1, False)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        ctx.blunder(fresh(inp, inp.images, resolution=0.25), 1, False)
        used = free - torch.cuda.mem_get_info()[0]
    finally:
        ctx.close()
    assert used < 3.25 * 16 * pixels, used / pixels
