"""The sampled-raster node passes (seed DEM, blunder) against the reference's
order of operations in numpy (ortho_oracle.py): the float NCC of the blunder
pass, values near zero among them."""
import numpy as np
import pytest

from tests import cases, ortho_oracle as oo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [
    dict(seed=11, size=512, nodes=40, res=6.0, template=5, blunder_level=1),
    dict(seed=11, size=512, nodes=40, res=6.0, template=7, blunder_level=1),
    dict(seed=12, size=512, nodes=40, res=6.0, template=11, blunder_level=1),
    dict(seed=13, size=512, nodes=24, res=9.0, template=15, blunder_level=0),
])
@pytest.mark.parametrize("content", ["scene", "flat", "holes"])
def test_blunder_floats(gpu_ctx, kw, content):
    """Within 1e-6 of the reference everywhere (the projection's last bit),
    and zero exactly where it is zero: one-pass sums may cancel to zero where
    the reference's two-pass ones leave 1e-17."""
    inp = cases.make_variant_case(**kw)
    rng = np.random.default_rng(kw["seed"])
    for im in inp.images:
        im.image_b, im.mag_b = im.image_b.copy(), im.mag_b.copy()
        h, w = im.image_b.shape
        if content == "flat":
            im.image_b[:, : w // 2], im.mag_b[:, : w // 2] = 321, 0
            y, x = rng.integers(0, h, 900), rng.integers(0, w // 2, 900)
            im.image_b[y, x] = rng.integers(300, 340, 900)
        elif content == "holes":   # windows of one, two and three samples
            im.image_b[rng.random((h, w)) < 0.8] = 0
    want = oo.blunder(inp)
    got = gpu_ctx.blunder(inp, 1, False)
    w32 = want.astype(np.float32)
    assert np.array_equal(got == 0, w32 == 0)
    assert np.abs(got.astype(np.float64) - want).max() < 1e-6
    assert np.count_nonzero(got != w32) <= 2
