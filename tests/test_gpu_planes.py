"""The preprocessing kernels against the oracle at the sizes where their tiles
end and on the images where a vote or a truncation is not decided by the
cheap sums: constant, near-empty, periodic and full-range images (exact
equality: the outputs are integers)."""
import numpy as np
import pytest

from oracle import oraclepy as op

pytestmark = pytest.mark.gpu

SIZES = [(3, 5), (13, 13), (14, 77), (29, 140), (28, 76), (131, 203)]


def image(kind, h, w):
    rng = np.random.default_rng(h * 1000 + w)
    y, x = np.mgrid[0:h, 0:w]
    a = {"bits11": rng.integers(0, 2048, (h, w)),
         "full": rng.integers(0, 65536, (h, w)) // 2,
         "flat": np.full((h, w), 777),
         "empty": (rng.random((h, w)) < 0.005) * 3,
         "check": ((x // 3 + y // 3) % 2) * 500}[kind]
    return np.ascontiguousarray(a.astype(np.uint16))


@pytest.mark.parametrize("kind", ["bits11", "full", "flat", "empty", "check"])
@pytest.mark.parametrize("h,w", SIZES)
def test_planes_match_oracle(gpu_ctx, kind, h, w):
    im = image(kind, h, w)
    mag, ori = gpu_ctx.preprocess(im)
    mag2, ori2 = op.preprocess(im)
    assert np.array_equal(mag, mag2)
    assert np.array_equal(ori, ori2)
    assert np.array_equal(gpu_ctx.pyramid_down(im), op.pyramid_down(im))
