"""FP32 windows of combined levels against the FP64 kernel, slot by slot: the
mean over the two pyramid levels, odd and even widths, and images with
saturated and constant areas, where a window may rest on a few samples.  The
kernel settles in FP32 the decisions further than 4e-6 from their boundary,
which holds while the error stays below half of that (a slot that FP32 does
not settle has its FP64 value here)."""
import numpy as np
import pytest

from oracle import oraclepy as op
from tests import cases

pytestmark = pytest.mark.gpu

CASES = {
    "l1_7": dict(L=1, it=2, nodes=64, res=6.0, n_heights=64, hs=0.5, size=1024),
    "l1_11": dict(L=1, it=2, nodes=64, res=6.0, n_heights=64, hs=0.5, size=1024, template=15),
    "l2_7": dict(L=2, it=2, nodes=56, res=8.0, n_heights=48, hs=1.0, size=1111),
    "l2_11": dict(L=2, it=4, nodes=56, res=8.0, n_heights=48, hs=1.0, size=1024, template=15),
    "l3_11": dict(L=3, it=2, nodes=40, res=12.0, n_heights=48, hs=2.0, size=1100, template=15),
}


def change(inp, content):
    rng = np.random.default_rng(1)
    for im in inp.images:
        for a, m in (("image", "mag"), ("image_next", "mag_next")):
            v = getattr(im, a).copy()
            h, w = v.shape
            if content == "saturated":
                v = np.minimum(v, np.uint16(np.quantile(v, 0.5)))
            elif content == "constant":
                y, x = np.arange(h)[:, None] // 31, np.arange(w)[None] // 31
                v[((y * 7 + x * 13) % 5) < 2] = 500
            elif content == "spikes":
                v[:] = 700
                v[rng.random((h, w)) < 0.004] = 60000
            setattr(im, a, v)
            setattr(im, m, op.sobel(v)[0])


@pytest.mark.parametrize("content", ["scene", "saturated", "constant", "spikes"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_fp32_rho_error(gpu_ctx, name, content):
    inp = cases.make_case(**CASES[name])
    if content != "scene":
        change(inp, content)
    r32, off = gpu_ctx.debug_slot_rho(inp, inp.new_nccresult(), "split")
    r64, off2 = gpu_ctx.debug_slot_rho(inp, inp.new_nccresult(), "plain")
    assert np.array_equal(off, off2) and np.array_equal(np.isnan(r32), np.isnan(r64))
    both = ~np.isnan(r32)
    assert both.sum() > 1000
    err = np.abs(r32[both] - r64[both])
    print(f"{name} {content}: {both.sum()} slots, max |dNCC| {err.max():.3e}")
    assert err.max() < 2e-6
