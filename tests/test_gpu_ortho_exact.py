"""The sampled-raster node passes (seed DEM, blunder) against the reference's
order of operations in numpy (ortho_oracle.py): the rounded NCC of nodes whose
window is constant but for a few texels, where it lies within 1e-6 of a
rounding boundary and rests on a sample that a coordinate error of 1e-8 pixel
moves by more; and the float NCC of the blunder pass, values near zero among
them."""
import numpy as np
import pytest

from tests import cases, ortho_oracle as oo

pytestmark = pytest.mark.gpu


def constant_but_for_texels(seed, matchtag=False):
    """A scene of constant images with single texels raised at the corners of
    some nodes' windows.  Returns the inputs and {node: NCC}."""
    inp = cases.make_variant_case(seed=seed, size=512, nodes=26, res=8.0, off_frac=0.0,
                                  void_frac=0.0, matchtag=matchtag)
    inp.gridpt3["Height"] = 150.0
    for im in inp.images:
        im.image, im.mag = np.full_like(im.image, 700), np.zeros_like(im.mag)
        im.image_b, im.mag_b = im.image, im.mag
    half = oo.seeddem_half(inp)
    r2max = (half + 1) ** 2
    ras = oo.Raster(inp, 0, False)
    rng = np.random.default_rng(seed)
    w = inp.grid_width

    def single(im, px):
        """{window pixel: (texel x, y, weight, 1 / smallest fraction)} of texels
        that one pixel of the window touches."""
        xy = ras.xy[im][px]
        lo, f = np.floor(xy).astype(int), xy - np.floor(xy)
        touched = {}
        for k in range(len(px)):
            for ox in (0, 1):
                for oy in (0, 1):
                    wx, wy = (f[k, 0] if ox else 1 - f[k, 0]), (f[k, 1] if oy else 1 - f[k, 1])
                    touched.setdefault((lo[k, 0] + ox, lo[k, 1] + oy), []).append(
                        (k, wx * wy, 1 / min(wx, wy)))
        out = {}
        for (x, y), t in touched.items():
            if len(t) == 1:
                out.setdefault(t[0][0], []).append((x, y, t[0][1], t[0][2]))
        return out

    found = []
    for pt in range(inp.n):
        if not (2 <= pt % w < w - 2 and 2 <= pt // w < inp.grid_height - 2):
            continue
        px, _ = ras.window(pt, half, r2max)
        L, R = single(0, px), single(1, px)
        for k, t in L.items():
            for x, y, wt, s in t:
                if s > 300 and wt * 64835 > 0.05 and k in R:
                    found.append((s, pt, px, k, (x, y, wt), L, R))
    found.sort(key=lambda c: -c[0])
    nodes = {}
    for s, pt, px, k, (x, y, wt), L, R in found:
        if pt in nodes or len(nodes) >= 40:
            continue
        other = [q for q in L if q in R and q != k]
        if not other:
            continue
        q = other[int(rng.integers(len(other)))]
        lq = max(L[q], key=lambda t: t[2])
        rk, rq = max(R[k], key=lambda t: t[2]), max(R[q], key=lambda t: t[2])
        n, dev = float(len(px)), wt * 64835
        a = np.zeros(2)
        a[0] = dev
        dl = max(1, min(64000, int(round(dev * rng.uniform(0.3, 2.0) / lq[2]))))
        a[1] = dl * lq[2]
        d1, d2 = rng.integers(500, 64000, (2, 400000))
        b1, b2 = d1 * rk[2], d2 * rq[2]
        sa, sb = a.sum() / n, (b1 + b2) / n
        r = ((a[0] * b1 + a[1] * b2 - n * sa * sb)
             / np.sqrt(((a * a).sum() - n * sa * sa) * (b1 * b1 + b2 * b2 - n * sb * sb)))
        side = 1 if len(nodes) & 1 else -1
        off = (r * 1000.0 - np.floor(r * 1000.0) - 0.5) / 1000.0 * side
        ok = np.flatnonzero((off > 3e-7) & (off < 8e-7) & (r > 0.35) & (r < 0.95))
        if not len(ok):
            continue
        i = ok[0]
        I0, I1 = inp.images[0].image, inp.images[1].image
        I0[y, x], I0[lq[1], lq[0]] = 65535, 700 + dl
        I1[rk[1], rk[0]], I1[rq[1], rq[0]] = 700 + d1[i], 700 + d2[i]
        nodes[pt] = None
    for pt in list(nodes):
        v = oo.Raster.ncc(ras, pt, 1, half, r2max)[0]
        d = abs(v * 1000.0 - np.floor(v * 1000.0) - 0.5) / 1000.0
        if 2.2e-7 < d < 1e-6:
            nodes[pt] = v
        else:
            del nodes[pt]   # another node's texel lies in its window
    return inp, nodes


@pytest.mark.parametrize("seed", [3, 5, 8])
def test_seeddem_rounds_as_the_reference(gpu_ctx, seed):
    inp, nodes = constant_but_for_texels(seed)
    assert len(nodes) >= 15
    gpu_ctx.seeddem(inp)
    got = {pt: int(inp.gridpt3["ortho_ncc"][pt, 1]) for pt in nodes}
    assert got == {pt: oo.quantize(v) for pt, v in nodes.items()}


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
