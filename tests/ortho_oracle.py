"""VerticalLineLocus_Ortho, VerticalLineLocus_seeddem and _blunder restated in
numpy, in the reference's FP64 operation order (setsm_code.cpp:8234-8533,
:7720-8026; Correlate and SetVecKernelValue, SubFunctions.cpp:974-1018,
:3281-3360): every height and every node evaluated, nothing screened.  The
projections are the C oracle's.  Sums run in the reference's order
(np.cumsum adds one term after the other)."""
from __future__ import annotations

import numpy as np

from oracle import oraclepy as op


def ordered_sum(v):
    return float(np.cumsum(v)[-1]) if len(v) else 0.0


def coords(im, adjust, lonlat, h, level, start):
    """Pyramid coordinates (n, 2) of points at the heights h."""
    xy = op.rpc_project(im.rpc, adjust, lonlat[:, 0], lonlat[:, 1], h)
    s = float(1 << level)
    return np.stack([xy[:, 0] / s - start[0], xy[:, 1] / s - start[1]], axis=1)


def inside(xy, img):
    hh, w = img.shape
    x, y = xy[:, 0], xy[:, 1]
    return (y >= 0) & (y + 1.0 < float(hh)) & (x >= 0) & (x + 1.0 < float(w))


def interp(img, xy):
    """InterpolatePatch at coordinates inside the image."""
    xi, yi = xy[:, 0].astype(np.int64), xy[:, 1].astype(np.int64)
    dx, dy = xy[:, 0] - xi, xy[:, 1] - yi
    t0 = (img[yi, xi].astype(np.float64) * (1.0 - dx)) * (1.0 - dy)
    t1 = (img[yi, xi + 1].astype(np.float64) * dx) * (1.0 - dy)
    t2 = (img[yi + 1, xi].astype(np.float64) * (1.0 - dx)) * dy
    t3 = (img[yi + 1, xi + 1].astype(np.float64) * dx) * dy
    return ((t0 + t1) + t2) + t3


def correlate(l, r):
    """Correlate: the correlation, or -99 where a variance sum is below 1e-8."""
    n = float(len(l))
    dl, dr = l - ordered_sum(l) / n, r - ordered_sum(r) / n
    lr, ll, rr = ordered_sum(dl * dr), ordered_sum(dl * dl), ordered_sum(dr * dr)
    return lr / np.sqrt(ll * rr) if ll > 1e-8 and rr > 1e-8 else -99.0


# ---- Ortho_blunder's search ------------------------------------------------------
class Triangle:
    """A triangle's inside cells (the reference's box and edge tests)."""

    def __init__(self, inp, three):
        self.inp, self.p = inp, [tuple(float(three[f][i]) for f in "xyz") for i in range(3)]
        gs, b = inp.grid_resolution, inp.boundary
        (x1, y1, _), (x2, y2, _), (x3, y3, _) = self.p
        xs, ys = (x1, x2, x3), (y1, y2, y3)
        c0 = max(0, int((min(xs) - b[0]) / gs + 0.5) - 1)
        r0 = max(0, int((min(ys) - b[1]) / gs + 0.5) - 1)
        c1 = min(inp.grid_width - 1, int((max(xs) - b[0]) / gs + 0.5) + 1)
        r1 = min(inp.grid_height - 1, int((max(ys) - b[1]) / gs + 0.5) + 1)
        self.cx = self.cy = np.zeros(0)
        if c1 - c0 > 0 and r1 - r0 > 0:
            cc, rr = np.meshgrid(np.arange(c0, c1 + 1), np.arange(r0, r1 + 1))
            cx, cy = cc.ravel() * gs + b[0], rr.ravel() * gs + b[1]
            n = ((x2 - x1) * (cy - y1) - (y2 - y1) * (cx - x1) > 0).astype(int)
            n += (x3 - x2) * (cy - y2) - (y3 - y2) * (cx - x2) > 0
            n += (x1 - x3) * (cy - y3) - (y1 - y3) * (cx - x3) > 0
            keep = (n == 0) | (n == 3)
            self.cx, self.cy = cx[keep], cy[keep]
        self.lonlat = op.ps2wgs(inp.param, np.stack([self.cx, self.cy], axis=1))

    def plane_z(self, iter_height):
        """The cells' heights on the plane through the third vertex at
        iter_height, or None."""
        (x1, y1, z1), (x2, y2, z2), (x3, y3, _) = self.p
        ax, ay, az = x2 - x1, y2 - y1, z2 - z1
        bx, by, bz = x3 - x1, y3 - y1, float(iter_height) - z1
        nx, ny, nz = ay * bz - az * by, az * bx - ax * bz, ax * by - ay * bx
        ln = float(np.sqrt(nx * nx + ny * ny + nz * nz))
        if not ln > 0:
            return None
        nx, ny, nz = nx / ln, ny / ln, nz / ln
        if nz == 0:
            return None
        d = -((nx * x1 + ny * y1) + nz * z1)
        return -((nx * self.cx + ny * self.cy) + d) / nz

    def coords(self, iter_height):
        """[reference, target 1, ...] pyramid coordinates of the cells (the
        targets with the reference image's adjustment, as the reference does)."""
        z = self.plane_z(iter_height)
        if z is None or not len(z):
            return None
        ims, ref = self.inp.images, self.inp.images[self.inp.reference_id]
        order = [ref] + [im for im in ims[1:] if im.selected]
        return [coords(im, ref.adjust, self.lonlat, z, self.inp.pyramid_step, im.startpos)
                for im in order], order

    def evaluate(self, iter_height):
        """(correlation, mean sample count as double, as int) or None."""
        c = self.coords(iter_height)
        if c is None:
            return None
        xy, ims = c
        total, n_img, n_sum = 0.0, 0, 0
        for k in range(1, len(ims)):
            ok = inside(xy[0], ims[0].image) & inside(xy[k], ims[k].image)
            if not ok.any():
                continue
            rho, cnt = 0.0, 0.0
            for a in ("image", "mag"):
                v = correlate(interp(getattr(ims[0], a), xy[0][ok]),
                              interp(getattr(ims[k], a), xy[k][ok]))
                if v != -99.0:
                    cnt += 1.0
                    rho += v
            total += rho / cnt if cnt > 0 else -1.0
            n_sum += int(ok.sum())
            n_img += 1
        return (total / n_img, n_sum / n_img, n_sum // n_img) if n_img else None


def heights(inp, mpp, node):
    lo, hi = int(inp.gridpt3["minHeight"][node]), int(inp.gridpt3["maxHeight"][node])
    step = inp.resolution * (1 << inp.pyramid_step) * min(max(mpp, 1.0), 3.0)
    return [np.float32(lo + k * step) for k in range(int((hi - lo) / step) + 1)]


def search(inp, mpp, three, node):
    """VerticalLineLocus_Ortho: (selected count, F_Height, F_sncc or NaN)."""
    t = Triangle(inp, three)
    low = inp.pyramid_step < 4
    min_n, min_rho = (0, 0.5) if low else (2, 0.2)
    best, out = -1.0, (0, -9999.0, float("nan"))
    for h in heights(inp, mpp, node):
        e = t.evaluate(h)
        if e is None:
            continue
        rho, n, n_int = e
        if n_int >= 10:
            if rho > min_rho and best < rho:
                best, out = rho, (int(n), float(h), rho)
        elif n_int > min_n:
            if rho > min_rho + 0.2 and best < rho:
                best, out = rho, (int(n), (t.p[0][2] + t.p[1][2]) / 2.0, rho)
    return out


# ---- the orthoimage window passes ------------------------------------------------
class Raster:
    """The sampled ortho pixels of a pass: im_res-spaced pixels at their grid
    cells' heights; blunder: the blunder level's images."""

    def __init__(self, inp, level, use_b):
        self.inp, g = inp, inp.gridpt3
        self.res = inp.resolution * float(1 << level)
        b, gs = inp.boundary, inp.grid_resolution
        self.w = int((b[2] - b[0]) / self.res) + 1
        self.h = int((b[3] - b[1]) / self.res) + 1
        x, y = b[0] + np.arange(self.w) * self.res, b[1] + np.arange(self.h) * self.res
        tc, tr = ((x - b[0]) / gs).astype(np.int64), ((y - b[1]) / gs).astype(np.int64)
        on = (tr < inp.grid_height)[:, None] & (tc < inp.grid_width)[None]
        cell = np.where(on, np.minimum(tr, inp.grid_height - 1)[:, None] * inp.grid_width
                        + np.minimum(tc, inp.grid_width - 1)[None], 0)
        hgt = g["Height"][cell].astype(np.float64)
        on &= hgt != -1000
        xx, yy = np.broadcast_arrays(x[None], y[:, None])
        ll = op.ps2wgs(inp.param, np.stack([xx.ravel(), yy.ravel()], axis=1))
        self.xy, self.planes = [], []
        for im in inp.images:
            c = coords(im, im.adjust, ll, hgt.ravel(),
                       inp.blunder_level if use_b else inp.pyramid_step,
                       im.startpos_b if use_b else im.startpos)
            c[~on.ravel()] = 0.0
            self.xy.append(c)
            self.planes.append((im.image_b, im.mag_b) if use_b else (im.image, im.mag))

    def window(self, pt, half, r2max):
        """(raster pixel, sub-window depth) of node pt's window, in the
        reference's order."""
        inp = self.inp
        b, gs = inp.boundary, inp.grid_resolution
        gx, gy = inp.grid_pts[pt]
        s1 = half // 2
        s2 = s1 + int(s1 / 2.0 + 0.5)
        out, dep = [], []
        for row in range(-half, half + 1):
            for col in range(-half, half + 1):
                r2 = row * row + col * col
                if r2 > r2max or r2 > (half + 1) ** 2:
                    continue
                tx, ty = gx + col * self.res, gy + row * self.res
                c, r = int((tx - b[0]) / self.res), int((ty - b[1]) / self.res)
                cc, cr = int((tx - b[0]) / gs), int((ty - b[1]) / gs)
                if not (0 <= c < self.w and 0 <= r < self.h and 0 <= cc < inp.grid_width
                        and 0 <= cr < inp.grid_height):
                    continue
                if inp.gridpt3["Height"][cr * inp.grid_width + cc] == -1000:
                    continue
                d = 0
                for k, s in ((1, s1), (2, s2)):
                    e = half - s
                    if r2 <= (e + 1) ** 2 and abs(row) <= e and abs(col) <= e:
                        d = k
                out.append(r * self.w + c)
                dep.append(d)
        return np.array(out, np.int64), np.array(dep)

    def ncc(self, pt, ti, half, r2max):
        """(NCC, samples of the whole window) of node pt against image ti."""
        px, dep = self.window(pt, half, r2max)
        if not len(px):
            return 0.0, 0
        ref = self.inp.reference_id
        p, q = self.xy[ref][px], self.xy[ti][px]
        ok = inside(p, self.planes[ref][0]) & inside(q, self.planes[ti][0])
        p, q, dep = p[ok], q[ok], dep[ok]
        v = [interp(self.planes[ref][0], p), interp(self.planes[ref][1], p),
             interp(self.planes[ti][0], q), interp(self.planes[ti][1], q)]
        ok = (v[0] > 0) & (v[2] > 0)
        v, dep = [a[ok] for a in v], dep[ok]
        if not all((dep >= k).any() for k in range(3)):
            return 0.0, len(dep)
        tot, n = 0.0, 0.0
        for k in range(3):
            m = dep >= k
            for a in (0, 1):
                r = correlate(v[a][m], v[a + 2][m])
                if r != -99.0:
                    n += 1.0
                    tot += r
        return (tot / n if n > 0 else 0.0), len(dep)


def seeddem_half(inp):
    t = int((5.0 / (inp.resolution * (1 << inp.pyramid_step))) / 2.0) * 2 + 1
    return max(inp.template_size, t) // 2


def blunder_half(inp):
    """Window half-size of the blunder pass with bblunder false."""
    t = int((5.0 / (inp.resolution * (1 << inp.blunder_level))) / 2.0) * 2 + 1
    return max(inp.template_size & 255, t) // 2


def quantize(v):
    """SignedCharToDouble_result's inverse: round half away from zero."""
    x = v * 1000.0
    return int(np.floor(abs(x) + 0.5) * (1 if x >= 0 else -1))


# ---- whole calls -----------------------------------------------------------------
def ortho_blunder(inp, mpp, pts, tris):
    """Ortho_blunder (setsm_code.cpp:8028-8232) on inp.gridpt3 and pts in place:
    rounds of searches over the triangles with two anchored vertices, then the
    results taken in triangle order (a point's height by the triangle with the
    most samples so far)."""
    b, gs, g = inp.boundary, inp.grid_resolution, inp.gridpt3
    node = (((pts["y"] - b[1]) / gs + 0.5).astype(np.int64) * inp.grid_width
            + ((pts["x"] - b[0]) / gs + 0.5).astype(np.int64))
    v = np.stack([tris[f].astype(np.int64) for f in "abc"], axis=1)
    done = np.zeros(len(tris), bool)
    flag = lambda t: [int(g["anchor_flag"][node[k]]) for k in v[t]]
    for _ in range(200):
        hits = {}
        for t in np.flatnonzero(~done):
            f = flag(t)
            nf = sum(x in (1, 3) for x in f)
            if nf == 3:
                done[t] = True
            elif nf == 2:
                k = 0 if f[0] == 2 else (1 if f[1] == 2 else 2)
                order = [v[t][i] for i in range(3) if i != k] + [v[t][k]]
                r = search(inp, mpp, pts[order], int(node[v[t][k]]))
                if r[1] != -9999.0:
                    hits[t] = (v[t][k], r)
        most, any_record = {}, False
        for t in np.flatnonzero(~done):
            if t in hits:
                k, r = hits[t]
                if most.get(k, 0) < r[0]:
                    most[k] = r[0]
                    pts["z"][k], pts["flag"][k] = r[1], 0
                    g["anchor_flag"][node[k]] = 3
                    done[t] = any_record = True
            f = flag(t)
            for k, x in zip(v[t], f):
                if x in (1, 3):
                    pts["flag"][k] = 0
            if sum(x in (1, 3) for x in f) == 3:
                done[t] = True
        if not any_record:
            return


def seeddem(inp):
    """VerticalLineLocus_seeddem on inp.gridpt3 (two images)."""
    half = seeddem_half(inp)
    ras = Raster(inp, inp.pyramid_step, inp.check_matchtag)
    lo, hi = inp.minmax_height
    g = inp.gridpt3
    for pt in range(inp.n):
        v, cnt = ras.ncc(pt, 1, half, (half + 1) ** 2)
        if cnt == 0:
            v = -10.0
        if v < 0.3 and not inp.check_matchtag:
            a, z = int(g["minHeight"][pt]) - 100, int(g["maxHeight"][pt]) + 100
            a = int(np.floor(lo)) if a < lo else a
            z = int(np.ceil(hi)) if z > hi else z
            g["minHeight"][pt], g["maxHeight"][pt] = (-9999, -9999) if v < 0.1 else (a, z)
        g["ortho_ncc"][pt, 1] = quantize(v)
        if inp.check_matchtag:
            g["roh"][pt] = quantize(v if v >= 0.2 else -0.2)


def blunder(inp):
    """VerticalLineLocus_blunder's NCC per node, bblunder false (two images)."""
    half = blunder_half(inp)
    ras = Raster(inp, inp.blunder_level, True)
    return np.array([ras.ncc(pt, 1, half, (half - 1) ** 2)[0] for pt in range(inp.n)])
