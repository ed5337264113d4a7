"""The listing of a staged box's zero texels (convert_tile and list_zeros,
setsm_b200/csrc/vll_window.cuh), emulated for 32 lanes on the CPU: the
conversion only takes the minimum of the texels it reads, which must be zero
exactly when the box [0, bw] x [0, bh) holds a zero texel, and the listing then
names each of them once."""
import numpy as np
import pytest


def zero_seen(tex, bw, bh):
    """Whether a lane of the conversion sees a zero: texels bx, bx + 1 and,
    for a whole pair, bx + 2 of each step."""
    bp = (bw + 1) >> 1
    seen = False
    for q in range(bp * bh):
        by, bx = divmod(q, bp)
        bx *= 2
        last = bx + 2 if bx + 1 < bw else bx + 1
        seen |= bool((tex[by, bx:last + 1] == 0).any())
    return seen


def listed(tex, bw, bh):
    return sorted((by, bx) for lane in range(32) for by in range(bh)
                  for bx in range(lane, bw + 1, 32) if tex[by, bx] == 0)


@pytest.mark.parametrize("bh", [1, 2, 9, 23])
def test_zeros_are_seen_and_listed_once(bh):
    rng = np.random.default_rng(bh)
    for bw in range(1, 100):
        for share in (0.0, 0.002, 0.3):
            tex = (rng.random((bh, bw + 9)) >= share).astype(np.uint16)
            tex[:, bw + 1:] = 0           # the tile's texels beyond the box
            want = sorted(map(tuple, np.argwhere(tex[:, :bw + 1] == 0)))
            assert zero_seen(tex, bw, bh) == bool(want), bw
            assert listed(tex, bw, bh) == want, bw
        for x in (0, bw - 1, bw):         # a single zero at each end
            tex = np.ones((bh, bw + 1), np.uint16)
            tex[bh - 1, x] = 0
            assert zero_seen(tex, bw, bh) and listed(tex, bw, bh) == [(bh - 1, x)]
