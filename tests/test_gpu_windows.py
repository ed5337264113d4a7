"""FP32 window statistics at every half-size of the window kernel: the records
against the C oracle, and the slots' rho against the FP64 kernel (half the
kernel's error band of 4e-6, as its decisions assume), with rotated target
windows, empty image areas whose borders cut the windows, and both parities
of the image width (tile copies and plain loads)."""
import copy

import numpy as np
import pytest

from oracle import oraclepy as op
from tests import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("zero_patch", [False, True])
@pytest.mark.parametrize("size", [512, 509])
@pytest.mark.parametrize("half", [2, 3, 4, 5, 6, 7])
def test_window(gpu_ctx, half, size, zero_patch):
    inp = cases.make_case(seed=40 + half, size=size, nodes=17, res=9.0, template=2 * half + 5,
                          n_heights=45, zero_patch=zero_patch)
    assert inp.template_size // 2 - 2 == half
    o = cases.run_cpu(op, inp, inp.iters)
    got = copy.copy(o["inputs"])
    got.gridpt3 = o["init_gp3"].copy()
    ncc = o["init_ncc"].copy()
    st = gpu_ctx.vertical_line_locus(got, ncc, None, "split")
    assert st.accessable_grid == o["acc"]
    assert cases.field_mismatch(ncc, o["vll_ncc"]) == {}
    r32, _ = gpu_ctx.debug_slot_rho(inp, inp.new_nccresult(), "split")
    r64, _ = gpu_ctx.debug_slot_rho(inp, inp.new_nccresult(), "plain")
    assert np.array_equal(np.isnan(r32), np.isnan(r64))
    both = ~np.isnan(r32)
    assert both.sum() > 1000
    assert np.abs(r32[both] - r64[both]).max() < 2e-6
