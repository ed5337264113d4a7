"""Slots without an FP32 value, listed over all nodes and evaluated in FP64
four per warp: at a window of half-size 2 every slot is one (its innermost
sub-window is a single sample).  Lists shorter than a warp's share, lists that
find no more room (the pending buffer's rest and 16 bytes a slot), levels and
window sizes mixed in one list; the records are the plain FP64 kernel's."""
import copy

import pytest

from setsm_b200 import abi
from tests import cases

pytestmark = pytest.mark.gpu


def records(ctx, inp, kernel):
    i = copy.copy(inp)
    i.gridpt3 = inp.gridpt3.copy()
    ncc = i.new_nccresult()
    ctx.vertical_line_locus(i, ncc, None, kernel)
    return ncc


@pytest.mark.parametrize("nodes, heights, pending", [
    (2, 5, None), (5, 33, None), (31, 64, None), (72, 100, None), (72, 100, "520000"),
    (72, 100, "300000")])
def test_every_slot_open(gpu_ctx, nodes, heights, pending, monkeypatch):
    if pending is not None:
        monkeypatch.setenv("SETSM_VLL_PENDING_SLOTS", pending)
    inp = cases.make_case(seed=51, size=512, nodes=nodes, res=300.0 / nodes, template=9,
                          n_heights=heights, hs=0.5)
    want = records(gpu_ctx, inp, "plain")
    assert cases.field_mismatch(records(gpu_ctx, inp, "split"), want) == {}


def test_mixed_levels(gpu_ctx):
    import torch
    kws = [dict(seed=52, template=9, nodes=9, n_heights=21),
           dict(seed=53, template=13, nodes=12, zero_patch=True),
           dict(seed=54, template=9, nodes=7, n_heights=10),
           dict(seed=55, L=2, it=2, nodes=14, res=16.0, zero_patch=True, ortho_frac=0.5),
           dict(seed=56, L=3, nodes=10, res=16.0, hs=2.0, template=13)]
    inps = [cases.make_case(**dict(dict(size=512, res=12.0, n_heights=40), **kw)) for kw in kws]
    want = [records(gpu_ctx, i, "plain") for i in inps]
    items = []
    for i in inps:
        i = copy.copy(i)
        i.gridpt3 = i.gridpt3.copy()
        items.append(cases.device_level(torch, i, i.new_nccresult()))
    gpu_ctx.batch([io for io, _ in items])
    for (_, held), w in zip(items, want):
        got = cases.from_device(held["ncc"], abi.NCCRESULT_DTYPE)
        assert cases.field_mismatch(got, w) == {}
