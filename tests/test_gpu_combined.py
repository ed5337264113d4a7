"""Combined levels (INCC over two pyramid levels) in FP32 windows against the
C oracle: every level and window size, odd image widths, node counts that do
not fill a warp or a block, more slots than a node holds in shared memory,
empty image areas, and a batch of combined and plain levels."""
import copy

import pytest

from oracle import oraclepy as op
from setsm_b200 import abi
from tests import cases

pytestmark = pytest.mark.gpu

CASES = {
    "l1": dict(L=1, it=2, nodes=37, res=8.0, n_heights=40, hs=1.0),
    "l2_7": dict(L=2, it=2, nodes=41, res=9.0, n_heights=33, hs=1.0, template=11, ortho_frac=0.6),
    "l2_odd": dict(L=2, it=3, nodes=29, res=12.0, n_heights=31, hs=1.0, size=701, ortho_frac=0.5),
    "l3_11": dict(L=3, it=4, nodes=24, res=16.0, n_heights=65, hs=2.0, template=15, ortho_frac=0.5),
    "l1_slots": dict(L=1, it=2, nodes=12, res=19.0, n_heights=600, hs=0.5, sigma=5.0),
    "l2_empty": dict(L=2, it=2, nodes=40, res=9.0, n_heights=40, hs=1.0, ortho_frac=0.6,
                     zero_patch=True),
    "plain": dict(L=2, it=1, nodes=24, res=16.0, n_heights=30, hs=2.0),
}

_runs = {}


def run(name):
    if name not in _runs:
        inp = cases.make_case(**CASES[name])
        _runs[name] = cases.run_cpu(op, inp, inp.iters)
    return _runs[name]


def fresh(o):
    inp = copy.copy(o["inputs"])
    inp.gridpt3 = o["init_gp3"].copy()
    return inp, o["init_ncc"].copy()


@pytest.mark.parametrize("name", sorted(CASES))
def test_combined_level(gpu_ctx, name):
    o = run(name)
    inp, ncc = fresh(o)
    st = gpu_ctx.vertical_line_locus(inp, ncc, None, "split")
    assert st.accessable_grid == o["acc"]
    assert cases.field_mismatch(ncc, o["vll_ncc"]) == {}


def test_batch_of_combined_and_plain_levels(gpu_ctx):
    import torch
    runs = [run(n) for n in ("l2_7", "plain", "l3_11", "plain", "l1")]
    items = [cases.device_level(torch, *fresh(o)) for o in runs]
    acc, _ = gpu_ctx.batch([io for io, _ in items])
    for o, (_, held), a in zip(runs, items, acc):
        assert a == o["acc"]
        ncc = cases.from_device(held["ncc"], abi.NCCRESULT_DTYPE)
        assert cases.field_mismatch(ncc, o["vll_ncc"]) == {}
