"""The numpy restatements of the orthoimage passes (ortho_oracle.py) against
the reference's fixtures in tests/golden."""
import numpy as np
import pytest

from setsm_b200 import abi
from tests import cases, ortho_oracle as oo
from tests.golden import make_golden as mg


def test_ortho_blunder_fixture():
    inp, pts, tris, z = mg.tin_case("tin_l0")
    oo.ortho_blunder(inp, mg.GOLDEN_TIN["tin_l0"]["mpp"], pts, tris)
    want = z["pts"].view(abi.POINT3_DTYPE)
    assert all(np.array_equal(pts[f], want[f]) for f in ("x", "y", "z", "flag"))
    assert cases.field_mismatch(mg.clean(inp.gridpt3), z["gp3"].view(abi.UGRID_DTYPE)) == {}


@pytest.mark.parametrize("name", ["sd_l0", "sd_mt_l1"])
def test_seeddem_fixture(name):
    inp, z = mg.variant_case(name)
    oo.seeddem(inp)
    want = z["gp3"].view(abi.UGRID_DTYPE)
    for f in ("minHeight", "maxHeight", "roh"):
        assert np.array_equal(inp.gridpt3[f], want[f])
    assert np.array_equal(inp.gridpt3["ortho_ncc"][:, 1], want["ortho_ncc"][:, 1])


def test_blunder_fixture():
    inp, z = mg.variant_case("bl_l0")
    assert np.abs(oo.blunder(inp) - z["ncc"].astype(np.float64)).max() < 1e-7
