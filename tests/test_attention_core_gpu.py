"""The tensor-memory attention core and its projection at the edges of their tiles: 128 queries, 64 keys, one to four
batch rows per work item, head sizes 8, 16 and 32, layers of 64 channels."""
import numpy as np
import pytest

from kutacc_b200 import api, runner
from kutacc_b200 import workloads as W
from . import helpers

pytestmark = pytest.mark.gpu

CASES = [(1, 1, 4, 32), (2, 63, 4, 32), (5, 65, 4, 32), (3, 129, 8, 32), (7, 200, 4, 32), (150, 130, 4, 32),
         (2, 64, 4, 16), (5, 129, 4, 16), (3, 100, 8, 16), (150, 70, 4, 16),
         (1, 8, 8, 8), (5, 65, 8, 8), (3, 200, 16, 8), (150, 129, 8, 8), (3, 70, 2, 32), (2, 66, 1, 64)]


@pytest.mark.parametrize("with_nb", [True, False])
@pytest.mark.parametrize("B,S,H,D", CASES)
def test_core_matches_faithful_oracle(kutacc_lib, B, S, H, D, with_nb):
    w = W.random_gating_case(seed=1000 + 7 * S + D, B=B, S=S, H=H, D=D, with_nb=with_nb, full_mask_rows=1 if B > 1 else 0)
    api.set_profile(True)
    api.profile_read()
    got = runner.out_to_f32(runner.DeviceCase(w).run())
    names = [n for n, _ in api.profile_read()]
    api.set_profile(False)
    assert [n for n in names if n != "repitch"] == ["proj_qkvg", "attn_core", "linear_bias"]
    assert np.isfinite(got).all()
    rows = slice(0, min(B, 6)) if B > 6 else slice(0, B)
    ref = w
    if B > 6:                                   # the oracle on the first and last rows only
        pick = [0, 1, 2, B - 3, B - 2, B - 1]
        ref = W.Workload(name="pick", kind="gating", dtype=w.dtype, B=len(pick), S=S, H=H, D=D, seed=0, has_nb=w.has_nb)
        ref.arrays = dict(w.arrays, x=w.arrays["x"][pick], mask=w.arrays["mask"][pick], bias=w.arrays["bias"][pick])
        got, rows = got[pick], slice(0, len(pick))
    assert helpers.rel_err(got[rows], helpers.oracle_faithful(ref)[rows]) <= helpers.BF16_TOL
