"""The streaming global attention at the edges of its steps (16 rows), records (32), partial sums (32 or 64) and output tiles
(128), with fewer and more columns than CTAs."""
import numpy as np
import pytest

from kutacc_b200 import runner
from kutacc_b200 import workloads as W
from . import helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,S", [(1, 1), (3, 16), (2, 17), (1, 33), (5, 127), (2, 129), (2, 1024), (2, 1025), (1, 1071), (300, 65),
                                 (1, 12000)])
def test_matches_faithful_oracle(kutacc_lib, B, S):
    w = W.random_global_case(seed=900 + S, B=B, S=S, zero_mask_rows=1 if B > 2 else 0)
    got = runner.out_to_f32(runner.DeviceCase(w).run())
    assert np.isfinite(got).all()
    assert helpers.rel_err(got, helpers.oracle_faithful(w)) <= helpers.BF16_TOL


def test_rows_whose_logits_grow_late(kutacc_lib):
    # masked rows first (-1e9), then ordinary ones, then a few with large activations: the running max rises in steps
    w = W.random_global_case(seed=77, B=2, S=700)
    mask = np.ones((2, 700), np.float32)
    mask[0, :300] = 0.0
    mask[1, 40:690] = 0.0
    w.arrays["mask"] = mask
    x = w.arrays["x"].copy()
    x[:, 600:610] *= 8.0
    w.arrays["x"] = W.as_f32(W.bf16_bits(x))
    got = runner.out_to_f32(runner.DeviceCase(w).run())
    assert helpers.rel_err(got, helpers.oracle_faithful(w)) <= helpers.BF16_TOL


def test_a_column_does_not_depend_on_the_number_of_columns(kutacc_lib):
    # few columns have an SM each, many share one
    w = W.random_global_case(seed=78, B=300, S=1500)
    many = runner.out_to_f32(runner.DeviceCase(w).run())
    few = W.Workload(name="few", kind="global", dtype=w.dtype, B=3, S=w.S, H=w.H, D=w.D, seed=0, has_nb=w.has_nb)
    few.arrays = dict(w.arrays, x=w.arrays["x"][:3], mask=w.arrays["mask"][:3])
    assert np.array_equal(many[:3], runner.out_to_f32(runner.DeviceCase(few).run()))


# sixteen warps a column in one wave; eight where two waves become one, up to their longest column and their last wave; sixteen past these
@pytest.mark.parametrize("B,S", [(200, 700), (297, 31), (297, 2048), (297, 2049), (444, 33), (445, 33), (593, 40)])
def test_columns_do_not_depend_on_the_warps_they_share(kutacc_lib, B, S):
    w = W.random_global_case(seed=79 + S, B=B, S=S, zero_mask_rows=1)
    many = runner.out_to_f32(runner.DeviceCase(w).run())
    pick = [0, 1, B // 2, B - 1]
    few = W.Workload(name="few", kind="global", dtype=w.dtype, B=len(pick), S=S, H=w.H, D=w.D, seed=0, has_nb=w.has_nb)
    few.arrays = dict(w.arrays, x=w.arrays["x"][pick], mask=w.arrays["mask"][pick])
    assert np.array_equal(many[pick], runner.out_to_f32(runner.DeviceCase(few).run()))
    assert helpers.rel_err(many[pick], helpers.oracle_faithful(few)) <= helpers.BF16_TOL
