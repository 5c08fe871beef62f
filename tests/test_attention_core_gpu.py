"""The tensor-memory attention core and its projection at the edges of their tiles: 128 queries, 64 keys, one to four
batch rows per work item, head sizes 8, 16 and 32, layers of 64 channels."""
import numpy as np
import pytest
import torch

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


LOWEST = float(np.finfo(np.float32).min)
LOWEST_BF16 = -float.fromhex("0x1.fep127")


def masked_case(value, through_nb, H, D, dtype):
    """Keys masked with `value` instead of -1e9: the first 70 (more than a tile) of batch row 0, or of all rows through the pair
    bias; all but the last; scattered ones."""
    w = W.random_gating_case(seed=77 + D, B=3, S=200, H=H, D=D, dtype=dtype, with_nb=through_nb, mask_frac=0.0)
    bias, nb = np.zeros((3, 200), np.float32), w.arrays.get("nb")
    if through_nb:
        w.arrays["nb"] = nb = nb.copy()
        nb[:, :, :70] = value
    else:
        bias[0, :70] = value
        bias[1, :199] = value
        bias[2, np.random.default_rng(1).random(200) < 0.5] = value
        bias[2, 9] = 0.0
    w.arrays["bias"] = bias
    return w


@pytest.mark.parametrize("through_nb", [True, False])
@pytest.mark.parametrize("value", [-np.inf, LOWEST_BF16, -3e9])
@pytest.mark.parametrize("H,D", [(4, 32), (4, 16), (8, 8)])
def test_other_mask_values(kutacc_lib, H, D, value, through_nb):
    w = masked_case(value, through_nb, H, D, "bf16")
    got = runner.out_to_f32(runner.DeviceCase(w).run())
    assert helpers.rel_err(got, helpers.oracle_faithful(w)) <= helpers.BF16_TOL


@pytest.mark.parametrize("H,D", [(4, 32), (4, 16), (8, 8)])
def test_fully_masked_rows_stay_uniform(kutacc_lib, H, D):
    w = W.random_gating_case(seed=78, B=3, S=200, H=H, D=D, mask_frac=0.0)
    w.arrays["bias"] = np.stack([np.full(200, v, np.float32) for v in (LOWEST_BF16, -1e9, 0.0)])
    w.arrays["nb"] = np.zeros_like(w.arrays["nb"])
    w.arrays["nb"][1] = -2.0e9                 # one head of a row that is masked twice
    w.arrays["bias"] = W.as_f32(W.bf16_bits(w.arrays["bias"]))
    w.arrays["nb"] = W.as_f32(W.bf16_bits(w.arrays["nb"]))
    got = runner.out_to_f32(runner.DeviceCase(w).run())
    assert helpers.rel_err(got, helpers.oracle_faithful(w)) <= helpers.BF16_TOL


@pytest.mark.parametrize("H,D", [(4, 32), (8, 8)])
def test_rescaling_of_rows_far_from_zero(kutacc_lib, H, D):
    # logits are zero, so that every x is exact: 64 keys at b, 66 at b + 6 (just past the threshold of the running max)
    w = W.random_gating_case(seed=79, B=6, S=130, H=H, D=D, mask_frac=0.0)
    w.arrays["wq"] = np.zeros_like(w.arrays["wq"])
    w.arrays["bias"] = W.as_f32(W.bf16_bits(np.repeat(np.array([[-0.7e7], [-0.9e7], [-1.1e7], [-1.3e7], [-1.5e7], [1.2e7]], np.float32), 130, 1)))
    w.arrays["nb"] = np.zeros_like(w.arrays["nb"])
    w.arrays["nb"][:, :, 64:] = 6.0
    got = runner.out_to_f32(runner.DeviceCase(w).run())
    assert helpers.rel_err(got, helpers.oracle_faithful(w)) <= helpers.BF16_TOL


# the last three take the sigmoid from tanh.approx, which is good to half a bf16 step down to -7
@pytest.mark.parametrize("H,D,low", [(4, 16, -10), (8, 8, -10), (2, 32, -10), (24, 16, -10), (48, 8, -10), (4, 32, -7), (8, 32, -7),
                                     (16, 32, -7)])
def test_nearly_closed_gates(kutacc_lib, H, D, low):
    # the gate is its bias, the output the gated average: each channel's error beside its own sigmoid
    w = W.random_gating_case(seed=81, B=2, S=70, H=H, D=D)
    C = H * D
    w.arrays["wg"], w.arrays["wo"] = np.zeros((C, C), np.float32), np.eye(C, dtype=np.float32)
    w.arrays["bg"], w.arrays["bo"] = np.linspace(low, low + 4, C).astype(np.float32).round(1), np.zeros(C, np.float32)
    w.arrays["bg"] = W.as_f32(W.bf16_bits(w.arrays["bg"]))
    sig = 1 / (1 + np.exp(-w.arrays["bg"].astype(np.float64)))
    got = runner.out_to_f32(runner.DeviceCase(w).run())
    assert helpers.rel_err(got / sig, helpers.oracle_exact(w) / sig) <= helpers.BF16_TOL


@pytest.mark.parametrize("H,D,dtype", [(4, 32, "bf16"), (4, 16, "bf16"), (8, 8, "bf16"), (2, 64, "bf16"), (4, 32, "fp32")])
@pytest.mark.parametrize("strides", [(0, 72, 1), (72, 0, 1), (0, 0, 1)])
def test_broadcast_pair_bias(kutacc_lib, H, D, dtype, strides):
    # one head, one query row, or one row for all
    w = W.random_gating_case(seed=90, B=3, S=72, H=H, D=D, dtype=dtype)
    case = runner.DeviceCase(w)
    store = case.nb[:, 0].contiguous() if strides[0] else case.nb[0].contiguous()      # [H, S] or [S, S]
    view = torch.as_strided(store, (H, 72, 72), strides)
    nb = api.tensor(store, sizes=[H, 72, 72], strides=list(strides))
    api.gating_attention(case.t_x, case.inputs, case.t_bias, nb, case.weights, case.t_out, 128)
    torch.cuda.synchronize()
    w.arrays["nb"] = view.float().cpu().contiguous().numpy()
    got = runner.out_to_f32(case.out)
    if dtype == "fp32":
        assert helpers.rel_err(got, helpers.oracle_exact(w)) <= helpers.FP32_TOL / 4
    else:
        assert helpers.rel_err(got, helpers.oracle_faithful(w)) <= helpers.BF16_TOL


@pytest.mark.parametrize("H,D", [(8, 8), (16, 8), (48, 8), (24, 16), (16, 32)])
def test_unaligned_gate_bias(kutacc_lib, H, D):
    w = W.random_gating_case(seed=91, B=2, S=40, H=H, D=D)
    case = runner.DeviceCase(w)
    store = torch.zeros(w.C + 4, device="cuda")
    store[1:w.C + 1] = case.bg
    weights = api.make_weights(w.C, H, D, case.wq, case.wk, case.wv, case.wg, store[1:w.C + 1], case.wo, case.bo)
    api.gating_attention(case.t_x, case.inputs, case.t_bias, case.t_nb, weights, case.t_out, 128)
    torch.cuda.synchronize()
    assert helpers.rel_err(runner.out_to_f32(case.out), helpers.oracle_faithful(w)) <= helpers.BF16_TOL


def test_more_than_2_25_work_items(kutacc_lib):
    # one key per row: the result is v times the gate, and with identity weights half of x
    B, H, D = 33000, 1024, 8
    C = H * D
    x = torch.randn(B, 1, C, device="cuda", dtype=torch.bfloat16)
    eye, zero = torch.eye(C, device="cuda", dtype=torch.bfloat16), torch.zeros(C, C, device="cuda", dtype=torch.bfloat16)
    vec, out = torch.zeros(C, device="cuda"), torch.empty_like(x)
    weights = api.make_weights(C, H, D, zero, zero, eye, zero, vec, eye, vec)
    api.gating_attention(api.tensor(x, sizes=[B, C], strides=[C, 1]), api.make_inputs(B, 1),
                         api.tensor(torch.zeros(B, 1, device="cuda", dtype=torch.bfloat16)), api.empty_tensor(), weights, api.tensor(out), 128)
    torch.cuda.synchronize()
    assert torch.equal(out, x * 0.5)
    del x, out, eye, zero
    api.lib().kutacc_b200_release_workspace()
    torch.cuda.empty_cache()


# (batch rows, positions): last query tile with one, two or three warps at work and its items at the end of the list; a last wave of
# items cut in two or in four; last key tiles of one to four pieces; a batch that does not fill its last item
@pytest.mark.parametrize("B,S,H,D,nb", [(301, 140, 4, 32, True), (75, 192, 4, 32, True), (161, 257, 4, 32, True), (298, 230, 2, 32, True),
                                        (77, 131, 8, 16, True), (150, 333, 8, 8, True), (160, 49, 4, 32, True), (297, 112, 8, 8, True),
                                        (600, 17, 2, 32, True), (299, 140, 4, 32, False), (101, 257, 4, 16, False), (85, 192, 8, 8, False), (85, 193, 8, 8, False),
                                        (193, 385, 8, 16, False), (300, 193, 8, 16, False)])
def test_rows_do_not_depend_on_the_item_list(kutacc_lib, B, S, H, D, nb):
    w = W.random_gating_case(seed=5 + S, B=B, S=S, H=H, D=D, with_nb=nb, full_mask_rows=1)
    got = runner.out_to_f32(runner.DeviceCase(w).run())
    pick = [0, 1, 2, 3, B // 2, B - 5, B - 4, B - 3, B - 2, B - 1]
    for rows in (pick[:1], pick[3:6], pick):                          # one row an item, three items, ...
        few = W.Workload(name="few", kind="gating", dtype=w.dtype, B=len(rows), S=S, H=H, D=D, seed=0, has_nb=nb)
        few.arrays = dict(w.arrays, x=w.arrays["x"][rows], mask=w.arrays["mask"][rows], bias=w.arrays["bias"][rows])
        assert np.array_equal(runner.out_to_f32(runner.DeviceCase(few).run()), got[rows])
    few.B, few.arrays = 3, {k: v[:3] if k in ("x", "mask", "bias") else v for k, v in few.arrays.items()}
    assert helpers.rel_err(got[:3], helpers.oracle_faithful(few)) <= helpers.BF16_TOL
