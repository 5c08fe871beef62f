"""The projection that keeps its rows in shared memory (64, 128 and 256 channels), with and without the LayerNorm in front,
at the edges of its row groups (32), row tiles (128) and blocks (256), from less than one tile to several blocks per SM."""
import numpy as np
import pytest
import torch

from kutacc_b200 import api, runner
from kutacc_b200 import workloads as W
from . import helpers
from .test_layernorm_fused_gpu import EPS, _ln_case, _oracle

pytestmark = pytest.mark.gpu

CASES = [(1, 1, 4, 32), (2, 32, 8, 32), (3, 33, 4, 16), (2, 128, 4, 32), (3, 129, 8, 8), (1, 257, 8, 32),
         (1300, 33, 2, 32), (1300, 33, 4, 32), (1300, 33, 8, 32), (320, 128, 8, 32)]


@pytest.mark.parametrize("ln", [False, True])
@pytest.mark.parametrize("B,S,H,D", CASES)
def test_projection_matches_faithful_oracle(kutacc_lib, B, S, H, D, ln):
    w, raw, gamma, beta = _ln_case(2000 + S + H, B, S, H, D, 1.0)
    case = runner.DeviceCase(w)
    api.set_profile(True)
    api.profile_read()
    if ln:
        x = runner._to_torch(raw, "bf16", "cuda:0")
        g, b = torch.from_numpy(gamma).cuda(), torch.from_numpy(beta).cuda()
        api.gating_attention_ln(api.tensor(x, sizes=[B * S, w.C], strides=[w.C, 1]), case.inputs, case.t_bias, case.t_nb,
                                case.weights, g.data_ptr(), b.data_ptr(), EPS, case.t_out)
        torch.cuda.synchronize()
        got = runner.out_to_f32(case.out)
    else:
        got = runner.out_to_f32(case.run())
    names = [n for n, _ in api.profile_read()]
    api.set_profile(False)
    assert [n for n in names if n != "repitch"] == ["proj_qkvg", "attn_core", "linear_bias"]
    assert np.isfinite(got).all()
    pick = sorted({0, B // 2, B - 1})                # the oracle on the first, a middle and the last batch row only
    ref = W.Workload(name="pick", kind="gating", dtype=w.dtype, B=len(pick), S=S, H=H, D=D, seed=0, has_nb=w.has_nb)
    ref.arrays = dict(w.arrays, x=w.arrays["x"][pick], mask=w.arrays["mask"][pick], bias=w.arrays["bias"][pick])
    want = _oracle(ref, raw[pick], gamma, beta) if ln else helpers.oracle_faithful(ref)
    assert helpers.rel_err(got.reshape(B, S, -1)[pick], want.reshape(len(pick), S, -1)) <= helpers.BF16_TOL
