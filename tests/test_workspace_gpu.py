"""Device memory that the operators take for themselves: what a call's path does not use is not reserved (the pool only grows)."""
import numpy as np
import pytest
import torch

from kutacc_b200 import api, runner
from kutacc_b200 import workloads as W

pytestmark = pytest.mark.gpu


def held_after(call):
    torch.cuda.synchronize()
    api.lib().kutacc_b200_release_workspace()
    call()
    torch.cuda.synchronize()
    return api.lib().kutacc_b200_workspace_bytes()


def test_attention_with_layernorm_in_the_projection(kutacc_lib):
    w = W.random_gating_case(seed=5, B=64, S=512, H=4, D=32)
    case = runner.DeviceCase(w)
    g, b = torch.ones(w.C, device="cuda"), torch.zeros(w.C, device="cuda")
    x_bytes = case.x.numel() * 2
    held = held_after(lambda: api.gating_attention_ln(case.t_x, case.inputs, case.t_bias, case.t_nb, case.weights, g.data_ptr(),
                                                      b.data_ptr(), 1e-5, case.t_out))
    assert held <= 5 * x_bytes * 9 / 8 + (3 << 20)          # q, k, v, gate, average; the pool adds an eighth and rounds up to 2 MB


def test_pair_bias_with_layernorm(kutacc_lib):
    z, wb = torch.randn(64, 64, 128, device="cuda").bfloat16(), torch.randn(4, 128, device="cuda").bfloat16()
    nb = torch.zeros(4, 64, 64, dtype=torch.bfloat16, device="cuda")
    g, b = torch.ones(128, device="cuda"), torch.zeros(128, device="cuda")
    tz, tw, tn = api.tensor(z), api.tensor(wb), api.tensor(nb)
    assert held_after(lambda: api.pair_bias_ln(tz, g.data_ptr(), b.data_ptr(), 1e-5, tw, tn)) == 0


@pytest.mark.parametrize("incoming", [False, True])
def test_triangle_product_of_aligned_operands(kutacc_lib, incoming):
    left, right = (torch.randn(8, 64, 64, device="cuda").bfloat16() for _ in range(2))
    center = torch.zeros(8, 64, 64, dtype=torch.bfloat16, device="cuda")
    tc, tl, tr = api.tensor(center), api.tensor(left), api.tensor(right)
    assert held_after(lambda: api.tm_equation(tc, tl, tr, 64, incoming)) == 0
