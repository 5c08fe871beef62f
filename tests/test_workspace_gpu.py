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


def test_global_attention_of_other_head_shapes(kutacc_lib):
    w = W.random_global_case(seed=6, B=64, S=4096, H=4, D=16)
    case = runner.DeviceCase(w)
    assert held_after(case.run) <= 4 << 20                  # split-softmax state, no k and v (9 MB)


def test_global_attention_in_groups_of_columns(kutacc_lib):
    # 382 MB of k, v and partial sums in groups of 26 columns; a column's result is that of a call of its own
    B, S, C = 40, 262144, 64
    g = torch.Generator("cuda").manual_seed(7)
    x = torch.randn(B, S, C, generator=g, device="cuda").bfloat16()
    mask = (torch.rand(B, S, generator=g, device="cuda") > 0.2).bfloat16()
    ws = [torch.randn(n, C, generator=g, device="cuda").bfloat16() / 8 for n in (C, 8, 8, C, C)]
    bg, bo = torch.ones(C, device="cuda"), torch.zeros(C, device="cuda")
    weights = api.make_weights(C, 8, 8, *ws[:4], bg, ws[4], bo)

    def run(cols):
        xs, ms, out = x[cols].contiguous(), mask[cols].contiguous(), torch.empty(len(cols), S, C, dtype=torch.bfloat16, device="cuda")
        api.global_attention(api.make_inputs(len(cols), S), api.tensor(xs), api.tensor(ms, sizes=[len(cols), S, 1], strides=[S, 1, 1]),
                             weights, api.tensor(out))
        torch.cuda.synchronize()
        return out

    whole = []
    assert held_after(lambda: whole.append(run(list(range(B))))) <= 256 * 9 / 8 * (1 << 20) + (3 << 20)
    for c in (0, 25, 26, 39):
        assert torch.equal(whole[0][c], run([c])[0])
