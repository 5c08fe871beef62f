"""fp32 attention core on tensor memory at the edges of its tiles (128 queries, 32 keys, one or two batch rows per work item),
with pair-bias strides that are and are not multiples of 16 bytes; the fp32 pair-bias projection."""
import numpy as np
import pytest
import torch

from kutacc_b200 import api, runner
from kutacc_b200 import workloads as W
from . import helpers
from .test_attention_core_gpu import LOWEST, masked_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("with_nb", [True, False])
# up to 8 heads its result leaves as plain rows, beyond (384 and 512 channels) as tf32 heads and tails
@pytest.mark.parametrize("B,S,H", [(1, 1, 4), (2, 31, 4), (3, 33, 8), (2, 64, 4), (5, 129, 4), (81, 130, 4), (40, 257, 8),
                                   (1, 1, 12), (3, 33, 12), (5, 129, 16), (40, 257, 12)])
def test_core_matches_exact_oracle(kutacc_lib, B, S, H, with_nb):
    w = W.random_gating_case(seed=2000 + S, B=B, S=S, H=H, D=32, dtype="fp32", with_nb=with_nb, full_mask_rows=1 if B > 1 else 0)
    api.set_profile(True)
    api.profile_read()
    got = runner.out_to_f32(runner.DeviceCase(w).run())
    names = [n for n, _ in api.profile_read()]
    api.set_profile(False)
    assert "attn_f32_tc" in names and np.isfinite(got).all()
    rows = list(range(B)) if B <= 6 else [0, 1, 2, B - 3, B - 2, B - 1]
    ref = W.Workload(name="pick", kind="gating", dtype=w.dtype, B=len(rows), S=S, H=H, D=32, seed=0, has_nb=w.has_nb)
    ref.arrays = dict(w.arrays, x=w.arrays["x"][rows], mask=w.arrays["mask"][rows], bias=w.arrays["bias"][rows])
    assert helpers.rel_err(got[rows], helpers.oracle_exact(ref)) <= helpers.FP32_TOL / 4


def test_running_max_that_grows_late(kutacc_lib):
    w = W.random_gating_case(seed=31, B=4, S=200, H=4, D=32, dtype="fp32", with_nb=True, mask_frac=0.0)
    mask = np.ones((4, 200), np.float32)
    mask[0, :40] = 0.0
    mask[1, :150] = 0.0
    mask[2, 5:190] = 0.0
    w.arrays["mask"], w.arrays["bias"] = mask, (1e9 * (mask - 1.0)).astype(np.float32)
    w.arrays["nb"] = w.arrays["nb"].copy()
    w.arrays["nb"][:, :, 100:110] += 40.0
    got = runner.out_to_f32(runner.DeviceCase(w).run())
    assert helpers.rel_err(got, helpers.oracle_exact(w)) <= helpers.FP32_TOL / 4


@pytest.mark.parametrize("H,large", [(4, 2.0 ** 45), (8, 1e30), (12, 2.0 ** 60)])
def test_a_large_channel_without_weights_changes_nothing(kutacc_lib, H, large):
    # its products are zeros; the elements beside it keep all their bits
    w = W.random_gating_case(seed=83, B=3, S=70, H=H, D=32, dtype="fp32")
    for name in ("wq", "wk", "wv", "wg"):
        w.arrays[name] = w.arrays[name].copy()
        w.arrays[name][:, 5] = 0
    out = []
    for v in (0.0, large):
        w.arrays["x"] = w.arrays["x"].copy()
        w.arrays["x"][..., 5] = v
        out.append(runner.out_to_f32(runner.DeviceCase(w).run()))
    assert np.array_equal(out[0], out[1])
    assert helpers.rel_err(out[0], helpers.oracle_exact(w)) <= helpers.FP32_TOL / 4


@pytest.mark.parametrize("through_nb", [True, False])
@pytest.mark.parametrize("value", [-np.inf, LOWEST, -3e9])
def test_other_mask_values(kutacc_lib, value, through_nb):
    w = masked_case(value, through_nb, 4, 32, "fp32")
    got = runner.out_to_f32(runner.DeviceCase(w).run())
    assert helpers.rel_err(got, helpers.oracle_exact(w)) <= helpers.FP32_TOL / 4


def test_rows_far_from_zero(kutacc_lib):
    # fully masked rows stay uniform; logits are zero in the other rows, so that every x is exact: 64 keys at b, 66 at b + 6
    w = W.random_gating_case(seed=80, B=5, S=130, H=4, D=32, dtype="fp32", mask_frac=0.0)
    w.arrays["wq"] = np.zeros_like(w.arrays["wq"])
    w.arrays["bias"] = np.repeat(np.array([[LOWEST], [-2e9], [-20000.0], [-30000.0], [25000.0]], np.float32), 130, 1)
    w.arrays["nb"] = np.zeros_like(w.arrays["nb"])
    w.arrays["nb"][:, :, 64:] = 6.0
    got = runner.out_to_f32(runner.DeviceCase(w).run())
    assert helpers.rel_err(got, helpers.oracle_exact(w)) <= helpers.FP32_TOL / 4


def test_pair_bias_with_the_heads_inside_its_rows(kutacc_lib):
    # [S, H, S] storage: copied once, not a second projection of k and v for another core
    w = W.random_gating_case(seed=82, B=4, S=136, H=4, D=32, dtype="fp32")
    case = runner.DeviceCase(w)
    store = case.nb.permute(1, 0, 2).contiguous()
    nb = api.tensor(store, sizes=[4, 136, 136], strides=[136, 4 * 136, 1])
    api.set_profile(True)
    api.profile_read()
    api.gating_attention(case.t_x, case.inputs, case.t_bias, nb, case.weights, case.t_out, 128)
    names = [n for n, _ in api.profile_read()]
    api.set_profile(False)
    assert names.count("gemm_f32_rows") == 2 and "attn_f32_tc" in names
    assert helpers.rel_err(runner.out_to_f32(case.out), helpers.oracle_exact(w)) <= helpers.FP32_TOL / 4


# 128 x 128 tiles, 128 x 256 tiles (enough of them to go round), ragged rows, K of one and several slabs
@pytest.mark.parametrize("M,N,K", [(1, 128, 32), (129, 384, 64), (20000, 256, 96), (9600, 512, 32)])
def test_linear_fp32(kutacc_lib, M, N, K):
    g = torch.Generator().manual_seed(M + N + K)
    a, w, b = torch.randn(M, K, generator=g), torch.randn(N, K, generator=g) / K ** 0.5, torch.randn(N, generator=g)
    ad, wd, bd, r = a.cuda(), w.cuda(), b.cuda(), torch.zeros(M, N, device="cuda")
    api.linear(api.tensor(ad), api.tensor(wd), bd.data_ptr(), api.tensor(r))
    torch.cuda.synchronize()
    ref = a.double() @ w.double().T + b.double()
    assert (r.cpu().double() - ref).abs().max() <= 4e-6 * ref.abs().max()


# The tensor core truncates: each of the K / 8 accumulations of the large product loses half a unit, 2^-24, of a partial sum on
# average; partial sums are two thirds of the result on average, and lie anywhere in their binade (0.72).
@pytest.mark.parametrize("M,N,K", [(300, 128, 512), (9600, 512, 512), (2000, 256, 128)])
def test_linear_fp32_accumulation(kutacc_lib, M, N, K):
    g = torch.Generator().manual_seed(M + N + K)
    a, w = torch.randn(M, K, generator=g), torch.randn(N, K, generator=g) / K ** 0.5
    ad, wd, bd, r = a.cuda(), w.cuda(), torch.zeros(N, device="cuda"), torch.zeros(M, N, device="cuda")
    api.linear(api.tensor(ad), api.tensor(wd), bd.data_ptr(), api.tensor(r))
    torch.cuda.synchronize()
    ref = a.double() @ w.double().T
    assert (r.cpu().double() - ref).norm() <= K / 8 * 2.0 ** -24 * 0.72 * 2 / 3 * ref.norm()


@pytest.mark.parametrize("R,Nk,Cz,H", [(8, 100, 128, 8), (3, 33, 64, 4), (1, 1, 32, 3), (40, 301, 128, 1)])
def test_pair_bias_fp32(kutacc_lib, R, Nk, Cz, H):
    g = torch.Generator().manual_seed(R * Nk + Cz)
    z, wb = torch.randn(R, Nk, Cz, generator=g), torch.randn(H, Cz, generator=g) / Cz ** 0.5
    store = torch.full((R, H + 1, Nk), 7.0, device="cuda")
    nb = torch.zeros(H, R, Nk, device="cuda")
    zd, wd = z.cuda(), wb.cuda()
    api.pair_bias(api.tensor(zd), api.tensor(wd), api.tensor(nb))
    api.pair_bias(api.tensor(zd), api.tensor(wd), api.Tensor(store.data_ptr(), [H, R, Nk], [Nk, (H + 1) * Nk, 1], api.DTYPE_FP32, keep=store))
    torch.cuda.synchronize()
    ref = torch.einsum("rkc,hc->hrk", z.double(), wb.double())
    assert (nb.cpu().double() - ref).abs().max() <= 1e-5 * ref.abs().max()
    assert torch.equal(store[:, :H].permute(1, 0, 2), nb) and bool((store[:, H] == 7.0).all())
