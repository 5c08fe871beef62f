"""kutacc_af2_linear, the fused pair-bias projection and the single-rank all-gather on the GPU."""
import numpy as np
import pytest
import torch

from kutacc_b200 import api
from kutacc_b200 import workloads as W
from oracle import cpu_oracle as O
from tests import helpers

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _bf16_cuda(a):
    return torch.from_numpy(W.bf16_bits(a).view(np.int16)).view(torch.bfloat16).to(DEV)


@pytest.mark.parametrize("M,N,K,bias,beta", [(300, 128, 128, True, 0), (513, 256, 192, False, 0), (1000, 4, 128, False, 0), (77, 8, 64, False, 0),
                                             (50, 24, 40, True, 0), (64, 64, 64, True, 1), (33, 5, 17, False, 2)])
def test_linear_bf16(kutacc_lib, M, N, K, bias, beta):
    rng = np.random.default_rng(M + N)
    a = W.as_f32(W.bf16_bits(rng.standard_normal((M, K)).astype(np.float32)))
    w = W.as_f32(W.bf16_bits(rng.standard_normal((N, K)).astype(np.float32) / np.sqrt(K)))
    b = rng.standard_normal(N).astype(np.float32) if bias else None
    prev = W.as_f32(W.bf16_bits(rng.standard_normal((M, N)).astype(np.float32)))
    ref = W.as_f32(O.linear_bf16(W.bf16_bits(a), W.bf16_bits(w), b, beta=beta, result=W.bf16_bits(prev)))
    ta, tw, tr = _bf16_cuda(a), _bf16_cuda(w), _bf16_cuda(prev)
    tb = torch.from_numpy(b).to(DEV) if bias else None
    api.linear(api.tensor(ta), api.tensor(tw), tb.data_ptr() if bias else None, api.tensor(tr), beta)
    got = tr.float().cpu().numpy()
    assert helpers.rel_err(got, ref) <= 5e-3


@pytest.mark.parametrize("M,N,K", [(1, 128, 64), (129, 256, 256), (4700, 256, 128), (4736, 256, 128), (4737, 256, 128)])
def test_linear_bf16_rows_do_not_depend_on_the_column_split(kutacc_lib, M, N, K):
    # few tiles are cut into halves of their columns: the same rows as in a call of many
    rng = np.random.default_rng(M)
    w = W.as_f32(W.bf16_bits(rng.standard_normal((N, K)).astype(np.float32) / np.sqrt(K)))
    tw, tb = _bf16_cuda(w), torch.randn(N, device=DEV)
    many = _bf16_cuda(rng.standard_normal((20000, K)).astype(np.float32))
    out = [torch.full((m + 1, N), 7.0, dtype=torch.bfloat16, device=DEV) for m in (20000, M)]
    for t in out:
        m = t.shape[0] - 1
        api.linear(api.tensor(many[:m].clone()), api.tensor(tw), tb.data_ptr(), api.tensor(t[:m]), 0)
    assert torch.equal(out[0][:M], out[1][:M]) and bool((out[1][M] == 7.0).all())
    ref = many[:M].float() @ tw.float().T + tb
    assert float((out[1][:M].float() - ref).abs().max()) <= 2.0 ** -8 * float(ref.abs().max()) * 1.01


def test_linear_fp32(kutacc_lib):
    rng = np.random.default_rng(5)
    a = rng.standard_normal((200, 96)).astype(np.float32)
    w = (rng.standard_normal((10, 96)) / 10).astype(np.float32)
    b = rng.standard_normal(10).astype(np.float32)
    ta, tw, tb = torch.from_numpy(a).to(DEV), torch.from_numpy(w).to(DEV), torch.from_numpy(b).to(DEV)
    tr = torch.zeros((200, 10), dtype=torch.float32, device=DEV)
    api.linear(api.tensor(ta), api.tensor(tw), tb.data_ptr(), api.tensor(tr), 0)
    assert helpers.rel_err(tr.cpu().numpy(), O.linear_exact(a, w, b)) <= helpers.FP32_TOL


@pytest.mark.parametrize("M,N,K,bias", [(300, 128, 96, True), (1000, 384, 256, False), (77, 256, 32, True)])
def test_linear_fp32_on_the_tensor_memory_gemm(kutacc_lib, M, N, K, bias):
    # fp32 with n % 128 == 0 and k % 32 == 0: tcgen05 on operands split into tf32 heads and tails, or for 128 and 256 columns into bf16
    # pieces; large values next to small ones in one row show a dropped tail at once
    rng = np.random.default_rng(M + N)
    a = (rng.standard_normal((M, K)) * rng.choice([1e-3, 1.0, 300.0], (M, K))).astype(np.float32)
    w = (rng.standard_normal((N, K)) / np.sqrt(K)).astype(np.float32)
    b = rng.standard_normal(N).astype(np.float32) if bias else None
    ta, tw = torch.from_numpy(a).to(DEV), torch.from_numpy(w).to(DEV)
    tb = torch.from_numpy(b).to(DEV) if bias else None
    tr = torch.full((M, N), 7.0, dtype=torch.float32, device=DEV)
    api.set_profile(True)
    api.profile_read()
    api.linear(api.tensor(ta), api.tensor(tw), tb.data_ptr() if bias else None, api.tensor(tr), 0)
    names = [k for k, _ in api.profile_read()]
    api.set_profile(False)
    assert ("gemm_f32_rows" if K == 256 else "gemm_tf32x3_tc") in names
    ref = O.linear_exact(a, w, b)
    got = tr.cpu().numpy()
    # against the magnitude of the terms of each dot product, not of the (possibly cancelling) result
    scale = (np.abs(a).astype(np.float64) @ np.abs(w).astype(np.float64).T).max()
    assert np.abs(got.astype(np.float64) - ref).max() <= 5e-6 * scale          # a dropped tail term would cost 2^-11


@pytest.mark.parametrize("R,Nk,Cz,H", [(8, 384, 128, 4), (5, 100, 128, 8), (3, 33, 64, 4), (2, 50, 40, 3)])
def test_pair_bias_matches_linear_then_permute(kutacc_lib, R, Nk, Cz, H):
    rng = np.random.default_rng(R * Nk)
    z = W.as_f32(W.bf16_bits(rng.standard_normal((R, Nk, Cz)).astype(np.float32)))
    wb = W.as_f32(W.bf16_bits(rng.standard_normal((H, Cz)).astype(np.float32) / np.sqrt(Cz)))
    lin = W.as_f32(O.linear_bf16(W.bf16_bits(z.reshape(-1, Cz)), W.bf16_bits(wb), None))      # [R*Nk, H]
    ref = lin.reshape(R, Nk, H).transpose(2, 0, 1)
    tz, tw = _bf16_cuda(z), _bf16_cuda(wb)
    nb = torch.zeros((H, R, Nk), dtype=torch.bfloat16, device=DEV)
    api.pair_bias(api.tensor(tz), api.tensor(tw), api.tensor(nb))
    got = nb.float().cpu().numpy()
    # same products, different summation order: at most one bf16 ulp apart
    assert helpers.rel_err(got, ref) <= 2.0 ** -7


def test_device_prepack_copies_rows(kutacc_lib):
    w = torch.arange(40 * 24, dtype=torch.int16, device=DEV).reshape(40, 24)
    packed = torch.zeros((40, 16), dtype=torch.int16, device=DEV)
    kutacc_lib.kutacc_af2_linear_weight_prepack(w.data_ptr(), packed.data_ptr(), 40, 16, 24, 0)
    api.raise_if_error()
    assert torch.equal(packed, w[:, :16])


def test_all_gather_single_rank_copies_with_byte_strides(kutacc_lib):
    # world_size == 1: the gather degenerates to a strided byte copy (all_gather.cpp:45-61)
    src = torch.arange(4 * 5 * 8, dtype=torch.uint8, device=DEV).reshape(4, 5, 8)
    dst = torch.zeros((4, 5, 16), dtype=torch.uint8, device=DEV)
    api.all_gather(api.tensor(src, sizes=[4, 5, 8], strides=[40, 8, 1]),
                   api.tensor(dst, sizes=[4, 5, 8], strides=[80, 16, 1]))
    assert torch.equal(dst[:, :, :8], src) and int(dst[:, :, 8:].sum()) == 0
    # host buffers, the reference's own grid for one rank
    grid = np.arange(20, dtype=np.uint8).reshape(4, 5, 1)
    out = np.zeros((4, 5, 1), dtype=np.uint8)
    api.all_gather(api.tensor(grid), api.tensor(out))
    assert np.array_equal(out, grid)


@pytest.mark.parametrize("R,Nk,Cz,H", [(8, 384, 128, 4), (5, 100, 64, 8)])
def test_pair_bias_written_with_the_heads_inside_the_rows(kutacc_lib, R, Nk, Cz, H):
    # nb [H, R, Nk] as a strided view of a [R, H, Nk] storage: the same values as the dense output, nothing else touched
    rng = np.random.default_rng(R + Nk)
    z = W.as_f32(W.bf16_bits(rng.standard_normal((R, Nk, Cz)).astype(np.float32)))
    wb = W.as_f32(W.bf16_bits((rng.standard_normal((H, Cz)) / np.sqrt(Cz)).astype(np.float32)))
    tz = torch.from_numpy(W.bf16_bits(z).view(np.int16)).view(torch.bfloat16).to(DEV)
    tw = torch.from_numpy(W.bf16_bits(wb).view(np.int16)).view(torch.bfloat16).to(DEV)
    dense = torch.zeros((H, R, Nk), dtype=torch.bfloat16, device=DEV)
    api.pair_bias(api.tensor(tz), api.tensor(tw), api.tensor(dense))
    store = torch.full((R, H + 1, Nk), 7.0, dtype=torch.bfloat16, device=DEV)       # one spare "head" of padding per row
    view = api.Tensor(store.data_ptr(), [H, R, Nk], [Nk, (H + 1) * Nk, 1], api.DTYPE_BF16, keep=store)
    api.pair_bias(api.tensor(tz), api.tensor(tw), view)
    torch.cuda.synchronize()
    assert torch.equal(store[:, :H, :].permute(1, 0, 2), dense)
    assert (store[:, H, :] == 7.0).all()


# rows around the 128-row block, calls of more blocks than SMs (whole blocks, then parts of blocks), one to three column tiles, the last
# size with tiles of half the width and the first without
@pytest.mark.parametrize("M,N,K", [(1, 128, 128), (127, 128, 256), (129, 384, 128), (300, 256, 256), (1152, 256, 256), (1153, 256, 128),
                                   (19200, 384, 128), (19201, 128, 256)])
def test_linear_fp32_rows_of_any_magnitude(kutacc_lib, M, N, K):
    # powers of two up to 2^60 between rows, channels and columns (the latter against their weights), a row of zeros
    rng = np.random.default_rng(M + N + K)
    col = np.exp2(rng.integers(-12, 13, K)).astype(np.float32)
    a = (rng.standard_normal((M, K)) * np.exp2(rng.integers(-60, 61, (M, 1)))).astype(np.float32) * col
    w = (rng.standard_normal((N, K)) * np.exp2(rng.integers(-20, 21, (N, 1)))).astype(np.float32) / col
    a[M // 2] = 0
    ta, tw = torch.from_numpy(a).to(DEV), torch.from_numpy(w).to(DEV)
    tr = torch.full((M, N), 7.0, dtype=torch.float32, device=DEV)
    api.linear(api.tensor(ta), api.tensor(tw), None, api.tensor(tr), 0)
    torch.cuda.synchronize()
    ref, terms = ta.double() @ tw.double().T, ta.double().abs() @ tw.double().abs().T
    # operands to 2^-23 each, the product of the tails dropped (2^-24): 3 * 2^-23; up to 2 K / 16 accumulations that truncate at 2^-23
    assert ((tr.double() - ref).abs() <= (3 + K / 8) * 2.0 ** -23 * terms).all()


# Elements of a row far apart: column factors up to 2^spread that the other operand takes back, so that every column counts the same; or
# one column 2^spread above the others whose partners are zero, so that only the small ones count
@pytest.mark.parametrize("spread", [30, 52, 56])
@pytest.mark.parametrize("M,N,K,way", [(300, 256, 256, "columns"), (3456, 256, 128, "columns"), (3457, 256, 256, "columns"), (300, 128, 128, "activation"), (19201, 256, 256, "activation"),
                                       (129, 128, 256, "weight"), (20000, 256, 128, "weight"), (300, 128, 512, "columns"),
                                       # runs of three of a block's eight column tiles: some begin in one block and end in the next
                                       (24001, 1024, 256, "columns"), (24001, 1024, 128, "weight")])
def test_linear_fp32_elements_of_any_magnitude_in_a_row(kutacc_lib, M, N, K, way, spread):
    g = torch.Generator().manual_seed(M + N + K + spread)
    a, w = torch.randn(M, K, generator=g).to(DEV), (torch.randn(N, K, generator=g) / K ** 0.5).to(DEV)
    if way == "columns":
        col = torch.exp2(torch.randint(-spread, spread + 1, (K,), generator=g).float()).to(DEV)
        a, w = a * col, w / col
    else:
        big, other = (a, w) if way == "activation" else (w, a)
        at = torch.randint(0, K, (8,), generator=g).to(DEV)
        big[:, at[0]] *= 2.0 ** spread
        big[:, at[1]] *= 2.0 ** (2 * spread)
        other[:, at] = 0
    tr = torch.full((M, N), 7.0, dtype=torch.float32, device=DEV)
    api.linear(api.tensor(a), api.tensor(w), None, api.tensor(tr), 0)
    torch.cuda.synchronize()
    ref, terms = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    # as above: three pieces of 8 bits hold an element whole, products below 2^-22 of the first one are dropped (tf32 pairs: 2^-22 too);
    # every accumulation of 16 (8) columns truncates at 2^-23
    assert ((tr.double() - ref).abs() <= (3 + K / 8) * 2.0 ** -23 * terms).all()


# M of one block and of blocks whose column tiles go to several CTAs
@pytest.mark.parametrize("M,K", [(100, 128), (1280, 256), (6000, 128), (30000, 256)])
def test_linear_fp32_over_its_own_input(kutacc_lib, M, K):
    g = torch.Generator().manual_seed(M + K)
    a, w, b = torch.randn(M, K, generator=g).to(DEV), (torch.randn(K, K, generator=g) / K ** 0.5).to(DEV), torch.randn(K, generator=g).to(DEV)
    ref = a.double() @ w.double().T + b
    store = torch.cat([a, torch.full((200, K), 7.0, device=DEV)])
    api.set_profile(True)
    api.profile_read()
    api.linear(api.tensor(store[:M]), api.tensor(w), b.data_ptr(), api.tensor(store[:M]), 0)
    names = [k for k, _ in api.profile_read()]
    api.set_profile(False)
    assert "split_weights" not in names and names.count("split_tf32") == 2          # through a copy of the activations
    assert helpers.rel_err(store[:M].cpu().numpy(), ref.cpu().numpy()) <= 4e-6 and bool((store[M:] == 7.0).all())
    # and a result that begins in the middle of them
    store = torch.cat([a, torch.zeros(200, K, device=DEV)])
    api.linear(api.tensor(store[:M]), api.tensor(w), b.data_ptr(), api.tensor(store[77:M + 77]), 0)
    assert helpers.rel_err(store[77:M + 77].cpu().numpy(), ref.cpu().numpy()) <= 4e-6 and torch.equal(store[:77], a[:77])


@pytest.mark.parametrize("M", [1, 129, 4000, 9472, 20000])
def test_linear_bf16_over_its_own_input(kutacc_lib, M):
    # 128 channels: a CTA has read the rows that it writes, whether few row tiles are to be had or many
    rng = np.random.default_rng(M)
    a, w = _bf16_cuda(rng.standard_normal((M, 128)).astype(np.float32)), _bf16_cuda(rng.standard_normal((128, 128)).astype(np.float32) / 11)
    b, out = torch.randn(128, device=DEV), torch.zeros(M, 128, dtype=torch.bfloat16, device=DEV)
    api.linear(api.tensor(a), api.tensor(w), b.data_ptr(), api.tensor(out), 0)
    for _ in range(5):
        x = a.clone()
        api.linear(api.tensor(x), api.tensor(w), b.data_ptr(), api.tensor(x), 0)
        assert torch.equal(x, out)


# more columns than a CTA writes, a result that begins in the middle of the activations, the kernels for other sizes, the old result added
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("M,K,off,beta", [(5000, 256, 0, 0), (5000, 128, 77, 0), (3000, 192, 0, 0), (700, 20, 3, 0), (700, 128, 0, 1), (900, 4, 0, 0)])
def test_linear_over_its_own_input(kutacc_lib, M, K, off, beta, dtype):
    g = torch.Generator().manual_seed(M + K + off)
    a, w, b = (torch.randn(M, K, generator=g)).to(DEV, dtype), (torch.randn(K, K, generator=g) / K ** 0.5).to(DEV, dtype), torch.randn(K, generator=g).to(DEV)
    store = torch.cat([a, torch.zeros(off + 1, K, device=DEV, dtype=dtype)])
    want = (a.double() @ w.double().T + b + beta * store[off:M + off].double()).cpu().numpy()
    api.linear(api.tensor(store[:M]), api.tensor(w), b.data_ptr(), api.tensor(store[off:M + off]), beta)
    assert helpers.rel_err(store[off:M + off].double().cpu().numpy(), want) <= (2.0 ** -7 if dtype == torch.bfloat16 else 4e-6)
    assert torch.equal(store[:off], a[:off])
