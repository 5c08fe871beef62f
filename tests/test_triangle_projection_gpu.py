"""The projection kernel of the triangle multiplication at the edges of its tiles (128 positions x 128 channels, 32 x 32 per
warp): rows that TMA stores and rows that it does not take, less than a tile, ragged last tiles, several tiles per SM."""
import pytest

from kutacc_b200 import workloads as W
from oracle import cpu_oracle as O
from tests import helpers
from tests.test_triangle_multiplication_gpu import _calc_proj, _case, _f32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,c_o,c_i", [(3, 64, 128), (4, 64, 128), (12, 128, 128), (33, 192, 128), (201, 128, 128), (204, 64, 256)])
def test_projection_matches_oracle(kutacc_lib, n, c_o, c_i):
    A = _case(700 + n, n, c_o, c_i)
    proj, gate = _calc_proj(A, n, c_o, c_i)
    want_p, want_g = O.tm_calc_proj_bf16(W.bf16_bits(A["x"]), W.bf16_bits(A["mask"]), W.bf16_bits(A["pw"]), A["pb"],
                                         W.bf16_bits(A["gw"]), A["gb"])
    assert helpers.rel_err(_f32(gate), W.as_f32(want_g)) <= 2.0 ** -7
    assert helpers.rel_err(_f32(proj), W.as_f32(want_p)) <= helpers.BF16_TOL
