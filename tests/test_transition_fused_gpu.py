"""The one-kernel transition MLP at the edges of its row tiles (128 or 256 rows per CTA) and hidden chunks (128)."""
import numpy as np
import pytest

from kutacc_b200 import api
from kutacc_b200.workloads import as_f32
from oracle import cpu_oracle as O
from . import helpers
from .test_transition_gpu import _case, _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,c_o,c_i", [(1, 128, 512), (127, 128, 128), (129, 128, 256), (38000, 128, 512), (37889, 128, 128),
                                          (1, 256, 1024), (128, 256, 128), (200, 256, 384), (19100, 256, 256)])
def test_matches_oracle(kutacc_lib, rows, c_o, c_i):
    arrays = _case(1, rows, c_o, c_i, 7 * rows + c_o)
    api.set_profile(True)
    api.profile_read()
    got = _run(1, rows, c_o, c_i, arrays)
    names = [n for n, _ in api.profile_read()]
    api.set_profile(False)
    assert names == ["transition"]
    assert np.isfinite(got).all()
    assert helpers.rel_err(got, as_f32(O.transition_bf16(*arrays))) <= helpers.BF16_TOL
