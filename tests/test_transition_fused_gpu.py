"""The one-kernel transition MLP at the edges of its row tiles (128 or 256 rows per CTA) and hidden chunks (128)."""
import numpy as np
import pytest
import torch

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


# few rows and many hidden channels: two products through the workspace, unless their aligned loads do not fit the biases
@pytest.mark.parametrize("rows,c_o,c_i,unaligned", [(129, 256, 1024, False), (2048, 256, 1024, False), (1, 128, 2048, False),
                                                    (130, 256, 2048, False), (130, 256, 2048, True)])
def test_few_rows(kutacc_lib, rows, c_o, c_i, unaligned):
    arrays = _case(1, rows, c_o, c_i, 7 * rows + c_o)
    api.set_profile(True)
    api.profile_read()
    if unaligned:
        x, w1, b1, w2, b2 = [torch.from_numpy(a.view(np.int16)).view(torch.bfloat16).cuda() if a.dtype == np.uint16 else torch.from_numpy(a).cuda()
                             for a in arrays]
        b1, b2 = (torch.cat([torch.zeros(1, device="cuda"), b])[1:] for b in (b1, b2))
        out = torch.zeros_like(x)
        api.transition(1, rows, c_o, c_i, *(api.tensor(t) for t in (x.view(1, rows, c_o), w1, b1, w2, b2, out.view(1, rows, c_o))))
        torch.cuda.synchronize()
        got = out.float().cpu().numpy()
    else:
        got = _run(1, rows, c_o, c_i, arrays)
    names = [n for n, _ in api.profile_read()]
    api.set_profile(False)
    assert names == (["transition"] if unaligned else ["linear_bias_relu", "linear_bias"])
    assert helpers.rel_err(got, as_f32(O.transition_bf16(*arrays))) <= helpers.BF16_TOL


# one kernel and two products
@pytest.mark.parametrize("rows,c_o,c_i", [(200, 128, 512), (200, 256, 2048), (19100, 256, 256)])
def test_relu_of_nan_is_zero(kutacc_lib, rows, c_o, c_i):
    x, w1, b1, w2, b2 = _case(1, rows, c_o, c_i, 3)
    clean = _run(1, rows, c_o, c_i, (x, w1, b1, w2, b2))
    x = x.copy()
    x[7, 3] = 0x7FC0
    got = _run(1, rows, c_o, c_i, (x, w1, b1, w2, b2))
    assert (got[7] == torch.from_numpy(b2).bfloat16().float().numpy()).all()
    assert (np.delete(got, 7, 0) == np.delete(clean, 7, 0)).all()


def test_few_rows_under_capture_without_a_workspace(kutacc_lib):
    rows, c_o, c_i = 2048, 256, 1024
    arrays = _case(1, rows, c_o, c_i, 5)
    x, w1, b1, w2, b2 = [(torch.from_numpy(a.view(np.int16)).view(torch.bfloat16) if a.dtype == np.uint16 else torch.from_numpy(a)).cuda() for a in arrays]
    out = torch.zeros_like(x)
    ts = [api.tensor(t) for t in (x.view(1, rows, c_o), w1, b1, w2, b2, out.view(1, rows, c_o))]
    torch.cuda.synchronize()
    api.lib().kutacc_b200_release_workspace()
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    api.set_async(True)
    try:
        with torch.cuda.graph(graph, stream=stream):
            api.set_stream(stream.cuda_stream)
            api.transition(1, rows, c_o, c_i, *ts)
    finally:
        api.set_stream(0)
        api.set_async(False)
    graph.replay()
    torch.cuda.synchronize()
    assert helpers.rel_err(out.float().cpu().numpy(), as_f32(O.transition_bf16(*arrays))) <= helpers.BF16_TOL
