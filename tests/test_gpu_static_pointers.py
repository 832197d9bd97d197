"""sr_gravity_solve_static on buffers a caller cuts out of its own: any of the four may begin on any float. The values are
those of a call on 16-byte boundaries, bit for bit, and nothing beside the outputs is written."""
import ctypes as C

import numpy as np
import pytest

from sandbox_reactions_b200.abi import Config
from sandbox_reactions_b200.engine import load_library

pytestmark = pytest.mark.gpu


def solve(cfg, sigma, at):
    """The outputs with the density and the three outputs `at` floats past a 16-byte boundary."""
    import torch

    lib, c, n = load_library(), cfg.to_c(), sigma.size
    bufs = [torch.full((n + 8,), -7.0, device="cuda") for _ in range(4)]
    bufs[0][at[0]:at[0] + n] = torch.from_numpy(sigma.ravel()).cuda()
    stream = torch.cuda.current_stream()
    st = lib.sr_gravity_solve_static(C.byref(c), *(b.data_ptr() + 4 * o for b, o in zip(bufs, at)),
                                     C.c_void_p(stream.cuda_stream))
    assert st == 0, lib.sr_last_error(None).decode()
    torch.cuda.synchronize()
    outs = [b.cpu().numpy() for b in bufs[1:]]
    for o, k in zip(outs, at[1:]):
        assert (o[:k] == -7.0).all() and (o[k + n:] == -7.0).all()
    return [o[k:k + n] for o, k in zip(outs, at[1:])]


@pytest.mark.parametrize("w,h", [(16, 16), (136, 104), (256, 256)])
@pytest.mark.parametrize("at", [(1, 0, 0, 0), (0, 1, 0, 0), (0, 0, 2, 0), (0, 0, 0, 3), (3, 1, 2, 3)])
def test_buffers_on_any_float(w, h, at):
    cfg = Config(width=w, height=h, gravity=True, hydro=False)
    sigma = np.random.default_rng(w + h).random((h, w), np.float32) + np.float32(0.05)
    for got, want in zip(solve(cfg, sigma, at), solve(cfg, sigma, (0, 0, 0, 0))):
        assert np.isfinite(want).all() and np.array_equal(got, want)


def test_a_steady_call_can_be_captured():
    """A call that uploads nothing (the last call's sizes and kernel), captured and replayed on another density."""
    import torch

    lib, rng = load_library(), np.random.default_rng(5)
    cfg = Config(width=136, height=104, gravity=True, hydro=False)
    first, second = (rng.random((104, 136), np.float32) + np.float32(0.05) for _ in range(2))
    want = solve(cfg, second, (0, 0, 0, 0))
    c = cfg.to_c()
    sigma = torch.from_numpy(first).cuda()
    outs = [torch.zeros((104, 136), device="cuda") for _ in range(3)]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        st = lib.sr_gravity_solve_static(C.byref(c), sigma.data_ptr(), *(o.data_ptr() for o in outs),
                                         C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == 0, lib.sr_last_error(None).decode()
    sigma.copy_(torch.from_numpy(second))
    graph.replay()
    torch.cuda.synchronize()
    for o, w in zip(outs, want):
        assert np.array_equal(o.cpu().numpy().ravel(), w)
