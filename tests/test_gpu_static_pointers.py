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
