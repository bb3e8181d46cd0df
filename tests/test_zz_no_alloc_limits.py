"""The allocation-free field sum at its per-receiver limit (2,048 paths): a
receiver over it gets a zero field, whatever the output buffer held, in a call
that reports the error and in a replayed CUDA graph, which cannot."""
import ctypes as C

import numpy as np
import pytest

from sbrsolver_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_long", [2048, 2049])
@pytest.mark.parametrize("captured", [False, True])
def test_receivers_at_the_path_limit(built, n_long, captured):
    torch = pytest.importorskip("torch")
    lib = _lib.load()
    n_rx, n = 3, n_long + 2
    recv = torch.full((n,), 1, dtype=torch.int32, device="cuda")
    recv[:2] = torch.tensor([0, 2], dtype=torch.int32)
    rank = torch.arange(n, dtype=torch.int64, device="cuda")
    pf = torch.ones(6 * n, dtype=torch.float64, device="cuda")  # sums are whole numbers: exact
    out = torch.full((6 * n_rx,), float("nan"), dtype=torch.float64, device="cuda")

    def call():
        return lib.sbr_receiver_field_sum_noalloc(
            C.c_void_p(recv.data_ptr()), C.c_void_p(rank.data_ptr()), C.c_void_p(pf.data_ptr()),
            n, n_rx, 0, C.c_void_p(out.data_ptr()),
            C.c_void_p(torch.cuda.current_stream().cuda_stream))

    torch.cuda.synchronize()
    st = call()
    over = n_long > 2048
    assert st == (_lib.ERR_INVALID_ARG if over else 0)
    if captured:
        g = torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(g):
            st = call()
        _lib.check(st)
        out.fill_(float("nan"))
        g.replay()
    torch.cuda.synchronize()
    want = np.repeat([1.0, 0.0 if over else float(n_long), 1.0], 6)
    np.testing.assert_array_equal(out.cpu().numpy(), want)
