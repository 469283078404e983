"""The bounded waits of the network's fused passes: in the give-up setting every wait for the tensor
cores gives up at once, the kernels drain and free what they hold, the count of timeouts says so,
and the next pass in the default setting gives the results of one before it."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,batch,width,modes,layers,hidden", [(32, 2, 8, 4, 2, 16), (256, 2, 32, 16, 1, 128),
                                                                (200, 1, 20, 12, 1, 40)])
def test_give_up_is_reported_and_the_next_pass_is_right(cuda_lib, n, batch, width, modes, layers, hidden):
    import torch

    from polarism_gb300 import _lib
    from polarism_gb300.fno import FNO2d

    rng = np.random.default_rng(n)
    net = FNO2d(n, c_in=3, c_out=3, width=width, modes=modes, layers=layers, hidden=hidden)
    assert net.fused
    a, d = (torch.tensor(rng.standard_normal((batch, 3, n, n)).astype(np.float32), device="cuda") for _ in range(2))

    def timeouts():
        count = ctypes.c_int32()
        _lib.check(cuda_lib.pg_gemm_timeouts(ctypes.byref(count), 1), "pg_gemm_timeouts")
        return count.value

    def run():
        out, cache = net.forward(a)
        grads = net.backward(cache, d)
        torch.cuda.synchronize()
        return [out.cpu().numpy()] + [grads[k].cpu().numpy() for k in net.names]

    want = run()
    assert timeouts() == 0
    with pytest.raises(RuntimeError, match="or 200000"):
        _lib.check(cuda_lib.pg_gemm_set_wait_limit(7), "pg_gemm_set_wait_limit")
    _lib.check(cuda_lib.pg_gemm_set_wait_limit(0), "pg_gemm_set_wait_limit")
    try:
        run()
        assert timeouts() > 0
    finally:
        _lib.check(cuda_lib.pg_gemm_set_wait_limit(200000), "pg_gemm_set_wait_limit")
    got = run()
    assert timeouts() == 0
    for g, w in zip(got, want):
        assert np.array_equal(g, w)
