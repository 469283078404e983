"""The fused passes of the Fourier neural operator against its general GEMMs.

Both round the same BF16 operands, multiply them in the same 16-wide steps of K in the same order and
apply the same FP32 operations to the products, so output and gradients agree bit for bit.  The sizes
reach the edges of the tiles: rows shorter and longer than 128 sites and not a multiple of it, K and
column counts that are padded, one and several slices of the plane, one sample."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(net, a, target):
    out, cache = net.forward(a)
    loss, grad = net.mse(out, target)
    grads = net.backward(cache, grad)
    return out.cpu().numpy(), loss, {k: v.cpu().numpy() for k, v in grads.items()}


@pytest.mark.parametrize("n,batch,width,modes,layers,hidden", [
    (32, 2, 8, 4, 2, 16), (64, 1, 32, 12, 1, 128), (200, 1, 32, 12, 1, 64), (136, 2, 20, 8, 2, 40),
    (128, 3, 32, 16, 2, 128), (256, 1, 32, 16, 1, 128), (24, 1, 1, 4, 1, 3)])
def test_fused_passes_match_the_general_gemms(cuda_lib, monkeypatch, n, batch, width, modes, layers, hidden):
    import torch

    from polarism_gb300.fno import FNO2d, init_params

    cfg = dict(c_in=3, c_out=3, width=width, modes=modes, layers=layers, hidden=hidden)
    rng = np.random.default_rng(n)
    params = init_params(seed=1, **cfg)
    for k in params:
        if "b" in k:
            params[k] = 0.1 * rng.standard_normal(params[k].shape)
    a = torch.tensor(rng.standard_normal((batch, 3, n, n)).astype(np.float32), device="cuda")
    target = torch.tensor(rng.standard_normal((batch, 3, n, n)).astype(np.float32), device="cuda")
    net = FNO2d(n, params=params, **cfg)
    assert net.fused
    got = _run(net, a, target)
    monkeypatch.setattr(FNO2d, "fused", property(lambda self: False))
    want = _run(FNO2d(n, params=params, **cfg), a, target)
    assert np.array_equal(got[0], want[0]) and got[1] == want[1]
    for k in want[2]:
        assert np.array_equal(got[2][k], want[2][k]), k
    import ctypes

    from polarism_gb300 import _lib

    count = ctypes.c_int32()
    _lib.check(net.lib.pg_gemm_timeouts(ctypes.byref(count), 1), "pg_gemm_timeouts")
    assert count.value == 0


@pytest.mark.parametrize("B,C,plane", [(1, 1, 1), (2, 3, 255), (1, 2, 257), (3, 2, 1000), (2, 4, 40960 + 17)])
def test_channel_sum_keeps_the_order_of_its_sum(cuda_lib, B, C, plane):
    """256 partial sums a channel (samples, then every 256th value), added by halves."""
    import torch

    from polarism_gb300 import _lib

    x = np.random.default_rng(plane).standard_normal((B, C, plane)).astype(np.float32)
    t, out = torch.tensor(x, device="cuda"), torch.empty(C, device="cuda")
    _lib.check(_lib.load().pg_fno_channel_sum(t.data_ptr(), out.data_ptr(), B, C, plane, 0, None), "channel_sum")
    part = np.zeros((C, 256), np.float32)
    for b in range(B):
        for i in range(0, plane, 256):
            row = x[b, :, i:i + 256]
            part[:, :row.shape[1]] += row
    part = part.reshape(C, 8, 32)
    for o in (16, 8, 4, 2, 1):
        part[:, :, :o] = part[:, :, :o] + part[:, :, o:2 * o]
    p = np.concatenate([part[:, :, 0], np.zeros((C, 24), np.float32)], axis=1)
    for o in (16, 8, 4, 2, 1):
        p[:, :o] = p[:, :o] + p[:, o:2 * o]
    assert np.array_equal(out.cpu().numpy(), p[:, 0])


def test_adam_takes_many_parameters_in_one_launch(cuda_lib):
    """More parameters than one launch takes, empty ones and lengths around a block's 1024 values,
    against the formula in FP64 (FP32 rounding of a few operations: 1e-6) and each one by itself."""
    import ctypes

    import torch

    from polarism_gb300 import _lib

    lib = _lib.load()
    sizes = [1, 1023, 1024, 1025, 0, 5000] + [7 + k for k in range(40)]
    rng = np.random.default_rng(0)
    host = [[rng.standard_normal(n).astype(np.float32) for _ in range(3)] +
            [rng.random(n).astype(np.float32)] for n in sizes]
    args = (1e-3, 0.9, 0.999, 1e-8, 3, 0.01)

    def run(many):
        dev = [[torch.tensor(a, device="cuda") for a in t] for t in host]
        bf = [torch.empty(max(n, 1), dtype=torch.bfloat16, device="cuda") for n in sizes]
        keep = [torch.empty(1, device="cuda")]
        ptr = lambda t: t.data_ptr() or keep[0].data_ptr()
        if many:
            cols = [(ctypes.c_void_p * len(sizes))(*(ptr(d[c]) for d in dev)) for c in (0, 1, 2, 3)]
            cols.append((ctypes.c_void_p * len(sizes))(*(b.data_ptr() for b in bf)))
            _lib.check(lib.pg_fno_adam_many(len(sizes), *cols, (ctypes.c_int64 * len(sizes))(*sizes), *args, None),
                       "pg_fno_adam_many")
        else:
            for d, b, n in zip(dev, bf, sizes):
                _lib.check(lib.pg_fno_adam(*(ptr(t) for t in d), b.data_ptr(), n, *args, None), "pg_fno_adam")
        return [[t.cpu().numpy() for t in d] for d in dev], [b[:n].float().cpu().numpy() for b, n in zip(bf, sizes)]

    got, got_bf = run(True)
    one, one_bf = run(False)
    for k, (w, g, m1, m2) in enumerate(host):
        assert all(np.array_equal(x, y) for x, y in zip(got[k], one[k])) and np.array_equal(got_bf[k], one_bf[k])
        w, g, m1, m2 = (x.astype(np.float64) for x in (w, g, m1, m2))
        gi = g + 0.01 * w
        a, b = 0.9 * m1 + 0.1 * gi, 0.999 * m2 + 0.001 * gi * gi
        v = w - 1e-3 * (a / (1 - 0.9 ** 3)) / (np.sqrt(b / (1 - 0.999 ** 3)) + 1e-8)
        np.testing.assert_allclose(got[k][0], v, rtol=1e-6, atol=1e-6)
