"""Calls of different sizes on several threads, each on its own stream: a call's shared memory does
not depend on what another thread asks for at the same time."""
from __future__ import annotations

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _together(*jobs):
    errors = []
    start = threading.Barrier(len(jobs))

    def run(job):
        try:
            start.wait()
            job()
        except Exception as e:  # noqa: BLE001 - reported by the test
            errors.append(e)

    threads = [threading.Thread(target=run, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


def _tensors(torch, rng, *shapes):
    return [torch.tensor(rng.standard_normal(s).astype(np.float32), device="cuda").to(torch.bfloat16) for s in shapes]


CALLS = 1500


def test_row_transforms_of_two_sizes(cuda_lib):
    import torch

    from polarism_gb300 import _lib

    rng = np.random.default_rng(0)

    def job(n, modes, rows):
        v, table = _tensors(torch, rng, (rows, n), (n, 2 * modes))
        out = torch.empty(rows, 2 * modes, dtype=torch.bfloat16, device="cuda")
        stream = torch.cuda.Stream()

        def run():
            for _ in range(CALLS):
                _lib.check(cuda_lib.pg_fno_dft_x(v.data_ptr(), table.data_ptr(), 0, out.data_ptr(), rows, n, modes,
                                                 stream.cuda_stream), "pg_fno_dft_x")
            stream.synchronize()
            want = v.float() @ table.float()
            assert torch.allclose(out.float(), want, rtol=2 ** -7, atol=2 ** -7 * float(want.abs().max()))

        return run

    torch.cuda.synchronize()
    _together(job(512, 16, 256), job(16, 4, 256))


def test_mode_mixing_of_two_sizes(cuda_lib):
    import torch

    from polarism_gb300 import _lib

    rng = np.random.default_rng(1)

    def job(B, channels, modes=4):
        y = torch.tensor(rng.standard_normal((B, channels, 2 * modes, 2 * modes)).astype(np.float32), device="cuda")
        wre, wim = _tensors(torch, rng, *[(2 * modes, modes, channels, channels)] * 2)
        out = torch.empty_like(y)
        stream = torch.cuda.Stream()

        def run():
            for _ in range(CALLS):
                _lib.check(cuda_lib.pg_fno_mode_mix(y.data_ptr(), wre.data_ptr(), wim.data_ptr(), out.data_ptr(), B,
                                                    channels, channels, modes, stream.cuda_stream), "pg_fno_mode_mix")
            stream.synchronize()
            yc = torch.complex(y[..., :modes].double(), y[..., modes:].double())
            want = torch.einsum("bikx,kxio->bokx", yc, torch.complex(wre.double(), wim.double()))
            got = torch.complex(out[..., :modes].double(), out[..., modes:].double())
            assert float((got - want).abs().max()) < 1e-5 * channels

        return run

    torch.cuda.synchronize()
    _together(job(8, 128), job(1, 8))
