"""Mode mixing and its adjoints with more channels than a block's shared memory holds values of.

Each of n sums rounds a partial sum of some 6 sqrt(n) at most by 2^-24; n such roundings as a random walk
stay below 6 n 2^-24."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,cin,cout", [(2, 30000, 2), (1, 3, 30000), (2, 20000, 1), (1, 1, 20000), (3, 15000, 3),
                                        (1, 15000, 14000)])
def test_many_channels(cuda_lib, B, cin, cout):
    import torch

    from polarism_gb300 import _lib

    m = 1
    rng = np.random.default_rng(cin + cout)
    f32 = lambda *s: torch.tensor(rng.standard_normal(s, dtype=np.float32), device="cuda")  # noqa: E731
    y, d = f32(B, cin, 2 * m, 2 * m), f32(B, cout, 2 * m, 2 * m)
    small = cin * cout < 10 ** 6
    wre, wim = ((f32(2 * m, m, cin, cout) if small else torch.randn(2 * m, m, cin, cout, device="cuda"))
                .to(torch.bfloat16) for _ in range(2))
    out, dy = torch.empty_like(d), torch.empty_like(y)
    dre, dim = (torch.empty(2 * m, m, cin, cout, device="cuda") for _ in range(2))
    st = torch.cuda.current_stream().cuda_stream
    ptr = lambda t: t.data_ptr()  # noqa: E731
    _lib.check(cuda_lib.pg_fno_mode_mix(ptr(y), ptr(wre), ptr(wim), ptr(out), B, cin, cout, m, st), "pg_fno_mode_mix")
    _lib.check(cuda_lib.pg_fno_mode_mix_backward(ptr(y), ptr(d), ptr(wre), ptr(wim), ptr(dy), ptr(dre), ptr(dim), B,
                                                 cin, cout, m, st), "pg_fno_mode_mix_backward")
    c64 = lambda t: torch.complex(t[..., :m].double(), t[..., m:].double())  # noqa: E731
    yc, dc = c64(y), c64(d)
    for k in range(2 * m):
        w = torch.complex(wre[k, 0].double(), wim[k, 0].double())
        assert float((c64(out)[:, :, k, 0] - yc[:, :, k, 0] @ w).abs().max()) < 6 * cin * 2 ** -24 + 1e-5
        assert float((c64(dy)[:, :, k, 0] - dc[:, :, k, 0] @ w.conj().T).abs().max()) < 6 * cout * 2 ** -24 + 1e-5
        dw = yc[:, :, k, 0].conj().T @ dc[:, :, k, 0]
        assert float((torch.complex(dre[k, 0].double(), dim[k, 0].double()) - dw).abs().max()) < 1e-5
