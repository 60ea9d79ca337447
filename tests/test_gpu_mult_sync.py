"""ed_bv_mult_real returns when its outputs are complete (the header's
"Synchronises the stream"), whatever the arithmetic: on a context with its own
non-blocking stream, a copy on another stream right after the call sees them."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('arith', [0, 1, 2, 3, 4])
@pytest.mark.parametrize('l', [1, 9])
def test_outputs_complete_on_return(arith, l):
    import torch
    from lsquantumed_gb300.build import build
    build()
    from lsquantumed_gb300 import capi
    ctx = ctypes.c_void_p()
    capi.call('ed_ctx_create', 0, None, ctypes.byref(ctx))
    m, n = 16, 8_000_000
    V = [torch.full((n,), float(i + 1), dtype=torch.float64, device='cuda') for i in range(m)]
    Y = np.zeros((m, l))
    Y[np.arange(l), np.arange(l)] = 0.5
    out = [torch.zeros(n, dtype=torch.float64, device='cuda') for _ in range(l)]
    torch.cuda.synchronize()
    vp = (ctypes.c_void_p * m)(*[v.data_ptr() for v in V])
    op = (ctypes.c_void_p * l)(*[o.data_ptr() for o in out])
    for scale in (1.0, 2.0, 4.0):  # each call overwrites the one before
        Yc = np.ascontiguousarray(Y * scale)
        capi.call('ed_bv_mult_real', ctx, vp, m, ctypes.c_void_p(Yc.ctypes.data), l, l, op, n, arith)
        got = torch.stack([o[-4:].clone() for o in out]).cpu().numpy()  # torch's stream, no wait for the context's
        want = np.repeat(0.5 * scale * np.arange(1, l + 1)[:, None], 4, axis=1)
        assert np.array_equal(got, want), (scale, got)
    torch.cuda.synchronize()
    capi.call('ed_ctx_destroy', ctx)
