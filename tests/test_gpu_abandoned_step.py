"""An expansion step that stops its queue leaves nothing behind in the operator:
when the solve is given up there (an error on the host), the next H.v of the
same operator still computes its product.

The stop is made with an exact eigenvector (equal amplitudes, total spin N / 2):
its invariant subspace ends the queue at step 0, and the host's part of that
step is then left out."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KR_STEP = '_Z10ed_kr_stepP6ed_hamPKPdibS1_P7KrState'  # ed_kr_step (ed_internal.h)


@pytest.mark.parametrize('per_bond', [False, True])
@pytest.mark.parametrize('N', [8, 16])
def test_hv_after_abandoned_step(N, per_bond):
    import torch
    from lsquantumed_gb300.build import build
    build()
    import lsquantumed_gb300 as ed
    from lsquantumed_gb300 import capi
    step = getattr(capi.lib(), KR_STEP)
    step.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_bool, ctypes.c_void_p, ctypes.c_void_p]
    env = ed.Environment(nspins=N)
    b = ed.Basis(env, 0)
    if per_bond:
        pairs = np.array([(i, (i + 1) % N) for i in range(N)], dtype=np.int32)
        h = ed.Hamiltonian.from_bonds(env, b, pairs, np.ones(N), np.ones(N))
    else:
        h = ed.Hamiltonian(env, b, ed.chain1D(env), 1.0, 1.0, 0.0, 0.0)
    h.build_diag(env)
    h.build_off_diag(env)
    x = torch.randn(b.size, dtype=torch.float64, device='cuda')
    want = h.apply_real(x).clone()
    cols = [torch.full((b.size,), b.size ** -0.5, dtype=torch.float64, device='cuda'), torch.zeros_like(x)]
    w = torch.zeros_like(x)
    state = torch.zeros(8192, dtype=torch.uint8, device='cuda')  # KrState, zeroed
    cp = (ctypes.c_void_p * 2)(*[c.data_ptr() for c in cols])
    assert step(h.handle, cp, 0, False, w.data_ptr(), state.data_ptr()) == 0
    torch.cuda.synchronize()
    assert float(cols[1].abs().max()) == 0.0  # the step stopped before its scaling
    y = torch.full_like(x, 7.0)
    h.apply_real(x, out=y)
    assert torch.equal(y, want)
    y2, xy, yy = h.apply_real_dot(x)
    assert torch.equal(y2, want) and abs(yy - float(want.dot(want))) <= 1e-12 * yy
