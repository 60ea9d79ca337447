"""ED_RESTART_FIXED takes the FP64 form beyond 32 columns: the default form's
results, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('m,l', [(33, 1), (40, 9), (127, 17)])
def test_fixed_beyond_32_columns(m, l):
    import torch
    from lsquantumed_gb300.build import build
    build()
    import lsquantumed_gb300 as ed
    env = ed.Environment(nspins=2)
    rng = np.random.default_rng(m)
    V = [torch.from_numpy(rng.standard_normal(5003)).cuda() for _ in range(m)]
    Y = np.ascontiguousarray(np.linalg.qr(rng.standard_normal((m, m)))[0][:, :l])
    a = ed.bv_mult_real(env, V, Y, arith='fp64')
    b = ed.bv_mult_real(env, V, Y, arith='fixed')
    assert all(torch.equal(x, y) for x, y in zip(a, b))
