"""The H.v variant that is reported is the one that runs: fewer rows than 256 per
SM take the form of 64 threads per block unless another is forced.  A forced
static variant keeps its own block shape (the blocks leave one partial sum each,
so a fused x.y differs in its last bits between the two shapes, H.v in none)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('N', [8, 16, 20])
def test_reported_variant(N):
    import torch
    from lsquantumed_gb300.build import build
    build()
    import lsquantumed_gb300 as ed
    env = ed.Environment(nspins=N)
    b = ed.Basis(env, 0)
    small = b.size < 256 * torch.cuda.get_device_properties(0).multi_processor_count
    h = ed.Hamiltonian(env, b, ed.chain1D(env), 1.0, 1.0, 0.3, 0.3)
    h.build_diag(env)
    h.build_off_diag(env)
    x = torch.randn(b.size, dtype=torch.float64, device='cuda')
    y, xy, yy = h.apply_real_dot(x)
    assert h.hv_variant(True) == ('u8-t64' if small else 'u4-b6')
    for v in ('u4-b6', 'u4-b4', 'u8-b4', 'u8-b1', 'u8-t64', 'jit', 'auto'):
        h.set_hv_variant(v)
        z, xz, zz = h.apply_real_dot(x)
        assert torch.equal(h.apply_real(x), y) and torch.equal(z, y)
        assert h.hv_variant(True) == (v if v != 'auto' else 'u8-t64' if small else 'u4-b6')
        # any order of at most dim additions
        assert abs(xz - xy) <= 2 * b.size * 2.0 ** -53 * float((x * y).abs().sum())
        assert abs(zz - yy) <= 2 * b.size * 2.0 ** -53 * yy
