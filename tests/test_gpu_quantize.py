"""Fixed-point copy of a short vector made by one cluster (up to 65536 entries)
against the two passes, which the allocation-free product still runs: a real
input gives the same exact integer sums, so the results agree bit for bit; a
complex one within the 1e-14 * ||x||_2 of the other products' tests.  Sizes
on both sides of the limit, one entry per thread and less, and vectors whose
maximum, zeros or non-finite entries decide the exponent and the flags.
"""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def ed():
    from lsquantumed_gb300.build import build
    build()
    import lsquantumed_gb300 as ed
    return ed


def _bits(t):
    import torch
    return t.contiguous().view(torch.int64)


@pytest.mark.parametrize('lx,ly,mag,dim', [
    (2, 2, 1, 4), (2, 4, 0, 70), (4, 4, 0, 12870), (4, 5, 4, 38760), (3, 6, 0, 48620), (4, 5, 3, 77520),
])
@pytest.mark.parametrize('kind', ['plain', 'zero', 'wide', 'last', 'nonfinite'])
def test_short_vector_fixed_point(ed, lx, ly, mag, dim, kind):
    import torch
    N = lx * ly
    env = ed.Environment(nspins=N)
    b = ed.Basis(env, mag)
    assert b.size == dim
    h = ed.Hamiltonian(env, b, ed.square2D(env, lx, ly), 1.0, 1.0, 0.5, 0.5)
    h.build_diag(env)
    h.build_off_diag(env)
    gen = torch.Generator(device='cuda').manual_seed(dim)

    def rand():
        return torch.rand(dim, dtype=torch.float64, device='cuda', generator=gen) * 2 - 1

    re, im = rand(), rand()
    if kind == 'zero':
        re, im = torch.zeros_like(re), torch.zeros_like(im)
    elif kind == 'wide':
        re = re * torch.exp2(-torch.arange(dim, device='cuda', dtype=torch.float64) % 60)
    elif kind == 'last':  # the largest entry, and the only imaginary one, is the last
        re[-1], im = 2.0 ** 70, torch.zeros_like(im)
        im[-1] = 2.0 ** 69
    elif kind == 'nonfinite':
        re[dim // 2] = float('inf')

    def noalloc(x):
        y = torch.empty_like(x)
        rc = ed.capi.lib().ed_ham_apply_noalloc(h.handle, ctypes.c_void_p(x.data_ptr()),
                                                ctypes.c_void_p(y.data_ptr()))
        assert rc == 0, ed.capi.last_error()
        torch.cuda.synchronize()
        return torch.view_as_real(y)

    xr = torch.complex(re, torch.zeros_like(re))
    want = noalloc(xr)
    got = torch.view_as_real(h.apply(xr))
    real = h.apply_real(re)
    if kind == 'nonfinite':
        bad = torch.isnan(want[:, 0])
        assert bad.any()
        assert torch.equal(torch.isnan(got[:, 0]), bad) and torch.equal(torch.isnan(real), bad)
        assert torch.equal(_bits(real[~bad]), _bits(want[:, 0][~bad]))
        return
    assert torch.equal(_bits(got), _bits(want))
    assert torch.equal(_bits(real), _bits(want[:, 0]))

    xc = torch.complex(re, im)
    err = (torch.view_as_real(h.apply(xc)) - noalloc(xc)).abs().max().item()
    assert err <= 1e-14 * torch.linalg.vector_norm(xc).item()
