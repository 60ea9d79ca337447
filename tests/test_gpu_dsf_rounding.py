"""Rounding of the S^z_q coefficients of long vectors of mostly one sign (as
ground states have), whose signed sums cancel: no more than that of FP64
multiply-add chains of signed products, one per thread of two blocks of 256 per
SM, joined in a tree.  Root mean square and largest error over all sites and
vectors; both are random, so a tenth more is allowed.  Also the vector counts
around one and two groups of five, and entries that are not finite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def ed():
    from lsquantumed_gb300.build import build
    build()
    import lsquantumed_gb300
    return lsquantumed_gb300


def _two_sum(a, b):
    s = a + b
    z = s - a
    return s, (a - (s - z)) + (b - z)


def _two_prod(a, b):
    def split(x):
        c = 134217729.0 * x
        h = c - (c - x)
        return h, x - h
    p = a * b
    ah, al = split(a)
    bh, bl = split(b)
    return p, ((ah * bh - p) + ah * bl + al * bh) + al * bl


def _tree(h, l):
    import torch
    while h.shape[-1] > 1:
        if h.shape[-1] % 2:
            h, l = torch.nn.functional.pad(h, (0, 1)), torch.nn.functional.pad(l, (0, 1))
        s, e = _two_sum(h[..., 0::2], h[..., 1::2])
        l = l[..., 0::2] + l[..., 1::2] + e
        h = s
    return h[..., 0], l[..., 0]


def _state(g, n, cplx, even=False):
    import torch
    a = torch.randn(n, dtype=torch.float64, device='cuda', generator=g)
    if even:
        a = 1.0 + 0.3 * a
    else:  # a few decades
        a = (1.0 + a) * torch.exp(1.5 * torch.randn(n, dtype=torch.float64, device='cuda', generator=g))
    a /= a.norm()
    ph = torch.rand(n, dtype=torch.float64, device='cuda', generator=g) * 1.5
    return torch.polar(a.abs(), ph) if cplx else torch.complex(a, torch.zeros_like(a))


@pytest.mark.parametrize('even', [False, True])
@pytest.mark.parametrize('N,cplx', [(18, False), (20, False), (20, True), (22, False)])
def test_sqz_rounding(ed, N, cplx, even):
    import torch
    env = ed.Environment(nspins=N)
    b = ed.Basis(env, 0)
    s = torch.from_numpy(b.int_basis.astype(np.int64)).cuda()
    threads = torch.cuda.get_device_properties(0).multi_processor_count * 2 * 256
    pad = -b.size % threads
    got, chains = [], []
    for seed in range(4):
        g = torch.Generator(device='cuda').manual_seed(100 * N + seed)
        psi = _state(g, b.size, cplx, even)
        V = torch.stack([_state(g, b.size, cplx, even) for _ in range(10)])
        c = np.asarray(ed.Phys.dsf_coefficients(env, b, b, 0, psi, V))
        for n in range(len(V)):
            terms = [(psi.real, V[n].real)] + ([(psi.imag, V[n].imag)] if cplx else [])
            prods = [_two_prod(x.contiguous(), y.contiguous()) for x, y in terms]
            e0, e1, top = [], [], 0.0
            for i in range(N):
                sg = torch.where((s >> i) & 1 == 1, 0.5, -0.5).to(torch.float64)
                acc = torch.zeros(threads, dtype=torch.float64, device='cuda')
                rows = [[torch.nn.functional.pad(sg * t, (0, pad)).view(-1, threads) for t in p] for p in prods]
                for k in range(rows[0][0].shape[0]):
                    for p, q in rows:
                        t, w = _two_sum(acc, p[k])
                        acc = t + (w + q[k])  # a multiply-add
                h, l = _tree(torch.cat([sg * p for p, _ in prods]), torch.cat([sg * q for _, q in prods]))
                a = acc.view(-1, 8, 32)  # blocks, warps, lanes: halves onto halves
                while a.shape[2] > 1:
                    a = a[:, :, :a.shape[2] // 2] + a[:, :, a.shape[2] // 2:]
                a = a[:, :, 0]
                while a.shape[1] > 1:
                    a = a[:, :a.shape[1] // 2] + a[:, a.shape[1] // 2:]
                a = a[:, 0]
                while a.numel() > 1:
                    a = torch.nn.functional.pad(a, (0, a.numel() % 2))
                    a = a[:a.numel() // 2] + a[a.numel() // 2:]
                e0.append(float((torch.tensor(c[i][n].real, dtype=torch.float64, device='cuda') - h) - l))
                e1.append(float((a[0] - h) - l))
                top = max(top, abs(float(h)))
            got += [e / top for e in e0]
            chains += [e / top for e in e1]
    got, chains = np.abs(got), np.abs(chains)
    assert np.sqrt((got ** 2).mean()) <= 1.1 * np.sqrt((chains ** 2).mean())
    assert got.max() <= 1.1 * chains.max()


@pytest.mark.parametrize('op', [0, 1])
@pytest.mark.parametrize('nev', [5, 6, 10, 11])
@pytest.mark.parametrize('cplx', [False, True])
def test_vector_groups(ed, op, nev, cplx):
    """Every vector of a call as it comes out alone."""
    import torch
    env = ed.Environment(nspins=14)
    b0, b1 = ed.Basis(env, 0), ed.Basis(env, op)
    g = torch.Generator(device='cuda').manual_seed(nev)
    psi = _state(g, b0.size, cplx)
    V = torch.stack([_state(g, b1.size, cplx) for _ in range(nev)])
    c = np.asarray(ed.Phys.dsf_coefficients(env, b0, b1, op, psi, V))
    for n in range(nev):
        assert np.array_equal(c[:, n], np.asarray(ed.Phys.dsf_coefficients(env, b0, b1, op, psi, V[n:n + 1]))[:, 0])


@pytest.mark.parametrize('bad', [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize('where', ['psi', 'vec'])
def test_sqp_nonfinite(ed, bad, where):
    """S^+_q with an entry that is not finite, as the sums in FP64 give it."""
    import torch
    env = ed.Environment(nspins=8)
    b0, b1 = ed.Basis(env, 0), ed.Basis(env, 1)
    psi = np.ones(b0.size, dtype=np.complex128)
    V = np.ones((3, b1.size), dtype=np.complex128)
    if where == 'psi':
        psi[5] = bad
    else:
        V[1, 7] = bad
    c = np.asarray(ed.Phys.dsf_coefficients(env, b0, b1, 1, psi, torch.from_numpy(V)))
    s0, s1 = b0.int_basis.astype(np.int64), b1.int_basis.astype(np.int64)
    for i in range(8):
        at = np.nonzero((s0 >> i) & 1 == 0)[0]
        to = np.searchsorted(s1, s0[at] | (1 << i))
        with np.errstate(invalid='ignore'):
            ref = (psi[at].real * V[:, to].real).sum(axis=1)
        ok = np.isfinite(ref)
        assert np.array_equal(np.isfinite(c[i].real), ok) and np.abs(c[i].real[ok] - ref[ok]).max(initial=0.0) <= 1e-13
