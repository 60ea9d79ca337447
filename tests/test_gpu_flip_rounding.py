"""Rounding of flip sums on long vectors (mixed expectations of two real vectors and
gradients over few bonds; lists of more than 16 pairs, also of vectors of a few
decades): no more than that of FP64 multiply-add chains over the rows of two blocks
of 256 threads per SM, joined in a tree.  Root mean square over 144 sums or more
each, whose ratio has a spread of 8%: two of those are allowed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


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


@pytest.mark.parametrize('what', ['mixed', 'gradient', 'pairs', 'pairs of a few decades'])
def test_flip_rounding(what):
    import torch
    from lsquantumed_gb300.build import build
    build()
    import lsquantumed_gb300 as ed
    N = 24
    env = ed.Environment(nspins=N)
    b = ed.Basis(env, 0)
    A = ed.Adjoint
    s = torch.from_numpy(b.int_basis.astype(np.int64)).cuda()
    threads = torch.cuda.get_device_properties(0).multi_processor_count * 2 * 256
    rng = np.random.default_rng(3)
    count = 17 if what.startswith('pairs') else 12
    bonds = [tuple(int(k) for k in rng.choice(N, 2, replace=False)) for _ in range(count)]
    rows = []
    for i, j in bonds:
        to = torch.arange(b.size, device='cuda')
        at = torch.nonzero(((s >> i) & 1) != ((s >> j) & 1))[:, 0]
        to[at] = torch.searchsorted(s, s[at] ^ ((1 << i) | (1 << j)))
        rows.append((at, to))
    pad = -b.size % threads
    got, chains = [], []
    for seed in range(12):
        g = torch.Generator(device='cuda').manual_seed(seed)
        psi = torch.randn(b.size, dtype=torch.float64, device='cuda', generator=g)
        if what.endswith('decades'):
            psi = (1.0 + psi) * torch.exp(1.5 * torch.randn(b.size, dtype=torch.float64, device='cuda', generator=g))
        psi /= psi.norm()
        lam = psi
        if what == 'mixed':
            lam = torch.randn(b.size, dtype=torch.float64, device='cuda', generator=g)
            lam /= lam.norm()
        cpsi, clam = torch.complex(psi, torch.zeros_like(psi)), torch.complex(lam, torch.zeros_like(lam))
        if what == 'mixed':
            xy = A.expect_mixed(b, [(A.XY, i, j) for i, j in bonds], clam, cpsi)
        elif what.startswith('pairs'):
            xy = ed.SpSm(env, b).ExpectValPairs(bonds, cpsi)
        else:  # a ratio: times the norm again, 2 roundings of a sum of 1e-3
            h, l = _tree(*_two_prod(psi, psi))
            xy = A.energy_gradient(b, bonds, cpsi)[0] * float(h)
        for (at, to), v in zip(rows, xy):
            on = torch.zeros_like(psi)
            on[at] = 0.5
            p, e = _two_prod(lam * on, psi[to])
            hi, lo = _tree(p, e)
            acc = torch.zeros(threads, dtype=torch.float64, device='cuda')
            for x, y in zip(*[torch.nn.functional.pad(t, (0, pad)).view(-1, threads) for t in (p, e)]):
                t, w = _two_sum(acc, x)
                acc = t + (w + y)  # a multiply-add
            acc = acc.view(-1, 8, 32)
            for dim in (2, 1):
                while acc.shape[dim] > 1:
                    k = acc.shape[dim] // 2
                    acc = acc.narrow(dim, 0, k) + acc.narrow(dim, k, k)
            acc = acc[:, 0, 0]
            while acc.numel() > 1:
                acc = torch.nn.functional.pad(acc, (0, acc.numel() % 2))
                acc = acc[:acc.numel() // 2] + acc[acc.numel() // 2:]
            got.append(float((torch.tensor(float(np.real(v)), dtype=torch.float64, device='cuda') - hi) - lo))
            chains.append(float((acc[0] - hi) - lo))
    r = np.sqrt(np.mean(np.square(got)) / np.mean(np.square(chains)))
    assert r <= 1.0 + 2 * 0.083, r
