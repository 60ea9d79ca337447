"""Rounding of the Gram-Schmidt dots on long vectors: no more than that of FP64
multiply-add chains over the rows of four blocks of 256 threads per SM, joined
in a tree.  The root mean square errors of both over 256 dots of random vectors
each have a spread of 1 / sqrt(512) = 4.4%, their ratio 6.3%: two of those are
allowed.  (Chains twice as long have 1.3 times the error.)"""
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


def _tree(h, l=None):
    """Pairwise sum along the last axis; as pairs where l is given."""
    import torch
    while h.shape[-1] > 1:
        if h.shape[-1] % 2:
            h = torch.nn.functional.pad(h, (0, 1))
            l = torch.nn.functional.pad(l, (0, 1)) if l is not None else None
        s, e = _two_sum(h[..., 0::2], h[..., 1::2])
        if l is not None:
            l = l[..., 0::2] + l[..., 1::2] + e
        h = s
    return h[..., 0], (l[..., 0] if l is not None else None)


def test_dots_rounding():
    import torch
    from lsquantumed_gb300.build import build
    build()
    import lsquantumed_gb300 as ed
    env = ed.Environment(nspins=2)
    threads = torch.cuda.get_device_properties(0).multi_processor_count * 4 * 256
    m, steps = 16, 64
    n = threads * steps
    g = torch.Generator(device='cuda').manual_seed(7)
    got, chains = [], []
    for _ in range(16):
        w = torch.randn(n, dtype=torch.float64, device='cuda', generator=g) / n ** 0.5
        V = [torch.randn(n, dtype=torch.float64, device='cuda', generator=g) / n ** 0.5 for _ in range(m)]
        h = ed.bv_dot_real(env, V, w)
        for v, x in zip(V, h):
            p, e = _two_prod(v, w)
            hi, lo = _tree(p, e)
            s = torch.zeros(threads, dtype=torch.float64, device='cuda')
            for a, b in zip(p.view(steps, threads), e.view(steps, threads)):
                t, c = _two_sum(s, a)
                s = t + (c + b)  # a multiply-add: one rounding of s + (a + b)
            got.append(float((torch.tensor(float(x), dtype=torch.float64, device='cuda') - hi) - lo))
            chains.append(float((_tree(s)[0] - hi) - lo))
    r = np.sqrt(np.mean(np.square(got)) / np.mean(np.square(chains)))
    assert r <= 1.0 + 2 * 0.063, r
