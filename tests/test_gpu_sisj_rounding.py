"""S_i.S_j of a real state is its two exact parts rounded once: the S^z sum of the
FP64 squares and the flip sum of entries rounded to 2^-63 of the largest one's
binade (below 2^-62 max|psi| sum|psi|), also where the parts cancel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('N,seed', [(10, 0), (12, 1), (14, 2), (16, 3)])
def test_sisj_rounded_once(N, seed):
    from lsquantumed_gb300.build import build
    build()
    import lsquantumed_gb300 as ed
    env = ed.Environment(nspins=N)
    b = ed.Basis(env, 0)
    s = b.int_basis.astype(np.int64)
    rng = np.random.default_rng(seed)
    neel = sum(1 << i for i in range(0, N, 2))
    away = np.array([bin(int(v) ^ neel).count('1') // 2 for v in s])
    psi = (-0.6) ** away * (1.0 + 0.2 * rng.random(b.size))  # S^z part and flips of either sign
    psi /= np.linalg.norm(psi)
    got = ed.SiSj(env, b).AllPairs(psi)
    x, w = psi.astype(np.longdouble), (psi * psi).astype(np.longdouble)
    slack = 2.0 ** -61 * np.abs(psi).max() * np.abs(psi).sum()
    for i in range(N):
        for j in range(i):
            bi, bj = (s >> i) & 1, (s >> j) & 1
            at = np.nonzero((bi == 1) & (bj == 0))[0]
            F = (x[at] * x[np.searchsorted(s, s[at] ^ ((1 << i) | (1 << j)))]).sum()
            ref = np.where(bi == bj, w, -w).sum() / 4 + F
            assert abs(got[i, j].real - ref) <= 2.0 ** -53 * abs(ref) * 1.01 + slack, (i, j)
