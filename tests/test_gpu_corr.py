"""Correlations of a real state through the all-pairs kernels (S^z moments
from half tables, flip sums as a Gram matrix of 8-bit digits): every pair,
every operator and the energy gradient against sums in extended precision, at
the edges of the kernels: sectors with no, one or all spins up, sizes below
one stage, ragged stages, several accumulation groups, states of very uneven
amplitudes, and pair lists just below and above the switch from the direct
flip kernel to the Gram kernel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def ed():
    from lsquantumed_gb300.build import build
    build()
    import lsquantumed_gb300
    return lsquantumed_gb300


def _state(dim, kind):
    rng = np.random.default_rng(dim)
    psi = rng.standard_normal(dim)
    if kind == 'wide':
        psi *= np.exp2(-rng.integers(0, 30, dim))
    elif kind == 'flat':  # every digit at its largest magnitude, one sign
        psi = np.ones(dim)
    elif kind == 'scaled':
        psi *= 2.0 ** 70
    return psi if kind == 'scaled' else psi / np.linalg.norm(psi)


@pytest.mark.parametrize('N,mag,kind', [
    (2, 0, 'plain'), (4, -2, 'plain'), (4, 2, 'plain'), (6, -2, 'plain'), (12, 0, 'flat'), (12, 5, 'plain'),
    (14, -3, 'wide'), (16, 0, 'wide'), (18, 1, 'plain'), (20, 0, 'flat'), (20, -2, 'scaled'),
])
def test_all_pairs_real_state(ed, N, mag, kind):
    env = ed.Environment(nspins=N)
    b = ed.Basis(env, mag)
    states = b.int_basis.astype(np.int64)
    psi = _state(b.size, kind)
    x = psi.astype(np.longdouble)
    w = x * x
    W = float(w.sum())
    bit = [(states >> i) & 1 for i in range(N)]
    F = np.zeros((N, N))
    Z = np.full((N, N), W)
    for i in range(N):
        for j in range(i):
            anti = bit[i] != bit[j]
            Z[i, j] = Z[j, i] = W - 2.0 * float(w[anti].sum())
            at = np.nonzero((bit[i] == 1) & (bit[j] == 0))[0]
            to = states[at] ^ ((1 << i) | (1 << j))
            rk = np.searchsorted(states, to)
            F[i, j] = F[j, i] = float((x[at] * x[rk]).sum())
    up = np.array([float(w[bt == 1].sum()) for bt in bit])
    # entries in 55-bit fixed point against the largest, products exact:
    # below 2^-54 max|psi| sum|psi|, and one rounding of the result
    tol = 2.0 ** -53 * np.abs(psi).max() * np.abs(psi).sum() + 2.0 ** -52 * W
    eye = np.eye(N, dtype=bool)
    want = {ed.SzSz: 0.25 * Z, ed.SiSj: np.where(eye, 0.75 * W, 0.25 * Z + F),
            ed.SpSm: np.where(eye, np.diag(up), F), ed.SmSp: np.where(eye, np.diag(W - up), F)}
    for cls, ref in want.items():
        got = cls(env, b).AllPairs(psi)
        assert np.abs(got - ref).max() <= tol, (cls.__name__, np.abs(got - ref).max(), tol)
    # short lists: the direct flip kernel below the switch, the Gram kernel above
    pairs = [(i, j) for i in range(N) for j in range(N) if i != j][:17]
    for n in (1, 16, 17):
        got = ed.SiSj(env, b).ExpectValPairs(pairs[:n], psi)
        ref = [0.25 * Z[i, j] + F[i, j] for i, j in pairs[:n]]
        assert np.abs(got - ref).max() <= tol
    bonds = pairs + [(0, 0)]
    dJ, dD, dh = ed.Adjoint.energy_gradient(b, bonds, psi)
    assert np.abs(dJ - [(0.5 * W if i == j else F[i, j]) / W for i, j in bonds]).max() <= tol / W
    assert np.abs(dD - [0.25 * Z[i, j] / W for i, j in bonds]).max() <= tol / W
    assert np.abs(dh - (up - 0.5 * W) / W).max() <= tol / W
