"""Correlations of real states at the ends of their range: states of tiny norm,
where the squares or their scale leave the exponents of FP64's normal range,
and pairs of vectors that are large where the other one is small.

Every sum here has at most dim additions, each rounding below 2^-53 of a partial
sum of at most sum |w|: dim 2^-53 sum |w| bounds the error of any order of FP64
additions, and the kernels with exact integer sums stay below it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def ed():
    from lsquantumed_gb300.build import build
    build()
    import lsquantumed_gb300
    return lsquantumed_gb300


def _basis(ed, N):
    env = ed.Environment(nspins=N)
    b = ed.Basis(env, 0)
    s = b.int_basis.astype(np.int64)
    return env, b, s, [(s >> i) & 1 for i in range(N)]


def _flip(s, bit, x, y, i, j):
    """sum over the antiparallel states of x_s y_flipped / 2 (i != j)."""
    at = np.nonzero(bit[i] != bit[j])[0]
    return 0.5 * (x[at] * y[np.searchsorted(s, s[at] ^ ((1 << i) | (1 << j)))]).sum()


@pytest.mark.parametrize('N', [8, 14])
@pytest.mark.parametrize('down', [0, 430, 452, 480])
def test_tiny_norm(ed, N, down):
    """psi 2^-down: expectation values scale by 2^(-2 down), the gradient of the
    energy, a ratio, not at all."""
    env, b, s, bit = _basis(ed, N)
    x = np.random.default_rng(N).standard_normal(b.size)
    psi = x * 2.0 ** -down
    X = x.astype(np.longdouble)
    w = X * X
    W = float(w.sum())
    tol = b.size * 2.0 ** -53 * W
    pairs = [(i, j) for i in range(N) for j in range(i + 1, N)]
    zz = np.array([float(np.where(bit[i] == bit[j], w, -w).sum()) / 4 for i, j in pairs])
    F = np.array([float(_flip(s, bit, X, X, i, j)) for i, j in pairs])
    up = 2.0 ** (2 * down)  # exact
    assert np.abs(ed.SzSz(env, b).ExpectValPairs(pairs, psi) * up - zz).max() <= tol
    assert np.abs(ed.SiSj(env, b).ExpectValPairs(pairs, psi) * up - zz - F).max() <= 2 * tol
    assert abs(ed.SpSm(env, b).ExpectValPairs([(1, 1)], psi)[0] * up - float(w[bit[1] == 1].sum())) <= tol
    dJ, dD, dh = ed.Adjoint.energy_gradient(b, pairs, psi)
    assert np.abs(dD - zz / W).max() <= 2 * tol / W
    assert np.abs(dJ - F / W).max() <= 2 * tol / W
    assert np.abs(dh - [float(np.where(t, w, -w).sum()) / 2 / W for t in bit]).max() <= 2 * tol / W
    A = ed.Adjoint
    lam = np.random.default_rng(N + 1).standard_normal(b.size)
    L = lam.astype(np.longdouble)
    terms = [(A.ZZ, i, j) for i, j in pairs] + [(A.Z, i, i) for i in range(N)]
    got = A.expect_mixed(b, terms, lam * 2.0 ** -down, psi) * up
    m = L * X
    ref = [float(np.where(bit[i] == bit[j], m, -m).sum()) / 4 for i, j in pairs]
    ref += [float(np.where(t, m, -m).sum()) / 2 for t in bit]
    assert np.abs(got - ref).max() <= b.size * 2.0 ** -53 * float(np.abs(m).sum())


@pytest.mark.parametrize('N', [8, 14])
@pytest.mark.parametrize('deep', [30, 110, 150, 400])
def test_vectors_on_different_states(ed, N, deep):
    """lam and psi each 2^-deep where the other is large: their products, and so
    every mixed S^z term, are 2^-deep of the product of the norms."""
    env, b, s, bit = _basis(ed, N)
    g = np.random.default_rng(deep)
    half = g.integers(0, 2, b.size).astype(bool)
    lam = g.standard_normal(b.size) * np.where(half, 1.0, 2.0 ** -deep)
    psi = g.standard_normal(b.size) * np.where(half, 2.0 ** -deep, 1.0)
    m = lam.astype(np.longdouble) * psi
    A = ed.Adjoint
    pairs = [(i, j) for i in range(N) for j in range(i + 1, N)]
    terms = [(A.ZZ, i, j) for i, j in pairs] + [(A.Z, i, i) for i in range(N)]
    got = A.expect_mixed(b, terms, lam, psi)
    ref = [float(np.where(bit[i] == bit[j], m, -m).sum()) / 4 for i, j in pairs]
    ref += [float(np.where(t, m, -m).sum()) / 2 for t in bit]
    assert np.abs(got - ref).max() <= b.size * 2.0 ** -53 * float(np.abs(m).sum())
