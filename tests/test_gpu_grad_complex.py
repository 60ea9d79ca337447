"""Energy gradient of a complex state: its parts are read for a real state once
(the pass over the state that finds the imaginary parts is not repeated by the
general kernel's own entry), and the values are those of the sums."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('N', [6, 14])
def test_gradient_of_complex_state(N):
    from lsquantumed_gb300.build import build
    build()
    import lsquantumed_gb300 as ed
    env = ed.Environment(nspins=N)
    b = ed.Basis(env, 0)
    rng = np.random.default_rng(N)
    psi = rng.standard_normal(b.size) + 1j * rng.standard_normal(b.size)
    s = b.int_basis.astype(np.int64)
    w = np.abs(psi) ** 2
    W = w.sum()
    bonds = [(i, j) for i in range(N) for j in range(N)]  # N^2 bonds, equal sites among them
    before = env.kernel_count()
    dJ, dD, dh = ed.Adjoint.energy_gradient(b, bonds, psi)
    # the look at the state, the terms with their sum (256 groups of 8 per launch), the norm with its sum
    launches = 1 + 2 * ((2 * len(bonds) + N + 2047) // 2048) + 2
    assert env.kernel_count() - before <= launches
    tol = 2.0 ** -52 * b.size
    for (i, j), a, z in zip(bonds, dJ, dD):
        si, sj = np.where((s >> i) & 1, 0.5, -0.5), np.where((s >> j) & 1, 0.5, -0.5)
        if i == j:
            ref = 0.5
        else:
            at = np.nonzero(si != sj)[0]
            to = np.searchsorted(s, s[at] ^ ((1 << i) | (1 << j)))
            ref = 0.5 * (psi[at] * psi[to].conj()).sum().real / W
        assert abs(a - ref) <= tol and abs(z - (si * sj * w).sum() / W) <= tol
    assert np.abs(dh - [(np.where((s >> i) & 1, 0.5, -0.5) * w).sum() / W for i in range(N)]).max() <= tol
