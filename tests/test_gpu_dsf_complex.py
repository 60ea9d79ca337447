"""DSF coefficients of vectors that are real but for one entry, wherever it is:
the search for imaginary parts ends at the first one found, and the kernels for
real vectors leave at once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('op', [0, 1])
@pytest.mark.parametrize('which,row', [(-1, 0), (-1, 5000), (-1, -1), (0, 0), (0, -1), (6, 777), (6, -1)])
def test_one_imaginary_entry(op, which, row):
    import torch
    from lsquantumed_gb300.build import build
    build()
    import lsquantumed_gb300 as ed
    N = 16
    env = ed.Environment(nspins=N)
    b0, b1 = ed.Basis(env, 0), ed.Basis(env, op)
    rng = np.random.default_rng(row % 97)
    psi = rng.standard_normal(b0.size).astype(np.complex128)
    V = rng.standard_normal((7, b1.size)).astype(np.complex128)
    (psi if which < 0 else V[which])[row] += 0.75j
    psi /= np.linalg.norm(psi)
    V /= np.linalg.norm(V, axis=1)[:, None]
    c = np.asarray(ed.Phys.dsf_coefficients(env, b0, b1, op, psi, torch.from_numpy(V)))
    s0, s1 = b0.int_basis.astype(np.int64), b1.int_basis.astype(np.int64)
    for i in range(N):
        if op == 0:
            ref = ((np.where((s0 >> i) & 1, 0.5, -0.5) * psi) * V.conj()).sum(axis=1)
        else:
            at = np.nonzero((s0 >> i) & 1 == 0)[0]
            ref = (psi[at] * V[:, np.searchsorted(s1, s0[at] | (1 << i))].conj()).sum(axis=1)
        # unit vectors: at most dim additions, each below 2^-53 of a partial sum of at most 1
        assert np.abs(c[i] - ref).max() <= 2.0 ** -52 * b0.size
