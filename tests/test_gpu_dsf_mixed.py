"""DSF coefficients and term expectations at the edges of their kernels: real
and complex vectors, both operators, vector counts around the groups of four
that share a read of the state, sectors with few states, more terms than one
group of eight, against sums in plain numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def ed():
    from lsquantumed_gb300.build import build
    build()
    import lsquantumed_gb300
    return lsquantumed_gb300


def _vec(rng, n, cplx):
    v = rng.standard_normal(n) + (1j * rng.standard_normal(n) if cplx else 0.0)
    return (v / np.linalg.norm(v)).astype(np.complex128)


@pytest.mark.parametrize('N,mag,nev,psi_c,vec_c', [
    (2, 0, 1, False, False), (4, -2, 3, False, False), (6, 1, 4, True, True), (12, 0, 5, False, True),
    (14, -3, 4, True, False), (16, 0, 9, False, False), (18, 2, 1, False, False),
])
def test_dsf_coefficients_runs(ed, N, mag, nev, psi_c, vec_c):
    import torch
    env = ed.Environment(nspins=N)
    b0 = ed.Basis(env, mag)
    rng = np.random.default_rng(N + nev)
    psi = _vec(rng, b0.size, psi_c)
    states = b0.int_basis.astype(np.int64)
    for op in (0, 1):
        if op == 1 and mag == N // 2:
            continue
        b1 = b0 if op == 0 else ed.Basis(env, mag + 1)
        V = np.stack([_vec(rng, b1.size, vec_c and n != 0) for n in range(nev)])
        c = ed.Phys.dsf_coefficients(env, b0, b1, op, psi, torch.from_numpy(V))
        target = b1.int_basis.astype(np.int64)
        for i in range(N):
            if op == 0:
                ref = ((np.where((states >> i) & 1, 0.5, -0.5) * psi) * V.conj()).sum(axis=1)
            else:
                at = np.nonzero(((states >> i) & 1) == 0)[0]
                to = np.searchsorted(target, states[at] | (1 << i))
                ref = (psi[at] * V[:, to].conj()).sum(axis=1)
            # unit vectors: each of at most dim additions rounds below 2^-53 of a partial sum of at most 1
            assert np.abs(c[i] - ref).max() <= 2.0 ** -52 * b0.size + 2.0 ** -51, (op, i)


def test_dsf_nonfinite(ed):
    """A NaN entry reaches every coefficient it enters, as in FP64."""
    import torch
    env = ed.Environment(nspins=8)
    b = ed.Basis(env, 0)
    psi = np.ones(b.size, dtype=np.complex128)
    psi[3] = np.nan
    V = torch.ones((2, b.size), dtype=torch.complex128)
    assert np.isnan(ed.Phys.dsf_coefficients(env, b, b, 0, psi, V).real).all()


@pytest.mark.parametrize('cplx', [False, True])
@pytest.mark.parametrize('N,nterms', [(2, 3), (4, 1), (12, 8), (12, 9), (16, 300), (18, 40)])
def test_expect_mixed_groups(ed, N, nterms, cplx):
    env = ed.Environment(nspins=N)
    b = ed.Basis(env, 0)
    rng = np.random.default_rng(nterms)
    lam, psi = _vec(rng, b.size, cplx), _vec(rng, b.size, cplx)
    states = b.int_basis.astype(np.int64)
    terms = [(int(k), int(i), int(j)) for k, i, j in
             zip(rng.integers(0, 4, nterms), rng.integers(0, N, nterms), rng.integers(0, N, nterms))]
    got = ed.Adjoint.expect_mixed(b, terms, lam, psi)
    for t, (kind, i, j) in enumerate(terms):
        bi, bj = (states >> i) & 1, (states >> j) & 1
        flip = np.zeros(b.size, dtype=np.complex128)
        if i == j:
            flip = psi
        else:
            at = np.nonzero(bi != bj)[0]
            flip[at] = psi[np.searchsorted(states, states[at] ^ ((1 << i) | (1 << j)))]
        zz = np.where(bi != bj, -0.25, 0.25) * psi
        o = {ed.Adjoint.XY: 0.5 * flip, ed.Adjoint.ZZ: zz, ed.Adjoint.Z: np.where(bi, 0.5, -0.5) * psi,
             ed.Adjoint.SISJ: zz + 0.5 * flip}[kind]
        assert abs(got[t] - np.vdot(lam, o)) <= 2.0 ** -52 * b.size, (t, terms[t])


@pytest.mark.parametrize('cplx', [False, True])
def test_dsf_infinite_entry(ed, cplx):
    """An infinite amplitude in row r gives sign(bit i of r) * conj(v_r) * inf
    at every site i, not NaN (real part; the imaginary part too where v and
    psi are complex with finite, nonzero parts)."""
    import torch
    N, r = 12, 7
    env = ed.Environment(nspins=N)
    b = ed.Basis(env, 0)
    g = np.random.default_rng(3)
    psi = g.standard_normal(b.size) + (1j * g.standard_normal(b.size) if cplx else 0j)
    V = g.standard_normal((2, b.size)) + (1j * g.standard_normal((2, b.size)) if cplx else 0j)
    psi[r] = complex(np.inf, psi[r].imag)
    c = ed.Phys.dsf_coefficients(env, b, b, 0, torch.tensor(psi, device='cuda'), torch.tensor(V, device='cuda'))
    s = int(b.int_basis[r])
    for i in range(N):
        sg = 1.0 if (s >> i) & 1 else -1.0
        for n in range(2):
            assert c[i, n].real == sg * np.sign(V[n, r].real) * np.inf
            if cplx:
                assert c[i, n].imag == -sg * np.sign(V[n, r].imag) * np.inf
