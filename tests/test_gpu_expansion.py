"""Expansion steps of the real Krylov-Schur solve over the column counts of the
update (one instance per count up to 16, the general form above): the Ritz
pair against the oracle's explicit-matrix product.

A pair the solver accepts at tolerance t has ||H x - theta x|| <= t |theta|;
twice that leaves the rounding of the products (1e-13 |theta|) ample room.  For
a unit x some eigenvalue lies within that residual of theta, so theta is also
compared with the dense spectrum's lowest value.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 1e-10


@pytest.fixture(scope='module')
def ed():
    from lsquantumed_gb300.build import build
    build()
    import lsquantumed_gb300 as ed
    return ed


# the last two: 319770 and 170544 rows, plain and dependent launches
@pytest.mark.parametrize('lx,ly,mag,ncv', [
    (lx, ly, mag, ncv) for lx, ly, mag in [(2, 4, 0), (4, 3, 0), (4, 3, 2), (4, 4, 0)]
    for ncv in [6, 8, 9, 10, 15, 16, 17, 18, 24, 40]
] + [(2, 11, 3, 16), (2, 11, 3, 18), (2, 11, 4, 16), (2, 11, 4, 18)])
def test_ground_state_over_subspace_sizes(ed, lx, ly, mag, ncv):
    import oracle
    N = lx * ly
    env = ed.Environment(nspins=N)
    b = ed.Basis(env, mag)
    h = ed.Hamiltonian(env, b, ed.square2D(env, lx, ly), 1.0, 1.0, 0.5, 0.5)
    h.build_diag(env)
    h.build_off_diag(env)
    eps = ed.Solver.SolverInit(h, 1, ncv)
    ed.Solver.EPSSetTolerances(eps, TOL, 2000)
    assert ed.Solver.solve(env, eps) >= 1
    theta, vec, _ = ed.Solver.solution(eps, 0)
    ed.Solver.SolverClean(eps)
    x = vec.cpu().numpy()
    M = oracle.Model(1, N, lx, ly, mag, 1.0, 1.0, 0.5, 0.5)
    M.build(3)
    assert abs(np.linalg.norm(x) - 1.0) <= 1e-12
    res = np.linalg.norm(M.apply(x) - theta * x)
    assert res <= 2 * TOL * abs(theta), (res, theta)
    if b.size <= 1000:
        H = np.array([M.apply(e) for e in np.eye(b.size, dtype=np.complex128)])
        assert abs(theta - np.linalg.eigvalsh(H)[0]) <= 2 * TOL * abs(theta)
