"""Flip sums <S+_i S-_j> of sharply peaked real states, far below the state's
largest amplitude: lists above 16 pairs (the Gram kernel) are as accurate as
lists of up to 16 (the direct FP64 kernel).

A direct sum over at most 924 rows adds fewer than 64 rounded partial sums in a
row: 64 2^-53 sum |psi_r psi_r'|.  The Gram kernel rounds the entries to 2^-63 of
the power of two above the largest and takes over at |F| >= 2^-9 of that power
and the norm: its error is below 2^-53 |F| sqrt(rows) < 31 2^-53 |F|, and one
rounding of F."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _peaked(states, N, per_flip):
    """Amplitude per_flip for every spin pair exchanged against the Neel state."""
    neel = sum(1 << i for i in range(0, N, 2))
    away = np.array([bin(int(s) ^ neel).count('1') // 2 for s in states])
    rng = np.random.default_rng(N)
    psi = per_flip ** away * (1.0 + 0.5 * rng.random(len(states)))
    return psi / np.linalg.norm(psi)


@pytest.mark.parametrize('N,mag', [(8, 0), (12, 0), (12, 1)])
@pytest.mark.parametrize('per_flip', [0.3, 1e-2, 1e-4, 1e-6])
def test_small_flip_sums(N, mag, per_flip):
    from lsquantumed_gb300.build import build
    build()
    import lsquantumed_gb300 as ed
    env = ed.Environment(nspins=N)
    b = ed.Basis(env, mag)
    states = b.int_basis.astype(np.int64)
    psi = _peaked(states, N, per_flip)
    x = psi.astype(np.longdouble)
    pairs = [(i, j) for i in range(N) for j in range(N) if i != j]
    ref, size = [], []
    for i, j in pairs:
        at = np.nonzero(((states >> i) & 1 == 1) & ((states >> j) & 1 == 0))[0]
        p = x[at] * x[np.searchsorted(states, states[at] ^ ((1 << i) | (1 << j)))]
        ref.append(p.sum())
        size.append(np.abs(p).sum())
    ref, size = np.array(ref), np.array(size)
    op = ed.SpSm(env, b)
    many = list(range(len(pairs))) * 5  # more than one launch of passes for the small ones
    for at in (many[:16], many[:17], many[:len(pairs)], many):
        got = op.ExpectValPairs([pairs[k] for k in at], psi).real
        assert (np.abs(got - ref[at]) <= 64 * 2.0 ** -53 * size[at]).all(), \
            (len(at), float((np.abs(got - ref[at]) / size[at]).max() * 2.0 ** 53))
    dJ = ed.Adjoint.energy_gradient(b, pairs, psi)[0]
    assert (np.abs(dJ - ref) <= 67 * 2.0 ** -53 * size).all()  # divided by the norm as well
