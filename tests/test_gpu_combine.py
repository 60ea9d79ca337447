"""The default restart combination (exact 10-bit digits on the tensor cores)
at its edges: column counts around 16 and 32, output counts around the groups
of 8 and 16, row counts around a tile of 16, columns that are not 16-byte
aligned, rows of very different scale, entries at the digit boundaries,
coefficients all alike (the largest level sums), and non-finite rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def ed():
    from lsquantumed_gb300.build import build
    build()
    import lsquantumed_gb300
    return lsquantumed_gb300


def _columns(V, shift):
    import torch
    out = []
    for v in V:
        t = torch.empty(len(v) + 1, dtype=torch.float64, device='cuda')[shift:shift + len(v)]
        t.copy_(torch.from_numpy(v))
        out.append(t)
    return out


def _check(ed, V, Y, shift=0):
    """Against extended precision: every entry within one rounding of the
    result and 2^-53 of (largest entry of the row) x (largest coefficient)."""
    import torch
    env = ed.Environment(nspins=2)
    n, l = V.shape[1], Y.shape[1]
    out = _columns(np.zeros((l, n)), shift)
    ed.bv_mult_real(env, _columns(V, shift), Y, out=out)
    got = np.stack([o.cpu().numpy() for o in out])
    # exact products of two 53-bit numbers need 106 bits: split the coefficients
    yh = Y.astype(np.float32).astype(np.longdouble)
    yl = (Y - Y.astype(np.float32)).astype(np.longdouble)
    Vl = V.astype(np.longdouble)
    ref = yh.T @ Vl + yl.T @ Vl
    bound = 2.0 ** -53 * np.abs(ref) + 2.0 ** -53 * np.abs(V).max(axis=0)[None, :] * np.abs(Y).max(axis=0)[:, None]
    assert (np.abs(got - ref) <= bound).all(), float((np.abs(got - ref) / np.maximum(bound, 1e-300)).max())


@pytest.mark.parametrize('m,l,n,shift', [
    (1, 1, 1, 0), (2, 1, 15, 0), (5, 4, 16, 1), (15, 8, 17, 0), (16, 9, 4099, 0), (16, 16, 1000, 1), (17, 16, 31, 0),
    (24, 17, 2048, 0), (31, 30, 4097, 1), (32, 31, 100003, 0), (33, 8, 1000, 0),
])
def test_combine_sizes(ed, m, l, n, shift):
    rng = np.random.default_rng(m * 100 + l)
    V = rng.standard_normal((m, n)) / np.sqrt(n)
    Y = np.linalg.qr(rng.standard_normal((m, m)))[0][:, :l]
    _check(ed, V, np.ascontiguousarray(Y), shift)


def test_combine_scales(ed):
    """Rows from 2^-900 to 2^900, rows with entries 60 binades apart, zero
    rows, and coefficients of different scale per column."""
    rng = np.random.default_rng(5)
    m, n = 16, 4000
    V = rng.standard_normal((m, n)) * np.exp2(rng.integers(-900, 900, n))[None, :].astype(np.float64)
    V[:, ::3] *= np.exp2(-rng.integers(0, 60, (m, len(V[0, ::3]))).astype(np.float64))
    V[:, 5] = 0.0
    Y = rng.standard_normal((m, 8)) * np.exp2(np.arange(8) * 9.0 - 36.0)[None, :]
    _check(ed, V, Y)


@pytest.mark.parametrize('m', [16, 32])
def test_combine_alike(ed, m):
    """All entries of a row and of a coefficient column equal, at values whose
    digits are the largest: every product of a level adds up."""
    top = [1.0 - 2.0 ** -53, 0.5 + 511 * 2.0 ** -18 + 511 * 2.0 ** -28, 1.0, 255.5 / 256, 0.75]
    V = np.repeat(np.array(top)[None, :], m, axis=0)
    Y = np.repeat(np.array(top)[None, :], m, axis=0)
    _check(ed, V, Y)
    _check(ed, -V, Y)


def test_combine_nonfinite_rows(ed):
    """A row with an infinity or a NaN gives what FP64 gives; its neighbours
    are not touched."""
    import torch
    env = ed.Environment(nspins=2)
    rng = np.random.default_rng(1)
    V = rng.standard_normal((6, 64))
    V[2, 10], V[3, 33], V[4, 34] = np.inf, np.nan, -np.inf
    Y = np.abs(rng.standard_normal((6, 9)))
    got = np.stack([o.cpu().numpy() for o in ed.bv_mult_real(env, _columns(V, 0), Y)])
    with np.errstate(invalid='ignore'):
        ref = Y.T @ V
    assert np.array_equal(np.isnan(got), np.isnan(ref)) and np.array_equal(np.isposinf(got), np.isposinf(ref))
    ok = np.isfinite(ref)
    assert np.abs(got[ok] - ref[ok]).max() <= 1e-14


def test_combine_nonfinite_coefficients(ed):
    """An infinite coefficient gives what FP64 gives in its output only."""
    env = ed.Environment(nspins=2)
    rng = np.random.default_rng(2)
    V = np.abs(rng.standard_normal((4, 40))) + 0.1
    Y = rng.standard_normal((4, 9))
    Y[1, 3] = np.inf
    got = np.stack([o.cpu().numpy() for o in ed.bv_mult_real(env, _columns(V, 0), Y)])
    assert np.isposinf(got[3]).all()
    rest = np.delete(np.arange(9), 3)
    assert np.abs(got[rest] - (Y.T @ V)[rest]).max() <= 1e-14
