"""The default restart combination keeps FP64's accuracy in every entry, however
small it is beside the row's largest entry and the column's largest
coefficient.

A chain of m FP64 multiply-adds is within (m + 1) 2^-53 sum_i |V_i Y_ic| of the
sum.  The digit form stays inside that bound: where the value or a product is at
least 2^-11 of (row scale) x (column scale) it has at most two roundings of 2^-53,
and cut digits below m 2^-64.6 of the scales, m 2^-53.6 of the products; where
neither is, it is an FP64 chain.
Coefficients that are 0 or a power of two alone in their column give exact
values, as in FP64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def ed():
    from lsquantumed_gb300.build import build
    build()
    import lsquantumed_gb300
    return lsquantumed_gb300


def _run(ed, V, Y, shift=0, **kw):
    import torch
    def cols(A):
        out = []
        for v in A:
            t = torch.empty(len(v) + 1, dtype=torch.float64, device='cuda')[shift:shift + len(v)]
            t.copy_(torch.from_numpy(v))
            out.append(t)
        return out
    out = cols(np.zeros((Y.shape[1], V.shape[1])))
    ed.bv_mult_real(ed.Environment(nspins=2), cols(V), np.ascontiguousarray(Y), out=out, **kw)
    return np.stack([o.cpu().numpy() for o in out])


def _check(ed, V, Y, shift=0, **kw):
    got = _run(ed, V, Y, shift, **kw)
    m = V.shape[0]
    yh = Y.astype(np.float32).astype(np.longdouble)
    yl = (Y - Y.astype(np.float32)).astype(np.longdouble)
    Vl = V.astype(np.longdouble)
    ref = yh.T @ Vl + yl.T @ Vl
    bound = (m + 1) * 2.0 ** -53 * (np.abs(Y).T.astype(np.longdouble) @ np.abs(Vl)) + (m + 1) * 2.0 ** -1074
    err = np.abs(got - ref)
    assert (err <= bound).all(), float((err / bound).max())


@pytest.mark.parametrize('m,l', [(2, 2), (8, 9), (16, 16), (17, 3), (32, 17), (33, 9), (64, 17), (127, 40)])
def test_selected_columns(ed, m, l):
    """Y selects columns (scaled by powers of two): the result is the column."""
    rng = np.random.default_rng(m)
    V = rng.standard_normal((m, 203)) * np.exp2(-rng.integers(0, 90, (m, 203)).astype(np.float64))
    V[rng.integers(0, m, 203), np.arange(203)] = 1.0
    at = rng.permutation(m)[:l] if l <= m else rng.integers(0, m, l)
    scale = np.exp2(rng.integers(-3, 4, l).astype(np.float64)) * rng.choice([-1.0, 1.0], l)
    Y = np.zeros((m, l))
    Y[at, np.arange(l)] = scale
    assert np.array_equal(_run(ed, V, Y), V[at] * scale[:, None])


@pytest.mark.parametrize('m,l,shift', [(2, 1, 0), (5, 4, 1), (16, 9, 0), (16, 16, 1), (31, 12, 0), (32, 8, 1), (33, 9, 0),
                                       (64, 17, 0), (127, 8, 1), (127, 33, 0)])
@pytest.mark.parametrize('spread', [0, 7, 40, 120])
def test_graded(ed, m, l, shift, spread):
    """Entries and coefficients spread over many binades, independently: the
    largest entry of a row often meets a small coefficient."""
    rng = np.random.default_rng(100 * m + spread)
    n = 331
    V = rng.standard_normal((m, n)) * np.exp2(-rng.integers(0, spread + 1, (m, n)).astype(np.float64))
    Y = rng.standard_normal((m, l)) * np.exp2(-rng.integers(0, spread + 1, (m, l)).astype(np.float64))
    Y[rng.integers(0, m, l // 2), np.arange(l // 2)] = 0.0
    _check(ed, V, Y, shift)


@pytest.mark.parametrize('m', [16, 64, 127])
def test_one_large_entry(ed, m):
    """One entry of 1 and the others 2^-7 .. 2^-6, alike in every row, with and
    without a coefficient on the large one."""
    V = np.repeat(np.linspace(2.0 ** -7, 2.0 ** -6, 50)[None, :], m, axis=0) * (1.0 - 2.0 ** -53)
    V[m // 2] = 1.0
    Y = np.repeat(np.linspace(0.3, 1.0 - 2.0 ** -53, 9)[None, :], m, axis=0)
    Y[m // 2, ::2] = 0.0
    Y[m // 2, 1::4] = 2.0 ** -30
    _check(ed, V, Y)


def test_end_of_range(ed):
    """Rows near and below the smallest normal number, and results there."""
    rng = np.random.default_rng(3)
    V = rng.standard_normal((6, 600)) * np.exp2(-rng.integers(900, 1074, 600).astype(np.float64))[None, :]
    V[:, ::7] = 0.0
    V[2, 14] = 2.0 ** -1074
    Y = rng.standard_normal((6, 9))
    _check(ed, V, Y)
    _check(ed, V * 2.0 ** 500, Y * 2.0 ** -560)
