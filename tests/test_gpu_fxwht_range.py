"""The fixed-point register FWHT on columns whose rounding errors or sizes do
not average out: one large element on a small background, data of one sign,
against exact sums in extended precision."""

import numpy as np
import pytest

torch = pytest.importorskip('torch')
pytestmark = pytest.mark.gpu


def _fwht(x):
    y = np.array(x, dtype=np.longdouble)
    n = y.shape[0]
    h = 1
    while h < n:
        v = y.reshape(n // (2 * h), 2, h, -1)
        y = np.stack((v[:, 0] + v[:, 1], v[:, 0] - v[:, 1]), 1)
        y = y.reshape(n, -1)
        h *= 2
    return y


def _apply(op, x):
    xt = torch.from_numpy(np.ascontiguousarray(x.T)).cuda().t()
    y = op.forward(xt)
    op.check()
    return y.cpu().numpy()


def _columns(n, rng):
    """Spikes at the head of every 4096 rows on a background of one sign
    (random, constant), and positive data."""
    cols = [np.abs(rng.standard_normal(n)), np.full(n, 1 / 3.0)]
    for b in (1e-2, 1e-3, 1e-6, 1e-10):
        for v in (np.abs(rng.standard_normal(n)), np.full(n, 1.0123456789)):
            v = v * b
            v[::4096] = 1.0
            cols.append(v)
    return np.stack(cols, axis=1)


# of the largest result: a level in double-float adds at most 2^-47 of the
# sums of magnitudes, of which every column holds one as a result; a pass of
# 4 levels in fixed point rounds its points once, which adds less
def _tol(order):
    return order * 2.0 ** -47


@pytest.mark.parametrize('order', [8, 9, 10, 11, 12, 13, 14, 17, 18, 20])
def test_contiguous(order):
    import fastmat_gb300 as fm
    x = _columns(1 << order, np.random.default_rng(order))
    y = _apply(fm.Hadamard(order), x)
    r = _fwht(x)
    assert (np.abs(y - r).max(axis=0) <= _tol(order) * np.abs(r).max(axis=0)).all()


@pytest.mark.parametrize('order', [5, 6, 7, 8, 9, 10])
def test_strided(order):
    import fastmat_gb300 as fm
    n = 1 << order
    x = _columns(n, np.random.default_rng(order))
    m = x.shape[1]
    # column j of x at every 32nd vector of a stride-32 mode
    z = np.zeros((n, 32))
    z[:, :m] = x
    y = _apply(fm.Kron(fm.Hadamard(order), fm.Eye(32)), z.reshape(-1, 1))
    y = y.reshape(n, 32)[:, :m]
    r = _fwht(x)
    assert (np.abs(y - r).max(axis=0) <= _tol(order) * np.abs(r).max(axis=0)).all()


@pytest.mark.parametrize('order', [8, 9, 10, 11, 12, 13, 17, 18])
@pytest.mark.parametrize('small', [1e-6, 1e-13, 1e-20, 1e-30])
def test_small_elements_survive_the_large_ones(order, small):
    """Two equal elements cancel in every second result: what remains are
    the small ones, with their own bits."""
    import fastmat_gb300 as fm
    rng = np.random.default_rng(order)
    n = 1 << order
    x = small * rng.standard_normal((n, 2))
    x[:2] = 1.0
    y = _apply(fm.Hadamard(order), x)
    x[:2] = 0.0
    r = _fwht(x)[1::2]
    # (in double-float: order levels of at most 2^-46, the bound of one of its
    # additions; elements 2^-74 of the largest and below have their heads'
    # 24 bits alone)
    tol = order * 2.0 ** -46 + (2.0 ** -23 if small < 1e-18 else 0.0)
    assert (np.abs(y[1::2] - r).max(axis=0) <=
            tol * np.abs(r).max(axis=0)).all()


@pytest.mark.parametrize('order', [6, 8, 10])
def test_small_elements_of_strided_vectors(order):
    import fastmat_gb300 as fm
    rng = np.random.default_rng(order)
    n = 1 << order
    x = 1e-13 * rng.standard_normal((n, 64))
    x[:2, ::3] = 1.0
    y = _apply(fm.Kron(fm.Hadamard(order), fm.Eye(64)),
               x.reshape(-1, 1)).reshape(n, 64)
    x[:2, ::3] = 0.0
    r = _fwht(x)[1::2]
    y = y[1::2]
    assert (np.abs(y - r).max(axis=0) <=
            order * 2.0 ** -46 * np.abs(r).max(axis=0)).all()


@pytest.mark.parametrize('order', [9, 13, 18])
def test_infinite_columns_beside_wide_ones(order):
    """Every vector of a CTA takes the form its widest one needs."""
    import fastmat_gb300 as fm
    rng = np.random.default_rng(order)
    n = 1 << order
    x = rng.standard_normal((n, 9))
    x[3, 1] = np.inf
    x[:, 4] *= 1e-14
    x[0, 4] = 1.0
    x[:, 6] = 0.0
    y = _apply(fm.Hadamard(order), x)
    assert not np.isfinite(y[:, 1]).any()
    keep = [0, 2, 3, 4, 5, 7, 8]
    r = _fwht(x[:, keep])
    assert (np.abs(y[:, keep] - r).max(axis=0) <=
            _tol(order) * np.abs(r).max(axis=0)).all()
    assert not y[:, 6].any()
