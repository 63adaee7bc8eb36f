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
