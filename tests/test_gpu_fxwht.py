"""The fixed-point register FWHT of float64 data (fm_rfwht.cuh): every built
length (contiguous, strided, two passes in one launch), vectors at the ends
of float64's exponent range, mixed magnitudes, exact integers, zero and
Inf / NaN columns, against a float64 butterfly."""

import numpy as np
import pytest

torch = pytest.importorskip('torch')
pytestmark = pytest.mark.gpu


def _fwht(x, tiny=0.0):
    """tiny: values below it vanish, as subnormal ones do between the
    passes of the transform (the first takes the low 12 bits)."""
    y = np.array(x, dtype=np.float64)
    n = y.shape[0]
    h = 1
    while h < n:
        if h == 1 << 12:
            y = np.where(np.abs(y) < tiny, 0.0, y)
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


@pytest.mark.parametrize('order', [8, 9, 10, 11, 12, 13, 17, 18, 19, 20])
@pytest.mark.parametrize('expo', [-1010, -940, -300, 0, 300, 980, 1000])
def test_contiguous(order, expo):
    import fastmat_gb300 as fm
    rng = np.random.default_rng(order)
    n = 1 << order
    x = rng.standard_normal((n, 4))
    x[:, 1] = 0.0
    x[:, 2] = rng.integers(-1000, 1001, n)  # exact sums
    x[:, 3] *= 10.0 ** rng.uniform(-20, 0, n)
    y = _apply(fm.Hadamard(order), np.ldexp(x, expo))
    # subnormal inputs and results flush to zero, in the oracle too
    tiny = np.ldexp(1.0, -1022 - expo) if expo < -900 else 0.0
    x = np.where(np.abs(x) < tiny, 0.0, x)
    r = _fwht(x, tiny)
    y = np.ldexp(y, -expo)
    top = np.abs(r).max(axis=0) + (np.arange(4) == 1)
    err = np.where(np.abs(r) > tiny, np.abs(y - r),
                   np.maximum(np.abs(y) - tiny, 0.0))
    assert (err.max(axis=0) <= 1e-14 * top).all()
    assert not y[:, 1].any()
    assert np.array_equal(y[:, 2], r[:, 2])


@pytest.mark.parametrize('order', [5, 6, 7, 8, 9, 10])
@pytest.mark.parametrize('cplx', [False, True])
def test_strided(order, cplx):
    import fastmat_gb300 as fm
    rng = np.random.default_rng(order)
    n = 1 << order
    op = fm.Kron(fm.Eye(3), fm.Hadamard(order), fm.Eye(64))
    x = rng.standard_normal((3 * n * 64, 2))
    if cplx:
        x = x + 1j * rng.standard_normal(x.shape)

    def ref(v):
        w = v.reshape(3, n, 64 * 2).transpose(1, 0, 2).reshape(n, -1)
        return _fwht(w).reshape(n, 3, 128).transpose(1, 0, 2).reshape(
            x.shape)

    y = _apply(op, x)
    r = ref(x.real) + (1j * ref(x.imag) if cplx else 0)
    assert np.abs(y - r).max() <= 1e-14 * np.abs(r).max()


@pytest.mark.parametrize('order', [9, 13, 18])
@pytest.mark.parametrize('bad', [np.inf, -np.inf, np.nan])
def test_non_finite(order, bad):
    import fastmat_gb300 as fm
    rng = np.random.default_rng(4)
    x = rng.standard_normal((1 << order, 3))
    x[5, 1] = bad
    y = _apply(fm.Hadamard(order), x)
    r = _fwht(x[:, ::2])
    assert np.abs(y[:, ::2] - r).max() <= 1e-14 * np.abs(r).max()
    assert not np.isfinite(y[:, 1]).any()


def test_results_beyond_the_range_overflow():
    import fastmat_gb300 as fm
    x = np.full((1 << 10, 1), 1e308)
    y = _apply(fm.Hadamard(10), x)
    assert y[0, 0] == np.inf and not y[1:].any()
