"""Packed double-float register kernels (register convolution, strided
register FFT): the float64 conversions at the edges of their range -- powers
of two, zero columns, magnitudes near the ends of float64's exponent range,
Inf / NaN columns -- against numpy in float64."""

import numpy as np
import pytest

torch = pytest.importorskip('torch')
pytestmark = pytest.mark.gpu


def _ops(kind, n, rng):
    import fastmat_gb300 as fm
    if kind == 'conv':
        c = rng.standard_normal(n) + 1j * rng.standard_normal(n)
        s = np.fft.fft(c)
        return fm.Circulant(c), lambda x: np.fft.ifft(
            s[:, None] * np.fft.fft(x, axis=0), axis=0)
    op = fm.Kron(fm.Fourier(n), fm.Eye(32))
    return op, lambda x: np.fft.fft(
        x.reshape(n, 32, -1), axis=0).reshape(n * 32, -1)


@pytest.mark.parametrize('kind', ['conv', 'strided'])
@pytest.mark.parametrize('n', [16, 128, 256])
@pytest.mark.parametrize('expo', [-1000, -895, -885, -300, 0, 300, 885, 895,
                                  1000])
def test_magnitudes(kind, n, expo):
    rng = np.random.default_rng(n)
    op, ref = _ops(kind, n, rng)
    rows = op.numCols
    x = rng.standard_normal((rows, 5)) + 1j * rng.standard_normal((rows, 5))
    x[:, 1] = 0.0
    x[:, 2] = 2.0 ** rng.integers(-3, 4, rows)  # exact powers of two
    x[:, 3] = 0.0
    x[rows // 3, 3] = -1.0
    # column maxima scaled to 2^expo; the transform of the unscaled column
    # is scaled exactly
    y = op.forward(np.asfortranarray(np.ldexp(x.real, expo) +
                                     1j * np.ldexp(x.imag, expo)))
    y = np.ldexp(y.real, -expo) + 1j * np.ldexp(y.imag, -expo)
    r = ref(x)
    # 1e-12 of the largest value, the engine's float64 bound
    assert np.abs(y - r).max(axis=0) == pytest.approx(
        np.zeros(5), abs=1e-12 * np.abs(r).max())
    assert not y[:, 1].any()


@pytest.mark.parametrize('kind', ['conv', 'strided'])
@pytest.mark.parametrize('bad', [np.inf, -np.inf, np.nan])
def test_non_finite_stay_in_their_vectors(kind, bad):
    rng = np.random.default_rng(3)
    op, ref = _ops(kind, 128, rng)
    rows = op.numCols
    x = rng.standard_normal((rows, 3)) + 1j * rng.standard_normal((rows, 3))
    z = x.copy()
    z[7, 1] = bad
    y = op.forward(np.asfortranarray(z))
    r = ref(x)
    hit = np.zeros((rows, 3), dtype=bool)
    if kind == 'conv':
        hit[:, 1] = True
    else:
        hit.reshape(128, 32, 3)[:, 7, 1] = True
    assert np.abs(y - r)[~hit].max() <= 1e-12 * np.abs(r).max()
    assert not np.isfinite(y[hit]).any()


@pytest.mark.parametrize('mag', [1e-30, 1e-24, 1e-10, 1e10, 1e24, 1e32])
def test_operator_magnitudes(mag):
    import fastmat_gb300 as fm
    rng = np.random.default_rng(5)
    c = rng.standard_normal(128) + 1j * rng.standard_normal(128)
    x = rng.standard_normal((128, 4)) + 1j * rng.standard_normal((128, 4))
    y = fm.Circulant(c * mag).forward(np.asfortranarray(x)) / mag
    r = np.fft.ifft(np.fft.fft(c)[:, None] * np.fft.fft(x, axis=0), axis=0)
    assert np.abs(y - r).max() <= 1e-12 * np.abs(r).max()
