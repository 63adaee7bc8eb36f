"""A conjugated factor inside a Kron next to a product of its launch's loader
or storer: conj(x) d is not conj(x d).  Every register kernel that takes a
conjugation and a product, against numpy in float64."""

import numpy as np
import pytest

torch = pytest.importorskip('torch')
pytestmark = pytest.mark.gpu

PREC = [('native', np.complex128, 1e-12), ('fp32', np.complex64, 1e-5)]


def _cplx(rng, *shape):
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


def _forward(op, x, backward=False):
    t = torch.from_numpy(np.ascontiguousarray(x.T)).cuda().t()
    y = (op.backward if backward else op.forward)(t)
    op.check()
    return y.cpu().numpy()


def _modes(v, a, b, shape):
    """a along axis 0 and b along axis 1 of the columns of v (callables on
    axis 0 of a matrix)."""
    f, g = shape
    w = v.reshape(f, g, -1)
    w = b(w.transpose(1, 0, 2).reshape(g, -1)).reshape(g, f, -1)
    w = a(w.transpose(1, 0, 2).reshape(f, -1))
    return w.reshape(v.shape)


@pytest.mark.parametrize('prec,dt,tol', PREC)
@pytest.mark.parametrize('n', [16, 64, 256, 1024, 4096])
def test_conjugated_circulant(n, prec, dt, tol):
    import fastmat_gb300 as fm
    rng = np.random.default_rng(n)
    c, d, e, x = _cplx(rng, n), _cplx(rng, 3 * n), _cplx(rng, 3 * n), None
    x = _cplx(rng, 3 * n, 2).astype(dt)
    C = fm.Circulant(c, precision=prec)

    def conv(k, adj=False):
        s = np.fft.fft(k)
        s = s.conj() if adj else s
        return lambda v: np.fft.ifft(
            s[:, None] * np.fft.fft(v.astype(np.complex128), axis=0), axis=0)

    def same(v):
        return v

    K = fm.Kron(fm.Eye(3), C.conj, precision=prec)
    for op, ref in (
            (fm.Product(K, fm.Diag(d), precision=prec),
             lambda v: _modes(d[:, None] * v, same, conv(c.conj()), (3, n))),
            (fm.Product(fm.Diag(e), K, precision=prec),
             lambda v: e[:, None] * _modes(v, same, conv(c.conj()), (3, n)))):
        r = ref(x)
        y = _forward(op, x)
        assert np.abs(y - r).max() <= tol * np.abs(r).max()
    op = fm.Product(K, fm.Diag(d), precision=prec)
    r = d.conj()[:, None] * _modes(x, same, conv(c.conj(), True), (3, n))
    y = _forward(op, x, True)
    assert np.abs(y - r).max() <= tol * np.abs(r).max()


@pytest.mark.parametrize('prec,dt,tol', PREC)
@pytest.mark.parametrize('n,inner', [(32, 32), (64, 3), (256, 9), (512, 2)])
def test_conjugated_fourier(n, inner, prec, dt, tol):
    import fastmat_gb300 as fm
    rng = np.random.default_rng(n)
    N = n * inner
    d, e = _cplx(rng, N), _cplx(rng, N)
    x = _cplx(rng, N, 2).astype(dt)

    def idft(v):  # conj(F) = n times the inverse transform
        return np.fft.ifft(v.astype(np.complex128), axis=0) * n

    def same(v):
        return v

    K = fm.Kron(fm.Fourier(n).conj, fm.Eye(inner), precision=prec)
    op = fm.Product(fm.Diag(e), K, fm.Diag(d), precision=prec)
    r = e[:, None] * _modes(d[:, None] * x, idft, same, (n, inner))
    y = _forward(op, x)
    assert np.abs(y - r).max() <= tol * np.abs(r).max()
