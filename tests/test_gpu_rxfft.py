"""The register transforms of long vectors (rxfft_kernel / rxconv_kernel,
fm_rfft.cuh) against numpy in float64: every built length, the edges of the
loader and storer (zero padding, clipped rows, gathers, scatters, products,
conjugation, accumulation, type conversion, padded leading dimensions),
both directions, both precisions.  Bounds: the engine's 1e-12 (complex128)
and 1e-5 (complex64) of the largest value."""

import numpy as np
import pytest

torch = pytest.importorskip('torch')
pytestmark = pytest.mark.gpu

PREC = [('native', np.complex128, 1e-12), ('fp32', np.complex64, 1e-5)]


def _cplx(rng, *shape):
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


def _conv(c, x, adjoint=False):
    s = np.fft.fft(c)
    s = s.conj() if adjoint else s
    return np.fft.ifft(s[:, None] * _fft(x), axis=0)


def _fft(x, axis=0):
    # (numpy transforms single-precision input in single precision)
    return np.fft.fft(x.astype(np.complex128), axis=axis)


def _ifft(x, axis=0):
    return np.fft.ifft(x.astype(np.complex128), axis=axis)


def _check(y, r, tol):
    y = y.cpu().numpy() if hasattr(y, 'cpu') else y
    assert y.shape == r.shape
    assert np.abs(y - r).max() <= tol * np.abs(r).max()


def _device(x, pad=0):
    n, m = x.shape
    t = torch.zeros((m, n + pad), dtype=torch.from_numpy(x[:1, :1]).dtype,
                    device='cuda')
    t[:, :n] = torch.from_numpy(np.ascontiguousarray(x.T)).cuda()
    return t[:, :n].t()


@pytest.mark.parametrize('prec,dt,tol', PREC)
@pytest.mark.parametrize('n', [257, 512, 1024, 1031, 2048, 4096, 8192, 16384,
                               20011, 1 << 15, 1 << 16, 1 << 17, 1 << 19])
@pytest.mark.parametrize('pad', [0, 3])
def test_circulant(n, prec, dt, tol, pad):
    import fastmat_gb300 as fm
    rng = np.random.default_rng(n)
    m = 5 if n <= 1 << 17 else 2
    c, x = _cplx(rng, n), _cplx(rng, n, m).astype(dt)
    op = fm.Circulant(c, precision=prec)
    assert ('rxconv' in op.plan(dt).describe(0)) == (
        n > (256 if dt == np.complex128 else 512) or n == 257)
    xt = _device(x, pad)
    _check(op.forward(xt), _conv(c, x), tol)
    _check(op.backward(xt), _conv(c, x, True), tol)
    if pad == 0:  # real input of another type, one column
        xr = x.real.astype(np.float32)[:, :1]
        _check(op.forward(_device(xr)), _conv(c, xr), tol)


@pytest.mark.parametrize('prec,dt,tol', PREC)
@pytest.mark.parametrize('n', [8192, 1 << 14, 1 << 15, 1 << 17, 1 << 19,
                               4099, 10007, 65521])
@pytest.mark.parametrize('m', [1, 7])
def test_fourier(n, prec, dt, tol, m):
    import fastmat_gb300 as fm
    rng = np.random.default_rng(n + m)
    x = _cplx(rng, n, m).astype(dt)
    op = fm.Fourier(n, precision=prec)
    assert 'rx' in op.plan(dt).describe(0)
    xt = _device(x)
    _check(op.forward(xt), _fft(x), tol)
    _check(op.backward(xt), _ifft(x) * n, tol)


@pytest.mark.parametrize('rows,cols', [(300, 301), (1000, 513), (513, 3000),
                                       (4097, 9000), (30000, 2)])
@pytest.mark.parametrize('prec,dt,tol', PREC)
def test_toeplitz(rows, cols, prec, dt, tol):
    import fastmat_gb300 as fm
    rng = np.random.default_rng(rows)
    vc, vr = _cplx(rng, rows), _cplx(rng, cols - 1)
    op = fm.Toeplitz(vc, vr, precision=prec)
    e = np.concatenate([vc, vr])
    for adj, n_in, n_out in ((False, cols, rows), (True, rows, cols)):
        x = _cplx(rng, n_in, 3).astype(dt)
        z = np.zeros((e.size, 3), dtype=np.complex128)
        z[:n_in] = x
        r = _conv(e, z, adj)[:n_out]
        xt = _device(x, 1)
        _check((op.backward if adj else op.forward)(xt), r, tol)


@pytest.mark.parametrize('prec,dt,tol', PREC)
@pytest.mark.parametrize('n', [1024, 8192, 1 << 16])
def test_chain_sum_conjugate(n, prec, dt, tol):
    import fastmat_gb300 as fm
    rng = np.random.default_rng(n)
    c, d, e = _cplx(rng, n), _cplx(rng, n), _cplx(rng, n)
    rows = np.sort(rng.permutation(n)[:n // 3])
    cols = rng.permutation(n)[:n // 2 + 1]
    C = fm.Circulant(c, precision=prec)
    op = fm.Product(fm.Partial(C, rows=rows, precision=prec),
                    fm.Diag(d, precision=prec), precision=prec)
    x = _cplx(rng, n, 3).astype(dt)
    _check(op.forward(_device(x)), _conv(c, d[:, None] * x)[rows], tol)
    y = _cplx(rng, rows.size, 3).astype(dt)
    z = np.zeros((n, 3), dtype=np.complex128)
    z[rows] = y
    _check(op.backward(_device(y)),
           d.conj()[:, None] * _conv(c, z, True), tol)
    # input selection, conjugated operator, complex scalar
    op = fm.Product(0.5 - 2j, fm.Partial(C, cols=cols, precision=prec).conj,
                    precision=prec)
    y = _cplx(rng, cols.size, 2).astype(dt)
    z = np.zeros((n, 2), dtype=np.complex128)
    z[cols] = y
    _check(op.forward(_device(y)), (0.5 - 2j) * _conv(c.conj(), z), tol)
    # accumulated terms
    op = fm.Sum(C, fm.Circulant(e, precision=prec), fm.Diag(d),
                precision=prec)
    _check(op.forward(_device(x)),
           _conv(c, x) + _conv(e, x) + d[:, None] * x, tol)


@pytest.mark.parametrize('prec,dt,tol', PREC)
@pytest.mark.parametrize('L', [32, 64, 128, 256, 512])
@pytest.mark.parametrize('inner', [2, 3, 9, 24, 33])
def test_strided_mode_with_ragged_stride(L, inner, prec, dt, tol):
    """A Fourier mode of a Kron at a stride that is no multiple of 32."""
    import fastmat_gb300 as fm
    rng = np.random.default_rng(L + inner)
    op = fm.Kron(fm.Eye(3), fm.Fourier(L), fm.Eye(inner), precision=prec)
    x = _cplx(rng, 3 * L * inner, 2).astype(dt)
    v = x.reshape(3, L, inner, 2)
    xt = _device(x)
    _check(op.forward(xt), _fft(v, 1).reshape(x.shape), tol)
    _check(op.backward(xt), (_ifft(v, 1) * L).reshape(x.shape),
           tol)
