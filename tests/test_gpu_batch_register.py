"""The register transforms of the batched kernel (fm_batch.cuh): every built
length of its FFTs and convolutions, with the column and vector counts that
leave a thread group or a tile partly empty, padded leading dimensions, and
the gather, scatter and product branches of the loader and storer.  Results
against the operator's own call and numpy in float64."""

import re

import numpy as np
import pytest

torch = pytest.importorskip('torch')
pytestmark = pytest.mark.gpu


def _cplx(rng, *shape):
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


def _device(x, pad=0):
    n, m = x.shape
    t = torch.full((m, n + pad), 7, dtype=torch.complex64, device='cuda')
    t[:, :n] = torch.from_numpy(
        np.ascontiguousarray(x.T.astype(np.complex64))).cuda()
    return t[:, :n].t()


def _conv(c, x, adj=False):
    s = np.fft.fft(c)
    s = s.conj() if adj else s
    return np.fft.ifft(s[:, None] * np.fft.fft(x.astype(np.complex128),
                                               axis=0), axis=0)


def _lengths(op, direction):
    """(kind, length) of the register steps of a plan that a batch runs."""
    text = op.plan(np.complex64).describe(direction)
    return {(k, int(n)) for k, n in re.findall(r'(rxfft|rxconv) L=(\d+)',
                                               text)}


def _operators(rng):
    """(operator, forward reference, adjoint reference)."""
    import fastmat_gb300 as fm
    p = dict(precision='fp32')
    out = []
    for n in (1024, 2048, 4096, 1 << 13, 1 << 14, 1 << 15, 1 << 16, 1 << 17,
              1 << 18):
        c, d, e = _cplx(rng, n), _cplx(rng, n), _cplx(rng, n)
        rows = np.sort(rng.permutation(n)[:n // 3])
        cols = rng.permutation(n)[:n // 2 + 1]
        C = fm.Circulant(c, **p)
        out.append((C, lambda x, c=c: _conv(c, x),
                    lambda x, c=c: _conv(c, x, True)))

        def chain(x, c=c, d=d, rows=rows):
            return _conv(c, d[:, None] * x)[rows]

        def chain_h(y, c=c, d=d, rows=rows, n=n):
            z = np.zeros((n, y.shape[1]), dtype=np.complex128)
            z[rows] = y
            return d.conj()[:, None] * _conv(c, z, True)
        out.append((fm.Product(fm.Partial(C, rows=rows, **p),
                               fm.Diag(d, **p), **p), chain, chain_h))

        def picked(x, c=c, e=e, cols=cols, n=n):
            z = np.zeros((n, x.shape[1]), dtype=np.complex128)
            z[cols] = x
            return e[:, None] * _conv(c, z)

        def picked_h(y, c=c, e=e, cols=cols):
            return _conv(c, e.conj()[:, None] * y, True)[cols]
        out.append((fm.Product(fm.Diag(e, **p),
                               fm.Partial(C, cols=cols, **p), **p),
                    picked, picked_h))
        if n > 4096:
            out.append((fm.Fourier(n, **p),
                        lambda x: np.fft.fft(x.astype(np.complex128),
                                             axis=0),
                        lambda x, n=n: n * np.fft.ifft(
                            x.astype(np.complex128), axis=0)))
    n = 10007  # chirp transform: products by row, clipped columns
    out.append((fm.Fourier(n, **p),
                lambda x: np.fft.fft(x.astype(np.complex128), axis=0),
                lambda x, n=n: n * np.fft.ifft(x.astype(np.complex128),
                                               axis=0)))
    return out


@pytest.mark.parametrize('backward', [False, True])
@pytest.mark.parametrize('m,pad', [(1, 0), (3, 5), (33, 0)])
def test_every_length_and_branch(backward, m, pad):
    import fastmat_gb300 as fm
    rng = np.random.default_rng(m)
    items, refs, seen = [], [], set()
    for op, fwd, adj in _operators(rng):
        n = op.numRows if backward else op.numCols
        if m == 33 and n > 1 << 15:
            continue
        x = _cplx(rng, n, m).astype(np.complex64)
        items.append((op, _device(x, pad)))
        refs.append((adj if backward else fwd)(x))
        seen |= _lengths(op, int(backward))
    want = {('rxfft', k) for k in (64, 128, 256, 512)}
    want |= {('rxconv', k) for k in (128, 256, 512, 1024, 2048, 4096)}
    if m != 33:
        assert want <= seen, want - seen
    b = fm.Batch(items, backward=backward)
    for y, r, (op, x) in zip(b.run(), refs, items):
        own = op.backward(x) if backward else op.forward(x)
        y, own = y.cpu().numpy(), own.cpu().numpy()
        top = np.abs(r).max()
        assert y.shape == r.shape
        assert np.abs(y - own).max() <= 1e-6 * top, repr(op)
        assert np.abs(y - r).max() <= 1e-5 * top, repr(op)
    b.check()
