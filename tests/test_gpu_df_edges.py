"""The double-float register kernels (register convolution, long-vector FFT
and convolution) where the operator, not the input, leaves the ordinary
range: NaN and Inf in an operator's own data, results that overflow, very
small results, and elements far below their vector's largest.  References
in float64 numpy."""

import numpy as np
import pytest

torch = pytest.importorskip('torch')
pytestmark = pytest.mark.gpu


def _cplx(rng, *shape):
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


def _conv(c, x):
    return np.fft.ifft(np.fft.fft(c)[:, None] * np.fft.fft(x, axis=0), axis=0)


def _forward(op, x):
    t = torch.from_numpy(np.ascontiguousarray(x.T)).cuda().t()
    y = op.forward(t)
    op.check()
    return y.cpu().numpy()


# rconv: one warp a vector; rxconv: whole columns; rxfft: the outer passes of
# long columns
ROUTES = [(16, 'rconv'), (128, 'rconv'), (512, 'rxconv'), (4096, 'rxconv'),
          (1 << 14, 'rxfft'), (1 << 17, 'rxfft')]


def _routed(op, route, direction=0):
    assert route in op.plan(np.complex128).describe(direction)
    return op


@pytest.mark.parametrize('bad', [np.nan, np.inf])
@pytest.mark.parametrize('n,route', ROUTES)
def test_non_finite_filter(n, route, bad):
    import fastmat_gb300 as fm
    rng = np.random.default_rng(n)
    c = _cplx(rng, n)
    c[3] = bad
    y = _forward(_routed(fm.Circulant(c), route), _cplx(rng, n, 2))
    assert not np.isfinite(y).any()


@pytest.mark.parametrize('bad', [np.nan, np.inf])
@pytest.mark.parametrize('n,route', ROUTES)
def test_non_finite_product_of_the_storer(n, route, bad):
    import fastmat_gb300 as fm
    rng = np.random.default_rng(n)
    c, d, x = _cplx(rng, n), _cplx(rng, n), _cplx(rng, n, 2)
    d[5] = bad
    y = _forward(_routed(fm.Product(fm.Diag(d), fm.Circulant(c)), route), x)
    assert not np.isfinite(y[5]).any()
    keep = np.arange(n) != 5
    r = d[keep, None] * _conv(c, x)[keep]
    assert np.abs(y[keep] - r).max() <= 1e-12 * np.abs(r).max()


@pytest.mark.parametrize('bad', [np.nan, np.inf])
@pytest.mark.parametrize('n,route', ROUTES)
def test_non_finite_product_of_the_loader(n, route, bad):
    import fastmat_gb300 as fm
    rng = np.random.default_rng(n)
    d = _cplx(rng, n)
    d[5] = bad
    op = fm.Product(fm.Circulant(_cplx(rng, n)), fm.Diag(d))
    y = _forward(_routed(op, route), _cplx(rng, n, 2))
    assert not np.isfinite(y).any()


@pytest.mark.parametrize('n,route', ROUTES)
def test_overflow_is_not_finite(n, route):
    """Results beyond the arithmetic's range (2^128 of the largest input) are
    Inf or NaN, never a wrong number."""
    import fastmat_gb300 as fm
    rng = np.random.default_rng(n)
    c, d, x = _cplx(rng, n), _cplx(rng, n), _cplx(rng, n, 2)
    op = fm.Product(fm.Diag(d * 1e25), fm.Circulant(c * 1e25))
    y = _forward(_routed(op, route), x)
    r = 1e50 * (d[:, None] * _conv(c, x))
    bad = np.abs(y - r) > 1e-12 * np.abs(r).max()
    assert not (bad & np.isfinite(y.real) & np.isfinite(y.imag)).any()


@pytest.mark.parametrize('e', range(-120, -99, 2))
@pytest.mark.parametrize('n,route', ROUTES)
def test_small_results_keep_their_tails(n, route, e):
    """Results of 2^e of the vector's largest element, by two factors of
    2^(e / 2): what float's subnormals hold of the tails is stored."""
    import fastmat_gb300 as fm
    rng = np.random.default_rng(n)
    c, d, x = _cplx(rng, n), _cplx(rng, n), _cplx(rng, n, 3)
    f = 2.0 ** (e // 2)
    C, D = fm.Circulant(c * f), fm.Diag(d * f)
    if route == 'rconv':
        # (its storer converts vectors with a product of its own as other
        # kernels do, which drops subnormal tails)
        op, r, terms = fm.Product(C, D), _conv(c, d[:, None] * x), n
    else:
        op, r, terms = fm.Product(D, C), d[:, None] * _conv(c, x), 1
    y = _forward(_routed(op, route), x)
    y = np.ldexp(y.real, -e) + 1j * np.ldexp(y.imag, -e)
    # the engine's 1e-12, and the tails of the products of that size, some
    # 10 roundings to multiples of 2^-149 of the column's largest element;
    # real and imaginary parts below 2^-126 of that element flush to zero
    top = np.abs(x).max()
    tails = np.ldexp(top * terms, -145 - e)
    gone = np.ldexp(top, -125 - e)
    for u, v in ((y.real, r.real), (y.imag, r.imag)):
        err = np.where((u == 0) & (np.abs(v) <= gone), 0.0, np.abs(u - v))
        assert err.max() <= 1e-12 * np.abs(r).max() + tails


@pytest.mark.parametrize('n,route', ROUTES[:3])
def test_results_up_to_the_range_of_float(n, route):
    """Results near 2^124 of the vector's largest element."""
    import fastmat_gb300 as fm
    rng = np.random.default_rng(n)
    c, x = np.zeros(n, dtype=np.complex128), _cplx(rng, n, 3)
    c[:2] = [1.0, 0.5j]
    x /= np.abs(x).max()
    # (2^121: the transform of x stays below 2^6.5 at 512 points, and the
    # spectrum's 1 / n returns what the sums of the inverse take)
    y = _forward(_routed(fm.Circulant(np.ldexp(c.real, 121) +
                                      1j * np.ldexp(c.imag, 121)), route), x)
    y = np.ldexp(y.real, -121) + 1j * np.ldexp(y.imag, -121)
    r = _conv(c, x)
    assert np.abs(y - r).max() <= 1e-12 * np.abs(r).max()


@pytest.mark.parametrize('n,route', ROUTES)
def test_elements_far_below_the_largest_keep_their_heads(n, route):
    """A Diag on the loader that removes the largest element: the others,
    2^-100 of it, keep the 24 bits of their heads."""
    import fastmat_gb300 as fm
    rng = np.random.default_rng(n)
    c, d, x = _cplx(rng, n), np.full(n, 2.0 ** 80, complex), _cplx(rng, n, 2)
    x = np.ldexp(x.real, -100) + 1j * np.ldexp(x.imag, -100)
    x[7] = 1.0
    d[7] = 0.0
    y = _forward(_routed(fm.Product(fm.Circulant(c), fm.Diag(d)), route), x)
    r = _conv(c, d[:, None] * x)
    # heads truncated to 24 bits: 2^-23 of each element, and at most
    # sum |c| / |y| ~ 1 / sqrt(n) .. 1 of that in the result
    assert np.abs(y - r).max() <= 2.0 ** -22 * np.abs(r).max()


def test_products_round_like_normalised_double_floats():
    """Complex products of the register kernels: both real products and their
    sum are normalised.  On a one-hot column the transforms are exact (sums of
    equal values), so the storer's product stands alone."""
    import fastmat_gb300 as fm
    rng = np.random.default_rng(6)
    m = 1 << 12
    err = []
    for k in range(16):
        for j in (0, 2, 4, 6):
            a, d = _cplx(rng, m), _cplx(rng, 8)
            op = fm.Product(fm.Diag(d), fm.Circulant(np.eye(8)[0] + 0j))
            x = np.zeros((8, m), dtype=np.complex128)
            x[j] = a
            y = _forward(_routed(op, 'rconv'), x)
            ld = np.clongdouble
            e = y[j].astype(ld) - a.astype(ld) * ld(d[j])
            err.append(np.abs(e) / np.abs(a * d[j]))
    # root mean square for these factors with the arithmetic emulated in
    # float32: 0.666 2^-48 with normalised products, 0.743 with products
    # renormalised once after their sum; the bound lies between
    assert np.sqrt(np.mean(np.square(err))) <= 0.70 * 2.0 ** -48


@pytest.mark.parametrize('real', [False, True])
@pytest.mark.parametrize('n,route', [(512, 'rxconv'), (4096, 'rxconv'),
                                     (1 << 17, 'rxfft')])
def test_inputs_keep_49_bits(n, route, real):
    """A one-hot column through the identity filter: every operation of the
    transforms is exact (sums of equal values, products with 1 and powers of
    two), what remains is the conversion of the input, heads rounded to 24
    bits and tails to 24 of 29."""
    import fastmat_gb300 as fm
    rng = np.random.default_rng(n)
    m = 2048 if n <= 4096 else 128
    c = np.zeros(n, dtype=np.complex128)
    c[0] = 1.0
    x = np.zeros((n, m), dtype=np.float64 if real else np.complex128)
    x[0] = rng.standard_normal(m) if real else _cplx(rng, m)
    y = _forward(_routed(fm.Circulant(c), route), x)
    assert (np.abs(y[0].real - x[0].real) <=
            2.0 ** -49 * np.abs(x[0].real)).all()
    if not real:
        # (a part below the vector's largest flushes no bits here: 2^-74)
        assert (np.abs(y[0].imag - x[0].imag) <=
                2.0 ** -49 * np.abs(x[0].imag)).all()
    assert not y[1:].any()


@pytest.mark.parametrize('n,route', ROUTES)
def test_nan_payloads(n, route):
    """NaN of any payload (all ones: a carry of the rounding) stays NaN."""
    import fastmat_gb300 as fm
    rng = np.random.default_rng(n)
    x = _cplx(rng, n, 2)
    x.view(np.float64).view(np.uint64).reshape(n, 2, 2)[1, 0, 1] = (
        0x7FFFFFFFFFFFFFFF)
    c = _cplx(rng, n)
    y = _forward(_routed(fm.Circulant(c), route), x)
    assert not np.isfinite(y[:, 0]).any()
    r = _conv(c, x[:, 1:])
    assert np.abs(y[:, 1:] - r).max() <= 1e-12 * np.abs(r).max()
