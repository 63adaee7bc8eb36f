"""The fused soft-thresholding step (fm_shrink_step) of ISTA / FISTA against
its formula in float64, at counts around a block and a grid, in every type;
and the iteration's fallback to separate operations."""

import numpy as np
import pytest

torch = pytest.importorskip('torch')
pytestmark = pytest.mark.gpu


def _rand(rng, n, dt):
    v = rng.standard_normal(n)
    if np.dtype(dt).kind == 'c':
        v = v + 1j * rng.standard_normal(n)
    return v.astype(dt)


@pytest.mark.parametrize('dt', [np.float32, np.float64, np.complex64,
                                np.complex128])
@pytest.mark.parametrize('n', [1, 255, 257, 152 * 8 * 256 + 3])
@pytest.mark.parametrize('momentum', [False, True])
def test_step(dt, n, momentum):
    import fastmat_gb300._native as nat
    rng = np.random.default_rng(n)
    y, g, xo = (_rand(rng, n, dt) for _ in range(3))
    t = [torch.from_numpy(a).cuda() for a in (y, g, xo)]
    out = [torch.full_like(t[0], 7) for _ in range(3)]
    l, alpha, beta = 0.37, 0.6, 0.81
    nat.shrink_step(n, nat.DTYPE_CODE[np.dtype(dt)], t[0].data_ptr(),
                    t[1].data_ptr(), t[2].data_ptr() if momentum else None,
                    out[0].data_ptr(), out[1].data_ptr(),
                    out[2].data_ptr() if momentum else None, l, alpha, beta,
                    torch.cuda.current_stream().cuda_stream)
    wide = np.complex128 if np.dtype(dt).kind == 'c' else np.float64
    s = y.astype(wide) - l * g.astype(wide)
    m = np.maximum(np.abs(s) - alpha, 0)
    x = m / (m + alpha) * s
    ref = [s, x, x + beta * (x - xo.astype(wide))]
    # a few roundings of values below max |y| + |g| + |xold|; the threshold
    # passes an error of |s| on with a factor of at most 1 + |s| / alpha
    scale = sum(np.abs(a).max() for a in (y, g, xo))
    tol = 8 * np.finfo(dt).eps * scale * (1 + scale / alpha)
    for k in range(3 if momentum else 2):
        assert np.abs(out[k].cpu().numpy() - ref[k]).max() <= tol
    if not momentum:
        assert bool((out[2] == 7).all())


def test_mixed_types_and_row_major_inputs_agree():
    import fastmat_gb300 as fm
    rng = np.random.default_rng(1)
    c = rng.standard_normal(300)
    C = fm.Circulant(c)
    b = torch.from_numpy(rng.standard_normal((300, 4)))
    alg = fm.algorithms.FISTA(C, numLambda=0.1, numMaxSteps=7)
    ref = alg.process(b.to(torch.complex128).cuda())
    # a real row-major right-hand side: the iterates change type, and the
    # separate operations run where the arrays differ
    y = alg.process(b.cuda())
    assert float((y - ref).abs().max()) <= 1e-11 * float(ref.abs().max())
