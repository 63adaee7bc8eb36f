"""Plans on a nearly full device: the tables that only the register transforms
of long vectors need are optional, the plan runs without them."""

import numpy as np
import pytest

torch = pytest.importorskip('torch')
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('kind,n', [('circulant', 1024), ('fourier', 1 << 14),
                                    ('circulant', 1 << 14)])
def test_plan_without_room_for_register_tables(kind, n):
    import fastmat_gb300 as fm
    from fastmat_gb300 import _native
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, 3)) + 1j * rng.standard_normal((n, 3))
    c = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    ref = np.fft.fft(x, axis=0)
    if kind == 'circulant':
        ref = np.fft.ifft(np.fft.fft(c)[:, None] * ref, axis=0)
    routes = []
    for k in range(60):
        op = fm.Circulant(c) if kind == 'circulant' else fm.Fourier(n)
        _native.fail_allocation(k)
        try:
            plan = op.plan(np.complex128)
        except MemoryError:
            continue
        finally:
            _native.fail_allocation(-1)
        routes.append(plan.describe(0).count(' rx'))
        y = op.forward(x)
        assert np.abs(y - ref).max() <= 1e-12 * np.abs(ref).max()
    # some plans were made although an allocation failed, with fewer register
    # launches, and the last ones (no failure) with all of them
    assert routes and min(routes) < routes[-1]
