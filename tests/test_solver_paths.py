"""ISTA / FISTA with operators and thresholds of a user's own: what ``forward``
returned is read, never written."""

import numpy as np
import pytest

torch = pytest.importorskip('torch')


class _Same(object):
    """Mixin: an operator whose products are its argument."""

    def forward(self, x):
        self.seen = (x, x.clone())
        return x

    def backward(self, x):
        return x


def _identity(n):
    import fastmat_gb300 as fm

    class Same(_Same, fm.Eye):
        largestSingularValue = 1.0
    return Same(n)


def test_the_products_of_a_user_operator_are_not_overwritten():
    from fastmat_gb300.algorithms import ISTA
    op = _identity(5)
    b = torch.arange(10, dtype=torch.float64).reshape(5, 2)
    ISTA(op, numMaxSteps=3)._process(b)
    assert torch.equal(*op.seen)


def test_iterates_of_a_user_operator():
    """A = 1: one FISTA run against the iteration written out."""
    from fastmat_gb300.algorithms import FISTA
    b = torch.linspace(-2, 2, 12, dtype=torch.float64).reshape(6, 2)
    got = FISTA(_identity(6), numLambda=0.4, numMaxSteps=4)._process(b)
    x = torch.zeros_like(b)
    y, t = x.clone(), 1.0
    for _ in range(4):
        old, z = x, y - (y - b)
        m = torch.clamp(z.abs() - 0.2, min=0)
        x = m / (m + 0.2) * z
        s, t = t, (1 + np.sqrt(1 + 4 * t * t)) / 2
        y = x + (s - 1) / t * (x - old)
    want = torch.where(x != 0, z, x)
    assert float((got - want).abs().max()) <= 1e-14


@pytest.mark.gpu
def test_a_threshold_set_as_a_parameter_is_used():
    import fastmat_gb300 as fm
    from fastmat_gb300.algorithms import ISTA

    def halve(x, alpha):
        halve.calls += 1
        return 0.5 * x

    halve.calls = 0
    rng = np.random.default_rng(0)
    op = fm.Circulant(rng.standard_normal(64))
    b = torch.from_numpy(rng.standard_normal((3, 64))).to(
        torch.complex128).cuda().t()
    alg = ISTA(op, numMaxSteps=3, softThreshold=halve)
    alg.process(b)
    assert halve.calls == 3
    assert torch.equal(alg.arrX, 0.5 * alg.arrStep)
