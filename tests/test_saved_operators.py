"""Operators stored as Python pickles by earlier versions of the package."""

import pickle

import numpy as np
import pytest

torch = pytest.importorskip('torch')


def test_state_without_the_type_table():
    """Earlier versions kept no table of input types on an operator."""
    import fastmat_gb300 as fm
    op = fm.Circulant(np.arange(8.0) + 1)
    new = pickle.loads(pickle.dumps(op))
    new.__dict__.pop('_io', None)
    code = new._io_types(torch.float64)
    assert code == op._io_types(torch.float64)
