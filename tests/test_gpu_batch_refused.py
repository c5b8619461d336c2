"""Lengths that the grouped passes are not built for are refused, not left out."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_batch_refuses_long_f64():
    from micromagnum_b200 import _lib
    from micromagnum_b200.batch import Batch, Instance
    q = Instance((600, 8, 1), (4e-9,) * 3, 8e5, 1.3e-11, 0.5, t_end=1e-14)
    b = Batch([], precision="f64")
    b.add(q, np.concatenate([np.ones((1, q.n)), np.zeros((2, q.n))]))
    with pytest.raises(_lib.MMError):
        b.relax(max_rounds=1)
