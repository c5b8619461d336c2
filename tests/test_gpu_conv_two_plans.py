"""Two plans alive whose mixed-radix passes need different amounts of shared memory: the first still runs after the
second, smaller one was made.  Both against numpy's FFT (test_gpu_conv_lengths)."""
import numpy as np
import pytest
import torch

from helpers import unit_random

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("first,second", [((1500, 3, 2), (1100, 3, 2)), ((3, 1040, 2), (3, 1030, 1)), ((4, 3, 200), (4, 3, 70)),
                                          ((3, 1500, 2), (3, 1100, 2))])
def test_smaller_plan_later(prec, first, second):
    from micromagnum_b200 import magneto as mg
    mg.enableCuda(mg.CUDA_64 if prec == "f64" else mg.CUDA_32)

    def make(dims):
        T = mg.GenerateDemagTensor(*dims, 3e-9, 4e-9, 2e-9, False, False, False, 1, mg.PADDING_ROUND_4)
        m, h = mg.VectorMatrix(dims), mg.VectorMatrix(dims)
        m.data.copy_(torch.as_tensor(unit_random(np.random.default_rng(1), int(np.prod(dims))).reshape(-1)))
        try:
            return mg.SymmetricMatrixVectorConvolution_FFT(T, *dims), m, h
        except Exception as e:  # a length too large for one block (FP64) is refused when the plan is made
            assert "too large" in str(e)
            pytest.skip("refused")

    a, m, h = make(first)
    a.execute(m, h)
    before = h.data.clone()
    b, mb, hb = make(second)
    b.execute(mb, hb)
    h.data.zero_()
    a.execute(m, h)
    assert torch.equal(h.data, before)
