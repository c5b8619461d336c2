"""2-D boxes with several columns per block of the fused y pass, FP32 and FP64, and single ones at the longest
length: against numpy's FFT; and a large film, whose FP32 evaluation (half the bytes) has to be the faster one."""
import numpy as np
import pytest
import torch

from test_gpu_conv_lengths import check

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mg():
    from micromagnum_b200 import magneto
    return magneto


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("dims", [(700, 250, 1), (770, 180, 1), (330, 500, 1), (330, 700, 1), (600, 90, 1), (310, 1000, 1)])
def test_tiles(mg, prec, dims):
    check(mg, prec, dims)


def test_f32_is_not_slower(mg):
    def time(mode):
        mg.enableCuda(mode)
        n = 1024
        T = mg.GenerateDemagTensor(n, n, 1, *(4e-9,) * 3, False, False, False, 1, mg.PADDING_ROUND_4)
        m, h = mg.VectorMatrix((n, n, 1)), mg.VectorMatrix((n, n, 1))
        m.data.copy_(torch.as_tensor(np.random.default_rng(0).standard_normal(3 * n * n)))
        conv = mg.SymmetricMatrixVectorConvolution_FFT(T, n, n, 1)
        best = []
        for _ in range(12):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            conv.execute(m, h)
            b.record()
            torch.cuda.synchronize()
            best.append(a.elapsed_time(b))
        return min(best)

    assert time(mg.CUDA_32) < time(mg.CUDA_64)
