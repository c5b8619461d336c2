"""Device memory that holds a plan at the tensor's own lengths but not at the longer ones of the plan's choice: the
calls succeed, with the same field to rounding (see test_gpu_conv_lengths for the tolerance)."""
import math

import numpy as np
import pytest
import torch

from helpers import rel_l2, unit_random

pytestmark = pytest.mark.gpu

DIMS = (520, 520, 8)  # 1040 x 1040 x 16 points: 0.55 GB; 1536 x 1536 x 16: 1.1 GB (FP64, with the set-up's scratch)


class Fill:
    """Leaves `free` bytes of device memory."""

    def __init__(self, free):
        torch.cuda.empty_cache()
        self.blocks = []
        for step in (1 << 30, 1 << 26, 1 << 24):
            while torch.cuda.mem_get_info()[0] > free + step:
                self.blocks.append(torch.empty(step, dtype=torch.uint8, device="cuda"))

    def __enter__(self):
        return self

    def __exit__(self, *_):
        self.blocks.clear()
        torch.cuda.empty_cache()


def test_convolution():
    from micromagnum_b200 import magneto as mg
    mg.enableCuda(mg.CUDA_64)
    T = mg.GenerateDemagTensor(*DIMS, *(4e-9,) * 3, False, False, False, 1, mg.PADDING_ROUND_4)
    m, h, h0 = (mg.VectorMatrix(DIMS) for _ in range(3))
    m.data.copy_(torch.as_tensor(unit_random(np.random.default_rng(1), int(np.prod(DIMS))).reshape(-1)))
    mg.SymmetricMatrixVectorConvolution_FFT(T, *DIMS).execute(m, h0)
    with Fill(780 << 20):
        c = mg.SymmetricMatrixVectorConvolution_FFT(T, *DIMS)
        c.execute(m, h)
        torch.cuda.synchronize()
    assert rel_l2(h.data.cpu().numpy(), h0.data.cpu().numpy()) < 4 * 2.0 ** -53 * math.log2(1536 * 1536 * 16)


def test_solver():
    from micromagnum_b200 import solver as sv
    make = lambda: sv.Solver(sv.RectangularMesh(DIMS, (4e-9,) * 3), [sv.Material(Ms=8e5, A=1.3e-11, alpha=0.1)], precision="f64")  # noqa: E731
    M = torch.as_tensor(unit_random(np.random.default_rng(1), int(np.prod(DIMS))) * 8e5)
    s = make()
    s.M = M
    H0 = s.eval()[2].cpu().numpy()
    s.close()
    # states and stages: 15 vectors of 52 MB; the plan 0.33 GB at its own lengths, 0.72 GB at the longer ones
    with Fill(1400 << 20):
        s = make()
    s.M = M
    H = s.eval()[2].cpu().numpy()
    assert rel_l2(H, H0) < 4 * 2.0 ** -53 * math.log2(1536 * 1536 * 16)
