"""Rounding of the compile-time transforms that adds up instead of averaging out.  With the unit tensor (identity at
offset 0) the field is M itself, so the projection of H - M on M is the gain of forward and inverse transform: the
moduli of the twiddles, which are the same in every line and both directions.

Bound: the constants inside the register transforms carry no rounding of modulus (two parts, or small relative to
one), and the pass tables take the pair of smallest modulus error among neighbours, under u / 6 on average over a
table's random angles; a length has at most two tables and three axes' tables enter twice, with random signs:
sqrt(6) * 2 * u / 6 < u.  The tensor's entry 1 / (px py pz) is rounded once in FP32 (known, taken out); the rounding of single
values averages out over the box as u / sqrt(3 n)."""
import math

import numpy as np
import pytest
import torch

from helpers import unit_random

pytestmark = pytest.mark.gpu

# (cells, FFT lengths of the plan)
BOXES = [((128, 32, 1), (256, 64, 1), ()), ((90, 45, 1), (192, 96, 1), ()), ((60, 60, 8), (128, 128, 16), ()),
         ((96, 48, 5), (192, 96, 12), ()), ((20, 20, 20), (48, 48, 64), ()), ((500, 100, 1), (1024, 256, 1), ()),
         ((90, 380, 3), (192, 768, 6), ()), ((128, 64, 4), (128, 128, 8), (0,)), ((96, 48, 12), (96, 48, 24), (0, 1))]


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("dims,lengths,pbc", BOXES)
def test_gain(prec, dims, lengths, pbc):
    from micromagnum_b200 import magneto as mg
    mg.enableCuda(mg.CUDA_64 if prec == "f64" else mg.CUDA_32)
    T = mg.GenerateDemagTensor(*dims, *(4e-9,) * 3, *(a in pbc for a in range(3)), 1, mg.PADDING_ROUND_4)
    T.data.zero_()
    T.data[:6] = torch.tensor([1.0, 0, 0, 1, 0, 1], dtype=torch.float64)
    M = unit_random(np.random.default_rng(1), int(np.prod(dims)))
    if prec == "f32":
        M = M.astype(np.float32).astype(np.float64)
    m, h = mg.VectorMatrix(dims), mg.VectorMatrix(dims)
    m.data.copy_(torch.as_tensor(M.reshape(-1)))
    mg.SymmetricMatrixVectorConvolution_FFT(T, *dims).execute(m, h)
    H = h.data.view(3, -1).cpu().numpy()
    u = 2.0 ** (-53 if prec == "f64" else -24)
    P = int(np.prod(lengths))
    scale = float(np.float32(1 / P)) * P - 1 if prec == "f32" else 0.0
    gain = math.fsum(((H - M) * M).reshape(-1)) / math.fsum((M * M).reshape(-1)) - scale
    assert abs(gain) < u, gain / u
