"""The convolution at every FFT length with compile-time passes (2^k and 3 * 2^k), at the edges of the
range of cell counts that each length serves, on 2-D and 3-D boxes, with few lines (narrow tiles) and
many, padded and circular, against the same convolution by numpy's FFT in FP64.

Tolerance: a length-n FFT of rounding unit u has a relative rms error of order u log2 n; forward and
inverse transforms of all three axes and the product add up to less than 4 u log2(px py pz)."""
import math

import numpy as np
import pytest
import torch

from helpers import rel_l2, unit_random

pytestmark = pytest.mark.gpu

D = (3e-9, 4e-9, 2e-9)
LENGTHS = [4, 8, 12, 16, 24, 32, 48, 64, 96, 128, 192, 256, 384, 512, 768, 1024, 1536, 2048]
# the largest cell count each length takes, and the smallest (one more than the next shorter length's)
COUNTS = sorted({n for q, p in zip(LENGTHS, LENGTHS[1:]) for n in (p // 2, q // 2 + 1)})


@pytest.fixture(scope="module")
def mg():
    from micromagnum_b200 import magneto
    return magneto


def check(mg, prec, dims, pbc=(False, False, False)):
    mg.enableCuda(mg.CUDA_64 if prec == "f64" else mg.CUDA_32)
    nx, ny, nz = dims
    T = mg.GenerateDemagTensor(nx, ny, nz, *D, *pbc, 2, mg.PADDING_ROUND_4)
    ex, ey, ez = T.shape[1:]
    rng = np.random.default_rng(nx * 131 + ny * 17 + nz)
    M = unit_random(rng, nx * ny * nz)
    if prec == "f32":
        M = M.astype(np.float32).astype(np.float64)
    m, h = mg.VectorMatrix(dims), mg.VectorMatrix(dims)
    m.data.copy_(torch.as_tensor(M.reshape(-1)))
    mg.SymmetricMatrixVectorConvolution_FFT(T, nx, ny, nz).execute(m, h)
    H = h.data.view(3, -1).cpu().numpy()
    N = T.data.cpu().numpy().reshape(ez, ey, ex, 6)
    S = [np.fft.rfftn(N[..., c]) for c in range(6)]
    F = [np.fft.rfftn(M[c].reshape(nz, ny, nx), s=(ez, ey, ex), axes=(0, 1, 2)) for c in range(3)]
    ref = [np.fft.irfftn(sum(S[a] * f for a, f in zip(row, F)), s=(ez, ey, ex), axes=(0, 1, 2))[:nz, :ny, :nx].reshape(-1)
           for row in ((0, 1, 2), (1, 3, 4), (2, 4, 5))]
    u = 2.0 ** (-53 if prec == "f64" else -24)
    err = rel_l2(H, np.stack(ref))
    assert err < 4 * u * math.log2(max(4, ex * ey * ez)), (dims, err)


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("n", COUNTS)
def test_lengths(mg, prec, n):
    for dims in ((n, 3, 1), (3, n, 1), (n, 3, 2), (3, n, 2)):
        check(mg, prec, dims)


@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_z_lengths(mg, prec):
    for nz in (2, 3, 4, 5, 6, 7, 8, 9, 12, 13, 16, 17, 32, 33):
        check(mg, prec, (10, 6, nz))


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("dims", [(190, 180, 5), (380, 90, 3), (96, 384, 2), (700, 700, 1), (320, 500, 1), (128, 128, 12)])
def test_many_lines(mg, prec, dims):  # the usual tiles and the staged passes
    check(mg, prec, dims)


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("dims,pbc", [((64, 12, 1), (1, 0, 0)), ((12, 64, 1), (0, 1, 0)), ((48, 24, 3), (1, 1, 0)),
                                      ((16, 10, 8), (0, 0, 1)), ((32, 16, 4), (1, 1, 1)), ((192, 256, 4), (1, 1, 0)),
                                      ((10, 12, 6), (1, 1, 1))])
def test_circular(mg, prec, dims, pbc):
    check(mg, prec, dims, tuple(bool(q) for q in pbc))


@pytest.mark.parametrize("padding", ["PADDING_ROUND_2", "PADDING_ROUND_POT", "PADDING_SMALL_PRIME_FACTORS", "PADDING_DISABLE"])
def test_other_paddings(mg, padding):  # the tensor's layout is longer or shorter than the plan's length
    mg.enableCuda(mg.CUDA_64)
    dims = (37, 22, 3)
    rng = np.random.default_rng(5)
    M = unit_random(rng, int(np.prod(dims)))
    out = []
    for pad in (getattr(mg, padding), mg.PADDING_ROUND_4):
        T = mg.GenerateDemagTensor(*dims, *D, False, False, False, 1, pad)
        m, h = mg.VectorMatrix(dims), mg.VectorMatrix(dims)
        m.data.copy_(torch.as_tensor(M.reshape(-1)))
        mg.SymmetricMatrixVectorConvolution_FFT(T, *dims).execute(m, h)
        out.append(h.data.cpu().numpy())
    assert rel_l2(*out) < 4 * 2.0 ** -53 * 20
