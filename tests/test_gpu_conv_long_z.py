"""Boxes of more than 32 layers, whose z passes are of the mixed-radix form: lengths of the plan's choice along x, y
and z against numpy's FFT at the tensor's lengths; and the time of an awkward number of layers (68 = 4 * 17 points)
against that of more layers of a smooth one."""
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
@pytest.mark.parametrize("dims", [(20, 18, 33), (100, 30, 34), (30, 70, 65), (33, 33, 37), (140, 20, 40), (12, 9, 101), (5, 5, 131)])
def test_long_z(mg, prec, dims):
    check(mg, prec, dims)


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("dims,pbc", [((50, 40, 33), (0, 0, 1)), ((65, 20, 11), (0, 0, 1)), ((16, 50, 34), (1, 0, 0)),
                                      ((70, 30, 5), (0, 1, 1))])
def test_periodic(mg, prec, dims, pbc):
    check(mg, prec, dims, tuple(bool(q) for q in pbc))


@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_awkward_layers(mg, prec):
    def time(nz):
        mg.enableCuda(mg.CUDA_64 if prec == "f64" else mg.CUDA_32)
        dims = (140, 140, nz)
        T = mg.GenerateDemagTensor(*dims, *(4e-9,) * 3, False, False, False, 1, mg.PADDING_ROUND_4)
        m, h = mg.VectorMatrix(dims), mg.VectorMatrix(dims)
        m.data.copy_(torch.as_tensor(np.random.default_rng(0).standard_normal(3 * int(np.prod(dims)))))
        conv = mg.SymmetricMatrixVectorConvolution_FFT(T, *dims)
        best = []
        for _ in range(12):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            conv.execute(m, h)
            b.record()
            torch.cuda.synchronize()
            best.append(a.elapsed_time(b))
        return min(best)

    assert time(34) < 1.3 * time(40)
