"""Tensors that are handed in and are not even or odd along each axis: the plan keeps the real part of the
transform over the tensor's own lengths at frequencies kx, ky, kz >= 0 and takes the negative ky and kz by the
components' parities (the real transform along x has no negative kx).  Against numpy's FFT of the whole tensor.

Tolerance: as for the convolution of a symmetric tensor, less than 4 u log2(px py pz) of the largest part."""
import math

import numpy as np
import pytest
import torch

from helpers import rel_l2, unit_random

pytestmark = pytest.mark.gpu

ODD = [(), (0, 1), (0, 2), (), (1, 2), ()]  # axes (x, y, z) along which xx, xy, xz, yy, yz, zz are odd


def parts(N, keep):
    """N[z, y, x, 6] reduced to its parts of relative parity in `keep` (bits x, y, z)."""
    out = np.zeros_like(N)
    for c in range(6):
        own = sum(1 << a for a in ODD[c])
        for q in keep:
            p = N[..., c]
            for a in range(3):
                ax = 2 - a
                mirror = np.roll(np.flip(p, ax), 1, ax)
                p = 0.5 * (p - mirror if (own ^ q) >> a & 1 else p + mirror)
            out[..., c] += p
    return out


def field(N, M, dims):
    nx, ny, nz = dims
    ez, ey, ex = N.shape[:3]
    ky, kz = np.arange(ey), np.arange(ez)
    sy, sz = (np.where(2 * k > e, -1.0, 1.0) for k, e in ((ky, ey), (kz, ez)))
    S = []
    for c in range(6):
        s = np.fft.fftn(N[..., c]).real[np.where(sz < 0, ez - kz, kz)][:, np.where(sy < 0, ey - ky, ky), :ex // 2 + 1]
        if 1 in ODD[c]:
            s = s * sy[None, :, None]
        if 2 in ODD[c]:
            s = s * sz[:, None, None]
        S.append(s)
    F = [np.fft.rfftn(M[c].reshape(nz, ny, nx), s=(ez, ey, ex), axes=(0, 1, 2)) for c in range(3)]
    H = [np.fft.ifft(np.fft.ifft(sum(S[a] * f for a, f in zip(row, F)), axis=0), axis=1)
         for row in ((0, 1, 2), (1, 3, 4), (2, 4, 5))]
    return np.stack([np.fft.irfft(h, n=ex, axis=2)[:nz, :ny, :nx].reshape(-1) for h in H])


def run(mg, prec, dims, pbc, change):
    mg.enableCuda(mg.CUDA_64 if prec == "f64" else mg.CUDA_32)
    T = mg.GenerateDemagTensor(*dims, 3e-9, 4e-9, 2e-9, *(bool(q) for q in pbc), 2, mg.PADDING_ROUND_4)
    ex, ey, ez = T.shape[1:]
    N = change(T.data.cpu().numpy().reshape(ez, ey, ex, 6).copy())
    T.data.copy_(torch.as_tensor(N.reshape(-1)))
    M = unit_random(np.random.default_rng(7), int(np.prod(dims)))
    if prec == "f32":
        M = M.astype(np.float32).astype(np.float64)
    m, h = mg.VectorMatrix(dims), mg.VectorMatrix(dims)
    m.data.copy_(torch.as_tensor(M.reshape(-1)))
    mg.SymmetricMatrixVectorConvolution_FFT(T, *dims).execute(m, h)
    tol = 4 * 2.0 ** (-53 if prec == "f64" else -24) * math.log2(max(4, ex * ey * ez))
    return h.data.view(3, -1).cpu().numpy(), field(N, M, dims), tol


def one_sided(N):
    """Images summed on one side of the x axis only: N(+i) and N(-i) differ."""
    f = np.ones(N.shape[2])
    f[1:(N.shape[2] + 1) // 2] = 1.7
    f[(N.shape[2] + 2) // 2:] = 0.5
    return N * f[None, None, :, None]


def noise(N):
    return N + 0.05 * np.random.default_rng(3).standard_normal(N.shape)


BOXES = [((24, 20, 1), (1, 0, 0)), ((16, 12, 5), (0, 1, 0)), ((24, 20, 3), (0, 0, 0)), ((37, 22, 1), (0, 0, 0)),
         ((48, 32, 4), (1, 1, 0)), ((10, 9, 8), (0, 0, 1)), ((15, 9, 5), (1, 1, 1))]


@pytest.fixture(scope="module")
def mg():
    from micromagnum_b200 import magneto
    return magneto


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("dims,pbc", BOXES)
def test_one_sided(mg, prec, dims, pbc):
    H, ref, tol = run(mg, prec, dims, pbc, one_sided)
    assert rel_l2(H, ref) < tol


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("dims,pbc", BOXES)
@pytest.mark.parametrize("keep", [range(8), (0, 1, 2, 4, 7), (0, 3), (5,), (6, 1)])
def test_any_parity(mg, prec, dims, pbc, keep):
    H, ref, tol = run(mg, prec, dims, pbc, lambda N: parts(noise(N), keep))
    assert rel_l2(H, ref) < tol


def test_solver_takes_it():
    from micromagnum_b200 import solver as sv
    dims = (16, 12, 2)
    s0 = sv.Solver(sv.RectangularMesh(dims, (4e-9,) * 3), [sv.Material(Ms=8e5, A=0.0)], precision="f64", terms=("demag",))
    from micromagnum_b200 import magneto as mg
    mg.enableCuda(mg.CUDA_64)
    T = mg.GenerateDemagTensor(*dims, *(4e-9,) * 3, False, False, False, 1, mg.PADDING_ROUND_4)
    ex, ey, ez = T.shape[1:]
    N = one_sided(T.data.cpu().numpy().reshape(ez, ey, ex, 6).copy())
    s = sv.Solver(sv.RectangularMesh(dims, (4e-9,) * 3), [sv.Material(Ms=8e5, A=0.0)], precision="f64", terms=("demag",), tensor=N.reshape(-1))
    M = unit_random(np.random.default_rng(2), int(np.prod(dims))) * 8e5
    for q in (s0, s):
        q.M = M
    assert rel_l2(s.eval()[2].cpu().numpy(), field(N, M, dims)) < 4 * 2.0 ** -53 * math.log2(ex * ey * ez)
    assert rel_l2(s.eval()[2].cpu().numpy(), s0.eval()[2].cpu().numpy()) > 1e-3
