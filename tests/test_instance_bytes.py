"""The device bytes that a request is charged are those that its set-up allocates: the octant of the tensor and two
half spectra (FP64) and the twiddles for a while, the working-precision tensor, spectra, vectors and twiddle tables to
stay (host-only)."""
import pytest

from micromagnum_b200.batch import Instance


def pot(n):
    p = 1
    while p < 2 * n - 1:
        p *= 2
    return p


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("dims", [(1024, 1024, 4), (40, 33, 2), (300, 17, 1)])
def test_bytes(prec, dims):
    nx, ny, nz = dims
    n, s = nx * ny * nz, 4 if prec == "f32" else 8
    px, py, pz = pot(nx), pot(ny), max(2, pot(nz))
    hx, qy, qz = px // 2 + 1, py // 2 + 1, pz // 2 + 1
    res, trans = Instance(dims, (4e-9,) * 3, 8e5, 1.3e-11, 0.5).device_bytes(prec)
    assert trans == 48 * (n + hx * ny * nz + hx * qy * nz) + 16 * (px + py + pz)
    tensor, vectors = 6 * hx * qy * qz * s, (13 if prec == "f32" else 11) * 3 * n * s + n
    spectra, twiddles = 3 * nz * py * hx * 2 * s, 3 * (px + py + pz) * 2 * s
    least = vectors + spectra + tensor + twiddles
    assert least <= res <= least + tensor + spectra / hx * 4 + (1 << 16)  # (a second tensor copy, rows rounded up)
