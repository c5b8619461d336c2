"""The demag tensor where the offsets next to the origin take their own kernel: flat and long cells,
whose quadrature orders stay high over many cells (past the table for the nearest), against the exact
(binary128 Newell) tensor; and the solver's own octant of it against the padded tensor handed in."""
import numpy as np
import pytest
import torch

from helpers import rel_l2, unit_random

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,d", [((12, 3, 2), (1e-9, 1e-9, 40e-9)), ((40, 1, 1), (2e-9, 2e-9, 2e-9)),
                                    ((2, 2, 2), (3e-9, 3e-9, 3e-9)), ((1, 1, 1), (1e-9, 2e-9, 3e-9)),
                                    ((24, 20, 2), (2e-9, 2e-9, 20e-9)), ((3, 30, 4), (50e-9, 2e-9, 3e-9))])
def test_tensor_flat_cells_vs_exact(oracle_mod, dims, d):
    from micromagnum_b200 import magneto as mg
    ref, pd = oracle_mod.demag_tensor(*dims, *d)
    T = mg.GenerateDemagTensor(*dims, *d, False, False, False, 1, mg.PADDING_ROUND_4)
    assert T.shape == (6,) + pd
    N = T.data.cpu().numpy()
    # Quadrature is good to about 1e-15 of an entry (1e-12 is the bound of the tensor test on ordinary cells).  Newell's
    # second difference sums 27 values (|weights| adding up to 64) of f, at most (asinh(L / s) + 1/3) L^3 for a longest
    # and a shortest edge L and s, and divides by 4 pi V: rounding each to 2^-53 leaves 64 / (4 pi) times that, over V,
    # in an entry, whose own size is of order 1/3.
    L, s, V = max(d), min(d), d[0] * d[1] * d[2]
    bound = 1e-12 + 3 * 64 / (4 * np.pi) * (np.arcsinh(L / s) + 1 / 3) * 2.0 ** -53 * L ** 3 / V
    assert np.abs(N - ref).max() < bound * np.abs(ref).max()
    assert rel_l2(N, ref) < bound


@pytest.mark.parametrize("prec,tol", [("f64", 1e-13), ("f32", 1e-6)])
@pytest.mark.parametrize("dims", [(20, 12, 1), (17, 9, 5), (64, 33, 2)])
def test_solver_octant_vs_given_tensor(prec, tol, dims):
    from micromagnum_b200 import magneto as mg, solver as sv
    d = (3e-9, 4e-9, 5e-9)
    T = mg.GenerateDemagTensor(*dims, *d, False, False, False, 1, mg.PADDING_ROUND_4)
    M = unit_random(np.random.default_rng(3), int(np.prod(dims))) * 8e5
    H = []
    for tensor in (None, T.data):
        s = sv.Solver(sv.RectangularMesh(dims, d), [sv.Material(Ms=8e5, A=1.3e-11, alpha=0.1)], terms=("demag",),
                      precision=prec, tensor=tensor)
        s.M = M
        H.append(s.eval()[2].cpu().numpy())
    assert rel_l2(*H) < tol
