"""Batch members large enough to run their convolution as passes of their own, beside a small grouped member,
with a mask: the same bits alone and in the mix, and the single-instance FP64 solver's trajectory.

Tolerances: FP64, the rounding of a few adaptive steps from a random state; FP32 (deviation form) against FP64,
about a hundred roundings of 2^-24 per step."""
import numpy as np
import pytest

from helpers import rel_l2, unit_random

pytestmark = pytest.mark.gpu

D, MS, A, T_END, H0 = (4e-9,) * 3, 8e5, 1.3e-11, 6e-14, 2e-14


def member(q, seed):
    from micromagnum_b200.batch import Instance
    y, x = np.mgrid[0:q[1], 0:q[0]]
    m = ((x + 0.5) / q[0] - 0.5) ** 2 + ((y + 0.5) / q[1] - 0.5) ** 2 <= 0.25
    mask = np.broadcast_to(m, q[::-1]).reshape(-1).astype(np.uint8)
    M = unit_random(np.random.default_rng(seed), int(np.prod(q))) * MS * mask
    return Instance(q, D, MS, A, 0.5, mask=mask, t_end=T_END), M


def run(members, prec):
    from micromagnum_b200.batch import Batch
    b = Batch([], precision=prec, h0=H0)
    slots = [b.add(q, M) for q, M in members]
    b.relax()
    assert all(b.results()[k]["status"] == 1 for k in slots)
    return [b.get_M(k).cpu().numpy() for k in slots]


@pytest.mark.parametrize("prec,dims,tol", [("f64", (512, 200, 4), 1e-10), ("f64", (500, 208, 4), 1e-10),
                                           ("f32", (512, 400, 4), 2e-5), ("f32", (500, 401, 4), 2e-5)])
def test_large_member(prec, dims, tol):
    from micromagnum_b200 import solver as sv
    large, small = member(dims, 1), member((40, 33, 2), 2)
    mixed, alone = run([small, large], prec), run([large], prec)
    assert np.array_equal(mixed[1], alone[0])
    assert np.array_equal(mixed[0], run([small], prec)[0])
    q, M = large
    s = sv.Solver(sv.RectangularMesh(dims, D), [sv.Material(), sv.Material(Ms=MS, A=A, alpha=0.5)], regions=q.mask,
                  precision="f64", h0=H0)
    s.M = M
    while s.t < T_END - 1e-22:  # the batch's step sequence: its last step is shortened and checked like any other
        h = s.stats["h_next"]
        if s.t + h > T_END:
            s.set_time(s.t, T_END - s.t)
        s.step()
    assert rel_l2(mixed[1], s.M.cpu().numpy()) < tol
