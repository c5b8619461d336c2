"""`attempt` waits for nothing: calls that follow while it is still pending (held back by a sleeping kernel on
the stream) give the bits that they give after a wait."""
import numpy as np
import pytest
import torch

from helpers import unit_random

pytestmark = pytest.mark.gpu

DIMS, D, MS = (48, 20, 2), (4e-9,) * 3, 8e5


def run(prec, what, wait):
    from micromagnum_b200 import solver as sv
    s = sv.Solver(sv.RectangularMesh(DIMS, D), [sv.Material(Ms=MS, A=1.3e-11, alpha=0.1)], precision=prec, h0=1e-14)
    s.M = unit_random(np.random.default_rng(3), int(np.prod(DIMS))) * MS
    torch.cuda._sleep(4_000_000)
    for h in (3e-14, 2e-15):
        s.attempt(h)
        if wait:
            torch.cuda.synchronize()
    if what == "step":
        s.step()
    elif what == "clamped":
        s.step(4e-15)
    else:
        s.solve(4e-14)
    torch.cuda.synchronize()
    q = s.stats
    return s.M.cpu().numpy(), [q[k] for k in ("t", "h", "h_next", "steps", "attempts", "rejected", "last_error")]


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("what", ["step", "clamped", "solve"])
def test_pending_attempt(prec, what):
    m, q = run(prec, what, False)
    m0, q0 = run(prec, what, True)
    assert q == q0
    assert np.array_equal(m, m0)
    assert np.abs(np.linalg.norm(m, axis=0) / MS - 1).max() < 1e-6
