"""Several batch members that run their convolution as passes of their own, with and without grouped ones beside
them, stopping at different times: each the same bits as alone.  That they run so shows in the launches of a
round: members of one size share the grouped launches, while each of these brings its own."""
import numpy as np
import pytest

from helpers import unit_random

pytestmark = pytest.mark.gpu

D, MS, A, H0 = (4e-9,) * 3, 8e5, 1.3e-11, 2e-14
LARGE = {"f32": (640, 512, 4), "f64": (512, 400, 4)}  # 1.6 and 2 times the line
SMALL = (40, 33, 2)


def member(dims, seed, t_end):
    from micromagnum_b200.batch import Instance
    return Instance(dims, D, MS, A, 0.5, t_end=t_end), unit_random(np.random.default_rng(seed), int(np.prod(dims))) * MS


def run(members, prec):
    from micromagnum_b200.batch import Batch
    b = Batch([], precision=prec, h0=H0)
    slots = [b.add(q, M) for q, M in members]
    b.relax()
    res = b.results()
    assert all(res[k]["status"] == 1 for k in slots)
    out = [(b.get_M(k).cpu().numpy(), res[k]["t"], res[k]["attempts"]) for k in slots], b.launches_per_round()
    b.close()
    return out


@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_own_launches(prec):
    launches = lambda dims, k: run([member(dims, i, 3e-14) for i in range(k)], prec)[1]  # noqa: E731
    one, two, five = (launches(LARGE[prec], k) for k in (1, 2, 5))
    assert two[1] > one[1] and five[1] - two[1] == 3 * (two[1] - one[1])
    assert launches(SMALL, 1) == launches(SMALL, 5)


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("large,small", [(2, 0), (2, 1), (5, 0), (5, 2)])
def test_same_bits_as_alone(prec, large, small):
    ends = [2e-14, 9e-14, 5e-14, 1.2e-13, 3e-14]
    members = [member(LARGE[prec], i, ends[i]) for i in range(large)] + [member(SMALL, 10 + i, ends[i + 1]) for i in range(small)]
    mixed, _ = run(members, prec)
    for q, got in zip(members, mixed):
        alone = run([q], prec)[0][0]
        assert got[1:] == alone[1:]
        assert np.array_equal(got[0], alone[0])
