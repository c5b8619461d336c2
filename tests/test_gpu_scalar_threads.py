"""Calls that return a scalar, made by several threads at once: each gets its own result, also when hundreds of
other calls begin and end while it is under way.

Tolerance: FP64 sums of n equal terms in another order, n * 2^-53."""
import ctypes
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu

F64 = 0


def norm(y, yerr, stream):
    """sqrt(mean((yerr / (1 + y))^2)) by mm_rk_scaled_error_norm"""
    from micromagnum_b200 import _lib
    out = ctypes.c_double()
    n = y.numel() // 3
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    _lib.check(_lib.lib().mm_rk_scaled_error_norm(F64, n, 1.0, 0.0, p(y), p(yerr), ctypes.byref(out),
                                                  ctypes.c_void_p(stream.cuda_stream)))
    return out.value


def fields(n, value):
    return torch.zeros(3 * n, dtype=torch.float64, device="cuda"), torch.full((3 * n,), value, dtype=torch.float64, device="cuda")


@pytest.mark.parametrize("between", [0, 63, 64, 255, 256])
def test_long_call_beside_short_ones(between):
    n = 1 << 21
    a, b, small = fields(n, 3.0), fields(n, 5.0), fields(5, 7.0)
    sa, sb, sc = (torch.cuda.Stream() for _ in range(3))
    torch.cuda.synchronize()
    asleep = torch.cuda.Event()
    with torch.cuda.stream(sa):
        torch.cuda._sleep(60_000_000)
        asleep.record()
    got = {}
    ta = threading.Thread(target=lambda: got.update(a=norm(*a, sa)))
    ta.start()
    for _ in range(between):
        assert norm(*small, sc) == pytest.approx(7.0, rel=1e-12)
    sb.wait_event(asleep)  # both long reductions start together
    got["b"] = norm(*b, sb)
    ta.join()
    assert got["a"] == pytest.approx(3.0, rel=3 * n * 2.0 ** -53) and got["b"] == pytest.approx(5.0, rel=3 * n * 2.0 ** -53)


def test_many_threads():
    bad = []

    def work(k):
        torch.cuda.set_device(0)
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            f = fields(1000 * (k + 1), float(k + 1))
        s.synchronize()
        for _ in range(300):
            v = norm(*f, s)
            if abs(v - (k + 1)) > 1e-9:
                bad.append((k, v))

    th = [threading.Thread(target=work, args=(k,)) for k in range(12)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not bad
