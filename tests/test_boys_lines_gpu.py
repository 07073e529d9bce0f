"""GPU test of the Boys row tables at the places where a class's evaluation changes: the
line between table and asymptote (36 for M = 0, up to 71 for M = 12), the last rows
below it and the rows past the plain table's end at 36, against mpmath."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from test_boys_gpu import _boys_mp  # noqa: E402

LINES = [36, 40, 44, 47, 50, 53, 56, 59, 61, 64, 66, 69, 71]


@pytest.mark.parametrize("M", range(13))
def test_boys_rows_at_the_lines(M):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from quick_b200._native import check, lib
    from quick_b200.basis import build_basis
    from quick_b200.get2e import Get2e
    from quick_b200.molecules import water_cluster
    L = lib()
    if M > 4 * L.qk_max_l():
        pytest.skip("M above the compiled maximum")
    t = float(LINES[M])
    T = np.concatenate([[0.0, 1.0 / 64, np.nextafter(1.0 / 64, 1), 0.024999, 0.025001, np.nextafter(t, 0), t, t + 1e-9,
                         t - 0.0249, t - 0.0251, t - 1.0 / 64, 35.99, 36.01], np.linspace(30.0, 80.0, 41)])
    eng = Get2e(build_basis(water_cluster(1, 3.0), "STO-3G"))
    n = len(T)
    Fr, F1 = np.zeros((n, M + 1)), np.zeros((n, M + 1))
    P = lambda a: ctypes.c_void_p(a.ctypes.data)  # noqa: E731
    check(L.qk_boys(ctypes.c_void_p(eng.h), M, P(T), n, P(Fr), P(F1)), "qk_boys")
    eng.close()
    for i, x in enumerate(T):
        for m in range(M + 1):
            ref = float(_boys_mp(m, float(x)))
            # a table value at 1.5e-15 (M = 12) and at most 2M + 2 roundings of a recursion
            assert abs(Fr[i, m] - ref) <= (1.5e-15 + (2 * M + 2) * 1.2e-16) * ref, (M, m, x)


def _boys_rows(M, T):
    """F_0..F_M at every T by the per-lane kernels' evaluation, one row per T."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from quick_b200._native import check, lib
    from quick_b200.basis import build_basis
    from quick_b200.get2e import Get2e
    from quick_b200.molecules import water_cluster
    L = lib()
    if M > 4 * L.qk_max_l():
        pytest.skip("M above the compiled maximum")
    eng = Get2e(build_basis(water_cluster(1, 3.0), "STO-3G"))
    n = len(T)
    Fr, F1 = np.zeros((n, M + 1)), np.zeros((n, M + 1))
    P = lambda a: ctypes.c_void_p(a.ctypes.data)  # noqa: E731
    check(L.qk_boys(ctypes.c_void_p(eng.h), M, P(T), n, P(Fr), P(F1)), "qk_boys")
    eng.close()
    return Fr


@pytest.mark.parametrize("M", range(13))
def test_boys_rows_at_the_end_of_the_range(M):
    """F_m = (2m-1)!!/(2T)^m sqrt(pi/T)/2 to where T overflows; at infinity every F_m is 0, as its limit is."""
    T = np.array([1e10, 1e100, 1e200, 1e300, 8.9e307, 9.1e307, 1.7e308, np.inf])
    Fr = _boys_rows(M, T)
    assert np.all(Fr[-1] == 0.0)
    assert np.all(np.isfinite(Fr))
    with np.errstate(under="ignore", over="ignore"):
        want = np.sqrt(np.pi / T) / 2
        for m in range(M + 1):
            # rsqrt is good to 2^-52, its factor and product add two roundings; a step has two and 1/(2T) to
            # two; products under 2^-1022 lose digits
            assert np.all(np.abs(Fr[:, m] - want) <= (4 + 4 * m) * 2.0 ** -53 * want + m * 2.0 ** -1022), m
            want = want * ((2 * m + 1) / (2 * T))


@pytest.mark.parametrize("M", [6, 8, 10, 12])
def test_boys_rows_low_orders_keep_their_precision(M):
    """The downward recursion may add one rounding a step to F_0, no more."""
    T = np.random.default_rng(M).uniform(0.0, 90.0, 8000)
    t, ref = T.astype(np.longdouble), np.zeros(len(T), dtype=np.longdouble)
    term = np.ones(len(T), dtype=np.longdouble)
    for j in range(1, 500):   # exp(T) F_0 = sum (2T)^j / (2j+1)!!
        ref += term
        term = term * (2 * t / (2 * j + 1))
    ref *= np.exp(-t)
    rms = float(np.sqrt(np.mean(((_boys_rows(M, T)[:, 0] - ref) / ref).astype(float) ** 2)))
    # a rounding's relative error is 4.71e-17 rms (uniform in the last place, significands
    # spread over their logarithm); the M steps and at most seven others: the table, the
    # interpolation's last steps, the scale
    assert rms <= 4.71e-17 * (M + 7) ** 0.5, rms
