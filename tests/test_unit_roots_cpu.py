"""The twiddle factors of the FP64 line pass: every value within half a unit in
the last place of the exact one (long double, which errs by 2^-11 of that), the
axes and diagonals exactly symmetric."""
import ctypes as C

import numpy as np
import pytest


@pytest.mark.parametrize("n", [64, 128, 256, 512, 1024])
def test_every_root_is_the_nearest_double(conan, n):
    if np.finfo(np.longdouble).nmant < 63:
        pytest.skip("needs an 80-bit long double")
    w = np.empty(2 * n)
    fn = C.CDLL(str(conan._lib.LIB_PATH))._ZN5conan10unit_rootsEiPd
    fn(C.c_int(n), w.ctypes.data_as(C.c_void_p))
    # reduced to the first octant, where the angle's rounding is below 2^-64
    k = np.arange(n)
    q, r = k // (n // 4), k % (n // 4)
    hi = r > n // 8
    pi = np.longdouble("3.14159265358979323846264338327950288")
    a = 2 * pi * np.where(hi, n // 4 - r, r).astype(np.longdouble) / n
    c, s = np.where(hi, np.sin(a), np.cos(a)), np.where(hi, np.cos(a), np.sin(a))
    re = np.choose(q, [c, -s, -c, s])
    im = np.choose(q, [-s, -c, s, c])
    for got, ref in ((w[0::2], re), (w[1::2], im)):
        ulp = np.spacing(np.abs(ref.astype(np.float64)))
        assert np.all(np.abs(got - ref) <= ulp * (0.5 + 2.0 ** -10))
    z = w[0::2] + 1j * w[1::2]
    assert z[0] == 1 and z[n // 4] == -1j and z[n // 2] == -1 and z[3 * n // 4] == 1j
    assert -z[n // 8].imag == z[n // 8].real == z[7 * n // 8].imag
    # what cos and sin of the rounded angle give is outside that bound
    old = np.cos(-2.0 * np.pi * k / n)
    assert np.any(np.abs(old - re) > np.spacing(np.abs(re.astype(np.float64))) * 2)
