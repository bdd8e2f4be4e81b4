"""The kernels' seeded and integer-pipe arithmetic over the whole exponent range,
on the GPU, against the IEEE operations (gb300_check_kernel_math): the bit-exact
mode's quotients and limited slopes, the mixed form's flux differences and
conversions, the totals' sums of eight, and the reciprocal seed.

Bounds: quotients, slopes, differences and conversions are the operations' bits.
A sum of eight is off by what it drops and one rounding (the kernel's test).
The seed's correction is rounded to 2^-43 of a reciprocal between 1/2 and 1, so
to 2^-43 of it at most, and its FP32 steps and the six mantissa bits it leaves
out take a quarter of that together: below 2^-42.  A Newton step squares that, so
the reciprocal misses the IEEE one only within 2^-84 of a tie, by one unit."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

N = 1 << 24


@pytest.mark.parametrize("seed", [1, 20261205])
def test_kernel_math_matches_ieee(seed):
    import flow_gb300 as fg
    counts = (ctypes.c_longlong * 6)()
    ulp = ctypes.c_longlong()
    err = ctypes.c_double()
    assert fg.lib().gb300_check_kernel_math(N, seed, counts, ctypes.byref(ulp),
                                            ctypes.byref(err)) == 0
    c = list(counts)
    print("mismatches", c, "max ulp", ulp.value, "seed rel err", err.value)
    assert c[:5] == [0, 0, 0, 0, 0], c
    assert c[5] <= N * 1e-6 and ulp.value <= 1, (c, ulp.value)
    assert err.value < 2.0 ** -42, err.value
