"""norm2 and scale over whole registers: every float class in complex64 (subnormals, zeros,
infinities, NaN), odd and single-word sizes, both storage types."""
import numpy as np
import pytest

from openqarp_b200 import Register

pytestmark = pytest.mark.gpu


def _filled(n, dtype, amps):
    reg = Register(n, dtype)
    reg.set_state(amps, validate=False)
    return reg


@pytest.mark.parametrize("dtype", ["complex128", "complex64"])
@pytest.mark.parametrize("n", [0, 1, 2, 9, 10, 13])
def test_norm_and_scale_against_numpy(dtype, n):
    """Sums of 2^(n+1) squares in float64, any order: within 2^(n+1) roundings of 2^-53 (and exact
    products of floats).  Scaling forms the product in float64 and rounds once to the storage type."""
    rng = np.random.default_rng(n)
    a = (rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)) * 10.0 ** rng.uniform(-18, 18, 1 << n)
    a = a.astype(dtype)
    part = np.float64 if dtype == "complex128" else np.float32
    reg = _filled(n, dtype, a)
    try:
        want = float(np.sum(a.real.astype(np.longdouble) ** 2 + a.imag.astype(np.longdouble) ** 2))
        assert abs(reg.norm2() - want) <= want * (2 << n) * 2.0 ** -53
        f = 1.0 + 1e-9
        reg.scale(f)
        want = (a.real.astype(np.float64) * f).astype(part) + 1j * (a.imag.astype(np.float64) * f).astype(part)
        np.testing.assert_array_equal(reg.get_state(), want.astype(np.complex128))
    finally:
        reg.close()


@pytest.mark.parametrize("where", [0, 1, 700, 1023])
def test_complex64_norm_of_special_values(where):
    """Zeros give exactly 0, subnormal floats their exact squares, an infinity infinity, a NaN NaN."""
    n = 10
    for value, want in ((0.0, 0.0), (2.0 ** -149, 2.0 ** -298), (2.0 ** -127, 2.0 ** -254), (-(2.0 ** 127), 2.0 ** 254),
                        (np.inf, np.inf), (-np.inf, np.inf), (np.nan, np.nan)):
        for amp in (complex(value, 0.0), complex(0.0, value)):
            a = np.zeros(1 << n, dtype=np.complex128)
            a[where] = amp
            reg = _filled(n, "complex64", a)
            try:
                got = reg.norm2()
            finally:
                reg.close()
            assert got == want or (np.isnan(want) and np.isnan(got)), (value, got)
