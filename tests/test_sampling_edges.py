"""Seeded terminal sampling on the device: the uniforms' engine at the edges of its twists (312 shots
each), half-warp searches with the last half partly empty, registers below one chunk, of one chunk and
of several, chunks of probability zero, and uniforms in any order."""
import numpy as np
import pytest

# the search compares u with FP64 cumulative sums: an index may differ from the sequential oracle's
# only where u lies within the sums' rounding (2^n * 2^-53) of a boundary
TIE = 1e-10


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["complex128", "complex64"])
@pytest.mark.parametrize("n,shots", [(0, 3), (1, 1), (5, 17), (11, 312), (12, 313), (13, 1000), (17, 2500)])
def test_seeded_shots_match_oracle(restatement, n, shots, dtype):
    from openqarp_b200 import Register, uniforms
    rng = np.random.default_rng([n, shots])
    a = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    if n == 17:                              # whole chunks without probability, first and last among them
        a.reshape(32, -1)[[0, 3, 4, 5, 30, 31]] = 0
    reg = Register(n, dtype)
    reg.set_state(a / np.linalg.norm(a))
    psi = reg.get_state()
    seed = 9000 + n
    u = uniforms(seed, shots)
    got = reg.sample_seeded(seed, shots)
    np.testing.assert_array_equal(got, reg.sample(u))
    order = rng.permutation(shots)
    np.testing.assert_array_equal(reg.sample(u[order]), got[order])
    want, cp = restatement.sample(psi, n, u, with_cdf=True)
    for k in np.flatnonzero(got != want):
        assert abs(cp[min(got[k], want[k])] - u[k]) < TIE
    odd = reg.sample_parities(seed, shots, [1, (1 << n) - 1] if n else [])
    for m, c in zip([1, (1 << n) - 1], odd):
        assert c == sum(bin(int(i) & m).count("1") & 1 for i in got)
    reg.close()


@pytest.mark.gpu
def test_device_uniforms_pick_every_index_of_a_uniform_register():
    """|a|^2 = 2^-n exactly: index = ceil(u 2^n) - 1, so the indices give back the uniforms' leading
    bits over many twists."""
    from openqarp_b200 import Register, uniforms
    n, shots = 16, 40000
    reg = Register(n)
    reg.set_state(np.full(1 << n, 2.0 ** (-n / 2)))
    for seed in (0, 1, 0xFFFFFFFF):
        u = uniforms(seed, shots)
        np.testing.assert_array_equal(reg.sample_seeded(seed, shots), np.maximum(np.ceil(u * 2 ** n), 1).astype(np.uint64) - 1)
    reg.close()
