"""<psi|H|psi> of real Pauli sums at the edges of its paths: the first tiled width, one tile and a
few, both sides of the width where partners come from shared memory, groups on lane, warp, slot and
outside qubits, odd numbers of Ys, one-group sums, and the general path where a coefficient is
complex."""
import numpy as np
import pytest


def _rows(n, seed):
    rng = np.random.default_rng([n, seed])
    rows = [(0, 0, 0.7), (0, (1 << n) - 1, -0.3), ((1 << n) - 1, 0, 0.4), ((1 << n) - 1, (1 << n) - 1, 0.9)]
    for q in range(n):                       # X, Y and XZ on every qubit: lanes, warps, slots, outside
        rows += [(1 << q, 0, 0.5), (1 << q, 1 << q, -0.8), (1 << q, 1 << ((q + 1) % n), 0.2)]
    for _ in range(60):                      # weight <= 4
        s = rng.choice(n, size=int(rng.integers(1, 5)), replace=False)
        l = rng.integers(1, 4, len(s))
        rows.append((sum(1 << int(q) for q, c in zip(s, l) if c < 3), sum(1 << int(q) for q, c in zip(s, l) if c > 1),
                     float(rng.normal())))
    for _ in range(12):                      # full weight
        rows.append((int(rng.integers(0, 1 << n)), int(rng.integers(0, 1 << n)), float(rng.normal())))
    return rows


def _masks(rows):
    from openqarp_b200 import PauliMasks
    c = np.zeros(2 * len(rows))
    c[0::2] = [complex(r[2]).real for r in rows]
    c[1::2] = [complex(r[2]).imag for r in rows]
    return PauliMasks(np.array([r[0] for r in rows], dtype=np.uint64), np.array([r[1] for r in rows], dtype=np.uint64), c)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["complex128", "complex64"])
@pytest.mark.parametrize("n", [11, 12, 13, 15, 21, 22])
def test_energy_matches_oracle(restatement, n, dtype):
    from openqarp_b200 import Register
    rng = np.random.default_rng(n)
    a = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    reg = Register(n, dtype)
    reg.set_state(a / np.linalg.norm(a))
    psi = reg.get_state()
    rows = _rows(n, 5)
    for part in (rows, rows[:1], rows[2:3], rows[5:6], [(r[0], r[1], r[2] * (1 - 0.5j)) for r in rows[:40]]):
        m = _masks(part)
        got, want = reg.expectation(m), restatement.transition(psi, psi, n, m)
        # |<P>| <= 1: 2^n-term FP64 sums of rounded products stay below 1e-13 per unit of coefficient
        assert abs(got - want) < 1e-12 * sum(abs(r[2]) for r in part)
    reg.close()


@pytest.mark.gpu
def test_transition_between_registers_keeps_both_states(restatement):
    from openqarp_b200 import Register
    n = 13
    rng = np.random.default_rng(3)
    a, b = (rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n) for _ in range(2))
    ra, rb = Register(n), Register(n)
    ra.set_state(a, validate=False)
    rb.set_state(b, validate=False)
    m = _masks(_rows(n, 6))
    want = restatement.transition(a, b, n, m)
    assert abs(ra.transition(rb, m) - want) < 1e-12 * np.linalg.norm(a) * np.linalg.norm(b) * np.abs(m.coeff).sum()
    ra.close()
    rb.close()
