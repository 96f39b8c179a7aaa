"""Registers held in one block's shared memory: gates and controls at every qubit place against the
gate-by-gate kernels, adjoint steps of every kind in the circuit batches' width classes, and shots
whose random engine runs through several generations."""
import numpy as np
import pytest

from openqarp_b200 import Command, GateType, Param, Register, circuits, ir, observable

pytestmark = pytest.mark.gpu


def _mixed(n, rng):
    """Dense and controlled gates, diagonals, Pauli rotations and swaps over random qubits."""
    G = GateType
    cmds = [Command(G.H, (q,)) for q in range(n)]
    for _ in range(12):
        q = [int(v) for v in rng.permutation(n)]
        a = rng.uniform(-3, 3, 4)
        cmds += [Command(G.U, (q[0],), tuple(a[:3])), Command(G.Rz, (q[-1],), (a[3],))]
        if n > 1:
            cmds += [Command(G.CX, (q[0], q[1])), Command(G.RXX, (q[1], q[0]), (a[0],)), Command(G.P, (q[1],), (a[1],)),
                     Command(G.SWAP, (q[0], q[-1])), Command(G.RZZ, (q[0], q[1]), (a[2],))]
        if n > 2:
            cmds += [Command(G.CCX, (q[2], q[0], q[1])), Command(G.CSWAP, (q[1], q[2], q[0]))]
        if n > 4:
            cmds.append(Command(G.MCZ, tuple(q[:5])))
    return cmds


@pytest.mark.parametrize("width", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("n", [1, 2, 3, 5, 9, 10, 12])
@pytest.mark.parametrize("dtype", ["complex128", "complex64"])
def test_gate_sequences_against_single_gates(dtype, n, width):
    """A stream of many gates runs in shared memory, streams of one gate each in the general
    kernels.  Roughly 150 gates, each within 4 roundings of its amplitudes: 600 eps, with eps of
    the register's type (complex64 stores round, double arithmetic)."""
    cmds = _mixed(n, np.random.default_rng(100 * n + width))
    a, b = Register(n, dtype), Register(n, dtype)
    try:
        a.configure(width, 0)
        a.apply(ir.pack(cmds).buf)
        for c in cmds:
            b.apply(ir.pack([c]).buf)
        tol = 600 * (2.0 ** -52 if dtype == "complex128" else 2.0 ** -23)
        np.testing.assert_allclose(a.get_state(), b.get_state(), rtol=0, atol=tol)
    finally:
        a.close()
        b.close()


def test_batch_classes_with_every_adjoint_kind(restatement):
    """One- and two-qubit parameters (adjoint steps on one and two qubits), fixed and controlled
    gates between them, in every width class: 1..9, 10..11, 12 and above."""
    from openqarp_b200.batch import CircuitBatch
    G, rng = GateType, np.random.default_rng(3)
    insts = []
    for n in (1, 2, 3, 9, 10, 11, 12, 13):
        cmds, names = [], []

        def sym():
            names.append(f"t{len(names)}")
            return Param.symbol(names[-1])
        for _ in range(2):
            cmds += [Command(G.Ry, (q,), (sym(),)) for q in range(n)]
            cmds += [Command(G.RXX, (q, (q + 3) % n), (sym(),)) for q in range(n) if (q + 3) % n != q]
            cmds += [Command(G.CX, (q + 1, q)) for q in range(n - 1)]
            cmds += [Command(G.CCX, (0, q, q + 1)) for q in range(1, n - 1)]
            cmds += [Command(G.RZZ, (n - 1, q), (sym(),)) for q in range(n - 1)]
            cmds.append(Command(G.GPhase, (), (sym(),)))
        obs = circuits.random_pauli_sum(n, 10, seed=n, max_weight=min(3, n))
        insts.append((cmds, n, obs, dict(zip(names, rng.uniform(-3, 3, len(names)))), names))
    b = CircuitBatch(with_gradient=True)
    try:
        for inst in insts:
            b.add(*inst)
        energies, grads, _ = b.run()
        for j, (cmds, n, obs, vals, names) in enumerate(insts):
            e, g = restatement.adjoint(ir.pack(cmds, vals, names), n, len(names), observable.to_masks(obs, n))
            assert abs(energies[j] - e) < 1e-10, (n, energies[j], e)
            np.testing.assert_allclose(grads[j], g, rtol=0, atol=1e-10, err_msg=f"n={n}")
    finally:
        b.close()


@pytest.mark.parametrize("n", [5, 9, 13, 16])
def test_engine_generations(n):
    """700 measurements of a fresh |+> per shot, 1400 words of the shot's mt19937: two generations
    and a part.  Each outcome is 1 exactly where the drawn uniform reaches p0 = 1/2 (a uniform
    within rounding of 1/2 is not among these seeds' draws)."""
    count, shots, seed = 700, 6, 77
    cmds = []
    for m in range(count):
        cmds += [Command(GateType.H, (1,)), Command(GateType.Measure, (1,), (), None, (m % 63,)),
                 Command(GateType.X, (1,), (), None, (), (m % 63,), (True,))]
    want = np.zeros(shots, dtype=np.uint64)
    for s in range(shots):
        words = np.random.RandomState(seed + s).randint(0, 2 ** 32, size=2 * count, dtype=np.uint32).astype(np.float64)
        u = (words[0::2] + words[1::2] * 2.0 ** 32) * 2.0 ** -64
        assert np.min(np.abs(u - 0.5)) > 1e-9
        for m in range(count):
            bit = np.uint64(1) << np.uint64(m % 63)
            want[s] = (want[s] | bit) if u[m] >= 0.5 else (want[s] & ~bit)
    reg = Register(n)
    try:
        _, regs, _ = reg.run_trajectories(ir.pack(cmds).buf, seed, shots)
    finally:
        reg.close()
    np.testing.assert_array_equal(regs, want)


@pytest.mark.parametrize("n,noisy,around", [(10, True, 441), (9, False, 815)])
def test_plans_that_just_fill_a_block(n, noisy, around):
    """Gates under alternating conditions (a step of 176 bytes each: a record and a 2 x 2 matrix), as many
    as fill a block's shared memory beside eight shots, and a few more and fewer: each plan runs, with
    the outcomes of the executor that keeps its shots in device memory."""
    from openqarp_b200 import NoiseModel
    shots, seed, G = 1300, 5, GateType
    for count in range(around - 10, around + 11):
        cmds = [Command(G.H, (q,)) for q in range(n)] + [Command(G.U, (0,), (0.7, 0.1, 0.4)),
                                                        Command(G.Measure, (0,), (), None, (0,))]
        cmds += [Command(G.X, (1 + i % (n - 1),), (), None, (), (0,), (i % 2 == 0,)) for i in range(count)]
        buf, got = ir.pack(cmds).buf, []
        for batch in (0, 512):
            reg = Register(n)
            try:
                reg.set_trajectory_batch(batch)
                if noisy:
                    reg.set_noise(NoiseModel.amplitude_damping(0.2, ["U"]))
                got.append(reg.run_trajectories(buf, seed, shots)[:2])
            finally:
                reg.close()
        np.testing.assert_array_equal(got[0][1], got[1][1])
        # a draw within rounding of a running sum may fall to either side
        assert np.mean(got[0][0] == got[1][0]) > 0.998, count
