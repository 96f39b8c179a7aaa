"""Compiled tile passes whose rotations turn by more than a quarter (their bits are left turned until
the pass's store): every kind of op that then acts on turned bits - phases of one, two and more qubits,
controlled gates of one and two controls, swaps, diagonals, Pauli rotations, dense blocks - on slot,
lane, warp and outside qubits, in chains of passes, against the CPU oracle."""
import numpy as np
import pytest

from openqarp_b200 import Command, GateType as G, Register, ir


def _circuit(n, seed, count=260):
    rng = np.random.default_rng([n, seed])
    one = [G.X, G.Y, G.H, G.SX, G.Z, G.S, G.T]
    rot = [G.Rx, G.Ry, G.Rz, G.P]
    two = [G.CX, G.CX, G.CZ, G.CZ, G.CY, G.SWAP, G.CH, G.CSX]
    tworot = [G.CP, G.CRx, G.CRz, G.RZZ, G.RXX, G.RYY]
    out = []
    for _ in range(count):
        q = [int(x) for x in rng.permutation(n)[:4]]
        pick = rng.integers(0, 12)
        if pick < 2:
            out.append(Command(one[rng.integers(len(one))], (q[0],)))
        elif pick < 6:
            out.append(Command(rot[rng.integers(len(rot))], (q[0],), (float(rng.uniform(-7, 7)),)))
        elif pick < 8:
            out.append(Command(two[rng.integers(len(two))], (q[0], q[1])))
        elif pick < 10:
            out.append(Command(tworot[rng.integers(len(tworot))], (q[0], q[1]), (float(rng.uniform(-7, 7)),)))
        elif pick == 10:
            out.append(Command([G.CCX, G.MCZ, G.CSWAP][rng.integers(3)], tuple(q[:3])))
        else:
            out.append(Command(G.U, (q[0],), tuple(float(x) for x in rng.uniform(-4, 4, 3))))
    return out


# a few hundred gates, each within 4 roundings of unit-norm amplitudes
@pytest.mark.gpu
@pytest.mark.parametrize("dtype,tol", [("complex128", 1e-12), ("complex64", 2e-5)])
@pytest.mark.parametrize("n,k", [(12, 0), (13, 1), (15, 0), (16, 2)])
def test_turned_bits_match_oracle(restatement, n, k, dtype, tol):
    for seed in (1, 2, 3):
        buf = ir.pack(_circuit(n, seed)).buf
        want = restatement.statevector(buf, n)
        reg = Register(n, dtype)
        reg.configure(k, 0, 3, 12)
        reg.apply(buf)
        assert np.max(np.abs(reg.get_state() - want)) < tol
        reg.close()


# one-qubit diagonals that are no phases (projectors, weights), on places of every kind, beside phases
# and turned bits, after the same circuit with a phase there: a hundred products of amplitudes below 1
@pytest.mark.gpu
@pytest.mark.parametrize("dtype,tol", [("complex128", 1e-12), ("complex64", 2e-5)])
@pytest.mark.parametrize("d", [(1.0, 1.0j), (0.0, 1.0), (1.0, 0.0), (0.0, 0.0), (0.25, 1.0), (-0.5j, 1e-30)])
def test_diagonals_of_any_modulus(restatement, d, dtype, tol):
    n, rng = 14, np.random.default_rng(8)
    for places in ([0], [5], [12, 13], list(range(n))):
        cmds = [Command(G.Ry, (q,), (float(rng.uniform(-7, 7)),)) for q in range(n)]
        for q in places:
            cmds += [Command(G.Rz, (q,), (0.3 + q,)), ir.custom((q,), np.diag(d)), Command(G.CZ, (q, (q + 1) % n)),
                     Command(G.Rx, ((q + 3) % n,), (4.0 - q,))]
        cmds += [Command(G.Ry, (q,), (float(rng.uniform(-7, 7)),)) for q in range(n)]
        buf = ir.pack(cmds).buf
        want = restatement.statevector(buf, n)
        reg = Register(n, dtype)
        reg.configure(0, 0, 3, 12)
        reg.apply(buf)
        assert np.max(np.abs(reg.get_state() - want)) < tol, places     # NaN fails too
        reg.close()


# what a complex128 pass reads of its coefficients is a whole pair (no device needed: the source is looked at)
@pytest.mark.parametrize("dtype", [0])
def test_coefficients_come_in_pairs(dtype, tmp_path, monkeypatch):
    import ctypes
    import re
    from openqarp_b200._lib import check, lib, u8ptr
    monkeypatch.setenv("QSV_JIT_DUMP", str(tmp_path / "passes.cu"))
    buf = ir.pack(_circuit(15, 4, 60)).buf
    passes, kernels, size = ctypes.c_int32(), ctypes.c_int32(), ctypes.c_uint64()
    check(lib.qsv_jit_check(u8ptr(buf), len(buf), 15, dtype, 0, 0, 10, 0, ctypes.byref(passes), ctypes.byref(kernels),
                            ctypes.byref(size)))
    src = (tmp_path / "passes.cu").read_text()
    singles = re.findall(r"const R t = P\.c\[(\d+)\]|\(P\.c\[(\d+)\] != 0\)", src)
    products = re.findall(r"= P\.c\[(\d+)\] \* xr - P\.c\[(\d+)\] \* xi", src)
    assert len(singles) > 20 and len(products) > 100
    assert all(int(a or b) % 2 == 0 for a, b in singles)
    assert all(int(a) % 2 == 0 and int(b) == int(a) + 1 for a, b in products)


# a pass of three-qubit blocks, a controlled one-qubit gate and a bit put back, whose amplitudes do not
# all stay in registers, against the executor of single passes: a dozen products of unit-norm amplitudes
@pytest.mark.gpu
@pytest.mark.parametrize("seed", [1, 2])
def test_pass_that_spills_amplitudes(seed):
    from openqarp_b200.ir import ControlledUnitaryRecord, PermutationRecord
    rng = np.random.default_rng(seed)

    def unitary(k):
        return np.linalg.qr(rng.standard_normal((1 << k, 1 << k)) + 1j * rng.standard_normal((1 << k, 1 << k)))[0]
    n = 12
    cmds = [Command(G.CH, (2, 11)), ir.custom((9, 7, 11, 10, 2), unitary(5)),
            PermutationRecord((8, 4, 11), rng.permutation(8).astype(np.uint64)), Command(G.Rz, (9,), (np.pi,)),
            Command(G.U, (7,), (1.2, 2.6, -np.pi)), ir.custom((1, 9, 5), unitary(3)), Command(G.Rx, (8,), (2 * np.pi,)),
            Command(G.CRz, (1, 8), (4.54,)), ir.custom((4,), unitary(1)), Command(G.iSWAP, (6, 7)),
            ControlledUnitaryRecord((5, 6, 9, 3), 7, unitary(4)), Command(G.Rx, (10,), (np.pi / 2,))]
    start = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    start /= np.linalg.norm(start)
    states = []
    for executor in (3, 0):
        reg = Register(n)
        reg.configure(1, 0, executor)
        reg.set_state(start)
        reg.apply(ir.pack(cmds).buf)
        states.append(reg.get_state())
        reg.close()
    assert np.max(np.abs(states[0] - states[1])) < 1e-13
