"""The compiled reverse sweep (complex128, executor 3) against the CPU oracle: every differentiable gate,
angles on both sides of a quarter turn, fixed gates of every form between them, parameters shared by
several gates, checkpoint restarts, a block no tile holds, and more steps than one pass accumulates."""
import numpy as np
import pytest

from openqarp_b200 import Command, GateType as G, Param, Register, circuits, ir, observable

ONE = [G.Rx, G.Ry, G.Rz, G.P]
TWO = [G.CRx, G.CRy, G.CRz, G.CP, G.RXX, G.RYY, G.RZZ]


def _circuit(n, seed, count, n_params=24, wide=False):
    rng = np.random.default_rng([n, seed])
    out = []
    for i in range(count):
        q = [int(x) for x in rng.permutation(n)[:3]]
        p = Param.linear(float(rng.choice([-1.5, 1.0, 2.0])), f"t{int(rng.integers(n_params))}", float(rng.uniform(-1, 1)))
        pick = int(rng.integers(0, 12))
        if pick < 5:
            out.append(Command(ONE[pick % 4], (q[0],), (p,)))
        elif pick < 7:
            out.append(Command(TWO[int(rng.integers(7))], (q[0], q[1]), (p,)))
        elif pick == 7:
            out.append(Command([G.H, G.X, G.Y, G.S, G.T, G.SX][int(rng.integers(6))], (q[0],)))
        elif pick == 8:
            out.append(Command([G.CX, G.CZ, G.SWAP, G.CH][int(rng.integers(4))], (q[0], q[1])))
        elif pick == 9:
            out.append(Command([G.CCX, G.MCZ][int(rng.integers(2))], tuple(q)))
        elif pick == 10:
            out.append(Command(G.GPhase, (), (p,)))
        else:
            out.append(Command(G.Ry, (q[0],), (float(rng.uniform(-7, 7)),)))
    if wide:
        z = rng.standard_normal((64, 64)) + 1j * rng.standard_normal((64, 64))
        out.insert(count // 2, ir.custom(tuple(int(x) for x in rng.permutation(n)[:6]), np.linalg.qr(z)[0]))
    names = [f"t{k}" for k in range(n_params)]
    return out, {k: float(v) for k, v in zip(names, rng.uniform(-4, 4, n_params))}, names


def _check(restatement, n, cmds, vals, names, checkpoint=-1):
    obs = circuits.tfim_chain(n) + circuits.random_pauli_sum(n, 12, seed=n, max_weight=3)
    masks = observable.to_masks(obs, n)
    stream = ir.pack(cmds, vals, names)
    want_e, want_g = restatement.adjoint(stream, n, len(names), masks)
    reg = Register(n)
    reg.configure(1, 0, 3)
    reg.set_checkpoint_interval(checkpoint)
    e, g = reg.adjoint(stream, len(names), masks)
    # sums of a few hundred steps' inner products, each below |H| ~ 40 with 1e-14 rounding
    assert abs(e - want_e) < 1e-10
    np.testing.assert_allclose(g, want_g, atol=1e-9)
    # the sweep leaves the state uncomputed
    psi = reg.get_state()
    psi[0] -= 1.0
    assert np.max(np.abs(psi)) < 1e-11
    reg.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n,seed,count", [(14, 1, 60), (14, 2, 200), (15, 3, 200), (17, 4, 120)])
def test_random_circuits_match_oracle(restatement, n, seed, count):
    _check(restatement, n, *_circuit(n, seed, count))


@pytest.mark.gpu
def test_checkpoints_and_wide_block(restatement):
    cmds, vals, names = _circuit(14, 5, 160)
    _check(restatement, 14, cmds, vals, names, checkpoint=45)
    cmds, vals, names = _circuit(15, 6, 80, wide=True)
    _check(restatement, 15, cmds, vals, names)


@pytest.mark.gpu
def test_ansatz_layers_and_many_steps_on_few_qubits(restatement):
    cmds, vals, names = circuits.hea(16, 4, seed=3)
    _check(restatement, 16, cmds, vals, names)
    # 200 steps on four qubits: one tile's pass is cut where its accumulators end
    rng = np.random.default_rng(9)
    names = [f"t{k}" for k in range(200)]
    cmds = [Command(ONE[int(rng.integers(4))], (int(rng.integers(4)),), (Param.symbol(nm),)) for nm in names]
    cmds = [Command(G.H, (q,)) for q in range(14)] + cmds
    _check(restatement, 14, cmds, {nm: float(v) for nm, v in zip(names, rng.uniform(-4, 4, 200))}, names)


def _phase_rich(n, seed, segments, length, block_in):
    """`segments` runs of `length` commands with many phase parameters; a fixed 4-qubit block, which the
    compiled sweep refuses, in the middle of segment `block_in`."""
    rng = np.random.default_rng([n, seed, block_in])
    out, names = [], [f"t{k}" for k in range(18)]
    for s in range(segments):
        for i in range(length):
            q = [int(x) for x in rng.permutation(n)[:4]]
            p = Param.linear(float(rng.choice([-1.5, 1.0])), names[int(rng.integers(18))], float(rng.uniform(-1, 1)))
            if s == block_in and i == length // 2:
                z = rng.standard_normal((16, 16)) + 1j * rng.standard_normal((16, 16))
                out.append(ir.custom(tuple(q), np.linalg.qr(z)[0]))
            elif i % 5 == 4:
                out.append(Command(G.CX, (q[0], q[1])))
            else:
                out.append(Command([G.Rz, G.Ry, G.P, G.Rx][i % 5], (q[0],), (p,)))
    return out, {k: float(v) for k, v in zip(names, rng.uniform(-4, 4, 18))}, names


# the tolerances of _check; the state a sweep leaves behind may lack a phase where it ends interpreted
@pytest.mark.gpu
@pytest.mark.parametrize("n", [14, 16])
@pytest.mark.parametrize("block_in", [0, 1, 2])
def test_segments_that_do_not_compile_beside_those_that_do(restatement, n, block_in, tmp_path, monkeypatch):
    cmds, vals, names = _phase_rich(n, 21, 3, 30, block_in)
    masks = observable.to_masks(circuits.tfim_chain(n) + circuits.random_pauli_sum(n, 12, seed=n, max_weight=3), n)
    stream = ir.pack(cmds, vals, names)
    want_e, want_g = restatement.adjoint(stream, n, len(names), masks)
    monkeypatch.setenv("QSV_JIT_CACHE", str(tmp_path))
    reg = Register(n)
    reg.configure(1, 0, 3)
    reg.set_checkpoint_interval(30)
    for k in range(3):      # the forward sweep's segments, compiled before the reverse sweep's are counted
        reg.apply(ir.pack(cmds[30 * k:30 * (k + 1)], vals))
    reg.reset()
    forward = len(list(tmp_path.iterdir()))
    e, g = reg.adjoint(stream, len(names), masks)
    reg.close()
    assert len(list(tmp_path.iterdir())) > forward      # two of the three segments in compiled passes
    assert abs(e - want_e) < 1e-10
    np.testing.assert_allclose(g, want_g, atol=1e-9)


# matrices rounded to 32 bits are unitary to 1e-7: the sweep that applies them as they are, the tolerances of _check
@pytest.mark.gpu
def test_matrices_of_fewer_digits(restatement):
    n = 14
    rng = np.random.default_rng(31)
    cmds, vals, names = _circuit(n, 7, 40)
    for q in range(0, n, 3):
        z = np.linalg.qr(rng.standard_normal((2, 2)) + 1j * rng.standard_normal((2, 2)))[0]
        at = 12 + 2 * q
        # the forward sweep takes it within a two-qubit block
        cmds[at:at] = [ir.custom((q,), z.astype(np.complex64)), Command(G.CX, (q, (q + 1) % n))]
    masks = observable.to_masks(circuits.tfim_chain(n), n)
    stream = ir.pack(cmds, vals, names)
    want_e, want_g = restatement.adjoint(stream, n, len(names), masks)
    reg = Register(n)
    reg.configure(2, 0, 3)
    e, g = reg.adjoint(stream, len(names), masks)
    reg.close()
    assert abs(e - want_e) < 1e-10
    np.testing.assert_allclose(g, want_g, atol=1e-9)


# a structure is compiled once for all angles: zeros (all of them, or some) compile nothing new
@pytest.mark.gpu
def test_angles_of_zero_compile_nothing(restatement, tmp_path, monkeypatch):
    n = 15
    names = [f"t{k}" for k in range(12)]
    fixed = [f"f{k}" for k in range(4)]
    rng = np.random.default_rng(41)
    cmds = []
    for i in range(90):
        q = [int(x) for x in rng.permutation(n)[:2]]
        sym = Param.symbol(names[int(rng.integers(12))])
        pick = i % 9
        if pick < 4:
            cmds.append(Command(ONE[pick], (q[0],), (sym,)))
        elif pick < 6:
            cmds.append(Command([G.Rx, G.Ry][pick - 4], (q[0],), (Param.symbol(fixed[int(rng.integers(4))]),)))
        elif pick < 8:
            cmds.append(Command(TWO[int(rng.integers(7))], (q[0], q[1]), (sym,)))
        else:
            cmds.append(Command(G.CX, (q[0], q[1])))
    masks = observable.to_masks(circuits.tfim_chain(n), n)
    monkeypatch.setenv("QSV_JIT_CACHE", str(tmp_path))
    reg = Register(n)
    reg.configure(0, 0, 3)
    files = 0
    for zero in (0.0, 0.5, 1.0):       # share of the angles that are 0
        vals = {k: 0.0 if rng.random() < zero else float(rng.uniform(-4, 4)) for k in names + fixed}
        stream = ir.pack(cmds, vals, names)
        want_e, want_g = restatement.adjoint(stream, n, len(names), masks)
        reg.reset()
        e, g = reg.adjoint(stream, len(names), masks)
        assert abs(e - want_e) < 1e-10
        np.testing.assert_allclose(g, want_g, atol=1e-9)
        files = files or len(list(tmp_path.iterdir()))
        assert len(list(tmp_path.iterdir())) == files > 0, zero
    reg.close()
