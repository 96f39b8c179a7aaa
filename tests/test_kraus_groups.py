"""Kraus channels decided and applied four qubits at a time, against a shot-by-shot simulation in numpy
that decides one channel after another: runs of 1..9 channels, qubits on lane, warp and block bits,
damping and dephasing, a channel with off-diagonal K^dag K (decided by itself), guarded runs, registers
at the width where the groups begin, complex64."""
import numpy as np
import pytest

from openqarp_b200 import Command, GateType as G, Register, ir
from openqarp_b200.noise import KrausChannel, NoiseModel

C, S = np.sqrt(0.9), np.sqrt(0.1)
DAMP_Y = [np.array([[1, 0], [0, np.sqrt(0.85)]]), np.array([[0, np.sqrt(0.15)], [0, 0]])]
DAMP_X = [np.array([[1, 0], [0, np.sqrt(0.95)]]), np.array([[0, np.sqrt(0.05)], [0, 0]])]
DEPHASE = [np.diag([1.0, C]), np.diag([0.0, S])]
MIXED = [np.array([[0.9, 0.1], [0.0, 0.8]])]      # columns not orthogonal
_w, _v = np.linalg.eigh(np.eye(2) - MIXED[0].T @ MIXED[0])
MIXED.append(_v @ np.diag(np.sqrt(_w)) @ _v.T)


class Draws:
    """std::mt19937(seed) through std::generate_canonical<double, 53>."""

    def __init__(self, seed):
        self.raw = np.frombuffer(np.random.RandomState(seed).bytes(8 * 400), dtype="<u8")
        self.at = 0

    def __call__(self):
        self.at += 1
        return float(self.raw[self.at - 1]) * 2.0 ** -64


def _one(psi, q, m):
    v = psi.reshape(-1, 2, 1 << q)
    a, b = v[:, 0].copy(), v[:, 1].copy()
    v[:, 0], v[:, 1] = m[0, 0] * a + m[0, 1] * b, m[1, 0] * a + m[1, 1] * b


def _simulate(n, cmds, channels, seed):
    psi = np.zeros(1 << n, dtype=complex)
    psi[0] = 1
    cbits, u = 0, Draws(seed)
    for c in cmds:
        g, q = int(c.gate), c.qubits
        if g == G.Measure:
            v = psi.reshape(-1, 2, 1 << q[0])
            p0 = float(np.sum(np.abs(v[:, 0]) ** 2))
            one = u() >= p0
            v[:, 0 if one else 1] = 0
            psi *= np.sqrt(1.0 / (1.0 - p0 if one else p0))
            cbits = (cbits & ~(1 << c.cbits[0])) | (int(one) << c.cbits[0])
            continue
        if c.condition_bits and not (cbits >> c.condition_bits[0]) & 1:
            continue
        if g == G.CX:
            i = np.arange(1 << n)
            psi[:] = psi[np.where((i >> q[0]) & 1, i ^ (1 << q[1]), i)]
        elif g == G.X:
            _one(psi, q[0], np.array([[0, 1], [1, 0]]))
        else:
            t = c.params[0] / 2
            cs, sn = np.cos(t), np.sin(t)
            _one(psi, q[0], np.array([[cs, -sn], [sn, cs]]) if g == G.Ry else np.array([[cs, -1j * sn], [-1j * sn, cs]]))
        for ops in ([channels[g]] if g in channels else []):
            v = psi.reshape(-1, 2, 1 << q[0])
            a, b = v[:, 0].ravel(), v[:, 1].ravel()
            rho = np.array([[np.vdot(a, a), np.vdot(b, a)], [np.vdot(a, b), np.vdot(b, b)]])
            p = np.array([max(0.0, np.trace(k @ rho @ k.conj().T).real) for k in ops])
            r, acc = u(), 0.0
            for k, w in zip(ops, p / p.sum()):
                acc += w
                if r < acc:
                    _one(psi, q[0], k / np.sqrt(w * p.sum()))
                    break
    w = np.abs(psi) ** 2
    return int(np.searchsorted(np.cumsum(w), u() * w.sum())), cbits


def _circuit(n, seed):
    rng = np.random.default_rng([n, seed])
    cmds = []
    for d in range(3):
        qs = [int(q) for q in rng.permutation(n)]
        cmds += [Command(G.Ry, (q,), (float(rng.uniform(-3, 3)),)) for q in qs[:int(rng.integers(1, n + 1))]]
        cmds += [Command(G.CX, (a, b)) for a, b in zip(qs[::2], qs[1::2])]
        cmds += [Command(G.Rx, (q,), (float(rng.uniform(-3, 3)),)) for q in qs[:int(rng.integers(1, 10))]]
        cmds.append(Command(G.Measure, (qs[0],), (), None, (d,)))
        cmds += [Command(G.X, (q,), (), None, (), (d,), (True,)) for q in qs[1:6]]
    return cmds


@pytest.mark.gpu
@pytest.mark.parametrize("n,mixed,dtype", [(11, False, "complex128"), (12, False, "complex128"), (12, True, "complex128"),
                                           (14, False, "complex128"), (13, False, "complex64")])
def test_groups_match_channel_by_channel(n, mixed, dtype):
    channels = {int(G.Ry): DAMP_Y, int(G.X): DAMP_X, int(G.Rx): MIXED if mixed else DEPHASE}
    model = NoiseModel()
    for g, ops in channels.items():
        model.set_channel(g, KrausChannel(tuple(np.asarray(k, dtype=complex) for k in ops)))
    shots, same = 20, 0
    for seed in (1, 2):
        cmds = _circuit(n, seed)
        reg = Register(n, dtype)
        reg.set_noise(model)
        reg.set_trajectory_batch(8)              # the batched executor, also where another is the default
        out, cbits, _ = reg.run_trajectories(ir.pack(cmds).buf, 50 * seed, shots)
        reg.close()
        want = [_simulate(n, cmds, channels, 50 * seed + s) for s in range(shots)]
        same += sum((int(o), int(c)) == w for o, c, w in zip(out, cbits, want))
    # complex64 may take the other side where a draw lies within FP32 rounding of a threshold
    assert same == 2 * shots if dtype == "complex128" else same >= 2 * shots - 2
