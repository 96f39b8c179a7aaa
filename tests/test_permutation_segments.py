"""Trajectory segments of X, CX and SWAP alone, moved in one pass, against a shot-by-shot simulation in
numpy: ladders and random runs over every qubit (more than one pass), targets and controls on lane,
block and shot-near bits, both storage types.  Amplitudes only move, so outcomes and classical bits
are those of the simulation (its uniforms lie away from every decision by more than rounding)."""
import numpy as np
import pytest

from openqarp_b200 import Command, GateType as G, Register, ir

pytestmark = pytest.mark.gpu


def _uniforms(seed):
    return np.frombuffer(np.random.RandomState(seed).bytes(8 * 200), dtype="<u8").astype(np.float64) * 2.0 ** -64


def _simulate(n, cmds, seed):
    psi = np.zeros(1 << n, dtype=complex)
    psi[0] = 1
    i, cbits, u = np.arange(1 << n), 0, iter(_uniforms(seed))
    near = 1.0
    for c in cmds:
        g, q = c.gate, c.qubits
        if g == G.Measure:
            v = psi.reshape(-1, 2, 1 << q[0])
            p0, r = float(np.sum(np.abs(v[:, 0]) ** 2)), next(u)
            near = min(near, abs(r - p0))
            one = r >= p0
            v[:, 0 if one else 1] = 0
            psi *= np.sqrt(1.0 / (1.0 - p0 if one else p0))
            cbits = (cbits & ~(1 << c.cbits[0])) | (int(one) << c.cbits[0])
        elif g == G.X:
            psi = psi[i ^ (1 << q[0])]
        elif g == G.CX:
            psi = psi[np.where((i >> q[0]) & 1, i ^ (1 << q[1]), i)]
        elif g == G.SWAP:
            d = ((i >> q[0]) ^ (i >> q[1])) & 1
            psi = psi[i ^ (d << q[0]) ^ (d << q[1])]
        elif g != G.Id:
            t = c.params[0] / 2
            v = psi.reshape(-1, 2, 1 << q[0])
            a, b = v[:, 0].copy(), v[:, 1].copy()
            v[:, 0], v[:, 1] = np.cos(t) * a - np.sin(t) * b, np.sin(t) * a + np.cos(t) * b
    w = np.cumsum(np.abs(psi) ** 2)
    r = next(u) * w[-1]
    near = min(near, np.min(np.abs(w - r)))
    return int(np.searchsorted(w, r)), cbits, near


def _moves(kind, n, rng):
    if kind == "ladder":
        return [Command(G.CX, (q, q + 1)) for q in range(n - 1)] + [Command(G.X, (n - 1,))]
    if kind == "disjoint":
        p = [int(v) for v in rng.permutation(n)]
        return [Command(G.CX, (a, b)) for a, b in zip(p[::2], p[1::2])]
    out = []
    for _ in range(30):
        a, b = (int(v) for v in rng.choice(n, 2, replace=False))
        out.append([Command(G.X, (a,)), Command(G.CX, (a, b)), Command(G.SWAP, (a, b)), Command(G.Id, (b,))][int(rng.integers(4))])
    return out


@pytest.mark.parametrize("dtype", ["complex128", "complex64"])
@pytest.mark.parametrize("kind", ["ladder", "disjoint", "random"])
@pytest.mark.parametrize("n", [14, 15])
def test_moved_segments_against_numpy(n, kind, dtype):
    rng = np.random.default_rng(n)
    cmds, shots, seed = [], 12, 5
    for layer in range(2):
        cmds += [Command(G.Ry, (q,), (float(rng.uniform(0.3, 2.8)),)) for q in range(n)]
        cmds += [Command(G.Measure, ((3 * layer) % n,), (), None, (layer,))]
        cmds += _moves(kind, n, rng)
        cmds += [Command(G.Measure, ((5 + layer) % n,), (), None, (2 + layer,))]
    reg = Register(n, dtype)
    try:
        reg.configure(1, 0)      # commands unfused: many operations to a segment, so it is moved
        idx, regs, _ = reg.run_trajectories(ir.pack(cmds).buf, seed, shots)
    finally:
        reg.close()
    # 4 n gates' rounding moves a probability or a running sum by less than this
    margin = 1e-12 if dtype == "complex128" else 1e-5
    compared = 0
    for s in range(shots):
        want_idx, want_bits, near = _simulate(n, cmds, seed + s)
        if near < margin:
            continue
        compared += 1
        assert (int(idx[s]), int(regs[s])) == (want_idx, want_bits), s
    assert dtype == "complex64" or compared == shots
