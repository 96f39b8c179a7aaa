"""Kraus channels on qubits 0..3 together (their amplitudes go through shared memory), in every
position of a run of groups and in any order of the four, against the shot-by-shot simulation."""
import numpy as np
import pytest

from openqarp_b200 import Command, GateType as G, Register, ir
from openqarp_b200.noise import KrausChannel, NoiseModel
from test_kraus_groups import DAMP_Y, _simulate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["complex128", "complex64"])
@pytest.mark.parametrize("order", [(0, 1, 2, 3), (2, 0, 3, 1), (3, 2, 1, 0)])
@pytest.mark.parametrize("n", [12, 14])
def test_lowest_four_qubits(n, order, dtype):
    rng = np.random.default_rng(n)
    high = [q for q in range(4, n)]
    runs = [list(order), list(order) + high, high[:4] + list(order), high[:4] + list(order) + high[4:7]]
    cmds = [Command(G.Rx, (q,), (float(rng.uniform(-3, 3)),)) for q in range(n)]
    for d, qs in enumerate(runs):
        cmds += [Command(G.Ry, (q,), (float(rng.uniform(-3, 3)),)) for q in qs]
        cmds += [Command(G.CX, (q, (q + 5) % n)) for q in order]
        cmds.append(Command(G.Measure, (d,), (), None, (d,)))
    channels = {int(G.Ry): DAMP_Y}
    model = NoiseModel()
    model.set_channel(int(G.Ry), KrausChannel(tuple(np.asarray(k, dtype=complex) for k in DAMP_Y)))
    shots = 20
    reg = Register(n, dtype)
    try:
        reg.set_noise(model)
        reg.set_trajectory_batch(8)          # the batched executor, also where another is the default
        out, cbits, _ = reg.run_trajectories(ir.pack(cmds).buf, 9, shots)
    finally:
        reg.close()
    same = sum((int(o), int(c)) == _simulate(n, cmds, channels, 9 + s) for s, (o, c) in enumerate(zip(out, cbits)))
    # complex64 may take the other side where a draw lies within FP32 rounding of a threshold
    assert same == shots if dtype == "complex128" else same >= shots - 2
