"""The native packer writes the bytes and dependency tables the general Python path writes: the same
commands as ir.Command and as duck-typed objects (which take that path), mixed streams, and the inputs
each refuses."""
import numpy as np
import pytest

from openqarp_b200 import Command, GateType as G, Param, ir


class Duck:
    def __init__(self, c):
        for k in ("gate", "qubits", "params", "unitary", "cbits", "condition_bits", "condition_values"):
            setattr(self, k, getattr(c, k))


def _commands(seed, count=120):
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(count):
        q = [int(x) for x in rng.permutation(9)[:5]]
        pick = int(rng.integers(0, 9))
        z = rng.standard_normal((4, 4)) + 1j * rng.standard_normal((4, 4))
        out.append([Command(G.H, (q[0],)), Command(G.Rx, (q[0],), (float(rng.normal()),)), Command(G.Rz, (q[0],), (2,)),
                    Command(G.Ry, (q[0],), (Param.symbol("a"),)), Command(G.RZZ, (q[0], q[1]), (Param.linear(-1.5, "b", 0.25),)),
                    Command(G.P, (q[0],), (Param.symbol("a") * 2.0 + Param.symbol("c") - 0.5,)),
                    Command(G.Custom, (q[0], q[1]), (), np.linalg.qr(z)[0]), Command(G.MCZ, tuple(q)),
                    Command(G.U, (q[0],), (0.1, Param(0.2), np.float64(0.3)))][pick])
    return out


@pytest.mark.parametrize("seed", range(4))
def test_bytes_and_dependencies_match_the_general_path(seed):
    cmds = _commands(seed)
    cmds.insert(5, Command(G.Measure, (2,), (), None, (1,)))
    cmds.insert(40, Command(G.X, (3,), (), None, (), (1,), (True,)))
    cmds.append(Command(G.Custom, (1,), (), np.asfortranarray(np.array([[0, 1], [1, 0]]))))
    values = {"a": 0.75, "b": np.float64(-2.5), "c": 3}
    for order in (None, ["c", "a"], ["b"]):
        got, want = ir.pack(cmds, values, order), ir.pack([Duck(c) for c in cmds], values, order)
        assert got.buf == want.buf and got.n_cmds == want.n_cmds == len(cmds)
        for k in ("dep_ptr", "dep_param", "dep_alpha"):
            np.testing.assert_array_equal(getattr(got, k), getattr(want, k))
    assert ir.pack(iter(cmds), values).buf == ir.pack([Duck(c) for c in cmds], values).buf
    back = ir.unpack(ir.pack(cmds, values).buf)
    skip = (G.Barrier, G.Measure, G.GPhase)
    assert ir.record_widths(ir.pack(cmds, values).buf) == [len(c.qubits) for c in back if c.gate not in skip and c.qubits]


@pytest.mark.parametrize("bad", [Command(G.Rx, (0,), (Param.symbol("missing"),)), Command(G.X, (-1,)), Command(G.X, (1 << 40,)),
                                 Command(G.Custom, (0, 1), (), np.eye(2)), Command(G.Custom, (0,)),
                                 Command(G.X, (0,), (), None, (), (), (True,))])
def test_refusals_are_the_general_path_s(bad):
    first = [Command(G.H, (0,))]
    errors = []
    for cmd in (bad, Duck(bad)):
        try:
            errors.append(ir.pack(first + [cmd], {"a": 1.0}).buf)
        except Exception as e:  # noqa: BLE001
            errors.append((type(e), str(e)))
    assert errors[0] == errors[1]


def test_trajectory_scan():
    plain = [Command(G.H, (0,)), Command(G.Measure, (0,))]
    for cmds in (plain, plain + [Command(G.Reset, (0,))], plain + [Command(G.Measure, (0,), (), None, (0,))],
                 plain + [Command(G.X, (0,), (), None, (), (0,), (True,))], plain + [Duck(Command(G.Reset, (0,)))], []):
        assert ir.any_needs_trajectory(cmds) == any(ir.needs_trajectory(c) for c in cmds)
