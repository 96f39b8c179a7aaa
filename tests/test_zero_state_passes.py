"""Compiled passes from |0...0> leave out the tiles a circuit has not reached: circuits that spread slowly,
all at once, or never to some qubits, against the CPU oracle; a register that is not |0...0> any more
takes whole passes, whatever came between the reset and the circuit."""
import numpy as np
import pytest

from openqarp_b200 import B200Simulator, Command, GateType as G, Register, circuits, ir


def _circuits(n):
    rng = np.random.default_rng(n)
    few = [Command(G.H, (q,)) for q in (0, n - 1, n // 2)] + [Command(G.CX, (n - 1, 5)), Command(G.RZZ, (5, 9), (0.4,))]
    spread = []
    for q in range(n):
        spread += [Command(G.Ry, (q,), (float(rng.uniform(-3, 3)),)), Command(G.CX, (q, (q + 1) % n))]
    neel = [Command(G.X, (q,)) for q in range(1, n, 2)] + circuits.heisenberg_trotter(n, 1, 0.1, rng.uniform(-1, 1, n), neel=False)
    swaps = [Command(G.X, (3,)), Command(G.SWAP, (3, n - 2)), Command(G.CP, (n - 2, 0), (0.3,)), Command(G.RXX, (n - 2, 4), (0.7,)),
             Command(G.CSWAP, (4, 7, n - 3))]
    return {"few": few, "spread": spread, "neel": neel, "swaps": swaps, "brickwork": circuits.brickwork(n, 5, seed=n), "none": []}


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,tol", [("complex128", 1e-12), ("complex64", 1e-5)])
@pytest.mark.parametrize("n", [12, 13, 17, 20])
def test_circuits_from_zero_match_oracle(restatement, n, dtype, tol):
    sim = B200Simulator(dtype=dtype)
    sim.executor, sim.fusion_max_qubits = 3, 1
    for name, cmds in _circuits(n).items():
        want = restatement.statevector(ir.pack(cmds).buf, n)
        for _ in range(2):          # the second time the register holds the first one's amplitudes
            assert np.max(np.abs(sim.statevector(cmds, n) - want)) < tol, name
    obs = circuits.tfim_chain(n)
    cmds, vals, names = circuits.hea(n, 2, seed=1)
    from openqarp_b200 import observable
    e, g = sim.energy_and_gradient(cmds, n, obs, vals, names)
    we, wg = restatement.adjoint(ir.pack(cmds, vals, names), n, len(names), observable.to_masks(obs, n))
    assert abs(e - we) < 1e3 * tol and np.max(np.abs(np.asarray(g) - wg)) < 1e3 * tol
    sim.close()


@pytest.mark.gpu
def test_whole_passes_once_the_register_was_touched(restatement):
    n = 15
    cmds = circuits.brickwork(n, 3, seed=2)
    buf = ir.pack(cmds).buf
    rng = np.random.default_rng(1)
    psi = rng.standard_normal(1 << n) + 1j * rng.standard_normal(1 << n)
    psi /= np.linalg.norm(psi)
    want = restatement.statevector(buf, n, psi)
    reg, other = Register(n), Register(n)
    other.set_state(psi)
    reg.configure(1, 0, 3)

    def through_pointer():
        import torch
        view = type("View", (), {"__cuda_array_interface__": {"shape": (1 << n,), "typestr": "<c16", "version": 3,
                                                              "data": (reg.device_pointer()[0], False)}})()
        torch.as_tensor(view, device="cuda").copy_(torch.from_numpy(psi))
        torch.cuda.synchronize()

    for touch in (lambda: reg.set_state(psi), lambda: reg.copy_from(other), through_pointer):
        reg._reset_async()
        reg.synchronize()
        touch()
        reg.apply(buf)
        assert np.max(np.abs(reg.get_state() - want)) < 1e-12
    # applied twice: the second circuit starts from the first one's state
    reg._reset_async()
    reg.apply(buf)
    reg.apply(buf)
    twice = restatement.statevector(buf, n, restatement.statevector(buf, n))
    assert np.max(np.abs(reg.get_state() - twice)) < 1e-12
    reg.close()
    other.close()
