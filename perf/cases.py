"""Performance cases: the work a user of the simulator has it do, through its public calls.

Twelve listed cases and a generator of more of the same ranges.  Each case is a dict of plain
values; ``prepare`` builds what a program holds before the call (commands, observable, simulator
or batch handle), ``run`` makes the call, ``work`` counts the bytes and operations the path
cannot do without, and ``exact`` computes the same outputs in 64 bits with plain torch.

Kinds
  call        one small circuit read back whole, and its <H>: the latency of a single call
  variational an ordinary ansatz: state on the device and <H>, the step of a VQE loop
  gates       random brickwork: one-qubit gates and CZ layers over a register larger than L2
  trotter     second-order Heisenberg steps: two-qubit Pauli rotations
  gradient    <H> and every parameter's derivative (forward, H|psi>, reverse sweep)
  energy      <H> of a random Pauli sum over a state already on the device
  sample      seeded terminal shots of a state already on the device
  shots       mid-circuit measurement with feed-forward, every shot its own trajectory
  qaoa        a batch of MaxCut instances of uneven width with gradients, one launch
  batch       a batch of small ansaetze with their own parameters and observables, one launch
Registers from 24 qubits up hold the plan the engine's autotuner picks for these circuits
(compiled tile passes of one-qubit layers), as a program that keeps its plan does.
"""
import math

import numpy as np
import torch

from openqarp_b200 import B200Simulator, Command, GateType, NoiseModel, Param, PauliMasks, Register
from openqarp_b200.batch import CircuitBatch, QaoaBatch, QaoaInstance
from openqarp_b200.ir import custom, pack

PLANNED_QUBITS = 24      # registers at least this wide pin the compiled-pass plan


def listed():
    return [
        # one small circuit at a time: the 12-qubit ansatz of 10 layers with a 64-term observable
        {"name": "call_12q", "kind": "call", "n": 12, "layers": 10, "terms": 64},
        # a VQE step on an ordinary register, smaller than L2
        {"name": "vqe_20q", "kind": "variational", "n": 20, "layers": 8, "terms": 100},
        # the headline circuit: 28 qubits, depth 20, a 4 GiB register, and its complex64 form
        {"name": "brickwork_28q_c128", "kind": "gates", "n": 28, "depth": 20, "dtype": "complex128"},
        {"name": "brickwork_28q_c64", "kind": "gates", "n": 28, "depth": 20, "dtype": "complex64"},
        # time evolution in bulk mode: a periodic Heisenberg chain from the Neel state
        {"name": "heisenberg_30q_c64", "kind": "trotter", "n": 30, "steps": 1, "dtype": "complex64"},
        # 384 derivatives of a 547-term sum (transverse-field Ising chain and 500 random terms)
        {"name": "gradient_24q", "kind": "gradient", "n": 24, "layers": 8, "terms": 500, "dtype": "complex128"},
        # <H> of many terms over a register larger than L2
        {"name": "energy_26q", "kind": "energy", "n": 26, "terms": 500},
        # the sampler: 100 000 shots of a register larger than L2
        {"name": "sample_26q", "kind": "sample", "n": 26, "shots": 100000},
        # noisy feed-forward trajectories on wide registers, noiseless ones on narrow registers
        {"name": "shots_16q_noisy", "kind": "shots", "n": 16, "depth": 8, "shots": 1024, "noisy": True},
        {"name": "shots_10q", "kind": "shots", "n": 10, "depth": 8, "shots": 20000, "noisy": False},
        # batched MaxCut QAOA, 10..20 qubits, depth 1..4, with gradients
        {"name": "qaoa_10_20q", "kind": "qaoa", "instances": 1024, "lo": 10, "hi": 20},
        # batched small ansaetze with gradients
        {"name": "batch_6_12q", "kind": "batch", "instances": 512, "lo": 6, "hi": 12},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["call", "variational", "gates", "trotter", "gradient", "energy", "sample", "shots",
                       "qaoa", "batch"])
    if kind == "call":
        return {"kind": kind, "n": rng.randint(4, 14), "layers": rng.randint(2, 12), "terms": _log_int(rng, 8, 128)}
    if kind == "variational":
        return {"kind": kind, "n": rng.randint(14, 23), "layers": rng.randint(2, 8), "terms": _log_int(rng, 16, 200)}
    if kind == "gates":
        return {"kind": kind, "n": rng.randint(20, 28), "depth": rng.randint(6, 20),
                "dtype": rng.choice(["complex128", "complex64"])}
    if kind == "trotter":
        dtype = rng.choice(["complex128", "complex64"])
        return {"kind": kind, "n": rng.randint(21, 29 if dtype == "complex64" else 28), "steps": rng.randint(1, 2),
                "dtype": dtype}
    if kind == "gradient":
        return {"kind": kind, "n": rng.randint(12, 24), "layers": rng.randint(2, 8), "terms": _log_int(rng, 8, 500),
                "dtype": rng.choice(["complex128", "complex64"])}
    if kind == "energy":
        return {"kind": kind, "n": rng.randint(16, 26), "terms": _log_int(rng, 8, 500)}
    if kind == "sample":
        return {"kind": kind, "n": rng.randint(16, 26), "shots": _log_int(rng, 1000, 100000)}
    if kind == "shots":
        n = rng.randint(5, 16)
        return {"kind": kind, "n": n, "depth": rng.randint(3, 8), "shots": _log_int(rng, 500, min(20000, 1 << (26 - n))),
                "noisy": rng.random() < 0.5}
    lo = rng.randint(8, 16) if kind == "qaoa" else rng.randint(4, 10)
    hi = min(lo + rng.randint(2, 6), 20 if kind == "qaoa" else 14)
    return {"kind": kind, "instances": _log_int(rng, 64, 700) if kind == "qaoa" else _log_int(rng, 32, 300),
            "lo": lo, "hi": hi}


# ------------------------------------------------------------------ circuits, as plain tuples
# ("ry" | "rz", q, slot): a rotation by parameter `slot`; ("u", q, 2x2); ("cx" | "cz", a, b);
# ("bond", a, b, t): exp(-i t (XX + YY + ZZ)); ("field", q, theta): Rz(theta)

def _hea(n, layers):
    gates, k = [], 0
    for _ in range(layers):
        for q in range(n):
            gates += [("ry", q, k), ("rz", q, k + 1)]
            k += 2
        gates += [("cx", q, q + 1) for q in range(n - 1)]
    return gates, k


def _haar(rng, count):
    z = rng.standard_normal((count, 2, 2)) + 1j * rng.standard_normal((count, 2, 2))
    q, r = np.linalg.qr(z)
    d = np.einsum("bii->bi", r)
    q = q * (d / np.abs(d))[:, None, :]
    return q / np.sqrt(np.linalg.det(q))[:, None, None]


def _brickwork(n, depth, rng):
    u = _haar(rng, n * depth)
    gates = []
    for l in range(depth):
        gates += [("u", q, u[l * n + q]) for q in range(n)]
        gates += [("cz", q, q + 1) for q in range(l % 2, n - 1, 2)]
    return gates


def _trotter(n, steps, fields, dt=0.05):
    bonds = [(i, (i + 1) % n) for i in range(n)]
    odd = [("bond", a, b, dt / 2) for a, b in bonds[1::2]]
    even = [("bond", a, b, dt) for a, b in bonds[0::2]]
    rz = [("field", q, 2.0 * float(fields[q]) * dt) for q in range(n)]
    return (odd + even + rz + odd) * steps


def _commands(gates, values=None):
    """The gates as commands: numbers where `values` has them, else symbols t0, t1, ..."""
    out = []
    for g in gates:
        if g[0] in ("ry", "rz"):
            p = Param.symbol("t%d" % g[2]) if values is None else float(values[g[2]])
            out.append(Command(GateType.Ry if g[0] == "ry" else GateType.Rz, (g[1],), (p,)))
        elif g[0] == "u":
            out.append(custom((g[1],), g[2]))
        elif g[0] in ("cx", "cz"):
            out.append(Command(GateType.CX if g[0] == "cx" else GateType.CZ, (g[1], g[2])))
        elif g[0] == "bond":
            out += [Command(t, (g[1], g[2]), (2.0 * g[3],)) for t in (GateType.RXX, GateType.RYY, GateType.RZZ)]
        else:
            out.append(Command(GateType.Rz, (g[1],), (g[2],)))
    return out


def _feedforward(n, depth, rng):
    cmds = []
    for d in range(depth):
        cmds += [Command(GateType.U, (q,), tuple(rng.uniform(-3, 3, 3))) for q in range(n)]
        qs = [int(x) for x in rng.permutation(n)]
        cmds += [Command(GateType.CX, (a, b)) for a, b in zip(qs[::2], qs[1::2])]
        cmds.append(Command(GateType.RZZ, (qs[0], qs[-1]), (float(rng.uniform(-3, 3)),)))
        cmds.append(Command(GateType.Measure, (d % n,), (), None, (d % 8,)))
        cmds.append(Command(GateType.X, ((d + 1) % n,), (), None, (), (d % 8,), (True,)))
    cmds += [Command(GateType.Measure, (q,), (), None, (q % 8,)) for q in range(n)]
    return cmds


def _pauli_sum(n, terms, rng, max_weight=None, std=1.0):
    """Random terms as (x mask, z mask, coefficient) rows."""
    rows = []
    for _ in range(terms):
        x = z = 0
        if max_weight is None:
            support = list(range(n))
            letters = rng.integers(0, 4, n)
        else:
            support = rng.choice(n, size=int(rng.integers(1, min(max_weight, n) + 1)), replace=False)
            letters = rng.integers(1, 4, len(support))
        for q, l in zip(support, letters):
            x |= (int(l) in (1, 2)) << int(q)
            z |= (int(l) in (2, 3)) << int(q)
        rows.append((x, z, float(rng.normal(0.0, std))))
    return rows


def _ising(n):
    return [(0, 3 << q, 1.0) for q in range(n - 1)] + [(1 << q, 0, 1.0) for q in range(n)]


def _masks(rows):
    c = np.zeros(2 * len(rows))
    c[0::2] = [r[2] for r in rows]
    return PauliMasks(np.array([r[0] for r in rows], dtype=np.uint64), np.array([r[1] for r in rows], dtype=np.uint64), c)


def _regular_graph(n, rng):
    while True:
        pairs = np.sort(rng.permutation(np.repeat(np.arange(n), 3)).reshape(-1, 2), axis=1)
        if np.all(pairs[:, 0] != pairs[:, 1]) and len(np.unique(pairs[:, 0] * n + pairs[:, 1])) == len(pairs):
            return [(int(a), int(b)) for a, b in pairs]


# the inputs of one case, from the seed alone (shared by prepare and exact)

def _inputs(case, seed):
    rng = np.random.default_rng([int(seed), 77])
    kind = case["kind"]
    if kind in ("call", "variational"):
        gates, k = _hea(case["n"], case["layers"])
        return {"gates": gates, "values": rng.uniform(0, 2 * math.pi, k),
                "obs": _pauli_sum(case["n"], case["terms"], rng)}
    if kind == "gates":
        return {"gates": _brickwork(case["n"], case["depth"], rng)}
    if kind == "trotter":
        return {"gates": _trotter(case["n"], case["steps"], rng.uniform(-1, 1, case["n"]))}
    if kind == "gradient":
        gates, k = _hea(case["n"], case["layers"])
        return {"gates": gates, "values": rng.uniform(0, 2 * math.pi, k),
                "obs": _ising(case["n"]) + _pauli_sum(case["n"], case["terms"], rng, 4, 0.1)}
    if kind == "energy":
        return {"obs": _ising(case["n"]) + _pauli_sum(case["n"], case["terms"], rng, 4, 0.1)}
    # a batch's widths and depths belong to the case; graphs, angles and observables to the seed
    if kind == "qaoa":
        out, shape = [], np.random.default_rng([case["instances"], case["lo"], case["hi"]])
        for _ in range(case["instances"]):
            n = 2 * int(shape.integers((case["lo"] + 1) // 2, case["hi"] // 2 + 1))
            p = int(shape.integers(1, 5))
            out.append((n, p, _regular_graph(n, rng), rng.uniform(0.0, math.pi, 2 * p)))
        return {"instances": out}
    if kind == "batch":
        out, shape = [], np.random.default_rng([case["instances"], case["lo"], case["hi"]])
        for _ in range(case["instances"]):
            n, layers = int(shape.integers(case["lo"], case["hi"] + 1)), int(shape.integers(1, 5))
            obs = _ising(n) + _pauli_sum(n, int(rng.integers(4, 32)), rng, 3)
            out.append((n, layers, rng.uniform(0, 2 * math.pi, 2 * n * layers), obs))
        return {"instances": out}
    return {"rng": rng}


def _random_state(n, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    a = torch.view_as_complex(torch.randn((1 << n, 2), generator=g, device="cuda", dtype=torch.float64))
    return a / math.sqrt(float(torch.view_as_real(a).square().sum()))


class _View:
    """A register's amplitudes on the device, as an array that torch reads in place."""

    def __init__(self, reg):
        self._reg = reg
        self.__cuda_array_interface__ = {"shape": (reg.dim,), "typestr": "<c16" if reg.dtype == "complex128" else "<c8",
                                         "data": (reg.device_pointer()[0], False), "version": 3}


def _amplitudes(reg):
    return torch.as_tensor(_View(reg), device="cuda")


def _simulator(case):
    sim = B200Simulator(dtype=case.get("dtype", "complex128"))
    if case["n"] >= PLANNED_QUBITS:
        sim.executor = 3
        sim.fusion_max_qubits = 1
    return sim


def prepare(case, seed):
    kind = case["kind"]
    d = _inputs(case, seed)
    s = {"case": case}
    if kind in ("call", "variational"):
        s.update(sim=_simulator(case), commands=_commands(d["gates"], d["values"]), obs=_masks(d["obs"]))
    elif kind == "gates":
        s.update(sim=_simulator(case), commands=_commands(d["gates"]))
    elif kind == "trotter":
        neel = [Command(GateType.X, (q,)) for q in range(1, case["n"], 2)]
        s.update(sim=_simulator(case), commands=neel + _commands(d["gates"]))
    elif kind == "gradient":
        names = ["t%d" % k for k in range(len(d["values"]))]
        s.update(sim=_simulator(case), commands=_commands(d["gates"]), obs=_masks(d["obs"]), names=names,
                 values={k: float(v) for k, v in zip(names, d["values"])})
    elif kind in ("energy", "sample"):
        reg = Register(case["n"])
        _amplitudes(reg).copy_(_random_state(case["n"], seed))
        s.update(reg=reg, obs=_masks(d["obs"]) if kind == "energy" else None, seed=int(seed) & 0xFFFFFF)
    elif kind == "shots":
        reg = Register(case["n"])
        if case["noisy"]:
            reg.set_noise(NoiseModel.depolarizing(0.01, "all") + NoiseModel.amplitude_damping(0.02, ["U"]))
        s.update(reg=reg, stream=pack(_feedforward(case["n"], case["depth"], d["rng"])), seed=int(seed) & 0xFFFFFF)
    elif kind == "qaoa":
        s.update(batch=QaoaBatch([QaoaInstance(n, p, e) for n, p, e, _ in d["instances"]]),
                 params=[v for _, _, _, v in d["instances"]])
    elif kind == "batch":
        b = CircuitBatch(with_gradient=True)
        built = {}
        for n, layers, values, obs in d["instances"]:
            if (n, layers) not in built:
                gates, k = _hea(n, layers)
                built[n, layers] = _commands(gates), ["t%d" % j for j in range(k)]
            commands, names = built[n, layers]
            b.add(commands, n, _masks(obs), {k: float(v) for k, v in zip(names, values)}, names)
        s.update(batch=b)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "call":
        return {"state": s["sim"].statevector(s["commands"], case["n"]),
                "energy": np.float64(s["sim"].expectation(s["commands"], case["n"], s["obs"]))}
    if kind == "variational":
        reg = s["sim"].prepared_register(s["commands"], case["n"])
        return {"state": _amplitudes(reg), "energy": np.float64(reg.expectation(s["obs"]).real)}
    if kind in ("gates", "trotter"):
        return {"state": _amplitudes(s["sim"].prepared_register(s["commands"], case["n"]))}
    if kind == "gradient":
        e, g = s["sim"].energy_and_gradient(s["commands"], case["n"], s["obs"], s["values"], s["names"])
        # a complex64 register's results carry 32-bit accuracy
        t = np.float64 if case["dtype"] == "complex128" else np.float32
        return {"energy": t(e), "gradient": np.asarray(g, dtype=t)}
    if kind == "energy":
        return {"energy": np.complex128(s["reg"].expectation(s["obs"]))}
    if kind == "sample":
        return {"outcomes": s["reg"].sample_seeded(s["seed"], case["shots"]).view(np.int64)}
    if kind == "shots":
        s["reg"].reset()
        out, cbits, _ = s["reg"].run_trajectories(s["stream"], s["seed"], case["shots"])
        return {"outcomes": out.view(np.int64), "cbits": cbits.view(np.int64)}
    e, g, _ = s["batch"].run(s["params"]) if kind == "qaoa" else s["batch"].run()
    return {"energies": e, "gradients": np.concatenate(g)}


# ------------------------------------------------------------------ work

# operations per amplitude: a general 2x2 gate 14, a real or diagonal rotation 6, exp(-i t (XX + YY + ZZ)) 8
_FLOPS = {"u": 14, "ry": 6, "rz": 6, "field": 6, "bond": 8, "cx": 0, "cz": 0}


def _gate_flops(gates, n):
    return float(sum(_FLOPS[g[0]] for g in gates)) * 2.0 ** n


def _sum_flops(rows, n):
    """<H> or H|psi>: one complex multiply-add per amplitude and X mask, one addition per term."""
    return (8.0 * len({r[0] for r in rows}) + len(rows)) * 2.0 ** n


def work(case):
    kind = case["kind"]
    if kind in ("qaoa", "batch"):
        d = _inputs(case, 1)
        flops = bytes_ = 0.0
        for inst in d["instances"]:
            if kind == "qaoa":
                n, p, edges, _ = inst
                # forward once, backward on two registers, an inner product per layer and register
                flops += 2.0 ** n * p * (3 * 6 * (n + 1) + 8 * (n + 1))
                bytes_ += 16.0 * len(edges) + 32.0 * p + 8
            else:
                n, layers, values, obs = inst
                flops += 3 * _gate_flops(_hea(n, layers)[0], n) + 8.0 * len(values) * 2.0 ** n + _sum_flops(obs, n)
                bytes_ += 16.0 * len(values) + 32.0 * len(obs) + 8
        return {"bytes": bytes_, "flops": flops}
    n = case["n"]
    amp = 8.0 if case.get("dtype") == "complex64" else 16.0
    if kind in ("call", "variational"):
        gates, _ = _hea(n, case["layers"])
        rows = _pauli_sum(n, case["terms"], np.random.default_rng(1))
        circuits = 2 if kind == "call" else 1
        return {"bytes": 16.0 * 2.0 ** n, "flops": circuits * _gate_flops(gates, n) + _sum_flops(rows, n)}
    if kind in ("gates", "trotter"):
        gates = _inputs(case, 1)["gates"]
        return {"bytes": amp * 2.0 ** n, "flops": _gate_flops(gates, n)}
    if kind == "gradient":
        d = _inputs(case, 1)
        # the register, its H|psi>, and both once more in the reverse sweep
        return {"bytes": 4 * amp * 2.0 ** n,
                "flops": 3 * _gate_flops(d["gates"], n) + 8.0 * len(d["values"]) * 2.0 ** n + _sum_flops(d["obs"], n)}
    if kind == "energy":
        return {"bytes": 16.0 * 2.0 ** n, "flops": _sum_flops(_inputs(case, 1)["obs"], n)}
    if kind == "sample":
        return {"bytes": 16.0 * 2.0 ** n + 16.0 * case["shots"], "flops": 4.0 * 2.0 ** n}
    gates = case["depth"] * (14.0 * n + 6.0 + 4.0)
    return {"bytes": 16.0 * case["shots"], "flops": case["shots"] * 2.0 ** n * gates}


# ------------------------------------------------------------------ the same in 64 bits, plain torch
# registers are (batch, 2^n) complex128 tensors; matrices (batch, 2, 2)

def _one(psi, q, u):
    v = psi.view(psi.shape[0], -1, 2, 1 << q)
    a, b = v[:, :, 0].clone(), v[:, :, 1]
    m = u.view(-1, 2, 2, 1, 1)
    v[:, :, 0] = m[:, 0, 0] * a + m[:, 0, 1] * b
    b.mul_(m[:, 1, 1]).add_(m[:, 1, 0] * a)


def _two(psi, a, b):
    """The register as (batch, ., bit of the higher qubit, ., bit of the lower one, .)."""
    lo, hi = min(a, b), max(a, b)
    return psi.view(psi.shape[0], -1, 2, 1 << (hi - lo - 1), 2, 1 << lo)


def _rotation(kind, theta):
    c, s = torch.cos(theta / 2), torch.sin(theta / 2)
    if kind == "ry":
        return torch.stack([c, -s, s, c], -1).view(-1, 2, 2).to(torch.complex128)
    z = torch.zeros_like(c, dtype=torch.complex128)
    return torch.stack([torch.complex(c, -s), z, z, torch.complex(c, s)], -1).view(-1, 2, 2)


def _apply(psi, gate, values=None, inverse=False):
    kind = gate[0]
    if kind in ("ry", "rz"):
        t = values[:, gate[2]]
        _one(psi, gate[1], _rotation(kind, -t if inverse else t))
    elif kind == "field":
        _one(psi, gate[1], _rotation("rz", torch.tensor([gate[2]], dtype=torch.float64, device=psi.device)))
    elif kind == "u":
        _one(psi, gate[1], torch.as_tensor(gate[2], device=psi.device))
    elif kind == "cz":
        _two(psi, gate[1], gate[2])[:, :, 1, :, 1].neg_()
    elif kind == "cx":
        v = _two(psi, gate[1], gate[2])
        if gate[1] > gate[2]:
            x, y = v[:, :, 1, :, 0], v[:, :, 1, :, 1]
        else:
            x, y = v[:, :, 0, :, 1], v[:, :, 1, :, 1]
        t = x.clone()
        x.copy_(y)
        y.copy_(t)
    else:
        # XX + YY + ZZ: 1 on |00> and |11>, -1 + 2 (exchange) on |01>, |10>
        t = gate[3]
        v = _two(psi, gate[1], gate[2])
        same = complex(math.cos(t), -math.sin(t))
        v[:, :, 0, :, 0].mul_(same)
        v[:, :, 1, :, 1].mul_(same)
        e = complex(math.cos(t), math.sin(t))
        c, s = e * math.cos(2 * t), e * complex(0.0, -math.sin(2 * t))
        x, y = v[:, :, 0, :, 1], v[:, :, 1, :, 0]
        a = x.clone()
        x.mul_(c).add_(y * s)
        y.mul_(c).add_(a * s)


def _parity(v):
    for s in (16, 8, 4, 2, 1):
        v = v ^ (v >> s)
    return v & 1


def _h_psi(psi, sums):
    """H_b |psi_b> for one list of (x, z, coefficient) rows per member of the batch."""
    dev = psi.device
    terms = max(len(r) for r in sums)
    rows = np.zeros((3, len(sums), terms))
    for b, r in enumerate(sums):
        if r:
            rows[:, b, :len(r)] = np.asarray(r, dtype=np.float64).T
    x = torch.tensor(rows[0].astype(np.int64), device=dev)
    z = torch.tensor(rows[1].astype(np.int64), device=dev)
    y = np.array([[bin(int(a) & int(c)).count("1") % 4 for a, c in zip(*m)] for m in zip(rows[0], rows[1])])
    c = torch.tensor(rows[2] * (1j ** y), device=dev)
    idx = torch.arange(psi.shape[1], device=dev).view(1, -1)
    out = torch.zeros_like(psi)
    for t in range(terms):
        src = idx ^ x[:, t:t + 1]
        sign = (1 - 2 * _parity(src & z[:, t:t + 1])).to(torch.float64)
        out += c[:, t:t + 1] * sign * torch.gather(psi, 1, src.expand(psi.shape))
    return out


def _dot(a, b):
    return (a.conj() * b).sum(dim=tuple(range(1, a.dim())))


def _zero_state(batch, n):
    psi = torch.zeros((batch, 1 << n), dtype=torch.complex128, device="cuda")
    psi[:, 0] = 1
    return psi


def _energy_gradient(n, gates, values, sums):
    values = torch.as_tensor(values, dtype=torch.float64, device="cuda")
    psi = _zero_state(values.shape[0], n)
    for g in gates:
        _apply(psi, g, values)
    lam = _h_psi(psi, sums)
    energy = _dot(psi, lam).real
    grad = torch.zeros_like(values)
    for g in reversed(gates):
        if g[0] in ("ry", "rz"):
            p, l = (r.view(r.shape[0], -1, 2, 1 << g[1]) for r in (psi, lam))
            if g[0] == "ry":     # <lam| Y psi>
                w = 1j * (_dot(l[:, :, 1], p[:, :, 0]) - _dot(l[:, :, 0], p[:, :, 1]))
            else:
                w = _dot(l[:, :, 0], p[:, :, 0]) - _dot(l[:, :, 1], p[:, :, 1])
            grad[:, g[2]] += w.imag
        _apply(psi, g, values, inverse=True)
        _apply(lam, g, values, inverse=True)
    return energy, grad


def _exact_qaoa(instances):
    energies = [None] * len(instances)
    grads = [None] * len(instances)
    groups = {}
    for i, (n, p, _, _) in enumerate(instances):
        groups.setdefault((n, p), []).append(i)
    for (n, p), members in groups.items():
        chunk = max(1, (1 << 26) >> n)
        for at in range(0, len(members), chunk):
            m = members[at:at + chunk]
            idx = torch.arange(1 << n, device="cuda")
            zz = torch.zeros((len(m), 1 << n), dtype=torch.float64, device="cuda")
            for b, i in enumerate(m):
                for u, v in instances[i][2]:
                    zz[b] += (1 - 2 * (((idx >> u) ^ (idx >> v)) & 1)).to(torch.float64)
            angles = torch.tensor(np.array([instances[i][3] for i in m]), device="cuda")
            edges = 1.5 * n
            psi = torch.full((len(m), 1 << n), 2.0 ** (-n / 2), dtype=torch.complex128, device="cuda")

            def mixer(reg, beta):
                c, s = torch.cos(beta), torch.sin(beta)
                u = torch.stack([c + 0j, -1j * s, -1j * s, c + 0j], -1).view(-1, 2, 2)
                for q in range(n):
                    _one(reg, q, u)

            for r in range(p):
                psi *= torch.exp(-1j * angles[:, 2 * r:2 * r + 1] * zz)
                mixer(psi, angles[:, 2 * r + 1])
            lam = 0.5 * (edges - zz) * psi
            e = _dot(psi, lam).real
            g = torch.zeros_like(angles)
            for r in reversed(range(p)):
                w = 0
                for q in range(n):
                    a, l = (t.view(len(m), -1, 2, 1 << q) for t in (psi, lam))
                    w = w + _dot(l[:, :, 0], a[:, :, 1]) + _dot(l[:, :, 1], a[:, :, 0])
                g[:, 2 * r + 1] = 2 * w.imag
                for reg in (psi, lam):
                    mixer(reg, -angles[:, 2 * r + 1])
                g[:, 2 * r] = 2 * _dot(lam, zz * psi).imag
                for reg in (psi, lam):
                    reg *= torch.exp(1j * angles[:, 2 * r:2 * r + 1] * zz)
            for b, i in enumerate(m):
                energies[i], grads[i] = float(e[b]), g[b].cpu().numpy()
    return {"energies": np.array(energies), "gradients": np.concatenate(grads)}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("sample", "shots"):
        return None          # whole numbers
    d = _inputs(case, seed)
    if kind == "qaoa":
        return _exact_qaoa(d["instances"])
    if kind == "batch":
        inst = d["instances"]
        groups, energies, grads = {}, [None] * len(inst), [None] * len(inst)
        for i, (n, layers, _, _) in enumerate(inst):
            groups.setdefault((n, layers), []).append(i)
        for (n, layers), m in groups.items():
            e, g = _energy_gradient(n, _hea(n, layers)[0], np.array([inst[i][2] for i in m]), [inst[i][3] for i in m])
            for b, i in enumerate(m):
                energies[i], grads[i] = float(e[b]), g[b].cpu().numpy()
        return {"energies": np.array(energies), "gradients": np.concatenate(grads)}
    n = case["n"]
    if kind == "energy":
        psi = _random_state(n, seed).view(1, -1)
        return {"energy": np.complex128(_dot(psi, _h_psi(psi, [d["obs"]])).cpu().numpy()[0])}
    if kind == "gradient":
        e, g = _energy_gradient(n, d["gates"], d["values"][None, :], [d["obs"]])
        return {"energy": np.float64(e.cpu().numpy()[0]), "gradient": g[0].cpu().numpy()}
    psi = _zero_state(1, n)
    if kind == "trotter":
        psi.zero_()
        psi[0, sum(1 << q for q in range(1, n, 2))] = 1
    values = torch.as_tensor(d["values"][None, :], device="cuda") if "values" in d else None
    for g in d["gates"]:
        _apply(psi, g, values)
    if kind in ("gates", "trotter"):
        return {"state": psi[0]}
    return {"state": psi[0], "energy": np.float64(_dot(psi, _h_psi(psi, [d["obs"]])).real.cpu().numpy()[0])}
