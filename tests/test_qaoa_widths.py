"""The batched QAOA kernel at the edges of its paths: one-thread half registers, layouts that the
width does not fill, the first width streamed through tiles, the last of 2^11-amplitude tiles and
both of 2^12; odd widths, repeated edges, no edges, and mixer angles on both sides of pi/4."""
import numpy as np
import pytest

from openqarp_b200 import circuits

# energies sum |C| <= E terms of unit-norm states: E * 2^-53 * (operations per amplitude, < 1e4)
TOL = 1e-10


def _instance(n, p, n_edges, seed):
    from openqarp_b200.batch import QaoaInstance
    rng = np.random.default_rng([n, p, seed])
    edges = [tuple(int(x) for x in rng.choice(n, size=2, replace=False)) for _ in range(n_edges)]
    if len(edges) > 2:
        edges[-1] = edges[0][::-1]          # the same edge again, its ends swapped
        edges[-2] = edges[0]
    return QaoaInstance(n, p, edges), rng.uniform(-7.0, 7.0, 2 * p)


@pytest.mark.gpu
@pytest.mark.parametrize("n,p", [(2, 3), (3, 2), (4, 1), (7, 4), (10, 3), (12, 2), (13, 3), (14, 2), (15, 3),
                                 (17, 1), (20, 2), (22, 1), (23, 2), (24, 1)])
def test_widths_match_per_circuit_adjoint(n, p):
    from openqarp_b200 import B200Simulator
    from openqarp_b200.batch import QaoaBatch
    made = [_instance(n, p, e, s) for s, e in enumerate((0, 1, n + n // 2) if n < 20 else (n,))]
    batch = QaoaBatch([i for i, _ in made])
    e, g, _ = batch.run([v for _, v in made])
    e2, _, _ = batch.run([v for _, v in made], with_gradient=False)
    batch.close()
    np.testing.assert_allclose(e2, e, atol=1e-12)
    sim = B200Simulator(autotune=False)
    for k, (inst, prm) in enumerate(made):
        cmds, names, cost = circuits.qaoa_maxcut(n, inst.edges, p)
        ew, gw = sim.energy_and_gradient(cmds, n, cost, dict(zip(names, prm)), names)
        assert abs(e[k] - ew) < TOL
        np.testing.assert_allclose(g[k], gw, atol=TOL)
    sim.close()


@pytest.mark.gpu
def test_cta_slots_are_shared_by_many_wide_instances():
    """More wide instances than CTAs: each CTA reuses one slot of the pool, and a second run of the
    same batch repeats the first bit for bit."""
    from openqarp_b200.batch import QaoaBatch
    made = [_instance(14 + k % 3, 1 + k % 3, 6, k) for k in range(320)]
    one = []
    for inst, prm in made[:4]:
        b = QaoaBatch([inst])
        one.append(b.run([prm])[0][0])
        b.close()
    batch = QaoaBatch([i for i, _ in made])
    e, g, _ = batch.run([v for _, v in made])
    e2, g2, _ = batch.run([v for _, v in made])
    batch.close()
    np.testing.assert_array_equal(e, e2)
    for a, b in zip(g, g2):
        np.testing.assert_array_equal(a, b)
    np.testing.assert_array_equal(e[:4], one)
