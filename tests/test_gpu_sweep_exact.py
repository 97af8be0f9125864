"""One-bead steps whose sum splits into exact parts only once an earlier step of
the group has been accepted: two crowders overlap so far that a move of either
changes the energy by about 8192 kcal/mol, less after the other has moved away.
Energies equal one launch per step bit for bit, as for every other grouping."""
import numpy as np
import pytest

from test_gpu_sweep_groups import _sweep, _system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed,turn", [(1, False), (2, False), (3, True)])
def test_sums_that_split_after_an_earlier_step(built_lib, seed, turn):
    from remcdockingsimulator_b200 import synth
    from remcdockingsimulator_b200.engine import Engine
    p, systems = synth.benchmark_params(), []
    for k in range(16):
        rng = np.random.default_rng(100 * seed + k)
        s = _system(100 * seed + k, [3, 4], 7, 12.0, 130.0, turn=turn)
        a, b = [m for m in s.molecules if m.crowder][:2]
        d = rng.normal(size=3)
        d /= np.linalg.norm(d)
        b.set_position((a.pos[0] + 10.0 * d).astype(np.float32))
        with Engine([s], 1, p) as eng:
            at10 = float(eng.energy_full()[0])  # r^-12, but for the other pairs
        r = 10.0 * (at10 / rng.uniform(1.5e4, 5e4)) ** (1.0 / 12.0)
        b.set_position((a.pos[0] + r * d).astype(np.float32))
        systems.append(s)
    got = _sweep(systems, 32, p, 60, 77, 128)
    want = _sweep(systems, 32, p, 60, 77, 128, plain=True)
    assert np.all(want[0] > 8192.0)
    for a, b in zip(got[1], want[1]):
        assert np.array_equal(a, b)
