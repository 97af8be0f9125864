"""Systems smaller than a CTA's virtual threads, and of one molecule, on every
cluster size, their beads in shared and in global memory: the oracle's
trajectory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

E_RTOL = 1e-5  # FP32 pair terms, FP64 sums: the bound of the other sweep tests


@pytest.mark.parametrize("chains,crowders", [([12, 8], 0), ([76, 24], 0), ([30], 0), ([9, 5], 6)])
@pytest.mark.parametrize("threads,cluster,in_smem", [
    (128, 1, True), (128, 4, True), (256, 8, True), (128, 2, False), (256, 4, False), (256, 8, False)])
def test_small_systems(built_lib, chains, crowders, threads, cluster, in_smem):
    from oracle import bindings as ob
    from remcdockingsimulator_b200 import synth
    from remcdockingsimulator_b200.engine import Engine
    from remcdockingsimulator_b200.model import geometric_ladder
    s = synth.build_system(np.random.default_rng(5), synth.contact_table(np.random.default_rng(1)),
                           chains, crowders, 6.0, 120.0)
    p, R, steps = synth.benchmark_params(), 2, 70
    lad = geometric_ladder(290.0, 480.0, R)
    with Engine([s], R, p) as eng:
        eng.set_replica_params([lad], np.full(1, 0.9, np.float32), np.full(1, 0.3))
        eng.set_schedule(threads, True)
        eng.set_bead_storage(in_smem)
        eng.set_cluster(cluster)
        e0 = eng.energy_full()
        eng.sweep(steps, 21, 0)
        got, energies, counters = eng.download_state(), eng.energies(), eng.counters()
        slices = eng.instance_slices()
    o = ob.FP64Oracle(s, p)
    for g in range(R):
        st, E, _, _, dE, cnt = o.mc_run(s.state(), float(lad[g]), float(np.float32(0.9)), 0.3, 21, 0,
                                        g, 0, steps, float(e0[g]), energy_mode=0)
        bs, ms = slices[g]
        assert tuple(c[g] for c in counters) == cnt
        for a, b in zip((got[0][bs], got[1][bs], got[2][ms], got[3][ms]), st):
            assert np.array_equal(a, b)
        assert abs(energies[g] - E) <= E_RTOL * max(np.abs(dE).sum(), abs(E), 1e-3)
