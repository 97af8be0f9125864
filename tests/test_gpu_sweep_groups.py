"""The sweep's groups of one-bead steps, its spread replicas and its split of
chain steps, at the edges of their sizes: against one launch per step (no
groups, single CTAs), bit for bit, and against the oracle's trajectory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

E_RTOL = 1e-5  # FP32 pair terms, FP64 sums: the bound of the other sweep tests


def _system(seed, chains, crowders, radius, box, radii=(), turn=False):
    from remcdockingsimulator_b200 import synth
    rng = np.random.default_rng(seed)
    s = synth.build_system(rng, synth.contact_table(np.random.default_rng(1)), chains, crowders,
                           radius, box, translate_only_crowders=not turn)
    k = 0
    for m in s.molecules:
        if m.crowder and radii:
            m.radius = radii[k % len(radii)]
            k += 1
    return s


def _sweep(systems, R, params, steps, seed, threads, cluster=1, plain=False, every=0):
    from remcdockingsimulator_b200.engine import Engine
    from remcdockingsimulator_b200.model import geometric_ladder
    n = len(systems)
    with Engine(systems, R, params) as eng:
        eng.set_replica_params([geometric_ladder(290.0, 480.0, R)] * n, np.full(n, 0.9, np.float32),
                               np.full(n, 0.3))
        eng.set_schedule(threads, True)
        if cluster > 1:
            eng.set_cluster(cluster)
        if every:
            eng.set_sampling(every, 0, -1.0)
        e0 = eng.energy_full()
        (eng.sweep_plain if plain else eng.sweep)(steps, seed, 3)
        out = list(eng.download_state()) + [eng.energies()] + list(eng.counters())
        out += list(eng.pair_evaluations())
        return e0, out, eng.instance_slices(), (list(eng.sample_counters()) if every else [])


def _check(systems, R, params, steps, threads, cluster=1, oracle=True, every=0):
    from oracle import bindings as ob
    from remcdockingsimulator_b200.model import geometric_ladder
    e0, got, slices, sampled = _sweep(systems, R, params, steps, 51, threads, cluster, every=every)
    if cluster == 1:
        want = _sweep(systems, R, params, steps, 51, threads, plain=True)[1]
        for a, b in zip(got, want):
            assert np.array_equal(a, b)
    if every:
        assert np.all(sampled[0] == steps // every)
    if not oracle:
        return
    lad = geometric_ladder(290.0, 480.0, R)
    for q, s in enumerate(systems):
        o = ob.FP64Oracle(s, params)
        for k in sorted({0, R - 1}):
            g = q * R + k
            st, E, _, _, dE, cnt = o.mc_run(s.state(), float(lad[k]), float(np.float32(0.9)), 0.3, 51,
                                            3, k, q, steps, float(e0[g]), energy_mode=0)
            bs, ms = slices[g]
            assert tuple(c[g] for c in got[5:8]) == cnt
            for a, b in zip((got[0][bs], got[1][bs], got[2][ms], got[3][ms]), st):
                assert np.array_equal(a, b)
            assert abs(got[4][g] - E) <= E_RTOL * max(np.abs(dE).sum(), abs(E), 1e-3)


@pytest.mark.parametrize("crowders", [1, 2, 7, 8, 9, 17, 83, 84, 85])
@pytest.mark.parametrize("model,turn", [("wall", False), ("reference", True)])
def test_groups_by_crowders(built_lib, crowders, model, turn):
    """Fewer crowders than a group's steps, as many, more; 127 to 129 beads."""
    from remcdockingsimulator_b200 import synth
    from remcdockingsimulator_b200.engine import make_params
    p = synth.benchmark_params() if model == "wall" else make_params()
    s = _system(crowders, [20, 24], crowders, 6.0, 130.0, turn=turn)
    _check([s], 3, p, 97, 128)


@pytest.mark.parametrize("threads,cluster", [(32, 1), (64, 1), (256, 1), (32, 2), (128, 2), (64, 4)])
@pytest.mark.parametrize("turn,radii", [(False, ()), (True, (6.0, 4.0))])
def test_groups_by_schedule(built_lib, threads, cluster, turn, radii):
    """Virtual threads and CTAs; turning crowders, crowders of two radii; the
    groups end at sampling chunks."""
    from remcdockingsimulator_b200 import synth
    s = _system(3, [1, 33, 40], 200, 6.0, 140.0, radii, turn)
    _check([s], 3, synth.benchmark_params(), 120, threads, cluster, every=12)


@pytest.mark.parametrize("chains,crowders,R", [
    ([90, 100], 60, 3), ([90, 100], 60, 40), ([90, 100], 60, 80),  # four, two and one CTA per replica
    ([1, 2], 0, 2), ([76, 24], 0, 2), ([200, 199], 0, 2), ([384, 130], 0, 2), ([380, 360], 0, 2),
])
def test_chain_steps(built_lib, chains, crowders, R):
    """Beads outside the moved chain fewer than the threads, about as many, more."""
    from remcdockingsimulator_b200 import synth
    s = _system(4, chains, crowders, 6.0, 220.0)
    _check([s], R, synth.benchmark_params(), 41, 128)


def test_costly_systems_apart(built_lib):
    """One large system among small ones, more replicas than SMs."""
    from remcdockingsimulator_b200 import synth
    systems = [_system(k, [20, 25 + k], 10 * k, 6.0, 120.0) for k in range(7)]
    systems.insert(3, _system(11, [250, 260, 240, 230], 80, 6.0, 300.0))
    _check(systems, 20, synth.benchmark_params(), 24, 128)


@pytest.mark.parametrize("gap", [2.0, 0.5])
def test_overlapping_crowders(built_lib, gap):
    """Crowders that start almost on top of one another: energies from 1e13 up,
    whose sums do not split into exact parts, so that the steps go singly."""
    from remcdockingsimulator_b200 import synth
    s = _system(6, [20, 24], 40, 12.0, 200.0)
    cr = [m for m in s.molecules if m.crowder]
    for a, b in zip(cr[0:12:2], cr[1:12:2]):
        b.set_position((a.pos[0] + np.array([gap, 0, 0], np.float32)).astype(np.float32))
    _check([s], 3, synth.benchmark_params(), 200, 128, oracle=False)


@pytest.mark.parametrize("inst,bead", [(0, 0), (5, 1500), (11, 1023), (23, 1601)])
def test_a_bad_bead_anywhere_is_refused(built_lib, inst, bead):
    from remcdockingsimulator_b200 import synth
    from remcdockingsimulator_b200._capi import RemcError
    from remcdockingsimulator_b200.engine import Engine
    s = _system(8, [400, 401, 400, 401], 0, 6.0, 320.0)
    with Engine([s] * 12, 2, synth.benchmark_params()) as eng:
        before = eng.download_state()
        flags = eng.fold_flags()
        pos, rel, cen, quat = [np.concatenate([a] * 24) for a in s.state()]
        bad = rel.copy()
        bad[inst * s.n_beads + bead, 2] = np.inf
        with pytest.raises(RemcError, match="instance %d bead %d: non-finite" % (inst, bead)):
            eng.upload_state(pos, bad, cen, quat)
        for a, b in zip(before, eng.download_state()):
            assert np.array_equal(a, b)
        eng.upload_state(pos, rel, cen, quat)
        assert np.array_equal(eng.fold_flags(), flags)
