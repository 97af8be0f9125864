"""Crowders that turn, over many refills of the ring of proposals: accumulated
rotations equal one launch per step bit for bit, in single CTAs, in replicas
spread over clusters of two and four, and beside costly systems, also where a
sampling chunk cuts the groups short."""
import numpy as np
import pytest

from test_gpu_sweep_groups import _check, _sweep, _system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chains,R,every", [
    ([20, 24], 12, 0), ([20, 24], 12, 20),      # a CTA per replica
    ([90, 100], 5, 0), ([90, 100], 5, 20),      # clusters of four
    ([90, 100], 40, 0), ([90, 100], 40, 7),     # clusters of two
])
def test_turns_over_many_refills(built_lib, chains, R, every):
    from remcdockingsimulator_b200.engine import make_params
    s = _system(2, chains, 70, 6.0, 170.0, turn=True)
    got = _sweep([s], R, make_params(), 800, 9, 128, every=every)
    want = _sweep([s], R, make_params(), 800, 9, 128, plain=True)
    for a, b in zip(got[1], want[1]):
        assert np.array_equal(a, b)
    if every:
        assert np.all(got[3][0] == 800 // every)


def test_turns_beside_costly_systems(built_lib):
    from remcdockingsimulator_b200.engine import make_params
    systems = [_system(k, [20, 25 + k], 10 + 10 * k, 6.0, 120.0, turn=True) for k in range(7)]
    systems.insert(3, _system(11, [250, 260, 240, 230], 80, 6.0, 300.0, turn=True))
    got = _sweep(systems, 20, make_params(), 160, 9, 128)
    want = _sweep(systems, 20, make_params(), 160, 9, 128, plain=True)
    for a, b in zip(got[1], want[1]):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("chains,crowders,turn", [
    ([20, 24], 0, False), ([90, 90], 0, False), ([20, 24], 12, False), ([20, 24], 40, True)])
@pytest.mark.parametrize("R,threads", [(160, 128), (340, 128), (340, 256)])
def test_cta_sizes(built_lib, chains, crowders, turn, R, threads):
    """More replicas than fit at once: CTAs of 512, 256 and 128 threads, fewer
    threads than virtual threads among them, against the oracle's trajectory and
    one launch per step."""
    from remcdockingsimulator_b200.engine import make_params
    s = _system(7, chains, crowders, 6.0, 140.0, turn=turn)
    _check([s], R, make_params(), 40, threads)


@pytest.mark.parametrize("R", [29, 30, 33, 34, 37, 60, 74])
def test_spread_where_clusters_just_fit(built_lib, R):
    """Replicas of long chain steps about as many as clusters of four and of two
    CTAs of 512 threads fit at once: the same results wherever they run."""
    from remcdockingsimulator_b200 import synth
    s = _system(9, [131, 130], 0, 6.0, 190.0)
    _check([s], R, synth.benchmark_params(), 12, 256, oracle=R == 34)


def test_replicas_about_as_many_as_clusters(built_lib):
    """Between a quarter and half as many replicas as CTAs fit: one CTA each or
    clusters apart, the same results."""
    from remcdockingsimulator_b200 import synth
    for R in (61, 76, 100):
        s = _system(9, [81, 80], 0, 6.0, 170.0)
        _check([s], R, synth.benchmark_params(), 16, 128, oracle=False)


def test_clusters_of_small_ctas(built_lib):
    """More clusters than fit with CTAs of 256 threads: of 128, fewer warps than
    virtual warps in each."""
    from remcdockingsimulator_b200.engine import make_params
    s = _system(7, [20, 24], 12, 6.0, 140.0)
    _check([s], 45, make_params(), 40, 256, cluster=8)
