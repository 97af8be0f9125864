"""dE/dlambda asked for alone is the full adjoint's sum, not another one: the
call's values lie in the full call's own scatter."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chains,crowders,box", [([76, 24], 400, 200.0), ([90, 130, 60], 100, 200.0)])
def test_lambda_alone_sums_as_the_adjoint(built_lib, chains, crowders, box):
    from remcdockingsimulator_b200 import synth
    from remcdockingsimulator_b200.engine import Engine
    rng = np.random.default_rng(17)
    table = synth.contact_table(rng)
    systems = [synth.build_system(rng, table, chains, crowders, 8.0, box) for _ in range(8)]
    full, only = [], []
    with Engine(systems, 4, synth.benchmark_params()) as eng:
        for _ in range(16):
            full.append(eng.adjoint()["dE_dlambda"])
            only.append(eng.dE_dlambda())
    full, only = np.array(full), np.array(only)
    # the sums are atomics' (their order is not fixed), so calls scatter: the
    # two means differ by some sqrt(2/16) of one call's deviation; four times
    # that is beyond chance. FP64 sums over the type pairs add 1e-12
    mean = full.mean(axis=0)
    size = np.linalg.norm(mean)
    scatter = np.sqrt(np.mean(np.sum((full - mean) ** 2, axis=1)))
    assert np.linalg.norm(only.mean(axis=0) - mean) <= 4.0 * np.sqrt(2.0 / 16.0) * scatter + 1e-12 * size
