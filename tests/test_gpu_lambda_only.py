"""dE/dlambda by itself (only the chains' tiles) against the full adjoint's:
chains within a tile, over its edge, over several tiles; with and without
crowders; and a system without residue pairs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chains,crowders", [
    ([20, 30], 0), ([64, 64], 50), ([64, 65], 0), ([1, 127], 10), ([100, 90, 80, 150], 120),
    ([40], 30),  # one chain: no residue pairs
])
def test_lambda_only_equals_adjoint(built_lib, chains, crowders):
    from remcdockingsimulator_b200 import synth
    from remcdockingsimulator_b200.engine import Engine
    rng = np.random.default_rng(sum(chains) + crowders)
    table = synth.contact_table(rng)
    systems = [synth.build_system(rng, table, chains, crowders, 8.0, 130.0) for _ in range(2)]
    with Engine(systems, [3, 2], synth.benchmark_params()) as eng:
        full = eng.adjoint()
        only = eng.dE_dlambda()
        # the full adjoint adds FP32 terms in FP32 over a tile of 128 x 128
        # pairs (2^-24 per addition, 2^14 of them at most, partly cancelling):
        # 1e-5 of the sum of magnitudes; its own check against FP64 holds 1e-4
        scale = np.abs(full["dE_deps"]).sum(axis=(1, 2)) * 10.0 + 1e-12
        assert np.all(np.abs(only - full["dE_dlambda"]) <= 1e-5 * scale)
        # the same FP32 sums over a tile again, by atomics in an order of their own
        assert np.all(np.abs(only - eng.dE_dlambda()) <= 1e-5 * scale)
        g = full["dE_deps"]
        assert np.array_equal(g, np.swapaxes(g, 1, 2))
        raw = table.pairs.astype(np.float64).reshape(20, 20) - np.float64(np.float32(-2.27))
        half = np.triu(g) * raw
        assert np.allclose(half.sum(axis=(1, 2)), full["dE_dlambda"], rtol=1e-9, atol=1e-9)
