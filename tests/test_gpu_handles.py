"""Many handles, alive at the same time and ended in another order, from two
host threads: the pinned blocks that ended handles leave to later ones are
never shared by two of them."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_handles_share_no_results(built_lib):
    from remcdockingsimulator_b200 import synth
    from remcdockingsimulator_b200.engine import Engine
    table = synth.contact_table(np.random.default_rng(2))
    systems = [synth.build_system(np.random.default_rng(k), table, [6 + k, 9], 3, 6.0, 90.0)
               for k in range(6)]
    p = synth.benchmark_params()
    # one replica, and so many that the results need a larger block
    sizes = [1, 3000]
    want = []
    for s in systems:
        with Engine([s], 1, p) as eng:
            want.append(eng.energy_full()[0])
    wrong = []

    def work(seed):
        rng = np.random.default_rng(seed)
        try:
            for _ in range(3):
                alive = []
                for _ in range(12):  # more blocks than are kept, over both threads
                    k = int(rng.integers(len(systems)))
                    alive.append((k, Engine([systems[k]], sizes[int(rng.integers(2))], p)))
                for k, eng in alive:
                    eng.energy_full_async()
                for k, eng in alive:
                    if not (np.all(eng.energies() == want[k]) and np.all(eng.energy_full() == want[k])):
                        wrong.append(k)
                for i in rng.permutation(len(alive)):
                    alive[i][1].close()
        except Exception as e:
            wrong.append(repr(e))

    threads = [threading.Thread(target=work, args=(s,)) for s in (1, 2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong[:3]
