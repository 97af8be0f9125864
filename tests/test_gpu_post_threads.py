"""DRMS from two host threads at once, of structures that need shared memory
beyond the default limit in different amounts: every call's result is what the
same call gives alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_two_threads_of_different_sizes(built_lib):
    from remcdockingsimulator_b200 import post
    rng = np.random.default_rng(4)
    jobs = []
    for n in (600, 1900):  # two molecules each: 1,200 and 3,800 beads, 58 and 182 KB
        ms = np.array([0, n, 2 * n], np.int32)
        ref = rng.uniform(0.0, 200.0, (2 * n, 3)).astype(np.float32)
        frames = (ref + rng.normal(0.0, 2.0, (3, 2 * n, 3))).astype(np.float32)
        jobs.append((frames, ref, ms, post.drms(frames, ref, ms)))
    wrong = []

    def work(job):
        try:
            for _ in range(150):
                got = post.drms(*job[:3])
                for a, b in zip(got, job[3]):
                    if not np.array_equal(a, b):
                        wrong.append("another result")
                        return
        except Exception as e:
            wrong.append(repr(e))

    threads = [threading.Thread(target=work, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong[:2]
