"""Orderings of the kernels that no run shows reliably, read from their source."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "remcdockingsimulator_b200", "csrc")


def _between(name, start, end):
    with open(os.path.join(CSRC, name)) as fh:
        text = fh.read()
    a = text.index(start) + len(start)
    return re.sub(r"//[^\n]*", "", text[a:text.index(end, a)])


def test_a_group_reads_its_records_before_its_closing_barrier():
    """Behind that barrier the other warps may request the ring half anew that
    holds the group's records (look reads later ones)."""
    tail = _between("remc_sweep.cuh", "__syncthreads();  // the group's installs and s_done",
                    "continue;")
    assert not re.search(r"\bmine\b|\bs_ring\b", tail)


def test_the_upload_scan_counts_a_finished_cta_between_fences():
    """Every thread may report a bad bead, so the fence before the count is
    behind the barrier that follows their reports, in the thread that counts;
    the last CTA's is before the barrier that lets its threads read them."""
    scan = _between("remc_engine.cu", "void __launch_bounds__(256) state_scan_kernel(",
                    "// the last CTA: systems by warp")
    count = scan.index("atomicAdd(&res->done")
    before = scan[scan.rindex("__syncthreads()", 0, count):count]
    after = scan[count:scan.index("__syncthreads()", count)]
    assert "__threadfence()" in before and "__threadfence()" in after
