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
