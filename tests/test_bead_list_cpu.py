"""Index arithmetic of a chain step's list of beads, compiled for the host: no
read outside a replica's beads, for any number of virtual threads and CTAs,
fewer beads than a CTA's virtual threads and one-molecule systems among them."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "remcdockingsimulator_b200", "csrc")

PROGRAM = r"""
#include "remc_sweep.cuh"
#include <cstdio>
#include <vector>
using remc::BeadList;

static int lg(int x) { int k = 0; while (1 << k < x) ++k; return k; }

int main() {
  const int sizes[] = {1, 2, 20, 31, 32, 33, 100, 127, 128, 129, 255, 257, 500, 1025, 2048, 2500};
  const int nthr = 512;
  long long fetched = 0, outside = 0;
  for (int N : sizes)
    for (int n : {1, 2, 24, 76, N / 2, N})
      for (int at = 0; at < 3; ++at)
        for (int vthr : {32, 64, 128, 256})
          for (int vsize : {1, 2, 4, 8}) {
            if (n < 1 || n > N) continue;
            const int m0 = at == 0 ? 0 : at == 1 ? (N - n) / 2 : N - n;
            const bool own = vsize > 1;
            std::vector<int> seen(N, 0);
            for (int r = 0; r < vsize; ++r) {
              const BeadList list(m0, n, own, vthr, lg(vthr), lg(vthr * vsize), r);
              const int end = list.positions(N);
              int before = -1, y;
              for (int x = 0; x < end; ++x) {
                const int j = list.bead(x, y);
                if (j <= before || j >= N || y < x || y >= list.place(N)) return 1;
                if (j >= m0 && j < m0 + n) return 2;
                ++seen[j];
                before = j;
              }
              // the residue pairs' beads, fetched by every thread of the CTA
              for (int ncb : {0, 1, 44, N}) {
                if (ncb > N) continue;
                const int xk = list.positions(ncb);
                if (xk > list.positions(N)) return 3;
                for (int spread = 0; spread < 2; ++spread) {
                  if (!remc::fetch_ahead(spread, xk, nthr / 2)) {
                    if (xk == 0 && list.bead(0, y) >= N) ++outside;
                    continue;
                  }
                  if (xk < 1) return 4;
                  for (int tid = 0; tid < nthr; ++tid) {
                    const int j = list.bead(tid - tid / xk * xk, y);
                    if (j < 0 || j >= N) return 5;
                    ++fetched;
                  }
                }
              }
            }
            for (int j = 0; j < N; ++j)
              if (seen[j] != (j >= m0 && j < m0 + n ? 0 : 1)) return 6;
          }
  // empty lists whose first position is no bead are among the cases
  if (!fetched || !outside) return 7;
  std::puts("ok");
  return 0;
}
"""


def test_bead_lists_stay_in_range(tmp_path):
    from remcdockingsimulator_b200 import build
    src, exe = tmp_path / "bead_list.cu", tmp_path / "bead_list"
    src.write_text(PROGRAM)
    r = subprocess.run([build.NVCC] + build.ARCH + ["-std=c++17", "--expt-relaxed-constexpr",
                                                    "-I" + CSRC, str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.returncode
