// The Metropolis sweep for r^-12 crowder walls.
#include "remc_sweep.cuh"

namespace {

template <bool CUT, bool FOLD>
remc::SweepFn layout(bool cluster, bool global_beads) {
  if (global_beads)
    return cluster ? remc::sweep_kernel<true, CUT, FOLD, true, true>
                   : remc::sweep_kernel<true, CUT, FOLD, false, true>;
  return cluster ? remc::sweep_kernel<true, CUT, FOLD, true, false>
                 : remc::sweep_kernel<true, CUT, FOLD, false, false>;
}

}  // namespace

remc::SweepFn remc::sweep_fn_wall(bool cut, bool fold, bool cluster, bool global_beads) {
  if (cut) return fold ? layout<true, true>(cluster, global_beads) : layout<true, false>(cluster, global_beads);
  return fold ? layout<false, true>(cluster, global_beads) : layout<false, false>(cluster, global_beads);
}
