// The Metropolis sweep: one CTA, or a cluster of CTAs, per replica-instance,
// persistent over a block of steps (Replica::MCSearch, Replica.cpp:368-478,
// with dE in place of the full E). Included by remc_engine.cu (host side) and
// by the files that instantiate the kernel, one per crowder model.
#pragma once

#include <cooperative_groups.h>

#include <type_traits>

#include "remc_device.cuh"

namespace remc {

struct SysDev {
  int n_beads, n_mol, n_rep, lmax;
  int inst0, bead_base, mol_base, mstart_off;
  float box, invbox;
  int translate_only_crowders;
  int n_chain_beads;  // beads of residue type; the rest are crowders
  int crowd_type;     // the one bead type of every crowder, or -1 (none or mixed)
  // 1: every bead pair is within 1.5 box lengths on each axis, for the state
  // uploaded last and every state the sweep can reach from it (set on the
  // device by state_pack_kernel at each upload; the sweep then folds the
  // minimum image)
  int fold_mi;
};

// Per-step proposal record: everything about step s of one replica that does
// not depend on the replica's state (Philox draws, chosen molecule, move type,
// translation vector, step quaternion). Written by proposal_kernel for a
// whole sweep, streamed through shared memory by sweep_kernel.
struct StepRec {
  double q[4];      // step quaternion (rotation)
  double thr;       // Metropolis threshold -log(u)/beta: accept iff dE < thr
  float t[3];       // translation vector
  int m;            // molecule
  int m0;           // its first bead
  int info;         // bits 0-29: its bead count; bit 30: rotation; bit 31: crowder
};
constexpr int kRecRotate = 1 << 30;
constexpr int kRecCrowd = (int)(1u << 31);
constexpr int kRecCount = kRecRotate - 1;
static_assert(sizeof(StepRec) == 64, "StepRec layout");

// A bound conformation recorded by Replica::sample (Replica.cpp:1717-1780):
// header + one pose (rotation quaternion, centre) per molecule.
struct SampleHeader {
  int inst;
  uint32_t label;     // step label (start of the sampling chunk, main.cpp:983-987)
  double e_nc;        // potential + chain-chain pair energy (the sample() sum)
  double e;           // potential
  float temperature;
  int n_mol;
  uint32_t pose_offset;
  int pad;
};
struct SamplePose {
  double q[4];
  float c[3];
  float pad;
};


constexpr int kRing = 64;          // proposal records held in shared memory (two halves)
constexpr int kLgGroup = 3;
constexpr int kGroup = 1 << kLgGroup;  // most one-bead moves evaluated together
constexpr int kWindow = 2 * kGroup;    // most steps of a group, one-bead rotations among them
constexpr int kSweepThreads = 512; // most threads of a sweep CTA
constexpr int kSweepWarps = kSweepThreads / 32;

// Sums a pass exchanges: for a group (hi, lo) of every warp of the replica,
// then of every step's corrections by the earlier steps, at b (b - 1) / 2 + a;
// for a chain step (dE, dcc) of 8 virtual warps per CTA.
__host__ __device__ constexpr int pass_sums(int csize) {
  return 2 * (kSweepWarps * csize + kGroup * (kGroup - 1) / 2);
}

// Sizes a sweep launch lays its shared memory out for.
struct SweepShape {
  int nmax, mmax, lmax;  // beads, molecules, beads of the longest molecule
  int nrel;              // beads up to the last one of a molecule of several
  int csize;             // CTAs per replica (a thread-block cluster), 1, 2, 4 or 8
  // virtual threads, which fix the order of the sums: vsize (1 or csize) times
  // vthreads, the schedule's CTAs and threads per replica
  int vthreads, vsize;
  int mol_in_smem;       // molecule centres in shared memory (else in global memory)
  int beads_in_smem;     // beads and trial buffers in shared memory (else in global memory)
  int aj_in_smem;        // a chain step's sums per bead in shared memory
  int rel_in_smem;       // positions relative to the centres in shared memory
  int term_cap;          // terms of a chain step's split passes (0: no split passes)
};
// A chain step's sums a CTA holds: those of its own beads, rounded up to whole
// rows, where CTAs and virtual CTAs are the same; else (a replica of one virtual
// CTA on a cluster) those of all beads, in two buffers
__host__ __device__ inline int local_beads(const SweepShape& s) {
  const int g = s.vthreads * s.vsize;
  return (s.nmax + g - 1) / g * s.vthreads;
}
__host__ __device__ inline int held_sums(const SweepShape& s) {
  return local_beads(s) * (s.csize > s.vsize ? 2 : 1);
}

// The beads whose sums a chain step takes, as one CTA goes through them: all but
// the moved molecule's n from m0 on, of a replica of one virtual CTA; else those
// of them that belong to the CTA's own virtual threads. A sum's place counts the
// CTA's beads, the molecule's among them.
struct BeadList {
  bool own;            // the CTA's own virtual threads' beads
  int vthr, lgv, lgs;  // virtual threads of a CTA, logarithms of it and of the replica's
  int vrank;
  int gap, skip;       // place and number of the molecule's beads
  __host__ __device__ BeadList(int m0, int n, bool own_, int vthr_, int lgv_, int lgs_, int vrank_)
      : own(own_), vthr(vthr_), lgv(lgv_), lgs(lgs_), vrank(vrank_) {
    gap = place(m0);
    skip = place(m0 + n) - gap;
  }
  // the CTA's beads below bead e
  __host__ __device__ int place(int e) const {
    if (!own) return e;
    const int rest = (e & ((1 << lgs) - 1)) - vrank * vthr;
    return ((e >> lgs) << lgv) + (rest < 0 ? 0 : rest > vthr ? vthr : rest);
  }
  // positions of the list below bead e: all that bead() may be asked for
  __host__ __device__ int positions(int e) const {
    const int p = place(e);
    return p <= gap ? p : (gap > p - skip ? gap : p - skip);
  }
  // the bead at position x of the list, and the place y of its sum
  __host__ __device__ int bead(int x, int& y) const {
    y = x < gap ? x : x + skip;
    return own ? ((y >> lgv) << lgs) + vrank * vthr + (y & (vthr - 1)) : y;
  }
};
// Are a step's xk residue pairs' beads fetched ahead? Only of a list that has
// some, and one the threads have split among them.
__host__ __device__ inline bool fetch_ahead(bool spread, int xk, int lim) {
  return !spread && xk > 0 && xk <= lim;
}

struct SweepArgs {
  const SysDev* sys;
  const int* inst_sys;
  const int* inst_list;  // instances, largest expected cost first
  int* queue;            // work counter (persistent grid), or null: CTA b runs inst_list[b]
  int n_list;
  float4* pos;
  float4* rel;
  float4* centre;
  double* quat;
  const float4* tab;
  const StepRec* recs;   // [n_inst][rec_stride]
  double* energy;
  double* ecc;           // chain-chain part of the energy (sample() sum)
  const int* temp_idx;
  const float* ladder;
  // sampling (Replica::sample): every `sample_every` steps, labels from step0
  int sample_every;
  uint32_t sample_after;
  double bound_thr;
  const uint32_t* ctrl;
  uint32_t step0;
  int* n_samples;
  int* n_bound;
  SampleHeader* sample_out;
  SamplePose* pose_out;
  unsigned* sample_cursor;  // [0] records, [1] poses, [2] dropped
  unsigned sample_cap, pose_cap;
  int* acc_neg;          // accepted with dE < 0
  int* acc_boltz;        // accepted by the Boltzmann test
  int* rej;
  unsigned long long* evals_kh;     // residue-residue pair evaluations
  unsigned long long* evals_crowd;  // pair evaluations involving a crowder
  int rec_stride, rec_offset;       // records of step s at rec_offset + s
  int n_steps;
  SweepShape shape;
  // global memory for what is not in shared memory, per (instance, CTA rank):
  // trial positions (2 lmax entries), trial relative positions (lmax), then a
  // chain step's sums per bead
  float4* scratch;
  long long scratch_stride;
  EnergyConsts K;
};

// Shared-memory layout of sweep_kernel, in bytes.
struct SweepSmem {
  size_t tab, beads, centres, trial_pos, trial_rel, ring, sums, aj, rel, terms, total;
  static __host__ __device__ size_t take(size_t& off, size_t bytes) {
    size_t o = off;
    off += (bytes + 15) & ~size_t(15);
    return o;
  }
  static __host__ __device__ SweepSmem make(const SweepShape& p) {
    SweepSmem s;
    size_t off = 0;
    s.tab = take(off, sizeof(float4) * kNT * kNT);
    s.beads = take(off, p.beads_in_smem ? sizeof(float4) * p.nmax : 0);
    s.centres = take(off, p.mol_in_smem ? sizeof(float4) * p.mmax : 0);
    s.trial_pos = take(off, p.beads_in_smem ? sizeof(float4) * 2 * p.lmax : 0);
    s.trial_rel = take(off, p.beads_in_smem ? sizeof(float4) * p.lmax : 0);
    s.ring = take(off, sizeof(StepRec) * kRing);
    // two buffers in a cluster, where another CTA may still read the last pass's
    s.sums = take(off, sizeof(double) * (p.csize > 1 ? 2 : 1) * pass_sums(p.csize));
    s.aj = take(off, p.aj_in_smem ? sizeof(float) * held_sums(p) : 0);
    s.rel = take(off, p.rel_in_smem ? sizeof(float4) * p.nrel : 0);
    s.terms = take(off, sizeof(float) * p.term_cap);
    s.total = off;
    return s;
  }
};

#ifdef __CUDACC__

// Sum of 8 FP64 partials (16-byte aligned) in a fixed pairwise order; the
// entries of warps a smaller CTA does not have hold an exact zero. Every
// thread evaluates it and gets the same value.
__device__ __forceinline__ double tree_sum8(const double* v) {
  const double2* v2 = reinterpret_cast<const double2*>(v);
  const double2 a = v2[0], b = v2[1], c = v2[2], d = v2[3];
  return ((a.x + a.y) + (b.x + b.y)) + ((c.x + c.y) + (d.x + d.y));
}

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(gmem_src));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n"); }


// ---- one-bead crowder steps, in groups
//
// A one-bead step is short (N pairs) against the fixed chain of a step: record,
// reduction, barrier, decision. Up to kGroup one-bead crowder moves in a row
// (rotations of one bead between them, which move nothing: dE = 0) are therefore
// evaluated at once, each by its own warps and against the state before the
// group, and decided in order afterwards: step b's dE is its sum
// over that state, plus, for every earlier step a of the group that was
// accepted, the change of its sum when bead a stands at its new place.
//
// A step's dE is defined by virtual threads: virtual thread t of the replica's
// gstride adds, in FP32 and ascending j, the pairs of beads j = t (mod
// gstride), and the threads' sums are added without rounding (split_sum) and
// rounded once. A lane keeps the FP32 sums of VW virtual threads; moving bead a
// changes one virtual thread's sum, which the correction evaluates again with
// both places, and a group ends before two of its beads share a virtual
// thread. So dE, and with it every decision, is the same bit for bit for any
// grouping and any number of warps.

// What the evaluation of a one-bead crowder step needs of its replica.
struct GroupView {
  const float4* beads;
  const float4* row;  // the moved bead's row of the type table
  int N, ncb;         // beads, chain beads
  int gstride, lgs;   // virtual threads (a power of two), and its logarithm
  float Tc;           // table entry of the system's one crowder species
  bool one_ct;
  float cut2;         // crowder cutoff^2, the same for every crowder pair
  float box, invbox;
};

// An FP32 sum as hi + lo, multiples of 2^-28 and 2^-71 (what lies below 2^-71
// is rounded off: sums down to 2^-47 keep all their bits). Sums of up to 2048
// such hi (or lo) parts of |x| < 2^13 have at most 53 bits, so FP64 adds them
// without rounding, in any order.
constexpr float kSplitMax = 8192.0f;
__device__ __forceinline__ void split_sum(float x, double& hi, double& lo) {
  const double kHi = 25165824.0;            // 1.5 * 2^24
  const double kLo = 2.86102294921875e-06;  // 1.5 * 2^-19
  const double d = (double)x;
  hi = __dsub_rn(__dadd_rn(d, kHi), kHi);
  lo = __dsub_rn(__dadd_rn(__dsub_rn(d, hi), kLo), kLo);
}
__device__ __forceinline__ bool split_fits(float x) { return fabsf(x) < kSplitMax; }  // no NaN either

// Sums of hi and of lo over the warp: hi in lanes 0-15, lo in lanes 16-31.
__device__ __forceinline__ double warp_sum_split(double hi, double lo, int lane) {
  const bool upper = lane >= 16;
  double v = (upper ? lo : hi) + __shfl_xor_sync(0xffffffffu, upper ? hi : lo, 16);
#pragma unroll
  for (int off = 8; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

// A one-bead move against two beads at a time.
template <bool R12, bool CUT, bool FOLD>
struct MovedBead {
  PackedBox B;
  float2 nx, ny, nz, ox, oy, oz, C2;  // new and old place, negated
  __device__ __forceinline__ MovedBead(const GroupView& G, float4 pn, float4 po)
      : B(packed_box(G.box, G.invbox)),
        nx(make_float2(-pn.x, -pn.x)), ny(make_float2(-pn.y, -pn.y)), nz(make_float2(-pn.z, -pn.z)),
        ox(make_float2(-po.x, -po.x)), oy(make_float2(-po.y, -po.y)), oz(make_float2(-po.z, -po.z)),
        C2(make_float2(G.cut2, G.cut2)) {}
  // change of the pair energies with beads at pa and pb
  __device__ __forceinline__ float2 change(float4 pa, float4 pb, float2 A2) const {
    const float2 xj = make_float2(pa.x, pb.x), yj = make_float2(pa.y, pb.y),
                 zj = make_float2(pa.z, pb.z);
    return crowd_change2<R12, CUT>(pair_r2_2<FOLD>(xj, yj, zj, nx, ny, nz, B),
                                   pair_r2_2<FOLD>(xj, yj, zj, ox, oy, oz, B), A2, C2);
  }
};

__device__ __forceinline__ float group_entry(const GroupView& G, float4 pj, int j) {
  return (G.one_ct && j >= G.ncb) ? G.Tc : G.row[bead_type(pj.w)].x;
}

// Sums of this lane's VW virtual threads t = 32 (v0 + u) + lane for the
// one-bead step that moves bead m0 from po to pn. Two beads per packed pass:
// neighbouring virtual warps, or (VW = 1) neighbouring rows of the one.
template <bool R12, bool CUT, bool FOLD, int VW>
__device__ __forceinline__ void group_rows(const GroupView& G, const MovedBead<R12, CUT, FOLD>& mv,
                                           int lane, int v0, int m0, float* sum) {
  // general: residues, the moved bead or the end of the beads among them
  auto masked = [&](int ja, int jb) {
    const float4 pa = G.beads[min(ja, G.N - 1)], pb = G.beads[min(jb, G.N - 1)];
    float2 d = mv.change(pa, pb, make_float2(group_entry(G, pa, ja), group_entry(G, pb, jb)));
    d.x = (ja < G.N && ja != m0) ? d.x : 0.0f;
    d.y = (jb < G.N && jb != m0) ? d.y : 0.0f;
    return d;
  };
  // rows of this warp's columns: row i holds beads [base + i gstride, + 32 VW).
  // Plain rows lie past the chains (of one crowder species) and before the end
  // of the beads and do not hold the moved bead
  const float2 Tc2 = make_float2(G.Tc, G.Tc);
  const int base = 32 * v0;
  const int rows = max(0, (G.N - base + G.gstride - 1) >> G.lgs);
  const int first = G.one_ct ? max(0, (G.ncb - base + G.gstride - 1) >> G.lgs) : rows;
  const int whole = max(0, (G.N - base - 32 * VW + G.gstride) >> G.lgs);
  const int own = (unsigned)(((m0 - base) & (G.gstride - 1))) < 32u * VW ? m0 >> G.lgs : -1;
  if constexpr (VW == 1) {
    float acc = 0.0f;
    for (int i = 0; i < rows; i += 2) {
      const int j = base + (i << G.lgs) + lane;
      float2 d;
      if (i >= first && i + 2 <= whole && i != own && i + 1 != own)
        d = mv.change(G.beads[j], G.beads[j + G.gstride], Tc2);
      else
        d = masked(j, j + G.gstride);
      acc += d.x;
      acc += d.y;
    }
    sum[0] = acc;
  } else {
    float2 acc[VW / 2];
#pragma unroll
    for (int u = 0; u < VW / 2; ++u) acc[u] = make_float2(0.0f, 0.0f);
    for (int i = 0;; ++i) {
      int stop = i < first ? i : whole;
      if (own >= i && own < stop) stop = own;
      const float4* b = G.beads + base + (i << G.lgs) + lane;
#pragma unroll 2
      for (; i < stop; ++i, b += G.gstride) {
#pragma unroll
        for (int u = 0; u < VW; u += 2)
          acc[u / 2] = __fadd2_rn(acc[u / 2], mv.change(b[32 * u], b[32 * u + 32], Tc2));
      }
      if (i >= rows) break;
      const int j = base + (i << G.lgs) + lane;
#pragma unroll
      for (int u = 0; u < VW; u += 2)
        acc[u / 2] = __fadd2_rn(acc[u / 2], masked(j + 32 * u, j + 32 * u + 32));
    }
#pragma unroll
    for (int u = 0; u < VW; u += 2) {
      sum[u] = acc[u / 2].x;
      sum[u + 1] = acc[u / 2].y;
    }
  }
}

// Change of the step's sum when bead qa stands at pa instead of its place in
// the state: its virtual thread's FP32 sum again, with both places. The lanes
// of a lane group (1 << lg_lanes) take that thread's beads side by side and
// add the terms in order. False if a sum does not split.
template <bool R12, bool CUT, bool FOLD>
__device__ __forceinline__ bool group_correction(const GroupView& G,
                                                 const MovedBead<R12, CUT, FOLD>& mv, int lane,
                                                 int lg_lanes, bool active, int qa, float4 pa,
                                                 double& hi, double& lo) {
  const int lanes = 1 << lg_lanes;
  const int h = lane & (lanes - 1);
  const int t = qa & (G.gstride - 1);
  const int rows = (G.N + G.gstride - 1) >> G.lgs;
  auto bead = [&](int i) {
    const int j = (i << G.lgs) + t;
    return j < G.N ? j : -1;
  };
  float s0 = 0.0f, s1 = 0.0f;
  // terms d of rows r, r + 1, ... in the lane group's lanes, dq in place of qa's
  auto add = [&](int r, int j, float d, float dq) {
    d = (active && j >= 0) ? d : 0.0f;
    const float e = j == qa ? dq : d;
    const int n = min(lanes, rows - r);
    for (int k = 0; k < n; ++k) {
      s0 += __shfl_sync(0xffffffffu, d, k, lanes);
      s1 += __shfl_sync(0xffffffffu, e, k, lanes);
    }
  };
  const int j0 = bead(h);
  const float4 p0 = G.beads[max(j0, 0)];
  const float2 first = mv.change(p0, pa, make_float2(group_entry(G, p0, j0), group_entry(G, pa, qa)));
  add(0, j0, first.x, first.y);
  for (int r = lanes; r < rows; r += 2 * lanes) {
    const int ja = bead(r + h), jb = bead(r + lanes + h);
    const float4 p1 = G.beads[max(ja, 0)], p2 = G.beads[max(jb, 0)];
    const float2 d = mv.change(p1, p2, make_float2(group_entry(G, p1, ja), group_entry(G, p2, jb)));
    add(r, ja, d.x, first.y);
    if (r + lanes < rows) add(r + lanes, jb, d.y, first.y);
  }
  double h0, l0, h1, l1;
  split_sum(s0, h0, l0);
  split_sum(s1, h1, l1);
  hi = h1 - h0;
  lo = l1 - l0;
  return split_fits(s0) && split_fits(s1);
}

// ---- chain steps
//
// dE of a step that moves a molecule of several beads (or a one-residue chain)
// is defined by beads: bead j outside the molecule has the FP32 sum a_j over
// the moved beads k in order; virtual thread t adds the a_j of its beads j = t
// (mod gstride) in ascending j, residue pairs apart from crowder pairs (their
// sum is the change of the chain-chain energy), and the virtual warps' FP64
// sums are added in a fixed tree. Any thread may evaluate any a_j; where too
// few beads are left for all threads, any thread may evaluate any term of a_j.

// Change of the crowder-wall energy of one pair: lanes of r2 are the new and
// the old distance. last: the bead is the odd one of its virtual thread, whose
// new energy's last product enters the difference unrounded.
template <bool R12, bool CUT, bool LAST>
__device__ __forceinline__ float wall_term(float2 r2, float A, float cut2, bool last) {
  if (CUT) {
    const float2 e = crowd_energy2<R12, true>(r2, make_float2(A, A), make_float2(cut2, cut2));
    return __fsub_rn(e.x, e.y);
  }
  const float2 rinv2 = make_float2(fast_rcp(r2.x), fast_rcp(r2.y));
  const float2 i6 = __fmul2_rn(__fmul2_rn(rinv2, rinv2), rinv2);
  float2 t = make_float2(A, A);
  if (R12) t = __fmul2_rn(t, i6);
  const float2 e = __fmul2_rn(t, i6);
  const float d = __fsub_rn(e.x, e.y);
  return (LAST && last) ? __fmaf_rn(t.x, i6.x, -e.y) : d;
}

// A trial entry's last word: its bead's row of the type table, and whether the
// row holds charges (a residue type without one needs no Debye-Hueckel terms:
// 16 of the 20, 8 of some 60 issue slots of a pair).
constexpr int kRowCharged = 1 << 16, kRowMask = kRowCharged - 1;

// a_j of NJ beads per lane over the moved beads [k0, k1); with `terms` (NJ = 1)
// the terms themselves go to terms[0], terms[stride], ...
template <bool R12, bool CUT, bool FOLD, bool KH, int NJ, bool LAST, bool TERMS>
__device__ __forceinline__ void chain_terms(const float4* tp, int k0, int k1, const float4* s_tab,
                                            const float4* pj, const bool* last, const PackedBox& B,
                                            float c_xi, float cut2, float* a, float* terms,
                                            int stride) {
  float2 nx[NJ], ny[NJ], nz[NJ];
  int tj[NJ];
#pragma unroll
  for (int q = 0; q < NJ; ++q) {
    nx[q] = make_float2(-pj[q].x, -pj[q].x);
    ny[q] = make_float2(-pj[q].y, -pj[q].y);
    nz[q] = make_float2(-pj[q].z, -pj[q].z);
    tj[q] = bead_type(pj[q].w);
    if constexpr (!TERMS) a[q] = 0.0f;
  }
  // two moved beads at a time, so that their chains of operations overlap
  auto step = [&](auto two, int k) {
    constexpr int NK = decltype(two)::value ? 2 : 1;
    float2 kx[NK], ky[NK], kz[NK];
    int off[NK], any = 0;
    float d[NK][NJ];
#pragma unroll
    for (int i = 0; i < NK; ++i) {
      const float4 P = tp[2 * (k + i)], Q = tp[2 * (k + i) + 1];
      kx[i] = make_float2(P.x, P.y);
      ky[i] = make_float2(P.z, P.w);
      kz[i] = make_float2(Q.x, Q.y);
      off[i] = __float_as_int(Q.w);
      any |= off[i];
    }
    auto residues = [&](auto charged) {
#pragma unroll
      for (int i = 0; i < NK; ++i)
#pragma unroll
        for (int q = 0; q < NJ; ++q) {
          const float2 e = kh_energy2<decltype(charged)::value>(
              pair_r2_2<FOLD>(kx[i], ky[i], kz[i], nx[q], ny[q], nz[q], B),
              s_tab[(off[i] & kRowMask) + tj[q]], c_xi);
          d[i][q] = __fsub_rn(e.x, e.y);
        }
    };
    if constexpr (KH) {
      // the same for every lane where the lanes share their moved beads
      if (TERMS || (any & kRowCharged))
        residues(std::true_type{});
      else
        residues(std::false_type{});
    } else {
#pragma unroll
      for (int i = 0; i < NK; ++i)
#pragma unroll
        for (int q = 0; q < NJ; ++q)
          d[i][q] = wall_term<R12, CUT, LAST>(
              pair_r2_2<FOLD>(kx[i], ky[i], kz[i], nx[q], ny[q], nz[q], B),
              s_tab[(off[i] & kRowMask) + tj[q]].x, cut2, last[q]);
    }
#pragma unroll
    for (int i = 0; i < NK; ++i)
#pragma unroll
      for (int q = 0; q < NJ; ++q) {
        if constexpr (TERMS) {
          *terms = d[i][q];
          terms += stride;
        } else {
          a[q] += d[i][q];
        }
      }
  };
  int k = k0;
  for (; k + 2 <= k1; k += 2) step(std::true_type{}, k);
  if (k < k1) step(std::false_type{}, k);
}

// One CTA (or cluster of csize CTAs) per replica-instance, persistent over the
// sweep: the instance's beads and molecule centres stay in shared memory for
// all n_steps steps. A pass of the loop is a group of one-bead crowder steps or
// one other step; its installs are behind a barrier when the next pass begins,
// so any thread may read any bead.
// In a cluster every CTA holds the whole replica and takes every step: the work
// is split over the cluster's warps (groups) or beads (chain steps: with csize
// virtual CTAs, CTA r evaluates the beads of its own virtual threads and the
// virtual warps' sums go to every CTA's shared memory; with one, it evaluates a
// part of the list and the sums per bead go there). One cluster barrier per
// pass shows the sums; every CTA then decides and installs the same. Rank 0 alone writes state that is not
// idempotent (rotations, counters, samples) and the final state.
// GB: the beads stay where they are in global memory (updated in place, no
// prologue copy and no write-back), the trial buffers in global scratch; every
// access pattern and barrier is the same (a CTA barrier orders global memory
// for the CTA, a cluster barrier for the cluster; the CTAs of a cluster write
// identical values).
// FOLD: the minimum image is folded (every system's fold flag is set).
template <bool R12, bool CUT, bool FOLD, bool CLUSTER, bool GB>
__global__ void __launch_bounds__(kSweepThreads, 1) sweep_kernel(const SweepArgs A) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const SweepSmem L = SweepSmem::make(A.shape);
  const int held = local_beads(A.shape);
  float4* const s_tab = reinterpret_cast<float4*>(smem_raw + L.tab);
  StepRec* const s_ring = reinterpret_cast<StepRec*>(smem_raw + L.ring);
  double* const s_sums = reinterpret_cast<double*>(smem_raw + L.sums);
  float* const s_terms = reinterpret_cast<float*>(smem_raw + L.terms);
  __shared__ int s_next, s_done, s_bound, s_mask[2];
  __shared__ double s_dE[2][kWindow];  // a group's dE by step, and which were accepted
  __shared__ long long s_pose_slot;

  const int tid = threadIdx.x, nthr = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5, nwarps = nthr >> 5;
  constexpr unsigned full = 0xffffffffu;
  const int csize = CLUSTER ? A.shape.csize : 1;
  const int crank = CLUSTER ? (int)cooperative_groups::this_cluster().block_rank() : 0;
  // virtual threads: vthr of a virtual CTA, gstride of the replica (powers of two)
  const int vthr = A.shape.vthreads, vsize = CLUSTER ? A.shape.vsize : 1;
  const int vrank = vsize > 1 ? crank : 0;
  const bool spread = CLUSTER && vsize < csize;  // one virtual CTA on a cluster
  const int gstride = vthr * vsize, gmask = gstride - 1;
  const int lgv = 31 - __clz(vthr), lgs = 31 - __clz(gstride);
  // warps of the replica, real and virtual
  const int lg_warps = 31 - __clz(nwarps * csize), lg_vwarps = lgs - 5;
  // a group: up to 1 << lg_most steps, P = 1 << lgP warps each, 1 << lg_vw
  // virtual warps per warp; its corrections: 1 << lg_lanes lanes each
  const int lg_most = min(kLgGroup, lg_warps);
  const int lgP = min(lg_warps - lg_most, lg_vwarps), P = 1 << lgP;
  const int lg_vw = lg_vwarps - lgP, lg_lanes = 5 - max(0, lg_most - lgP);
  const int gw = crank * nwarps + warp;
  auto cluster_barrier = [&] {
    if (CLUSTER)
      cooperative_groups::this_cluster().sync();
    else
      __syncthreads();
  };

  // a work queue launched beside these clusters may start once all have
  if (CLUSTER) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  for (int it = 0;; ++it) {
  int idx;
  if (A.queue) {
    if (tid == 0) s_next = atomicAdd(A.queue, 1);
    __syncthreads();
    idx = s_next;
    __syncthreads();  // every thread has read s_next before it is rewritten
    if (idx >= A.n_list) break;
  } else {
    if (it > 0) break;
    idx = blockIdx.x / csize;
  }
  const int inst = A.inst_list[idx];
  const SysDev S = A.sys[A.inst_sys[inst]];
  const int slot = inst - S.inst0;
  const int N = S.n_beads, M = S.n_mol;
  const int bead_off = S.bead_base + slot * N;
  const int mol_off = S.mol_base + slot * M;
  const float box = S.box, invbox = S.invbox;
  const StepRec* const recs = A.recs + (size_t)inst * A.rec_stride + A.rec_offset;
  const int n_steps = A.n_steps;
  const int ncb = S.n_chain_beads;  // beads [0, ncb) belong to chains
  const int ctype = S.crowd_type;   // the crowders' one type, or -1
  float4* const scratch = A.scratch + ((size_t)inst * csize + crank) * A.scratch_stride;
  float4* const s_beads = GB ? A.pos + bead_off : reinterpret_cast<float4*>(smem_raw + L.beads);
  // trial positions of a chain step, two entries per moved bead k:
  // s_tpos[2 k] = (new x, old x, new y, old y), s_tpos[2 k + 1] = (new z,
  // old z, meta word, table row offset), so that each (new, old) coordinate
  // pair is a register pair of the packed pair loops as loaded; the rotated
  // relative positions; and a chain step's sums a_j by local bead
  float4* const s_tpos = GB ? scratch : reinterpret_cast<float4*>(smem_raw + L.trial_pos);
  float4* const s_trel =
      GB ? scratch + 2 * A.shape.lmax : reinterpret_cast<float4*>(smem_raw + L.trial_rel);
  float* const sums_aj = A.shape.aj_in_smem ? reinterpret_cast<float*>(smem_raw + L.aj)
                                            : reinterpret_cast<float*>(scratch + 3 * A.shape.lmax);
  float4* const rel =
      A.shape.rel_in_smem ? reinterpret_cast<float4*>(smem_raw + L.rel) : A.rel + bead_off;
  float4* const cent = A.shape.mol_in_smem ? reinterpret_cast<float4*>(smem_raw + L.centres)
                                           : A.centre + mol_off;

  // residue types with charges: the word behind the type table
  const unsigned charged = __float_as_uint(A.tab[kNT * kNT].x);

  // ---- prologue: make the instance resident in shared memory
  for (int i = tid; i < kNT * kNT; i += nthr) s_tab[i] = A.tab[i];
  if (!GB)
    for (int i = tid; i < N; i += nthr) s_beads[i] = A.pos[bead_off + i];
  if (A.shape.mol_in_smem)
    for (int i = tid; i < M; i += nthr) cent[i] = A.centre[mol_off + i];
  const int nrel = min(N, A.shape.nrel);
  if (A.shape.rel_in_smem)
    for (int i = tid; i < nrel; i += nthr) rel[i] = A.rel[bead_off + i];
  {
    // first ring fill: records of steps 0..min(kRing, n_steps)-1, 16 B per copy
    const int nrec = min(kRing, n_steps);
    const int chunks = nrec * (int)(sizeof(StepRec) / 16);
    for (int c = tid; c < chunks; c += nthr)
      cp_async16(reinterpret_cast<char*>(s_ring) + 16 * c,
                 reinterpret_cast<const char*>(recs) + 16 * c);
    cp_async_commit();
    cp_async_wait_all();
  }
  // energies: kept by warp 2 of every CTA; counters: by the lanes of warp 0
  double energy = A.energy[inst], ecc = A.ecc[inst];
  int n_neg = 0, n_boltz = 0, n_rej = 0, n_one = 0, n_samp = 0, n_bnd = 0;
  unsigned long long ev_kh = 0, ev_crowd = 0;
  const uint32_t step0 = A.ctrl ? A.ctrl[0] : A.step0;
  int to_sample = A.sample_every;  // steps left in the current sampling chunk
  // every CTA of a cluster has started before any writes another's shared memory
  cluster_barrier();
  // one-bead crowders sit at their centres, bit for bit (moves keep it so):
  // a group then reads one place per moved bead instead of two
  bool same_place = true;
  for (int i = ncb + tid; i < N; i += nthr) {
    const float4 p = s_beads[i];
    const float4 c = cent[bead_mol(p.w)];
    same_place = same_place && p.x == c.x && p.y == c.y && p.z == c.z;
  }
  const bool at_centre = __syncthreads_and(same_place);

  // A group's energies, in step order, by warp 2 (the buffer before the next one)
  int pending = 0;  // bit 0: the next group's buffer; bit 1: the other one is not added yet
  auto add_energies = [&] {
    if (warp == 2 && (pending & 2)) {
      const int at = (pending & 1) ^ 1;
      const int accepted = s_mask[at];
      for (int m = accepted; m; m &= m - 1) energy += s_dE[at][__ffs(m) - 1];
    }
    pending &= 1;
  };
  // Replica::sample at the end of the sampling chunk that ends before step
  // `done` (main.cpp:975-989): bound if potential (+ chain-chain energy when
  // crowders exist) < threshold.
  auto sample = [&](int done) {
    to_sample = A.sample_every;
    const uint32_t label = step0 + (uint32_t)(done - A.sample_every);
    if (label < A.sample_after) return;
    add_energies();
    const double enc = (ncb < N) ? energy + ecc : energy;
    if (tid == 64) {
      const bool bound = enc < A.bound_thr;
      s_bound = bound;
      ++n_samp;
      n_bnd += bound ? 1 : 0;
    }
    __syncthreads();
    if (s_bound && A.sample_out && crank == 0) {
      if (tid == 64) {
        const unsigned r = atomicAdd(&A.sample_cursor[0], 1u);
        const unsigned p0 = atomicAdd(&A.sample_cursor[1], (unsigned)M);
        if (r < A.sample_cap && (unsigned long long)p0 + M <= A.pose_cap) {
          SampleHeader hd;
          hd.inst = inst;
          hd.label = label;
          hd.e_nc = enc;
          hd.e = energy;
          hd.temperature = A.ladder[S.inst0 + A.temp_idx[inst]];
          hd.n_mol = M;
          hd.pose_offset = p0;
          hd.pad = 0;
          A.sample_out[r] = hd;
          s_pose_slot = p0;
        } else {
          atomicAdd(&A.sample_cursor[2], 1u);
          s_pose_slot = -1;
        }
      }
      __syncthreads();
      const long long p0 = s_pose_slot;
      if (p0 >= 0) {
        for (int i = tid; i < M; i += nthr) {
          const double* qd = A.quat + 4 * (size_t)(mol_off + i);
          const float4 c = cent[i];
          SamplePose ps;
          ps.q[0] = qd[0];
          ps.q[1] = qd[1];
          ps.q[2] = qd[2];
          ps.q[3] = qd[3];
          ps.c[0] = c.x;
          ps.c[1] = c.y;
          ps.c[2] = c.z;
          ps.pad = 0.0f;
          A.pose_out[p0 + i] = ps;
        }
      }
      __syncthreads();  // poses read before the next step moves anything
    }
  };

  // new centre of a translated molecule (Replica::translate); c + t + L
  // almost always lies in [0, 2L), where wrap_box subtracts L or nothing: one
  // test for all three, selects instead of branches
  auto translated = [&](float4 c, const float* t) {
    const float x0 = __fadd_rn(__fadd_rn(c.x, t[0]), box);
    const float x1 = __fadd_rn(__fadd_rn(c.y, t[1]), box);
    const float x2 = __fadd_rn(__fadd_rn(c.z, t[2]), box);
    const float L2 = 2.0f * box;  // exact
    if (x0 >= 0.0f && x0 < L2 && x1 >= 0.0f && x1 < L2 && x2 >= 0.0f && x2 < L2)
      return make_float4(x0 < box ? x0 : __fsub_rn(x0, box), x1 < box ? x1 : __fsub_rn(x1, box),
                         x2 < box ? x2 : __fsub_rn(x2, box), c.w);
    return make_float4(wrap_box(x0, box), wrap_box(x1, box), wrap_box(x2, box), c.w);
  };
  // What the next pass does, looked at ahead (it does not depend on the state):
  // lane i's record of the steps from s on, how many of them form a group (0:
  // step s is not a one-bead crowder step), and which of them move their bead.
  // The group ends before another kind of step, at the sampling chunk's end,
  // before a second move in a virtual thread or a second rotation of a
  // molecule, and before the move it has no warps for.
  int run = 0, my_m0 = 0, my_m = 0;
  unsigned movers = 0u;
  bool my_rot = false;
  float my_t[3];
  const int window = S.translate_only_crowders ? kGroup : kWindow;
  auto look = [&](int s, int readable, int chunk) {
    const bool there = lane < window && s + lane < readable && (chunk <= 0 || lane < chunk);
    const StepRec& r = s_ring[(there ? s + lane : s) & (kRing - 1)];
    my_m0 = r.m0;
    my_m = r.m;
    my_rot = (r.info & kRecRotate) != 0;
    my_t[0] = r.t[0];
    my_t[1] = r.t[1];
    my_t[2] = r.t[2];
    const bool one = there && (r.info & kRecCrowd) && (r.info & kRecCount) == 1;
    const int key = !one ? -1 - lane : my_rot ? kRecRotate | my_m0 : my_m0 & gmask;
    const unsigned moves = __ballot_sync(full, one && !my_rot);
    const unsigned before = (1u << lane) - 1u;
    // lanes from the window's end on always stop it
    bool stop = !one || (!my_rot && __popc(moves & before) >= (1 << lg_most));
    auto alike = [&](int k) {
      const int other = __shfl_up_sync(full, key, k);
      stop = stop || (lane >= k && other == key);
    };
#pragma unroll
    for (int k = 1; k < kGroup; ++k) alike(k);
    if (window > kGroup)
#pragma unroll
      for (int k = kGroup; k < kWindow; ++k) alike(k);
    run = __ffs(__ballot_sync(full, stop)) - 1;
    movers = moves & ((1u << run) - 1u);
  };

  // Records up to `avail` can be read, up to `filled` are requested. The
  // records before this pass are read by nobody any more (a pass takes what it
  // needs of its own before the barrier that ends it), and a ring half that
  // lies before it is requested anew.
  int avail = min(kRing, n_steps), filled = avail;
  int parity = 0;      // buffer of this pass's sums (clusters alternate)
  bool alone = false;  // the next step's sum does not split: taken like a chain step
  if (ncb < N && n_steps > 0) look(0, avail, to_sample);  // without crowders run stays zero
  for (int s = 0; s < n_steps;) {
    if (filled == avail && filled < n_steps && s >= filled - 32) {
      const int nrec = min(32, n_steps - filled);
      const int chunks = nrec * (int)(sizeof(StepRec) / 16);
      char* dst = reinterpret_cast<char*>(s_ring + (filled & (kRing - 1)));
      const char* src = reinterpret_cast<const char*>(recs + filled);
      for (int c = tid; c < chunks; c += nthr) cp_async16(dst + 16 * c, src + 16 * c);
      cp_async_commit();
      filled += nrec;
    }
    // requested records are waited for, and visible, at this pass's barrier
    const bool landing = filled != avail;
    if (alone) run = 0;
    alone = false;
    double* const sums = s_sums + parity * pass_sums(csize);
    float* const s_aj = sums_aj + (spread && parity ? held : 0);
    if (CLUSTER) parity ^= 1;

    if (run > 0) {
      // ---- a group of one-bead crowder steps. Lane i holds step s + i; move b
      // of the group is that of lane at(b). Warp gw takes virtual warps [p VW,
      // (p + 1) VW) of move b, gw = b P + p
      const int gsize = run, n_moves = __popc(movers);
      const int b = gw >> lgP, p = gw & (P - 1);
      int my_at = lane;  // lane b: the lane of move b
      if (n_moves < gsize) {
        unsigned m = movers;
#pragma unroll
        for (int k = 0; k < kGroup - 1; ++k)
          if (k < lane) m &= m - 1u;
        my_at = max(__ffs(m) - 1, 0);
      }
      const float4 my_old = s_beads[my_m0];
      const float4 my_new = translated(at_centre ? my_old : cent[my_m], my_t);
      if (b < n_moves) {
        const int at_b = __shfl_sync(full, my_at, b);
        const int b_m0 = __shfl_sync(full, my_m0, at_b);
        const float4 po = s_beads[b_m0];
        const float4 pn = make_float4(__shfl_sync(full, my_new.x, at_b), __shfl_sync(full, my_new.y, at_b),
                                      __shfl_sync(full, my_new.z, at_b), 0.0f);
        GroupView G;
        G.beads = s_beads;
        G.row = s_tab + bead_type(po.w) * kNT;
        G.N = N;
        G.ncb = ncb;
        G.gstride = gstride;
        G.lgs = lgs;
        G.one_ct = ctype >= 0;
        G.Tc = G.row[ctype >= 0 ? ctype : 0].x;
        G.cut2 = G.row[0].z;  // every entry of a crowder's row holds the cutoff
        G.box = box;
        G.invbox = invbox;
        // corrections by earlier moves a = p, p + P, ...: a lane group each
        const int a = ((lane >> lg_lanes) << lgP) + p;
        const bool active = a < b;
        const int at_a = __shfl_sync(full, my_at, a & (kGroup - 1));
        const int qa = __shfl_sync(full, my_m0, at_a);
        const float4 pa =
            make_float4(__shfl_sync(full, my_new.x, at_a), __shfl_sync(full, my_new.y, at_a),
                        __shfl_sync(full, my_new.z, at_a), __shfl_sync(full, my_old.w, at_a));
        double hi = 0.0, lo = 0.0, c_hi = 0.0, c_lo = 0.0;
        bool fits = true, c_fits = true;
        {
          const MovedBead<R12, CUT, FOLD> mv(G, pn, po);
          auto split = [&](float x) {
            double h, l;
            split_sum(x, h, l);
            hi += h;
            lo += l;
            fits = fits && split_fits(x);
          };
          if (lg_vw == 2) {
            float sum[4];
            group_rows<R12, CUT, FOLD, 4>(G, mv, lane, p << 2, b_m0, sum);
#pragma unroll
            for (int u = 0; u < 4; ++u) split(sum[u]);
          } else {
            for (int u = 0; u < (1 << lg_vw); ++u) {
              float sum;
              group_rows<R12, CUT, FOLD, 1>(G, mv, lane, (p << lg_vw) + u, b_m0, &sum);
              split(sum);
            }
          }
          if (__any_sync(full, active))
            c_fits = group_correction<R12, CUT, FOLD>(G, mv, lane, lg_lanes, active, qa, pa, c_hi, c_lo);
        }
        // a sum that does not split is passed on as NaN
        double tot = warp_sum_split(hi, lo, lane);
        if (!__all_sync(full, fits)) tot = NAN;
        if (!c_fits) c_hi = NAN;
        const int at_tot = 2 * gw + (lane >> 4);
        const int at_cor = 2 * kSweepWarps * csize + b * (b - 1) + 2 * a;
        const bool writes = active && (lane & ((1 << lg_lanes) - 1)) == 0;
        for (int k = 0; k < csize; ++k) {
          double* dst = sums;
          if (CLUSTER) dst = cooperative_groups::this_cluster().map_shared_rank(sums, k);
          if ((lane & 15) == 0) dst[at_tot] = tot;
          if (writes) {
            dst[at_cor] = c_hi;
            dst[at_cor + 1] = c_lo;
          }
        }
      }
      if (landing) cp_async_wait_all();
      cluster_barrier();
      if (landing) avail = filled;

      // ---- warp 0 decides the steps in order (lane b holds step b) and
      // installs; meanwhile warp 2 adds up the last group's energies, the last
      // warp fetches rotations, and all but warp 0 look at the next steps
      const StepRec& mine = s_ring[(s + (lane < gsize ? lane : 0)) & (kRing - 1)];
      const unsigned group_movers = movers;
      const bool turns = warp == nwarps - 1 && crank == 0 && lane < gsize && my_rot;
      double4 quat = make_double4(0.0, 0.0, 0.0, 0.0), turn = quat;
      double* const my_quat = A.quat + 4 * (size_t)(mol_off + my_m);
      bool accepts = false;
      if (turns) {  // the record too: behind the closing barrier its place may be refilled
        quat = make_double4(my_quat[0], my_quat[1], my_quat[2], my_quat[3]);
        turn = make_double4(mine.q[0], mine.q[1], mine.q[2], mine.q[3]);
        accepts = mine.thr > 0.0;
      }
      if (warp == 0) {
        double hi = 0.0, lo = 0.0;
        const bool moves = lane < gsize && !my_rot;
        const int my_b = __popc(group_movers & ((1u << lane) - 1u));  // moves before this lane's step
        if (moves)
          for (int w = 0; w < P; ++w) {
            const double2 x = *reinterpret_cast<const double2*>(sums + 2 * ((my_b << lgP) + w));
            hi += x.x;
            lo += x.y;
          }
        // corrections by the earlier moves of the group
        const double2* const mine_c =
            reinterpret_cast<const double2*>(sums + 2 * kSweepWarps * csize + my_b * (my_b - 1));
        double2 c[kGroup - 1];
#pragma unroll
        for (int k = 0; k < kGroup - 1; ++k) c[k] = moves && k < my_b ? mine_c[k] : make_double2(0.0, 0.0);
        const double thr = fmax(mine.thr, 0.0);  // accepted: dE < 0 or dE < thr
        double dE = hi + lo;
        unsigned left_movers = group_movers;
#pragma unroll
        for (int k = 0; k < kGroup - 1; ++k) {
          const unsigned accepted = __ballot_sync(full, dE < thr);
          if (accepted & left_movers & (0u - left_movers)) {  // move k: the lowest left (none past the end)
            hi += c[k].x;
            lo += c[k].y;
            dE = hi + lo;
          }
          left_movers &= left_movers - 1u;
        }
        // a sum that did not split (NaN) ends the group before its step
        const unsigned broke = __ballot_sync(full, lane < gsize && isnan(dE));
        const int done = broke ? __ffs(broke) - 1 : gsize;
        const bool acc = lane < done && dE < thr;
        if (acc && !my_rot) {
          s_beads[my_m0] = make_float4(my_new.x, my_new.y, my_new.z, my_old.w);
          cent[my_m] = make_float4(my_new.x, my_new.y, my_new.z, 0.0f);
        }
        const unsigned accepted = __ballot_sync(full, acc);
        if (lane < gsize) s_dE[pending & 1][lane] = dE;
        if (lane == 0) {
          s_done = done;
          s_mask[pending & 1] = (int)accepted;
        }
        // counters by lane, added up at the end
        n_neg += acc && dE < 0.0;
        n_boltz += acc && !(dE < 0.0);
        n_rej += lane < done && !acc;
        n_one += lane < done && !my_rot;
      } else if (warp == 2) {
        add_energies();
      }
      // one more look below where it cannot be right: warp 0 has been busy, or
      // the group has ended early
      const int left = to_sample <= 0 ? 0 : to_sample == gsize ? A.sample_every : to_sample - gsize;
      const bool moved_on = s + gsize < n_steps;
      if (warp != 0 && moved_on) look(s + gsize, avail, left);
      __syncthreads();  // the group's installs and s_done
      const int done = s_done;
      pending = 2 + (pending & 1 ^ 1);  // the sums just left for warp 2, the next buffer
      if (accepts && lane < done) {
        double out[4];
        quat_mul(turn.x, turn.y, turn.z, turn.w, quat.x, quat.y, quat.z, quat.w, out);
        my_quat[0] = out[0];
        my_quat[1] = out[1];
        my_quat[2] = out[2];
        my_quat[3] = out[3];
      }
      // a group's first step is evaluated against its own state: if its sum does
      // not split there, it goes alone; a later one first begins a new group
      alone = done == 0;
      s += done;
      if (to_sample > 0 && (to_sample -= done) == 0) sample(s);
      if ((warp == 0 || done < gsize) && s < n_steps) look(s, avail, to_sample);
      continue;
    }

    // ---- any other step: trial positions by bead
    const StepRec& r = s_ring[s & (kRing - 1)];  // stable for the whole pass
    const int m0 = r.m0, n = r.info & kRecCount;
    const bool rot = (r.info & kRecRotate) != 0, crowd = (r.info & kRecCrowd) != 0;
    const bool skip = rot && n == 1;  // a one-bead rotation moves nothing: dE = 0
    // the rotation a turned molecule has had, fetched ahead
    const bool turns = tid == 32 && crank == 0 && rot;
    double4 quat = make_double4(0.0, 0.0, 0.0, 0.0);
    double* const my_quat = A.quat + 4 * (size_t)(mol_off + r.m);
    if (turns) quat = make_double4(my_quat[0], my_quat[1], my_quat[2], my_quat[3]);
    const float4 c_old = cent[r.m];
    const float4 c_new = rot ? c_old : translated(c_old, r.t);
    const BeadList list(m0, n, CLUSTER && !spread, vthr, lgv, lgs, vrank);
    // is crowder pair j the odd one of its virtual thread's last pass (see
    // wall_term)? Alone in a pass: a one-residue chain's pairs, and the
    // chain beads a moved crowder meets
    auto odd_last = [&](int j) {
      if (n == 1 || j < ncb) return true;
      const int a = j < m0 ? ncb : max(m0 + n, ncb), e = j < m0 ? m0 : N;
      return j + gstride >= e && ((((j - a) >> lgs) & 1) == 0);
    };
    // At least two threads for every bead: `parts` threads per bead, each with a
    // run of the moved beads. With one thread per bead the terms' way through
    // shared memory, in rounds of a few moved beads, only costs: 300 beads on
    // 512 threads 90,000 cycles a step split, 70,000 whole
    const int cap = A.shape.term_cap, lim = min(nthr / 2, cap / 8);
    struct Split {
      int rest, part, parts, most, y;
      bool last;
      float4 pj;
    };
    // quotients of small integers: the half keeps them off the roundings
    auto quotient = [](int a, int b) { return __float2int_rd(((float)a + 0.5f) * fast_rcp((float)b)); };
    auto split = [&](bool kh, int x, int rest) {
      Split S;
      S.rest = rest;
      S.part = quotient(tid, rest);
      S.parts = quotient(nthr, rest);
      S.most = quotient(cap, rest) & ~7;  // moved beads per round
      const int j = list.bead(x + tid - S.part * rest, S.y);
      S.pj = s_beads[j];
      S.last = !kh && !CUT && odd_last(j);
      return S;
    };
    const int xk = crowd || skip ? 0 : list.positions(ncb), xe = list.positions(N);
    // Where that is all there is to the residue pairs (two short chains) it is
    // worked out, and the beads are fetched, beside the trial positions, which
    // a few warps are busy with: for 76 + 24 residues 900 to 450 cycles between
    // them and the first pair, 2.96 to 2.79 us a step with the counters of this
    // path on a warp of their own
    const bool ahead = fetch_ahead(spread, xk, lim);
    Split S0{};
    if (ahead) S0 = split(true, 0, xk);
    {
      QuatProducts qp{};
      if (rot) qp = quat_products(r.q[0], r.q[1], r.q[2], r.q[3]);
      for (int k = tid; k < n; k += nthr) {
        float3 rl = make_float3(0.0f, 0.0f, 0.0f);  // a one-bead molecule sits at its centre
        if (n > 1) {
          const float4 v = rel[m0 + k];
          rl = make_float3(v.x, v.y, v.z);
        }
        const float4 ol = s_beads[m0 + k];
        if (rot) {
          rl = rotate_rel(qp, rl.x, rl.y, rl.z);
          s_trel[k] = make_float4(rl.x, rl.y, rl.z, 0.0f);
        }
        const float4 np = make_float4(__fadd_rn(rl.x, c_new.x), __fadd_rn(rl.y, c_new.y),
                                      __fadd_rn(rl.z, c_new.z), ol.w);
        s_tpos[2 * k] = make_float4(np.x, ol.x, np.y, ol.y);
        s_tpos[2 * k + 1] = make_float4(np.z, ol.z, ol.w, __int_as_float((bead_type(ol.w) * kNT) |
                                                         (((charged >> bead_type(ol.w)) & 1u) ? kRowCharged : 0)));
      }
    }
    __syncthreads();  // trial positions
    // records this pass waits for are not readable yet: a shorter run
    if (ncb < N && s + 1 < n_steps)
      look(s + 1, avail, to_sample <= 0 ? 0 : to_sample == 1 ? A.sample_every : to_sample - 1);

    // ---- a_j of the beads outside the molecule, residue pairs then crowder pairs
    if (!skip) {
      const PackedBox PB = packed_box(box, invbox);
      const float cut2 = s_tab[(kNT - 1) * kNT].z;
      auto put_sum = [&](int y, float a) {
        if (spread)
          for (int k = 0; k < csize; ++k)
            cooperative_groups::this_cluster().map_shared_rank(s_aj, k)[y] = a;
        else
          s_aj[y] = a;
      };
      auto run_class = [&](auto kh, int x, int end) {
        constexpr bool KH = decltype(kh)::value;
        if (spread) {  // this CTA's part of the list
          const int part = (end - x + csize - 1) / csize;
          x = min(x + crank * part, end);
          end = min(x + part, end);
        }
        // one or two beads per lane, all moved beads
        auto whole = [&](auto two) {
          constexpr int NJ = decltype(two)::value ? 2 : 1;
          float4 pj[NJ];
          bool last[NJ], put[NJ];
          int y[NJ];
          float a[NJ];
          bool any_last = false;
#pragma unroll
          for (int q = 0; q < NJ; ++q) {
            const int at = x + tid + q * nthr;
            const int j = list.bead(min(at, end - 1), y[q]);
            put[q] = at < end;
            pj[q] = s_beads[j];
            last[q] = !KH && !CUT && odd_last(j);
            any_last = any_last || last[q];
          }
          if (KH || CUT || (NJ == 2 && !__any_sync(full, any_last)))
            chain_terms<R12, CUT, FOLD, KH, NJ, false, false>(s_tpos, 0, n, s_tab, pj, last, PB,
                                                              A.K.c_xi, cut2, a, nullptr, 0);
          else
            chain_terms<R12, CUT, FOLD, KH, NJ, !KH && !CUT, false>(s_tpos, 0, n, s_tab, pj, last, PB,
                                                                    A.K.c_xi, cut2, a, nullptr, 0);
#pragma unroll
          for (int q = 0; q < NJ; ++q)
            if (put[q]) put_sum(y[q], a[q]);
        };
        Split S = S0;
        if (!KH || !ahead) {
          // two beads per lane while that keeps most threads at work, then one;
          // what is left, fewer beads than threads, is split by terms
          while (end - x > nthr + nthr / 2) {
            if (x + warp * 32 + nthr < end)
              whole(std::true_type{});
            else
              whole(std::false_type{});
            x += 2 * nthr;
          }
          while (end - x > lim) {
            if (x + warp * 32 < end) whole(std::false_type{});
            x += nthr;
          }
          if (end > x) S = split(KH, x, end - x);
        }
        // the parts' threads leave the terms, and one adds them in order
        const int rest = S.rest;
        if (end > x) {
          const int part = S.part, parts = S.parts, most = S.most;
          const float4 pj = S.pj;
          const bool last = S.last;
          float a = 0.0f;
          for (int k0 = 0; k0 < n; k0 += most) {
            const int nk = min(most, n - k0);
            const int per = quotient(nk + parts - 1, parts);
            const int ka = min(part * per, nk), kb = min(ka + per, nk);
            // whole eights: terms past the last moved bead are zero
            for (int e = nk * rest + tid; e < ((nk + 7) & ~7) * rest; e += nthr) s_terms[e] = 0.0f;
            if (part < parts)
              chain_terms<R12, CUT, FOLD, KH, 1, !KH && !CUT, true>(
                  s_tpos, k0 + ka, k0 + kb, s_tab, &pj, &last, PB, A.K.c_xi, cut2, nullptr,
                  s_terms + ka * rest + tid - part * rest, rest);
            __syncthreads();
            if (tid < rest) {  // eight terms ahead of the chain of additions
              const float* t = s_terms + tid;
              float now[8];
#pragma unroll
              for (int q = 0; q < 8; ++q) now[q] = t[q * rest];
              for (int k = 8; k < nk; k += 8) {
                t += 8 * rest;
                float next[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) next[q] = t[q * rest];
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                  a += now[q];
                  now[q] = next[q];
                }
              }
#pragma unroll
              for (int q = 0; q < 8; ++q) a += now[q];
            }
            __syncthreads();
          }
          if (tid < rest) put_sum(S.y, a);
        }
      };
      if (xk > 0) run_class(std::true_type{}, 0, xk);
      if (xe > xk) run_class(std::false_type{}, xk, xe);
    }
    if (spread)  // every a_j
      cluster_barrier();
    else
      __syncthreads();

    // ---- virtual threads' sums, virtual warps' FP64 sums, one fixed tree
    // sums of residue and of crowder pairs, the first in lanes 16-31, the other
    // in 0-15, each in warp_sum's order; zero for virtual warps there are none of
    for (int w = warp; w < 8; w += nwarps) {
      double v = 0.0;
      if (32 * w < vthr) {
        float acc_c = 0.0f, acc_o = 0.0f;
        if (!skip)
          for (int y = 32 * w + lane, j = vrank * vthr + y; j < N; j += gstride, y += vthr) {
            if ((unsigned)(j - m0) < (unsigned)n) continue;
            const float a = s_aj[y];
            if (j < ncb && !crowd)
              acc_c += a;
            else
              acc_o += a;
          }
        v = warp_sum_split((double)acc_o, (double)acc_c, lane);
      }
      if ((lane & 15) == 0)
        for (int k = 0; k < vsize; ++k) {
          double* dst = sums;
          if (CLUSTER && !spread) dst = cooperative_groups::this_cluster().map_shared_rank(sums, k);
          dst[16 * vrank + (lane >> 1) + w] = v;
        }
    }
    if (landing) cp_async_wait_all();
    if (spread)
      __syncthreads();
    else
      cluster_barrier();
    if (landing) avail = filled;

    // ---- every thread takes the same decision
    double dE = tree_sum8(sums), dE_cc = 0.0;
    if (!crowd) dE_cc = tree_sum8(sums + 8);
    for (int k = 1; k < vsize; ++k) {  // the other CTAs' sums, in rank order
      dE += tree_sum8(sums + 16 * k);
      if (!crowd) dE_cc += tree_sum8(sums + 16 * k + 8);
    }
    if (!crowd) dE += dE_cc;
    const int acc = dE < 0.0 ? 1 : (dE < r.thr ? 2 : 0);
    if (acc && !skip)
      for (int k = tid; k < n; k += nthr) {
        const float4 P = s_tpos[2 * k], Q = s_tpos[2 * k + 1];
        s_beads[m0 + k] = make_float4(P.x, P.z, Q.x, Q.z);
        if (rot) rel[m0 + k] = s_trel[k];  // every CTA of a cluster: each reads its own write
      }
    add_energies();
    if (warp == 2 && acc) {
      energy += dE;
      ecc += dE_cc;
    }
    if (turns && acc) {
      double out[4];
      quat_mul(r.q[0], r.q[1], r.q[2], r.q[3], quat.x, quat.y, quat.z, quat.w, out);
      my_quat[0] = out[0];
      my_quat[1] = out[1];
      my_quat[2] = out[2];
      my_quat[3] = out[3];
    }
    if (tid == 96) {  // warps 0 to 2 have installs, the rotation, the energies
      if (acc && !rot) cent[r.m] = make_float4(c_new.x, c_new.y, c_new.z, 0.0f);
      n_neg += acc == 1;
      n_boltz += acc == 2;
      n_rej += acc == 0;
      if (!skip) {
        // two evaluations (old and new position) per pair
        const unsigned nn2 = 2u * (unsigned)n;
        if (crowd) {
          ev_crowd += (unsigned long long)nn2 * (unsigned)(N - n);
        } else {
          ev_kh += (unsigned long long)nn2 * (unsigned)(ncb - n);
          ev_crowd += (unsigned long long)nn2 * (unsigned)(N - ncb);
        }
      }
    }
    ++s;
    __syncthreads();  // the step's installs
    if (to_sample > 0 && --to_sample == 0) sample(s);
  }

  add_energies();

  // ---- epilogue: write the instance back (every CTA of a cluster holds the
  // same state; rank 0 writes it)
  if (crank == 0) {
    if (!GB)
      for (int i = tid; i < N; i += nthr) A.pos[bead_off + i] = s_beads[i];
    if (A.shape.mol_in_smem)
      for (int i = tid; i < M; i += nthr) A.centre[mol_off + i] = cent[i];
    if (A.shape.rel_in_smem)
      for (int i = tid; i < nrel; i += nthr) A.rel[bead_off + i] = rel[i];
    if (warp == 0) {
      n_neg = (int)__reduce_add_sync(full, (unsigned)n_neg);
      n_boltz = (int)__reduce_add_sync(full, (unsigned)n_boltz);
      n_rej = (int)__reduce_add_sync(full, (unsigned)n_rej);
      ev_crowd += 2ull * (unsigned)(N - 1) * __reduce_add_sync(full, (unsigned)n_one);
    }
    if (tid == 64) {
      A.energy[inst] = energy;
      A.ecc[inst] = ecc;
      A.n_samples[inst] += n_samp;
      A.n_bound[inst] += n_bnd;
    }
    if (tid == 0 || tid == 96) {  // the groups' counts, the other steps'
      atomicAdd(&A.acc_neg[inst], n_neg);
      atomicAdd(&A.acc_boltz[inst], n_boltz);
      atomicAdd(&A.rej[inst], n_rej);
      atomicAdd(&A.evals_kh[inst], ev_kh);
      atomicAdd(&A.evals_crowd[inst], ev_crowd);
    }
  }
  __syncthreads();  // shared memory is reused by the next instance
  }  // instance loop
  // no CTA leaves while another may still write into its shared memory; a work
  // queue launched beside clusters ends after them
  if (CLUSTER)
    cooperative_groups::this_cluster().sync();
  else
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

#endif  // __CUDACC__

// The sweep kernel for a crowder model: cutoff, folded minimum image, single
// CTAs or clusters of CTAs per replica, beads in shared or in global memory.
using SweepFn = void (*)(SweepArgs);
SweepFn sweep_fn_wall(bool cut, bool fold, bool cluster, bool global_beads);       // A r^-12
SweepFn sweep_fn_reference(bool cut, bool fold, bool cluster, bool global_beads);  // A r^-6

}  // namespace remc
