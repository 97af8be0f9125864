// Batched post-processing (include/remc_post.h): pose reconstruction of bound
// conformations and DRMS against a reference conformation.
//
// Reconstruction follows pdbgen (post processor/pdbgensrc/pdbgen.cpp:166-215)
// in the reference's precisions: the pose quaternion is normalised twice in
// FP64 (pdbgen, then Molecule::setRotation), relative positions are rotated
// by Quaternion::rotateVector (FP64, rounded to FP32), the centre of a shifted
// molecule moves by box * round(v / box) with v its FP32 offset from molecule
// 0's position, and bead = rel + centre in FP32. All with explicit rounding
// intrinsics, so the result is bit-identical to the host arithmetic.
//
// DRMS follows drms.cpp:7-57 (FP32 Vector3f::magnitude of the FP32 difference,
// |d_sim - d_ref| in FP32, summed in FP64); the lanes' sums are added in a fixed
// order.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <mutex>
#include <vector>

#include "../../include/remc_b200.h"
#include "../../include/remc_post.h"
#include "remc_device.cuh"
#include "remc_internal.h"

using namespace remc;

namespace {

int fail(int code, const char* msg) {
  record_error(msg);
  return code;
}

// Quaternion::normalize (Quaternion.cpp:18-27) in FP64, exact rounding.
__device__ __forceinline__ void normalize_q(double q[4]) {
  const double m = __dsqrt_rn(__dadd_rn(
      __dadd_rn(__dadd_rn(__dmul_rn(q[0], q[0]), __dmul_rn(q[1], q[1])), __dmul_rn(q[2], q[2])),
      __dmul_rn(q[3], q[3])));
  q[0] = __ddiv_rn(q[0], m);
  q[1] = __ddiv_rn(q[1], m);
  q[2] = __ddiv_rn(q[2], m);
  q[3] = __ddiv_rn(q[3], m);
}

// The image of c nearest p: c - box * round((c - p) / box), per axis in FP32
// (pdbgen.cpp:196-203, round half away from zero).
__device__ __forceinline__ float3 nearest_image(float3 c, float3 p, float box) {
  const float vx = __fsub_rn(c.x, p.x), vy = __fsub_rn(c.y, p.y), vz = __fsub_rn(c.z, p.z);
  return make_float3(__fsub_rn(c.x, __fmul_rn(box, roundf(__fdiv_rn(vx, box)))),
                     __fsub_rn(c.y, __fmul_rn(box, roundf(__fdiv_rn(vy, box)))),
                     __fsub_rn(c.z, __fmul_rn(box, roundf(__fdiv_rn(vz, box)))));
}

__global__ void rebuild_kernel(const float* __restrict__ rel0, const int* __restrict__ ms,
                               int n_mol, const int* __restrict__ shift, float3 centre0,
                               float box, const double* __restrict__ quat,
                               const float* __restrict__ centre, int n_beads,
                               float* __restrict__ pos, float* __restrict__ centre_out) {
  const int f = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const float* cf = centre + (size_t)f * n_mol * 3;
  const double* qf = quat + (size_t)f * n_mol * 4;
  // molecule 0's position after its own shift (every warp derives it)
  float3 p0 = make_float3(cf[0], cf[1], cf[2]);
  if (shift[0]) p0 = nearest_image(p0, centre0, box);
  for (int m = warp; m < n_mol; m += nw) {
    double q[4] = {qf[4 * m], qf[4 * m + 1], qf[4 * m + 2], qf[4 * m + 3]};
    normalize_q(q);  // pdbgen.cpp:191
    normalize_q(q);  // Molecule::setRotation
    const QuatProducts qp = quat_products(q[0], q[1], q[2], q[3]);
    float3 c = make_float3(cf[3 * m], cf[3 * m + 1], cf[3 * m + 2]);
    if (m == 0)
      c = p0;
    else if (shift[m])
      c = nearest_image(c, p0, box);
    if (centre_out && lane == 0) {
      float* o = centre_out + ((size_t)f * n_mol + m) * 3;
      o[0] = c.x;
      o[1] = c.y;
      o[2] = c.z;
    }
    for (int b = ms[m] + lane; b < ms[m + 1]; b += 32) {
      const float3 r = rotate_rel(qp, rel0[3 * b], rel0[3 * b + 1], rel0[3 * b + 2]);
      float* o = pos + ((size_t)f * n_beads + b) * 3;
      o[0] = __fadd_rn(r.x, c.x);
      o[1] = __fadd_rn(r.y, c.y);
      o[2] = __fadd_rn(r.z, c.z);
    }
  }
}

// The length of (dx, dy, dz) as Vector3f::magnitude computes it: FP32 squares
// summed left to right, FP32 square root.
__device__ __forceinline__ float length3(float dx, float dy, float dz) {
  return __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz)));
}
__device__ __forceinline__ float dist3(const float* a, const float* b) {
  return length3(__fsub_rn(a[0], b[0]), __fsub_rn(a[1], b[1]), __fsub_rn(a[2], b[2]));
}

constexpr int kDrmsThreads = 256;
constexpr int kDrmsFrames = 4;  // frames a CTA takes against one evaluation of the reference: a float4

// Per (group of kDrmsFrames frames, part of the i beads): a warp takes one bead
// i at a time and its lanes the beads j of later molecules, side by side. A
// reference distance (two with REVERSE) serves all frames of the group. The
// frames sit in shared memory by coordinate, the four values of a bead in one
// load (SHARED; frames too large for it are read from global memory). Bound by
// issue slots, the square roots' among them: 4 chains of 150, 500 frames, both
// orders, ran 378 us with one CTA per frame, a thread per bead i and both
// distances evaluated per frame and pair, 229 us in two CTAs per SM with a load
// per frame and a last round of 33 CTAs, 165 us now.
// out[frame][part]: sums; counts[frame][part]: native, recovered, binding pairs.
struct DrmsOut {
  double a, b;
  unsigned long long native, recovered, binding;
};
template <bool REVERSE, bool SHARED>
__global__ void __launch_bounds__(kDrmsThreads, 3) drms_kernel(
    const float* __restrict__ frames, int n_frames, const float* __restrict__ ref,
    const int* __restrict__ ms, const int* __restrict__ mol_of, int n_beads, float native_cut,
    float recovered_cut, DrmsOut* __restrict__ out) {
  extern __shared__ float4 s_x[];  // [coordinate][bead], the frames side by side
  __shared__ DrmsOut s_out[kDrmsThreads / 32][kDrmsFrames];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int f0 = blockIdx.x * kDrmsFrames, nf = min(kDrmsFrames, n_frames - f0);
  const float* x = frames + (size_t)f0 * n_beads * 3;
  if (SHARED) {
    for (int e = tid; e < n_beads * 3; e += kDrmsThreads) {
      const int bead = e / 3;
      float v[kDrmsFrames];
#pragma unroll
      for (int f = 0; f < kDrmsFrames; ++f)  // past the last frame: repeated, not written out
        v[f] = x[(size_t)min(f, nf - 1) * n_beads * 3 + e];
      s_x[(e - 3 * bead) * n_beads + bead] = make_float4(v[0], v[1], v[2], v[3]);
    }
    __syncthreads();
  }
  // coordinate c of a bead in every frame
  auto at = [&](int c, int bead, float (&v)[kDrmsFrames]) {
    if (SHARED) {
      const float4 q = s_x[c * n_beads + bead];
      v[0] = q.x;
      v[1] = q.y;
      v[2] = q.z;
      v[3] = q.w;
    } else {
#pragma unroll
      for (int f = 0; f < kDrmsFrames; ++f) v[f] = x[((size_t)min(f, nf - 1) * n_beads + bead) * 3 + c];
    }
  };
  double sa[kDrmsFrames] = {}, sb[kDrmsFrames] = {};
  unsigned cn = 0, cr[kDrmsFrames] = {}, cb[kDrmsFrames] = {};
  const int warps = (kDrmsThreads / 32) * gridDim.y;
  for (int i = blockIdx.y * (kDrmsThreads / 32) + warp; i < n_beads; i += warps) {
    const int I = mol_of[i], li = i - ms[I];
    float xi[3][kDrmsFrames];
#pragma unroll
    for (int c = 0; c < 3; ++c) at(c, i, xi[c]);
    for (int j = ms[I + 1] + lane; j < n_beads; j += 32) {  // beads of molecules J > I
      const float de = dist3(ref + 3 * i, ref + 3 * j);
      float dr = 0.0f;
      if (REVERSE) {
        // drms.cpp:45-46: the reference's molecules I and J swapped
        const int J = mol_of[j], lj = j - ms[J];
        dr = dist3(ref + 3 * (ms[J] + li), ref + 3 * (ms[I] + lj));
      }
      const bool near = de < native_cut;
      cn += near;
      float xj[3][kDrmsFrames];
#pragma unroll
      for (int c = 0; c < 3; ++c) at(c, j, xj[c]);
#pragma unroll
      for (int f = 0; f < kDrmsFrames; ++f) {
        const float ds = length3(__fsub_rn(xi[0][f], xj[0][f]), __fsub_rn(xi[1][f], xj[1][f]),
                                 __fsub_rn(xi[2][f], xj[2][f]));
        sa[f] += (double)fabsf(__fsub_rn(ds, de));
        if (REVERSE) sb[f] += (double)fabsf(__fsub_rn(ds, dr));
        cr[f] += near && ds < recovered_cut;
        cb[f] += ds < native_cut;
      }
    }
  }
  auto total = [](unsigned v) {  // 64 bits: a warp may meet 2^32 pairs
    unsigned long long t = v;
    for (int off = 16; off > 0; off >>= 1) t += __shfl_xor_sync(0xffffffffu, t, off);
    return t;
  };
#pragma unroll
  for (int f = 0; f < kDrmsFrames; ++f) {
    DrmsOut o;
    o.a = warp_sum(sa[f]);
    o.b = REVERSE ? warp_sum(sb[f]) : 0.0;
    o.native = total(cn);
    o.recovered = total(cr[f]);
    o.binding = total(cb[f]);
    if (lane == 0) s_out[warp][f] = o;
  }
  __syncthreads();
  if (tid < nf) {
    DrmsOut t = s_out[0][tid];
    for (int w = 1; w < kDrmsThreads / 32; ++w) {
      const DrmsOut o = s_out[w][tid];
      t.a += o.a;
      t.b += o.b;
      t.native += o.native;
      t.recovered += o.recovered;
      t.binding += o.binding;
    }
    out[(size_t)(f0 + tid) * gridDim.y + blockIdx.y] = t;
  }
}

// Parts a group of frames is split into, of `most`: the fewest rounds of `slots`
// resident CTAs, weighed by a part's length, which is the group's pairs over
// the parts plus the loading of the frames, some 1.5 pairs a bead. About four
// CTAs per SM instead, 625 of them for 125 groups, left a third round on 296
// slots with 33.
int drms_parts(int groups, int slots, int most, double beads_per_pair) {
  int best = 1;
  double least = INFINITY;
  for (int p = 1; p <= std::min(most, 64); ++p) {
    const long long rounds = ((long long)groups * p + slots - 1) / slots;
    const double t = (double)rounds * (1.0 / p + 1.5 * beads_per_pair);
    if (t < least) {
      least = t;
      best = p;
    }
  }
  return best;
}

// One slab of device memory for a call, from a pool per device that keeps up to
// kPoolKeep bytes between calls (the rest goes back to the driver at the next
// synchronisation). Seven allocations and frees of their own had taken most of
// a call on 1000 small frames. Stream-ordered on the legacy default stream, on
// which the calls run, so several host threads may use it at once.
constexpr size_t kPoolKeep = (size_t)64 << 20;
class Slab {
 public:
  ~Slab() {
    if (base_) cudaFreeAsync(base_, 0);
  }
  // offsets first (take), then the memory (get)
  size_t take(size_t bytes) {
    const size_t at = size_;
    size_ += (bytes + 255) & ~(size_t)255;
    return at;
  }
  int get() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices)
      return fail(REMC_ERR_CUDA, "post: no current device");
    {
      std::lock_guard<std::mutex> lock(mutex_);
      if (!pools_[dev]) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool;
        if (cudaMemPoolCreate(&pool, &props) != cudaSuccess)
          return fail(REMC_ERR_NOMEM, "post: no memory pool");
        unsigned long long keep = kPoolKeep;
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
        pools_[dev] = pool;
      }
    }
    if (cudaMallocFromPoolAsync((void**)&base_, size_ ? size_ : 1, pools_[dev], 0) != cudaSuccess) {
      base_ = nullptr;
      cudaGetLastError();
      return fail(REMC_ERR_NOMEM, "post: device allocation failed");
    }
    return REMC_OK;
  }
  template <class T>
  T* at(size_t offset) const {
    return reinterpret_cast<T*>(base_ + offset);
  }

 private:
  static constexpr int kMaxDevices = 64;
  static std::mutex mutex_;
  static cudaMemPool_t pools_[kMaxDevices];
  unsigned char* base_ = nullptr;
  size_t size_ = 0;
};
std::mutex Slab::mutex_;
cudaMemPool_t Slab::pools_[Slab::kMaxDevices] = {};

template <class T>
int copy_in(T* d, const T* h, size_t n) {
  if (n && cudaMemcpyAsync(d, h, sizeof(T) * n, cudaMemcpyHostToDevice, 0) != cudaSuccess)
    return fail(REMC_ERR_CUDA, "post: host to device copy failed");
  return REMC_OK;
}

int check_starts(const int* mol_start, int n_mol) {
  if (!mol_start || n_mol <= 0 || mol_start[0] != 0)
    return fail(REMC_ERR_INVALID, "post: mol_start must start at 0");
  for (int m = 0; m < n_mol; ++m)
    if (mol_start[m + 1] <= mol_start[m])
      return fail(REMC_ERR_INVALID, "post: every molecule needs at least one bead");
  return REMC_OK;
}

}  // namespace

extern "C" {

int remc_post_rebuild(const float* rel0, const int* mol_start, int n_mol, const int* shift,
                      const float* centre0, float box, const double* quat, const float* centre,
                      int n_frames, float* pos, float* centre_out) {
  int rc = check_starts(mol_start, n_mol);
  if (rc) return rc;
  if (!rel0 || !shift || !centre0 || !quat || !centre || !pos || n_frames < 0)
    return fail(REMC_ERR_INVALID, "post_rebuild: null argument");
  if (!(box > 0.0f) || !std::isfinite(box)) return fail(REMC_ERR_INVALID, "post_rebuild: bad box");
  if (n_frames == 0) return REMC_OK;
  const int nb = mol_start[n_mol];
  const size_t nm = (size_t)n_mol * n_frames, np = (size_t)nb * n_frames;
  Slab B;
  const size_t o_rel = B.take(sizeof(float) * 3 * nb), o_ms = B.take(sizeof(int) * (n_mol + 1)),
               o_shift = B.take(sizeof(int) * n_mol), o_q = B.take(sizeof(double) * 4 * nm),
               o_cen = B.take(sizeof(float) * 3 * nm), o_pos = B.take(sizeof(float) * 3 * np),
               o_cout = B.take(centre_out ? sizeof(float) * 3 * nm : 0);
  if ((rc = B.get())) return rc;
  float *d_rel = B.at<float>(o_rel), *d_cen = B.at<float>(o_cen), *d_pos = B.at<float>(o_pos),
        *d_cout = centre_out ? B.at<float>(o_cout) : nullptr;
  int *d_ms = B.at<int>(o_ms), *d_shift = B.at<int>(o_shift);
  double* d_q = B.at<double>(o_q);
  if ((rc = copy_in(d_rel, rel0, 3 * (size_t)nb)) || (rc = copy_in(d_ms, mol_start, n_mol + 1)) ||
      (rc = copy_in(d_shift, shift, n_mol)) || (rc = copy_in(d_q, quat, 4 * nm)) ||
      (rc = copy_in(d_cen, centre, 3 * nm)))
    return rc;
  rebuild_kernel<<<n_frames, 256>>>(d_rel, d_ms, n_mol, d_shift,
                                    make_float3(centre0[0], centre0[1], centre0[2]), box, d_q,
                                    d_cen, nb, d_pos, d_cout);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpy(pos, d_pos, sizeof(float) * 3 * np, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && centre_out)
    e = cudaMemcpy(centre_out, d_cout, sizeof(float) * 3 * nm, cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) {
    char msg[256];
    snprintf(msg, sizeof(msg), "post_rebuild: %s", cudaGetErrorString(e));
    return fail(REMC_ERR_CUDA, msg);
  }
  return REMC_OK;
}

int remc_post_drms(const float* frames, int n_frames, const float* ref, const int* mol_start,
                   int n_mol, int reverse, float native_cut, float recovered_cut, double* drms,
                   long long* native, long long* recovered, long long* binding) {
  int rc = check_starts(mol_start, n_mol);
  if (rc) return rc;
  if (!frames || !ref || !drms || n_frames < 0) return fail(REMC_ERR_INVALID, "post_drms: null argument");
  if (n_mol < 2) return fail(REMC_ERR_INVALID, "post_drms: needs at least two molecules");
  if (reverse)
    for (int m = 1; m < n_mol; ++m)
      if (mol_start[m + 1] - mol_start[m] != mol_start[1] - mol_start[0])
        return fail(REMC_ERR_INVALID, "post_drms: reverse order needs molecules of equal length");
  if (n_frames == 0) return REMC_OK;
  const int nb = mol_start[n_mol];
  std::vector<int> mol_of(nb);
  double n_pairs = 0.0;
  for (int m = 0; m < n_mol; ++m) {
    for (int b = mol_start[m]; b < mol_start[m + 1]; ++b) mol_of[b] = m;
    n_pairs += (double)(mol_start[m + 1] - mol_start[m]) * (double)(nb - mol_start[m + 1]);
  }
  // groups of frames, each in parts of the i beads
  int dev = 0, sms = 148, smem_max = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  const int groups = (n_frames + kDrmsFrames - 1) / kDrmsFrames;
  const int most = std::max(1, nb / (2 * (kDrmsThreads / 32)));
  const size_t smem = sizeof(float) * 3 * (size_t)nb * kDrmsFrames;
  const bool shared = smem + 4096 <= (size_t)smem_max;
  auto kernel = reverse ? (shared ? drms_kernel<true, true> : drms_kernel<true, false>)
                        : (shared ? drms_kernel<false, true> : drms_kernel<false, false>);
  cudaError_t e = cudaSuccess;
  if (shared && smem > 48 * 1024) {
    // always the same limit, whatever this call needs: another host thread's
    // call may be between setting it and its launch
    cudaFuncAttributes attr;
    e = cudaFuncGetAttributes(&attr, kernel);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               smem_max - (int)attr.sharedSizeBytes);
  }
  int per_sm = 0;
  if (e != cudaSuccess || cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                              &per_sm, kernel, kDrmsThreads, shared ? smem : 0) != cudaSuccess)
    per_sm = 1;
  const int parts = drms_parts(groups, std::max(1, per_sm) * sms, most, nb / n_pairs);
  const size_t n_out = (size_t)n_frames * parts;
  Slab B;
  const size_t o_x = B.take(sizeof(float) * 3 * (size_t)nb * n_frames), o_ref = B.take(sizeof(float) * 3 * nb),
               o_ms = B.take(sizeof(int) * (n_mol + 1)), o_mol = B.take(sizeof(int) * nb),
               o_out = B.take(sizeof(DrmsOut) * n_out);
  if ((rc = B.get())) return rc;
  float *d_x = B.at<float>(o_x), *d_ref = B.at<float>(o_ref);
  int *d_ms = B.at<int>(o_ms), *d_mol = B.at<int>(o_mol);
  DrmsOut* d_out = B.at<DrmsOut>(o_out);
  if ((rc = copy_in(d_ref, ref, 3 * (size_t)nb)) || (rc = copy_in(d_ms, mol_start, n_mol + 1)) ||
      (rc = copy_in(d_mol, (const int*)mol_of.data(), (size_t)nb)) ||
      (rc = copy_in(d_x, frames, 3 * (size_t)nb * n_frames)))
    return rc;
  std::vector<DrmsOut> out(n_out);
  if (e == cudaSuccess) {
    kernel<<<dim3(groups, parts), kDrmsThreads, shared ? smem : 0>>>(
        d_x, n_frames, d_ref, d_ms, d_mol, nb, native_cut, recovered_cut, d_out);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out.data(), d_out, sizeof(DrmsOut) * n_out, cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) {
    char msg[256];
    snprintf(msg, sizeof(msg), "post_drms: %s", cudaGetErrorString(e));
    return fail(REMC_ERR_CUDA, msg);
  }
  for (int f = 0; f < n_frames; ++f) {
    // drms.cpp:32 and :52: drms /= N; reverse: min(drms, drms2 / N)
    DrmsOut t = out[(size_t)f * parts];
    for (int p = 1; p < parts; ++p) {
      const DrmsOut& o = out[(size_t)f * parts + p];
      t.a += o.a;
      t.b += o.b;
      t.native += o.native;
      t.recovered += o.recovered;
      t.binding += o.binding;
    }
    double d = t.a / n_pairs;
    if (reverse) d = std::min(d, t.b / n_pairs);
    drms[f] = d;
    if (native) native[f] = (long long)t.native;
    if (recovered) recovered[f] = (long long)t.recovered;
    if (binding) binding[f] = (long long)t.binding;
  }
  return REMC_OK;
}

}  // extern "C"
