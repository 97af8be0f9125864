// Drop-in replacements for the reference's CUDA C ABI (include/remc_reference_abi.h),
// in the reference's own device data layout.
//
// Energy: tiled upper-triangle pair sum, one CTA per item of 128 beads i by 32
// or 128 beads j; each CTA stages its beads j (positions + metadata) in shared
// memory, each thread keeps one i bead in registers, pair terms are FP32 (MUFU
// rsqrt/ex2) and each item's sum goes to a per-item FP64 partial; the last CTA
// to finish adds the partials in a fixed order (deterministic result). Follows Replica::E (Replica.cpp:603-745) and the
// reference kernel's masking rules (CudaFunctions.cu:483-548): padding beads
// have position w < 0, beads of the same molecule share w, a pair involving a
// crowder (metadata w = -1) is (6/r)^6 inside 15 A.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <utility>

#include "../../include/remc_reference_abi.h"
#include "remc_device.cuh"
#include "remc_internal.h"

using namespace remc;

namespace {

constexpr int kRefTile = 128;
constexpr int kMaxDevices = 64;

struct RefConsts {
  float lambda_, e0, c_xi;
  float lj_scale, dh_scale;  // LJ_CF * KBT_CF, DH constant * KBT_CF
  float box, invbox;
  float cutoff2;             // crowder cutoff squared (inf: none)
};

thread_local int g_status = REMC_OK;
std::mutex g_mutex;
float g_box = 150.0f;  // BOUNDING_VALUE until CUDA_setBoxDimension (definitions.h:68)
float* g_bound_table = nullptr;
bool g_params_set = false;
remc_params g_params;

// Scratch for the per-item partials of the allocating energy calls, one
// buffer per (device, stream). A call holds its buffer's lock from the
// lookup until its last launch (and, on the synchronous path, its result
// copy) is enqueued, so calls on one stream take their turns in stream order,
// and calls on different streams or host threads never share partials.
// cudaStreamPerThread is one handle for another stream in every host thread:
// each thread has a slot of its own for it, which goes to a later thread once
// its last call has ended on the GPU, so there are as many as threads at a time.
struct ScratchSlot {
  std::mutex mu;
  double* ptr = nullptr;
  size_t cap = 0;
  cudaEvent_t used = nullptr;  // behind the last call, of a thread's slot
};
std::mutex g_slots_mutex;
std::map<std::pair<int, cudaStream_t>, std::unique_ptr<ScratchSlot>> g_slots;
// slots of threads that have ended, by device (never destroyed: threads may end late)
std::multimap<int, ScratchSlot*>& idle_slots() {
  static auto* idle = new std::multimap<int, ScratchSlot*>();
  return *idle;
}
struct ThreadSlots {
  std::map<int, ScratchSlot*> by_device;
  ~ThreadSlots() {
    std::lock_guard<std::mutex> g(g_slots_mutex);
    for (const auto& s : by_device)
      if (s.second) idle_slots().insert(s);
  }
};
thread_local ThreadSlots t_slots;

// This thread's slot for cudaStreamPerThread; null on failure.
ScratchSlot* thread_slot(int dev) {
  ScratchSlot*& mine = t_slots.by_device[dev];
  if (mine) return mine;
  std::lock_guard<std::mutex> g(g_slots_mutex);
  const auto range = idle_slots().equal_range(dev);
  for (auto it = range.first; it != range.second; ++it) {
    if (cudaEventQuery(it->second->used) == cudaSuccess) {
      mine = it->second;
      idle_slots().erase(it);
      return mine;
    }
    cudaGetLastError();  // not ready is no error
  }
  std::unique_ptr<ScratchSlot> made(new ScratchSlot());
  if (cudaEventCreateWithFlags(&made->used, cudaEventDisableTiming) != cudaSuccess) return nullptr;
  mine = made.release();
  return mine;
}

void set_status(int code, const char* what, cudaError_t e = cudaSuccess) {
  g_status = code;
  if (code != REMC_OK) {
    char buf[256];
    snprintf(buf, sizeof(buf), "%s%s%s", what, e != cudaSuccess ? ": " : "",
             e != cudaSuccess ? cudaGetErrorString(e) : "");
    record_error(buf);
  }
}

RefConsts make_consts(float* unscale = nullptr) {
  std::lock_guard<std::mutex> lock(g_mutex);
  if (!g_params_set) {
    remc_default_params(&g_params);
    g_params_set = true;
  }
  if (unscale) *unscale = 1.0f / (float)((double)g_params.kbt_cf);
  RefConsts C;
  C.lambda_ = g_params.lambda_;
  C.e0 = g_params.e0;
  C.c_xi = (float)(-1.4426950408889634 / (double)g_params.debye_length);
  C.lj_scale = (float)((double)g_params.lj_cf * (double)g_params.kbt_cf);
  C.dh_scale = (float)((double)g_params.dh_const * (double)g_params.kbt_cf);
  C.box = g_box;
  C.invbox = 1.0f / g_box;
  C.cutoff2 = g_params.crowder_cutoff > 0.0f ? g_params.crowder_cutoff * g_params.crowder_cutoff
                                             : INFINITY;
  return C;
}

// The upper triangle in items of 128 beads i by `jt` beads j (a chunk): with
// T tiles of i and C chunks of j, tile ti meets the chunks from ti * kRefTile /
// jt on. Items of a tile are numbered one after the other, tile by tile.
struct RefItems {
  int P, T, C, per;  // beads, i tiles, j chunks, chunks per tile
  __host__ __device__ int first(int ti) const { return ti * per; }
  __host__ __device__ int offset(int ti) const { return ti * C - per * (ti * (ti - 1) / 2); }
  __host__ __device__ int count() const { return offset(T); }
};
// Chunks of 32 beads while items of 128 x 128 would leave the GPU idle (a
// thread then adds 32 pairs one after the other instead of 128: 1,312 beads
// took 22.3 us in 66 items, half of them empty CTAs beside them), whole tiles
// for larger structures, whose items are many anyway.
constexpr int kRefChunk = 32;
constexpr int kRefSmallTiles = 48;
// Counters of finished items, one per number of items: the word of the items'
// counter, or -1 for structures beyond some 112,000 beads, whose call of
// milliseconds adds its partials in a second launch. A call that another one
// overlaps (a captured call replayed on another stream) shares its partials
// and may get a wrong sum, but leaves no counter off for later calls: each
// word goes round from zero to zero with every call's items, and only calls
// of as many items count in it.
constexpr int kRefCounters = 1024;
RefItems ref_items(int P, bool chunks = true) {
  RefItems it;
  it.P = P;
  it.T = (P + kRefTile - 1) / kRefTile;
  const int jt = chunks && it.T <= kRefSmallTiles ? kRefChunk : kRefTile;
  it.per = kRefTile / jt;
  it.C = (P + jt - 1) / jt;
  return it;
}

int ref_counter(const RefItems& it) {
  const int word = it.per > 1 ? it.C : kRefSmallTiles * (kRefTile / kRefChunk - 1) + it.C;
  return word < kRefCounters ? word : -1;
}

// Fixed-order sum of n partials by one CTA; thread 0 has it.
template <int THREADS>
__device__ double sum_partials(const volatile double* partials, int n, double* s) {
  double v = 0.0;
  for (int i = threadIdx.x; i < n; i += THREADS) v += partials[i];
  s[threadIdx.x] = v;
  __syncthreads();
  for (int w = THREADS / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) s[threadIdx.x] += s[threadIdx.x + w];
    __syncthreads();
  }
  return s[0];
}

// Where the total goes: *out, and the reference's per-block layout (the host
// sums it and scales by KBT_CF).
struct RefTotal {
  double* out;
  float* grid_out;
  int grid_n;
  float unscale;
};
__device__ void put_total(double total, const RefTotal& R) {
  if (threadIdx.x == 0 && R.out) *R.out = total;
  if (R.grid_out)
    for (int i = threadIdx.x; i < R.grid_n; i += blockDim.x)
      R.grid_out[i] = (i == 0) ? (float)(total * (double)R.unscale) : 0.0f;
}

// One item per CTA (chunk blockIdx.x, tile blockIdx.y). With `done` the last CTA
// to finish adds the partials, in a fixed order; the counter is then at zero.
template <int JT>
__global__ void __launch_bounds__(kRefTile) ref_energy_tiles(
    const float4* __restrict__ pos, const float4* __restrict__ meta,
    const float* __restrict__ lj_table, RefItems it, double* __restrict__ partials, RefConsts C,
    unsigned* __restrict__ done, RefTotal total) {
  const int ti = blockIdx.y, c = blockIdx.x;
  if (c < it.first(ti)) return;
  __shared__ float s_eps[400];
  __shared__ float4 s_jp[JT], s_jm[JT];
  __shared__ double s_red[kRefTile];
  __shared__ bool s_last;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < 400; i += kRefTile) s_eps[i] = C.lambda_ * (lj_table[i] - C.e0);
  const int j0 = c * JT, jn = min(JT, it.P - j0);
  if (tid < JT) {  // places past the last bead hold padding
    s_jp[tid] = tid < jn ? pos[j0 + tid] : make_float4(0.0f, 0.0f, 0.0f, -2.0f);
    s_jm[tid] = tid < jn ? meta[j0 + tid] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  }
  const int i = ti * kRefTile + tid;
  const bool valid = i < it.P;
  const float4 pi = valid ? pos[i] : make_float4(0.0f, 0.0f, 0.0f, -2.0f);
  const float4 mi = valid ? meta[i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  const bool counts = pi.w > -2.0f;  // not a padding bead
  const bool icrowd = mi.w == -1.0f;
  const float row = 20.0f * mi.x;
  const float two_third = 1.2599210498948732f;  // 2^(1/3)
  __syncthreads();
  float lj = 0.0f, dh = 0.0f;
#pragma unroll 4
  for (int jj = 0; jj < JT; ++jj) {
    const float4 pj = s_jp[jj], mj = s_jm[jj];
    // padding, the same molecule, or (diagonal) an earlier bead
    const bool use = counts && j0 + jj > i && !(pj.w < 0.0f) && pj.w != pi.w;
    const float r2 = pair_r2(pi, pj, C.box, C.invbox);
    const float rinv = fast_rsqrt(r2);
    const float rinv2 = rinv * rinv;
    if (icrowd || mj.w == -1.0f) {
      const float i6 = rinv2 * rinv2 * rinv2;
      if (use && r2 < C.cutoff2) lj += 46656.0f * i6;  // (6/r)^6
    } else if (use) {
      // rint of the index in [0, 399] (no number: 0), without a conversion
      const float in = fminf(fmaxf(__fadd_rn(row, mj.x), 0.0f), 399.0f);
      const float eps = s_eps[__float_as_int(__fadd_rn(in, 12582912.0f)) - 0x4b400000];
      const float sig = (mi.z + mj.z) * 0.5f;
      const float sig2 = sig * sig;
      const float s2 = sig2 * rinv2;
      const float s6 = s2 * s2 * s2;
      float L = 4.0f * eps * fmaf(-s6, s6, s6);
      if (eps > 0.0f && r2 < sig2 * two_third) L = 2.0f * eps - L;
      lj += L;
      const float r = r2 * rinv;
      dh += mi.y * mj.y * fast_ex2(r * C.c_xi) * rinv;
    }
  }
  double v = (double)lj * (double)C.lj_scale + (double)dh * (double)C.dh_scale;
  v = warp_sum(v);
  if (lane == 0) s_red[warp] = v;
  __syncthreads();
  if (tid == 0) {
    double t = 0.0;
    for (int w = 0; w < kRefTile / 32; ++w) t += s_red[w];
    partials[it.offset(ti) + c - it.first(ti)] = t;
    if (done) {
      const unsigned last = (unsigned)it.count() - 1u;
      __threadfence();
      s_last = atomicInc(done, last) == last;
      __threadfence();
    }
  }
  if (!done) return;
  __syncthreads();
  if (!s_last) return;
  const double sum = sum_partials<kRefTile>(partials, it.count(), s_red);
  put_total(sum, total);
}

// Fixed-order sum of n partials (one CTA), for calls without a counter.
__global__ void ref_energy_sum(const double* __restrict__ partials, int n, RefTotal total) {
  __shared__ double s[256];
  put_total(sum_partials<256>(partials, n, s), total);
}

// Launch the items and the sum of their partials: by the last CTA with `done`,
// by a launch of its own without.
cudaError_t launch_energy(const float4* pos, const float4* meta, const float* table,
                          const RefItems& it, double* partials, const RefConsts& C,
                          unsigned* done, const RefTotal& total, cudaStream_t stream) {
  const dim3 grid(it.C, it.T);
  if (it.per == 1)
    ref_energy_tiles<kRefTile><<<grid, kRefTile, 0, stream>>>(pos, meta, table, it, partials, C, done, total);
  else
    ref_energy_tiles<kRefChunk><<<grid, kRefTile, 0, stream>>>(pos, meta, table, it, partials, C, done, total);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || done) return e;
  ref_energy_sum<<<1, 256, 0, stream>>>(partials, it.count(), total);
  return cudaGetLastError();
}

__global__ void rotate_molecule_kernel(float4* pos, const int* start, const int* length,
                                       const float4* rv, const float4* center) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= *length) return;
  const float4 r = *rv;
  const float4 c = *center;
  // unit quaternion of the axis-angle (CudaFunctions.cu:798-840)
  float qw = cosf(r.w * 0.5f), sh = sinf(r.w * 0.5f);
  float qx = r.x * sh, qy = r.y * sh, qz = r.z * sh;
  const float inv = rsqrtf(qx * qx + qy * qy + qz * qz + qw * qw);
  qw *= inv;
  qx *= inv;
  qy *= inv;
  qz *= inv;
  float4& p = pos[*start + k];
  const float vx = p.x - c.x, vy = p.y - c.y, vz = p.z - c.z;
  p.x = vx * (qw * qw + qx * qx - qy * qy - qz * qz) + vy * (qx * qy - qw * qz) * 2.0f +
        vz * (qw * qy + qx * qz) * 2.0f + c.x;
  p.y = vx * (qw * qz + qx * qy) * 2.0f + vy * (qw * qw - qx * qx + qy * qy - qz * qz) +
        vz * (qy * qz - qw * qx) * 2.0f + c.y;
  p.z = vx * (qx * qz - qw * qy) * 2.0f + vy * (qy * qz + qw * qx) * 2.0f +
        vz * (qw * qw - qx * qx - qy * qy + qz * qz) + c.z;
}

__global__ void translate_molecule_kernel(float4* pos, const int* start, const int* length,
                                          const float4* t) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= *length) return;
  const float4 v = *t;
  float4& p = pos[*start + k];
  p.x += v.x;
  p.y += v.y;
  p.z += v.z;
}

// Runs after translate_molecule_kernel in stream order: the centre moves once.
__global__ void translate_center_kernel(float4* center, const float4* t) {
  const float4 v = *t;
  center->x += v.x;
  center->y += v.y;
  center->z += v.z;
}

// Sets a new buffer's counters to zero before the stream's next work: on the
// stream, or, where that is being captured (it would happen in the graph only),
// now.
bool clear_counters(double* scratch, cudaStream_t stream) {
  const size_t bytes = sizeof(unsigned) * kRefCounters;
  cudaStreamCaptureStatus capture;
  if (cudaStreamIsCapturing(stream, &capture) != cudaSuccess) return false;
  if (capture == cudaStreamCaptureStatusNone)
    return cudaMemsetAsync(scratch, 0, bytes, stream) == cudaSuccess;
  cudaStream_t s;
  if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess) return false;
  const bool ok = cudaMemsetAsync(scratch, 0, bytes, s) == cudaSuccess &&
                  cudaStreamSynchronize(s) == cudaSuccess;
  cudaStreamDestroy(s);
  return ok;
}

// The scratch buffer of (current device, stream), locked by `lock`, holding
// at least n doubles. Growing it first waits for the work already queued on
// the stream (the only work that can still read the old buffer) and frees it.
// Returns null on failure.
double* stream_scratch(cudaStream_t stream, size_t n, std::unique_lock<std::mutex>& lock) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) return nullptr;
  ScratchSlot* slot;
  if (stream == cudaStreamPerThread) {
    slot = thread_slot(dev);
    if (!slot) return nullptr;
  } else {
    std::lock_guard<std::mutex> g(g_slots_mutex);
    std::unique_ptr<ScratchSlot>& p = g_slots[std::make_pair(dev, stream)];
    if (!p) p.reset(new ScratchSlot());
    slot = p.get();
  }
  lock = std::unique_lock<std::mutex>(slot->mu);
  if (slot->cap < n) {
    if (slot->ptr) {
      if (cudaStreamSynchronize(stream) != cudaSuccess) return nullptr;
      cudaFree(slot->ptr);
      slot->ptr = nullptr;
      slot->cap = 0;
    }
    const size_t cap = std::max<size_t>(n, 4096);
    if (cudaMalloc(&slot->ptr, cap * sizeof(double)) != cudaSuccess ||
        !clear_counters(slot->ptr, stream)) {
      cudaFree(slot->ptr);
      slot->ptr = nullptr;
      return nullptr;
    }
    slot->cap = cap;
  }
  return slot->ptr;
}

// ---- allocation-free energy (CUDA_EonDevice_noalloc)
// Fixed scratch for the per-item partials: a file-scope device array, so the
// entry point never allocates. Every GPU that loads this library holds it
// (256 KiB) until the process exits. REMC_NOALLOC_MAX_ITEMS items of 128 x 128
// beads cover up to 255 tiles, i.e. 32640 beads.
constexpr int kNoAllocMaxItems = REMC_NOALLOC_MAX_ITEMS;
static __device__ __align__(256) double g_noalloc_scratch[kNoAllocMaxItems];

// Device address of g_noalloc_scratch, looked up once per device (the host
// name of a __device__ array is only a host-side stand-in).
double* g_noalloc_ptr[kMaxDevices] = {nullptr};

bool energy_args_ok(const float4* pos, const float4* meta, const float* table, int P) {
  if (!pos || !meta) {
    set_status(REMC_ERR_INVALID, "null position or metadata pointer");
    return false;
  }
  if (!table) {
    set_status(REMC_ERR_STATE, "no contact table: pass LJPotentials or call bindLJTexture");
    return false;
  }
  if (P <= 0) {
    set_status(REMC_ERR_INVALID, "datasetSize must be positive");
    return false;
  }
  return true;
}

// A call's scratch, in doubles: the counters of finished items (zero between
// calls, which take turns on their stream), the total, the partials.
constexpr size_t kRefTotal = sizeof(unsigned) * kRefCounters / sizeof(double);
size_t ref_scratch(int P) { return kRefTotal + 1 + (size_t)ref_items(P).count(); }

// Enqueue the energy of P beads on `stream`; the total goes to scratch[kRefTotal]
// and, optionally, to the reference's per-block grid.
int enqueue_energy(const float4* pos, const float4* meta, const float* table, int P,
                   double* scratch, float* grid_out, int grid_n, cudaStream_t stream) {
  RefTotal total{scratch + kRefTotal, grid_out, grid_n, 1.0f};
  const RefConsts C = make_consts(&total.unscale);
  const RefItems it = ref_items(P);
  const int word = ref_counter(it);
  const cudaError_t e =
      launch_energy(pos, meta, table, it, scratch + kRefTotal + 1, C,
                    word < 0 ? nullptr : reinterpret_cast<unsigned*>(scratch) + word, total, stream);
  if (e != cudaSuccess) {
    set_status(REMC_ERR_CUDA, "energy kernel launch", e);
    return REMC_ERR_CUDA;
  }
  return REMC_OK;
}

}  // namespace

extern "C" {

int remc_reference_abi_status(void) { return g_status; }

int remc_reference_abi_set_params(const remc_params* p) {
  if (!p || !(p->debye_length > 0.0f)) {
    set_status(REMC_ERR_INVALID, "bad parameters");
    return REMC_ERR_INVALID;
  }
  std::lock_guard<std::mutex> lock(g_mutex);
  g_params = *p;
  g_params_set = true;
  g_status = REMC_OK;
  return REMC_OK;
}

float* LJPotentialDataToDevice(const float* table) {
  float* d = nullptr;
  if (!table) {
    set_status(REMC_ERR_INVALID, "null table");
    return nullptr;
  }
  cudaError_t e = cudaMalloc(&d, 400 * sizeof(float));
  if (e != cudaSuccess) {
    set_status(REMC_ERR_NOMEM, "cudaMalloc", e);
    return nullptr;
  }
  e = cudaMemcpy(d, table, 400 * sizeof(float), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    cudaFree(d);
    set_status(REMC_ERR_CUDA, "cudaMemcpy", e);
    return nullptr;
  }
  set_status(REMC_OK, "");
  return d;
}

void copyLJPotentialDataToDevice(float* dev, const float* table) {
  if (!dev || !table) {
    set_status(REMC_ERR_INVALID, "null pointer");
    return;
  }
  cudaError_t e = cudaMemcpy(dev, table, 400 * sizeof(float), cudaMemcpyHostToDevice);
  set_status(e == cudaSuccess ? REMC_OK : REMC_ERR_CUDA, "cudaMemcpy", e);
}

void MCSearchOnDevice(void) { set_status(REMC_OK, ""); }

void CUDA_rotateMolecule(float4* d_pos, int* d_start, int* d_len, int moleculeLength,
                         float4* d_rot, float4* d_center, cudaStream_t stream) {
  if (!d_pos || !d_start || !d_len || !d_rot || !d_center || moleculeLength < 0) {
    set_status(REMC_ERR_INVALID, "bad argument");
    return;
  }
  if (moleculeLength == 0) return;
  rotate_molecule_kernel<<<(moleculeLength + 255) / 256, 256, 0, stream>>>(d_pos, d_start, d_len,
                                                                           d_rot, d_center);
  cudaError_t e = cudaGetLastError();
  set_status(e == cudaSuccess ? REMC_OK : REMC_ERR_CUDA, "rotate launch", e);
}

void CUDA_translateMolecule(float4* d_pos, int* d_start, int* d_len, int moleculeLength,
                            float4* d_t, float4* d_center, cudaStream_t stream) {
  if (!d_pos || !d_start || !d_len || !d_t || !d_center || moleculeLength < 0) {
    set_status(REMC_ERR_INVALID, "bad argument");
    return;
  }
  if (moleculeLength > 0)
    translate_molecule_kernel<<<(moleculeLength + 255) / 256, 256, 0, stream>>>(d_pos, d_start,
                                                                              d_len, d_t);
  translate_center_kernel<<<1, 1, 0, stream>>>(d_center, d_t);
  cudaError_t e = cudaGetLastError();
  set_status(e == cudaSuccess ? REMC_OK : REMC_ERR_CUDA, "translate launch", e);
}

void CUDA_EonDevice(float4* pos, float4* meta, int* residueCount, int* moleculePositions,
                    int* moleculeCount, float* LJPotentials, double* result, int blockSize,
                    int datasetSize, int sharedMemSize) {
  (void)residueCount;
  (void)moleculePositions;
  (void)moleculeCount;
  (void)blockSize;
  (void)sharedMemSize;
  const float* table = LJPotentials ? LJPotentials : g_bound_table;
  if (!result) {
    set_status(REMC_ERR_INVALID, "null result pointer");
    return;
  }
  if (!energy_args_ok(pos, meta, table, datasetSize)) return;
  // the reference's synchronous path runs on the legacy default stream; the
  // result copy is made under the scratch lock, before another host thread
  // can queue its energy on the same buffer
  std::unique_lock<std::mutex> lock;
  double* scratch = stream_scratch(0, ref_scratch(datasetSize), lock);
  if (!scratch) {
    set_status(REMC_ERR_NOMEM, "scratch allocation failed");
    return;
  }
  if (enqueue_energy(pos, meta, table, datasetSize, scratch, nullptr, 0, 0) != REMC_OK) return;
  cudaError_t e = cudaMemcpy(result, scratch + kRefTotal, sizeof(double), cudaMemcpyDeviceToHost);
  set_status(e == cudaSuccess ? REMC_OK : REMC_ERR_CUDA, "result copy", e);
}

void CUDA_EonDevice_async(float4* pos, float4* meta, int* residueCount, int* moleculePositions,
                          int* moleculeCount, float* LJPotentials, float* device_result,
                          int resultSize, int blockSize, int datasetSize, int sharedMemSize,
                          cudaStream_t stream) {
  (void)residueCount;
  (void)moleculePositions;
  (void)moleculeCount;
  (void)blockSize;
  (void)sharedMemSize;
  const float* table = LJPotentials ? LJPotentials : g_bound_table;
  if (!device_result || resultSize <= 0) {
    set_status(REMC_ERR_INVALID, "bad result buffer");
    return;
  }
  if (!energy_args_ok(pos, meta, table, datasetSize)) return;
  // the stream's own scratch: energies queued on other streams run
  // concurrently on other buffers, and the next call on this stream reuses
  // this one only after this call's kernels, in stream order
  std::unique_lock<std::mutex> lock;
  double* scratch = stream_scratch(stream, ref_scratch(datasetSize), lock);
  if (!scratch) {
    set_status(REMC_ERR_NOMEM, "scratch allocation failed");
    return;
  }
  if (enqueue_energy(pos, meta, table, datasetSize, scratch, device_result,
                     resultSize * resultSize, stream) != REMC_OK)
    return;
  if (stream == cudaStreamPerThread) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaEventRecord(thread_slot(dev)->used, stream);
    if (e != cudaSuccess) {
      set_status(REMC_ERR_CUDA, "event record", e);
      return;
    }
  }
  set_status(REMC_OK, "");
}

void CUDA_Esum_async(float*, float*, int, int, cudaStream_t) { set_status(REMC_OK, ""); }

int CUDA_memcpy_to_device(void* dst, void* src, int n) {
  return (int)cudaMemcpy(dst, src, (size_t)n, cudaMemcpyHostToDevice);
}
int CUDA_memcpy_to_host(void* dst, void* src, int n) {
  return (int)cudaMemcpy(dst, src, (size_t)n, cudaMemcpyDeviceToHost);
}
int CUDA_memcpy_to_device_async(void* dst, void* src, int n, cudaStream_t s) {
  return (int)cudaMemcpyAsync(dst, src, (size_t)n, cudaMemcpyHostToDevice, s);
}
int CUDA_memcpy_to_host_async(void* dst, void* src, int n, cudaStream_t s) {
  return (int)cudaMemcpyAsync(dst, src, (size_t)n, cudaMemcpyDeviceToHost, s);
}

void printCudaError(int code) { printf("CUDA error: %s\n", cudaGetErrorString((cudaError_t)code)); }

void cudaInfo(void) {
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0) {
    printf("ERROR: no devices supporting CUDA.\n");
    set_status(REMC_ERR_CUDA, "no CUDA device");
    return;
  }
  for (int i = 0; i < n; ++i) {
    cudaDeviceProp p;
    cudaGetDeviceProperties(&p, i);
    printf("CUDA Device %d: %s, %zu MB, %d SMs, sm_%d%d\n", i, p.name, p.totalGlobalMem >> 20,
           p.multiProcessorCount, p.major, p.minor);
  }
  set_status(REMC_OK, "");
}

void CUDA_setBoxDimension(float value) {
  if (!(value > 0.0f) || !std::isfinite(value)) {
    set_status(REMC_ERR_INVALID, "box edge must be positive");
    return;
  }
  std::lock_guard<std::mutex> lock(g_mutex);
  g_box = value;
  g_status = REMC_OK;
}

void CUDA_freeBoxDimension(void) { set_status(REMC_OK, ""); }

void bindLJTexture(float* ljp) {
  std::lock_guard<std::mutex> lock(g_mutex);
  g_bound_table = ljp;
  g_status = REMC_OK;
}

void unbindLJTexture(void) {
  std::lock_guard<std::mutex> lock(g_mutex);
  g_bound_table = nullptr;
  g_status = REMC_OK;
}

int CUDA_EonDevice_noalloc(const float4* pos, const float4* meta, const float* LJPotentials,
                           int datasetSize, double* d_result, cudaStream_t stream) {
  const float* table = LJPotentials ? LJPotentials : g_bound_table;
  if (!d_result) {
    set_status(REMC_ERR_INVALID, "null result pointer");
    return REMC_ERR_INVALID;
  }
  if (!energy_args_ok(pos, meta, table, datasetSize)) return g_status;
  // chunks while their items fit the fixed scratch
  RefItems it = ref_items(datasetSize);
  if (it.count() > kNoAllocMaxItems) it = ref_items(datasetSize, false);
  if ((long long)it.T * (it.T + 1) / 2 > kNoAllocMaxItems) {
    char buf[160];
    snprintf(buf, sizeof(buf),
             "datasetSize %d exceeds the allocation-free limit of %d beads (%d tile pairs)",
             datasetSize, REMC_NOALLOC_MAX_BEADS, kNoAllocMaxItems);
    set_status(REMC_ERR_INVALID, buf);
    return REMC_ERR_INVALID;
  }
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    set_status(REMC_ERR_CUDA, "cudaGetDevice", e);
    return REMC_ERR_CUDA;
  }
  double* scratch = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_mutex);
    if (!g_noalloc_ptr[dev]) {
      // once per device, with that device current
      void* p = nullptr;
      e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
      if (e != cudaSuccess || !p) {
        set_status(REMC_ERR_CUDA, "cudaGetSymbolAddress(scratch)", e);
        return REMC_ERR_CUDA;
      }
      g_noalloc_ptr[dev] = static_cast<double*>(p);
    }
    scratch = g_noalloc_ptr[dev];
  }
  // every item writes its partial before the sum reads it: no clearing needed
  const RefConsts C = make_consts();
  e = launch_energy(pos, meta, table, it, scratch, C, nullptr, RefTotal{d_result, nullptr, 0, 1.0f},
                    stream);
  if (e != cudaSuccess) {
    set_status(REMC_ERR_CUDA, "energy kernel launch", e);
    return REMC_ERR_CUDA;
  }
  set_status(REMC_OK, "");
  return REMC_OK;
}

}  // extern "C"
