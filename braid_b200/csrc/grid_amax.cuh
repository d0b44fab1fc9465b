// Grid-wide NaN-propagating max of |x| for the quantizer kernels: CTA reduction, one atomicMax
// per CTA on the float's bit pattern, a released arrival counter, and a BOUNDED polled wait.
// All CTAs of the grid must be co-resident (the launchers size grids accordingly).
#pragma once
#include <cuda_runtime.h>

#include "ptx.cuh"
#include "quant_device.cuh"

namespace bq {
namespace qd {

// Scratch words shared by all quantizer kernels (16 bytes, zero between launches).
struct QuantWs {
  unsigned int amax_bits;  // running max of |x| as a float bit pattern
  unsigned int arrive;     // CTAs that published their max
  unsigned int depart;     // CTAs that consumed the global max
  unsigned int status;     // sticky: non-zero once a bounded wait ran out
};

// One thread of each of `expected` CTAs: publishes w (>= 0, or NaN with the sign cleared) and returns the largest of all,
// once all have published theirs (bounded).  It owes exchange_leave() and exchange_end() afterwards.
// words: [0] the maximum's bits [1] arrivals [2] departures.
__device__ __forceinline__ float exchange_max(float w, unsigned int* words, unsigned int expected, unsigned int* status) {
  // The unsigned order of the bit patterns is the order of the values, NaN on top.  The max is published first; the
  // release on the counter orders it before the arrival.
  atomicMax(&words[0], __float_as_uint(w));
  asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&words[1]) : "memory");
  // amax word and arrival counter sit in one aligned 8-byte pair: one acquire load sees both
  unsigned int amax_bits = 0, arrived = 0;
  const long long t0 = clock64();
  bool ok = true;
  for (;;) {
    asm volatile("ld.acquire.gpu.global.v2.u32 {%0, %1}, [%2];" : "=r"(amax_bits), "=r"(arrived) : "l"(words) : "memory");
    if (arrived >= expected) break;
    if (clock64() - t0 > bq::kSpinLimitCycles) { ok = false; break; }
  }
  if (!ok) atomicExch(status, (unsigned int)bq::kErrDeviceWait);
  return __uint_as_float(amax_bits);
}
// The place among those that check out.  Asked for before the codes are written and looked at behind them, so that a launch does
// not end a trip to L2 (0.7 us) later: with the barrier at the end of gemm_wide_kernel, four graphed layers of 128 rows 304.5 ->
// 297.8 us, 64 rows 273.0 -> 271.1; hidden 1024, 256 rows 180.6 -> 173.0.  The K-sliced gate/up launch asks behind its
// codes: earlier 16 rows lose (217.0 -> 218.9), the warp that asks also prefetches.
__device__ __forceinline__ unsigned int exchange_leave(unsigned int* words) { return atomicAdd(&words[2], 1u); }
// True for the last one, which has returned the words to zero, so that the next launch (and a graph replay) starts
// clean.
__device__ __forceinline__ bool exchange_end(unsigned int* words, unsigned int expected, unsigned int ticket) {
  if (ticket != expected - 1u) return false;
  words[0] = 0u; words[1] = 0u; words[2] = 0u;
  __threadfence();
  return true;
}

// The largest of a warp's values, each >= 0 or NaN with the sign cleared.
__device__ __forceinline__ float warp_amax(float m) {
  return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(m)));
}

// CTA-wide max, then the grid-wide exchange.  Returns the global amax to every
// thread.  A single-CTA grid never touches global memory here.  Thread 0 of every
// CTA of a multi-CTA grid owes the scratch a grid_depart() call afterwards.
struct WholeCta {
  static constexpr bool live = true;
  __device__ int warp() const { return threadIdx.x >> 5; }
  __device__ int warps() const { return (blockDim.x + 31) >> 5; }
  __device__ int slot() const { return 0; }
  __device__ void sync() const { __syncthreads(); }
};

// A CTA of THREADS working threads and, where it was launched with 32 more, a warp that only rehearses
// (see norm_quant.cu): that one runs the code of warp 0 on its own words of shared memory, and the
// others never wait for it.
template <int THREADS>
struct RehearsingCta {
  bool live;
  __device__ int warp() const { return live ? threadIdx.x >> 5 : 0; }
  __device__ int warps() const { return live ? THREADS / 32 : 1; }
  __device__ int slot() const { return live ? 0 : 1; }
  __device__ void sync() const {
    if (live) asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory");
    else __syncwarp();
  }
};

// `cta.live` = false: this warp's own max without the exchange.  `late`: the ticket is drawn by grid_depart.
template <typename Cta = WholeCta>
__device__ __forceinline__ float grid_amax(float m, QuantWs* ws, unsigned int& ticket, const Cta& cta = Cta{}, bool late = false) {
  __shared__ float s_warp_of[2][32];
  __shared__ float s_amax_of[2];
  float* const s_warp = s_warp_of[cta.slot()];
  float& s_amax = s_amax_of[cta.slot()];
  m = warp_amax(m);
  const int lane = threadIdx.x & 31, warp = cta.warp();
  if (lane == 0) s_warp[warp] = m;
  cta.sync();
  if (warp == 0) {
    float w = warp_amax(lane < cta.warps() ? s_warp[lane] : 0.0f);
    if (lane == 0) {
      if (gridDim.x > 1 && cta.live) {
        w = exchange_max(w, &ws->amax_bits, gridDim.x, &ws->status);
        if (!late) ticket = exchange_leave(&ws->amax_bits);
      }
      s_amax = w;
    }
  }
  cta.sync();
  return s_amax;
}

// The exchange of a grid that is ONE cluster: every CTA stores its max into every other's shared memory, where the
// bytes are counted, and no word of global memory is involved.  A grid-wide exchange is three trips to L2 one after the
// other (max, arrival, poll), each 0.7 us and more while the next GEMM's weights stream.
constexpr int kMaxCluster = 16;      // beyond 8 a kernel has to allow it
struct ClusterAmax {
  uint64_t full;
  uint32_t slot[kMaxCluster];        // one word per CTA of the cluster
};

// All threads of the CTA, before anything else.
__device__ __forceinline__ void cluster_amax_begin(ClusterAmax& s) {
  if (threadIdx.x == 0) {
    bq::mbar_init(bq::smem_u32(&s.full), 1);
    bq::fence_mbar_init();
    bq::mbar_expect_tx(bq::smem_u32(&s.full), 4u * gridDim.x);
  }
  __syncwarp();
  bq::cluster_arrive();              // says that this CTA runs and its barrier is set up
}

// As grid_amax; nothing is owed to the scratch afterwards.  A CTA has every other's word when it leaves, so none is
// stored to that has ended.
template <typename Cta>
__device__ __forceinline__ float cluster_amax(float m, ClusterAmax& s, QuantWs* ws, const Cta& cta) {
  __shared__ uint32_t s_warp_of[2][32];
  uint32_t* const s_warp = s_warp_of[cta.slot()];
  const int lane = threadIdx.x & 31, warp = cta.warp();
  // |x| >= 0 or NaN with the sign cleared: bit patterns order like the values, NaN on top
  const uint32_t mine = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
  if (lane == 0) s_warp[warp] = mine;
  cta.sync();
  uint32_t all = __reduce_max_sync(0xffffffffu, lane < cta.warps() ? s_warp[lane] : 0u);
  if (!cta.live) return __uint_as_float(all);
  if (warp == 0) {
    bq::cluster_wait();              // every CTA's barrier is set up
    if (lane < gridDim.x)
      bq::st_async_cluster(bq::map_to_cta(bq::smem_u32(&s.slot[blockIdx.x]), lane), all,
                           bq::map_to_cta(bq::smem_u32(&s.full), lane));
  }
  if (!bq::mbar_wait_cluster(bq::smem_u32(&s.full), 0) && threadIdx.x == 0)
    atomicExch(&ws->status, (unsigned int)bq::kErrDeviceWait);
  all = lane < gridDim.x ? *static_cast<volatile uint32_t*>(&s.slot[lane]) : 0u;
  return __uint_as_float(__reduce_max_sync(0xffffffffu, all));
}

// CTA-wide max alone, to every thread.  Blocks of whole warps, 1024 threads at most.
__device__ __forceinline__ float cta_amax(float m) {
  __shared__ float s_warp[32];
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) m = nan_max(m, __shfl_xor_sync(0xffffffffu, m, off));
  if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = m;
  __syncthreads();
  m = s_warp[0];
  for (unsigned int i = 1; i < blockDim.x / 32; ++i) m = nan_max(m, s_warp[i]);
  return m;
}

// Column-parallel form: every CTA waits (bounded, thread 0 polls with a system-scope acquire)
// until the arrival counter has advanced by `count` beyond *seen -- i.e. until every rank's push
// launch has stored its share of the buffer this kernel is about to read.  *seen is advanced by
// grid_depart once every CTA has read it for the last time.
__device__ __forceinline__ void grid_wait_arrivals(const unsigned int* flag, const unsigned int* seen,
                                                   unsigned int count, QuantWs* ws) {
  if (threadIdx.x == 0) {
    unsigned int base;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(base) : "l"(seen) : "memory");
    const unsigned int target = base + count;
    const long long t0 = clock64();
    for (;;) {
      unsigned int v;
      asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
      if (static_cast<int>(v - target) >= 0) break;
      if (clock64() - t0 > bq::kSpinLimitCycles) {
        atomicExch(&ws->status, (unsigned int)bq::kErrDeviceWait);
        break;
      }
    }
  }
  __syncthreads();
}

// Called by all threads when grid_amax is behind them, with the ticket it gave; `late`: behind the last read of what was waited
// for, so that the last one to leave knows that every CTA has read it, and the old *wait_seen.
__device__ __forceinline__ void grid_depart(QuantWs* ws, unsigned int ticket, unsigned int* wait_seen = nullptr,
                                            unsigned int wait_count = 0u, bool late = false) {
  if (threadIdx.x != 0) return;
  if (late && gridDim.x > 1) ticket = exchange_leave(&ws->amax_bits);
  if ((gridDim.x == 1 || exchange_end(&ws->amax_bits, gridDim.x, ticket)) && wait_seen != nullptr) *wait_seen += wait_count;
}

// Host side: CTAs of a kernel that an SM of the current device holds at once, 0 where CUDA cannot say.  The
// answer is a property of the compiled kernel; asking costs a launch's host time a third over, so
// each thread keeps the last few.
template <typename Kernel>
inline int resident_per_sm(Kernel kernel, int threads, size_t dynamic_smem) {
  struct Known { const void* kernel; int dev, threads; size_t smem; int per_sm; };
  static thread_local Known known[32];
  static thread_local unsigned int next = 0;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) { (void)cudaGetLastError(); return 0; }
  const void* const key = reinterpret_cast<const void*>(kernel);
  for (const Known& k : known)
    if (k.kernel == key && k.dev == dev && k.threads == threads && k.smem == dynamic_smem) return k.per_sm;
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, dynamic_smem) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  known[next++ % 32] = Known{key, dev, threads, dynamic_smem, per_sm};
  return per_sm;
}

// Host side: can a cluster of `n` CTAs of this kernel be scheduled at all?  Asked once per thread, kernel and size.
extern bool g_cluster_exchange;       // quant_act.cu: option "quant_cluster"

template <typename Kernel>
inline bool cluster_fits(Kernel kernel, int threads, int n) {
  struct Known { const void* kernel; int dev, threads, n; bool fits; };
  static thread_local Known known[32];
  static thread_local unsigned int next = 0;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) { (void)cudaGetLastError(); return false; }
  const void* const key = reinterpret_cast<const void*>(kernel);
  for (const Known& k : known)
    if (k.kernel == key && k.dev == dev && k.threads == threads && k.n == n) return k.fits;
  bool fits = n <= 8 || cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
  if (fits) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(n), 1, 1);
    cfg.blockDim = dim3(static_cast<unsigned>(threads), 1, 1);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = static_cast<unsigned>(n);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    fits = cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) == cudaSuccess && clusters > 0;
  }
  if (!fits) (void)cudaGetLastError();
  known[next++ % 32] = Known{key, dev, threads, n, fits};
  return fits;
}

// Host side: launches a grid that is one cluster of `ctas` CTAs; kErrTooLarge where such a cluster cannot be scheduled.
template <typename Kernel, typename Params>
inline int launch_cluster(Kernel kernel, int ctas, int threads, cudaStream_t stream, Params p, bool pdl = true) {
  if (!cluster_fits(kernel, threads, ctas)) return bq::kErrTooLarge;
#ifdef BQ_PHASES
  p.phase_ring = bq::phase_ring_for_launch(&p.phase_seq);
#endif
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(ctas), 1, 1);
  cfg.blockDim = dim3(static_cast<unsigned>(threads), 1, 1);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(ctas);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, p);
  if (e != cudaSuccess) { (void)cudaGetLastError(); return bq::kErrLaunch; }
  return bq::kOk;
}

// Host side: launches a grid-stride kernel with at most as many CTAs as the device holds at
// once (`want` CTAs if that is fewer), so that no partial second wave trails the first -- a grid
// of 8 CTAs per SM where five fit ran 1.6 waves.  Programmatic dependent launch on request.
template <typename Kernel, typename... Args>
inline cudaError_t launch_resident_smem(Kernel kernel, long long want, int threads, int sms, bool pdl,
                                        size_t dynamic_smem, cudaStream_t stream, Args... args) {
  int per_sm = resident_per_sm(kernel, threads, dynamic_smem);
  if (per_sm < 1) per_sm = 4;
  const long long cap = static_cast<long long>(per_sm) * sms;
  long long grid = want < cap ? want : cap;
  if (grid < 1) grid = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(grid), 1, 1);
  cfg.blockDim = dim3(static_cast<unsigned>(threads), 1, 1);
  cfg.dynamicSmemBytes = dynamic_smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}
template <typename Kernel, typename... Args>
inline cudaError_t launch_resident(Kernel kernel, long long want, int threads, int sms, bool pdl,
                                   cudaStream_t stream, Args... args) {
  return launch_resident_smem(kernel, want, threads, sms, pdl, 0, stream, args...);
}

}  // namespace qd
}  // namespace bq
