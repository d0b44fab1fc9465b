// RMSNorm fused into the FP8 activation quantizer, one launch each:
//
//   bq_rmsnorm_quant        h = rms_norm(x, gamma, eps)            -> (h), e4m3 codes, scale
//                           braid/model/norm.py:31-45 feeding `project` / the MLP
//                           (braid/model/layer.py:49,59 -> gdn.py:254, attention.py:173, mlp.py:45)
//   bq_gated_rmsnorm_quant  core = rms_norm_gated(y, z, gamma, eps) -> e4m3 codes, scale
//                           braid/model/norm.py:48-71 feeding out_proj (braid/model/gdn.py:373-387)
//
// The result has to be bit-identical to the reference's torch spelling on a CUDA device, and a
// sum of squares is not order-free, so the reduction restates the arithmetic of the kernel torch
// runs for `F.rms_norm` on an fp32 row (its vectorized layer-norm kernel in the rms_norm mode,
// one CTA of 32 x 4 threads per row): thread t accumulates the 4-element vectors t, t+128, ...
// in order as s = fma(v, v, s); lanes combine by shuffle-down (16, 8, 4, 2, 1); the four warps
// combine as (w0 + w2) + (w1 + w3); sigma2 = s / float(N) (IEEE division);
// rstd = rsqrtf(sigma2 + eps); y = gamma * (rstd * x) in fp32, then ONE rounding to the
// activation type.  The gated form normalises without gamma, rounds to the activation type,
// multiplies by gamma in fp32, multiplies by silu(z) evaluated in fp32 (x / (1 + expf(-x))) and
// rounds once more.  tests/test_norm_quant_gpu.py pins all of this against torch on the device.
//
// After the norm the values stay in registers; amax, exchange and cast are the activation quantizer's (quant_act.cu).
// The exchange of up to 64 rows stays inside one cluster; beyond it is grid-wide: a CTA holds one token row, or from 257 rows on
// four or eight (rmsnorm_rows_quant_kernel), and all of them are co-resident for it; larger inputs are refused, and the caller takes the norm with its rows
// looped (bq_rmsnorm_scale, bq_gated_rmsnorm_scale) and the cast pass.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/braid_b200.h"
#include "ptx.cuh"
#include "quant_device.cuh"
#include "grid_amax.cuh"

namespace {

using namespace bq::qd;

constexpr int kNormThreads = 128;   // 32 x 4, the block shape whose reduction order is restated
constexpr int kVec = 4;

struct NormParams {
  const void* x;
  const float* gamma;
  void* h_out;        // optional normalised activation in the activation type
  uint8_t* q;
  float* scale;
  float* rstd;        // prefill: [rows], from the first launch to the second
  void* ws;
  int rows, cols;
  int beside;         // rmsnorm_cast_kernel: rows next to one another in a CTA
  long long ld_x, ld_h;
  float eps;
  unsigned long long* phase_ring;   // development builds (BQ_PHASES) only, else nullptr
  int phase_seq;
};

constexpr int kWideRows = 256;      // batches whose rows get four times the threads
constexpr int kRehearseRows = 128;   // see rmsnorm_quant_kernel; one CTA per row
constexpr int with_rehearsal(int threads) { return threads < 1024 ? threads + 32 : threads; }    // CTAs of 1024 have no room for it

template <typename T> struct Vec4 { T v[kVec]; };

// Coherent loads on purpose (see load8).
template <typename T>
__device__ __forceinline__ Vec4<T> load4(const T* p) {
  Vec4<T> r;
  if constexpr (sizeof(T) == 4) {
    const float4 f = __ldcg(reinterpret_cast<const float4*>(p));
    r.v[0] = f.x; r.v[1] = f.y; r.v[2] = f.z; r.v[3] = f.w;
  } else {
    const uint2 raw = __ldcg(reinterpret_cast<const uint2*>(p));
    *reinterpret_cast<uint2*>(&r) = raw;
  }
  return r;
}

template <typename T>
__device__ __forceinline__ void store4(T* p, const Vec4<T>& v) {
  if constexpr (sizeof(T) == 4) {
    *reinterpret_cast<float4*>(p) = make_float4(v.v[0], v.v[1], v.v[2], v.v[3]);
  } else {
    *reinterpret_cast<uint2*>(p) = *reinterpret_cast<const uint2*>(&v);
  }
}

template <typename T>
__device__ __forceinline__ void emit4(const Vec4<T>& v, const ScaleDiv& sc, uint8_t* dst, bool live) {
  float f[4] = {widen(v.v[0]), widen(v.v[1]), widen(v.v[2]), widen(v.v[3])};
  divide_group<T, 4, true>(sc, f);   // the scale is that of these very values
  const uint32_t a = __nv_cvt_float2_to_fp8x2(make_float2(f[0], f[1]), __NV_SATFINITE, __NV_E4M3);
  const uint32_t b = __nv_cvt_float2_to_fp8x2(make_float2(f[2], f[3]), __NV_SATFINITE, __NV_E4M3);
  const uint32_t w = (a & 0xFFFFu) | ((b & 0xFFFFu) << 16);
  if (live) *reinterpret_cast<uint32_t*>(dst) = w;
}

// Lane 0 of the warp ends up with the shuffle-down tree sum (the other lanes hold partial
// garbage, as in the kernel this restates).
__device__ __forceinline__ float warp_tree_sum(float s) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) s = __fadd_rn(s, __shfl_down_sync(0xffffffffu, s, off));
  return s;
}

// ---------------------------------------------------------------------------------------------
// plain RMSNorm -> quantize.  R rows per CTA (more than one only where the grid is one cluster, see launch_rmsnorm_cluster),
// each of G groups of 128 threads; VPT = vectors that a thread would hold if a row were 128 threads in all.
// ---------------------------------------------------------------------------------------------
template <typename T, int VPT, int G, int R, bool CLUSTER>
__global__ void __launch_bounds__(with_rehearsal(R * G * kNormThreads)) rmsnorm_quant_kernel(const NormParams p) {
  static_assert(R == 1 || CLUSTER, "several rows per CTA: one cluster");
  // G groups of 128 threads share a row; a thread holds VG vectors of it
  static_assert(VPT % G == 0, "whole vectors per thread");
  constexpr int VG = VPT / G;
  if (threadIdx.x == 0) { BQ_STAMP(p, 0); BQ_STAMP_META(p, 1); }
  bq::pdl_launch_dependents();
  __shared__ float s_red_of[1 + R][4];
  __shared__ __align__(16) Vec4<T> s_x_of[G > 1 ? R * VPT * kNormThreads + 32 : 1];   // the last 32: the rehearsing warp's
  __shared__ ClusterAmax s_cluster;
  if constexpr (CLUSTER) cluster_amax_begin(s_cluster);
  const RehearsingCta<R * G * kNormThreads> cta{threadIdx.x < R * G * kNormThreads};
  const bool live = cta.live;
  const int lane = threadIdx.x & 31, of_row = (cta.warp() * 32 + lane) / (G * kNormThreads);   // row of this CTA
  const int t = cta.warp() * 32 + lane - of_row * (G * kNormThreads), warp = t >> 5;            // thread of that row
  const int group = t / kNormThreads;
  float* const s_red = s_red_of[live ? of_row : R];
  Vec4<T>* const s_x = s_x_of + (G > 1 && live ? of_row * (VPT * kNormThreads) : 0);
  // vector i of this thread
  auto vec = [&](int i) { return (t - group * kNormThreads) + (group * VG + i) * kNormThreads; };
  const int row = blockIdx.x * R + of_row;
  const bool row_ok = live && (R == 1 || row < p.rows);
  const int n_vec = p.cols / kVec;
  const T* xr = reinterpret_cast<const T*>(p.x) + static_cast<long long>(row) * p.ld_x;
  // gamma is a weight, not the previous kernel's output: fetch it before the dependency wait
  float g[VG][kVec];
#pragma unroll
  for (int i = 0; i < VG; ++i) {
    const int v = vec(i);
    if (v < n_vec) {
      const float4 f = __ldg(reinterpret_cast<const float4*>(p.gamma) + v);
      g[i][0] = f.x; g[i][1] = f.y; g[i][2] = f.z; g[i][3] = f.w;
    }
  }
  // What bounds this kernel at a decode batch is neither bytes nor arithmetic but one dependent chain
  // run once.  Two things shorten it.
  //
  // The row is shared by G groups of 128 threads instead of one, so that a thread normalises and casts a
  // quarter of the values; a lone warp per scheduler issues an instruction every few clocks, and the
  // chain's length is what it has to issue.  Only the sum of squares stays with 128 threads, whose order it
  // restates; they read the other groups' values from shared memory.  Together with 16 instead of 8 warps in
  // the gated kernel (four graphed layers of hidden 4096, before -> gated -> both): 1 row 246 -> 238 -> 232 us,
  // 27 rows 286 -> 281 -> 274, 128 rows 333 -> 323 -> 317; hidden 5120, 64 rows 434 -> 435 -> 421.  32 warps
  // in the gated kernel gave no more.
  //
  // A further warp rehearses: it runs the same instructions on zeros and words of its own, without an access to
  // global memory and without the exchange, while the others wait for the previous kernel, and they find the
  // code in the instruction cache, where the previous kernel's code was.  A warp of its own, because there may be nothing to wait for (behind a
  // kernel that was not launched with early starts).  Only up to kRehearseRows rows: beyond, the
  // rehearsal competes with the GEMM that is waited for.
  Vec4<T> x[VG];
  if (live) {
    bq::pdl_wait_prior_grids();
    if (threadIdx.x == 0) BQ_STAMP(p, 2);
  }
#pragma unroll
  for (int i = 0; i < VG; ++i) {
    const int v = vec(i);
    if (row_ok && v < n_vec) x[i] = load4(xr + v * kVec);
    else x[i] = Vec4<T>{};
  }
  float s = 0.0f;
  if constexpr (G == 1) {
#pragma unroll
    for (int i = 0; i < VG; ++i) {
      const int v = vec(i);
      if (v < n_vec) {
#pragma unroll
        for (int j = 0; j < kVec; ++j) {
          const float f = widen(x[i].v[j]);
          s = __fmaf_rn(f, f, s);
        }
      }
    }
  } else {
    // the sum's order is that of 128 threads: the first group walks the others' vectors (the rehearsing warp,
    // which passes no barrier with them, words of its own)
    const int put = live ? vec(0) : R * VPT * kNormThreads + lane, get = live ? t : put, step = live ? kNormThreads : 0;
#pragma unroll
    for (int i = 0; i < VG; ++i) s_x[put + i * step] = x[i];
    cta.sync();
    if (group == 0) {
      Vec4<T> all[VPT];
#pragma unroll
      for (int i = 0; i < VPT; ++i) all[i] = s_x[get + i * step];
#pragma unroll
      for (int i = 0; i < VPT; ++i) {
        if (t + i * kNormThreads < n_vec) {
#pragma unroll
          for (int j = 0; j < kVec; ++j) {
            const float f = widen(all[i].v[j]);
            s = __fmaf_rn(f, f, s);
          }
        }
      }
    }
  }
  if (group == 0) {
    s = warp_tree_sum(s);
    if (lane == 0) s_red[warp] = s;
  }
  cta.sync();
  // every thread adds the four warps' sums up in the restated order
  s = __fadd_rn(__fadd_rn(s_red[0], s_red[2]), __fadd_rn(s_red[1], s_red[3]));
  s = __fdiv_rn(s, static_cast<float>(p.cols));
  const float rstd = rsqrtf(__fadd_rn(s, p.eps));

  float m = 0.0f;
#pragma unroll
  for (int i = 0; i < VG; ++i) {
    const int v = vec(i);
    if (v < n_vec && (R == 1 || row_ok || !live)) {
#pragma unroll
      for (int j = 0; j < kVec; ++j) {
        const float y = __fmul_rn(g[i][j], __fmul_rn(rstd, widen(x[i].v[j])));
        x[i].v[j] = narrow<T>(y);
        m = nan_max(m, fabsf(widen(x[i].v[j])));
      }
    }
  }
  if (row_ok && p.h_out != nullptr) {
    T* hr = reinterpret_cast<T*>(p.h_out) + static_cast<long long>(row) * p.ld_h;
#pragma unroll
    for (int i = 0; i < VG; ++i) {
      const int v = vec(i);
      if (v < n_vec) store4(hr + v * kVec, x[i]);
    }
  }
  if (live && threadIdx.x == 0) BQ_STAMP(p, 3);
  float amax;
  unsigned int ticket = 0u;
  if constexpr (CLUSTER) amax = cluster_amax(m, s_cluster, static_cast<QuantWs*>(p.ws), cta);
  else amax = grid_amax(m, static_cast<QuantWs*>(p.ws), ticket, cta);
  const float sc = scale_from_amax(amax);
  if (live && threadIdx.x == 0) BQ_STAMP(p, 4);
  const ScaleDiv dv(sc);
  if (blockIdx.x == 0 && threadIdx.x == 0) p.scale[0] = sc;
  uint8_t* qr = p.q + static_cast<long long>(row) * p.cols;
#pragma unroll
  for (int i = 0; i < VG; ++i) {
    const int v = vec(i);
    if (v < n_vec) emit4(x[i], dv, qr + v * kVec, row_ok);
  }
  if constexpr (!CLUSTER) grid_depart(static_cast<QuantWs*>(p.ws), ticket);
  if (threadIdx.x == 0) BQ_STAMP(p, 7);
}

// ---------------------------------------------------------------------------------------------
// plain RMSNorm -> quantize of a short prompt: CTAs of four groups of 128 threads, R rows per group.  A row's
// arithmetic is that of rmsnorm_quant_kernel.  Gamma is in shared memory, not in registers, so that more rows are
// resident at once, and a quarter or an eighth of the CTAs meet in the exchange (three atomics each on one word pair).
// What bounds it are the rows' loads in flight, so the registers decide: held to 40 for a third CTA per SM, the compiler asks
// for a row's vectors one after the other; with two it takes the 47 to 50 that it wants.  The form of 40 (PER_SM = 3) is taken
// where two CTAs per SM do not hold the rows.
// One CTA per row / 40 registers / 50, us: 16-bit 512 x 4096 7.5 / 9.2 / 7.0, 768 x 4096 8.9 / 10.8 / 7.4, 1036 x 4096 - / 10.3 /
// 7.5, 1500 x 4096 - / 10.5 / - (two rows per group 11.7); 600 x 1024 5.8 / 4.9 / 4.5.
// Resident on 148 SMs: 16-bit rows of up to 2048 columns 3552, up to 4096 columns 2368, up to 8192 columns 1184; fp32
// 3552 (1024 columns), 2368 (2048), 1184 (4096), longer ones never.  Beyond, the two launches, from HBM: 2600 x 4096
// bf16 14.5, 1300 x 5120 bf16 13.7, 1300 x 4096 fp32 13.9.
// Of few rows a block has four to wait for where one would do.  One CTA per row and this, us: 16-bit 257 x 2048 4.8 and
// 4.7, 333 x 4096 6.3 and 6.4, 413 x 4096 6.8 and 6.6, fp32 333 x 4096 6.3 and 6.3, 413 x 4096 6.7 and 6.6; bf16
// 257 x 8192 8.5 and 8.7, 600 x 8192 9.8 and 11.1, 900 x 8192 12.3 and 11.5.
// ---------------------------------------------------------------------------------------------
constexpr int kRowGroups = 4;
// more rows than these, for rows of up to 2048, 4096 and 8192 columns
constexpr int grouped_rows(int per_thread) { return per_thread <= 4 ? 256 : per_thread <= 8 ? 384 : 768; }
// The forms that hold more rows than the one before them (of R = 1, PER_SM 2 and then 3).  A thread has VPT * sizeof(T) registers of a row: two rows of
// 32 make 80 registers and one CTA of eight rows per SM, no more than two CTAs of four; one row of 64 makes one CTA of
// four, 592 rows in all.
template <typename T, int VPT> constexpr bool kOneRowPerGroup = VPT * sizeof(T) <= 32;
template <typename T, int VPT> constexpr bool kTwoRowsPerGroup = VPT * sizeof(T) <= 16;
template <typename T, int VPT, int R, int PER_SM>
__global__ void __launch_bounds__(kRowGroups * kNormThreads, PER_SM) rmsnorm_rows_quant_kernel(const NormParams p) {
  bq::pdl_launch_dependents();
  __shared__ float s_red[kRowGroups][R][4];
  extern __shared__ float4 s_gamma[];
  const int group = threadIdx.x / kNormThreads, t = threadIdx.x - group * kNormThreads, lane = t & 31, warp = t >> 5;
  const int n_vec = p.cols / kVec;
  for (int v = threadIdx.x; v < n_vec; v += kRowGroups * kNormThreads) s_gamma[v] = __ldg(reinterpret_cast<const float4*>(p.gamma) + v);
  __syncthreads();
  const int row0 = (blockIdx.x * kRowGroups + group) * R;
  bq::pdl_wait_prior_grids();
  Vec4<T> x[R][VPT];
#pragma unroll
  for (int k = 0; k < R; ++k) {
    const T* xr = reinterpret_cast<const T*>(p.x) + static_cast<long long>(row0 + k) * p.ld_x;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int v = t + i * kNormThreads;
      x[k][i] = Vec4<T>{};
      if (row0 + k < p.rows && v < n_vec) x[k][i] = load4(xr + v * kVec);
    }
  }
#pragma unroll
  for (int k = 0; k < R; ++k) {
    float s = 0.0f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      if (t + i * kNormThreads < n_vec) {
#pragma unroll
        for (int j = 0; j < kVec; ++j) {
          const float f = widen(x[k][i].v[j]);
          s = __fmaf_rn(f, f, s);
        }
      }
    }
    s = warp_tree_sum(s);
    if (lane == 0) s_red[group][k][warp] = s;
  }
  asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(kNormThreads) : "memory");
  float m = 0.0f;
#pragma unroll
  for (int k = 0; k < R; ++k) {
    const float* const r = s_red[group][k];
    float s = __fadd_rn(__fadd_rn(r[0], r[2]), __fadd_rn(r[1], r[3]));
    s = __fdiv_rn(s, static_cast<float>(p.cols));
    const float rstd = rsqrtf(__fadd_rn(s, p.eps));
    T* hr = reinterpret_cast<T*>(p.h_out) + static_cast<long long>(row0 + k) * p.ld_h;
    const bool row_ok = row0 + k < p.rows;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int v = t + i * kNormThreads;
      if (row_ok && v < n_vec) {
        const float4 gv = s_gamma[v];
        const float g[kVec] = {gv.x, gv.y, gv.z, gv.w};
#pragma unroll
        for (int j = 0; j < kVec; ++j) {
          const float y = __fmul_rn(g[j], __fmul_rn(rstd, widen(x[k][i].v[j])));
          x[k][i].v[j] = narrow<T>(y);
          m = nan_max(m, fabsf(widen(x[k][i].v[j])));
        }
        if (p.h_out != nullptr) store4(hr + v * kVec, x[k][i]);
      }
    }
  }
  unsigned int ticket = 0u;
  const float sc = scale_from_amax(grid_amax(m, static_cast<QuantWs*>(p.ws), ticket));
  const ScaleDiv dv(sc);
  if (blockIdx.x == 0 && threadIdx.x == 0) p.scale[0] = sc;
#pragma unroll
  for (int k = 0; k < R; ++k) {
    uint8_t* qr = p.q + static_cast<long long>(row0 + k) * p.cols;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int v = t + i * kNormThreads;
      if (v < n_vec) emit4(x[k][i], dv, qr + v * kVec, row0 + k < p.rows);
    }
  }
  grid_depart(static_cast<QuantWs*>(p.ws), ticket);
}

// ---------------------------------------------------------------------------------------------
// plain RMSNorm at prefill sizes: more rows than one co-resident grid has CTAs.  Two launches, and nobody waits for
// anybody.  The first finds every row's rstd and max |h|: each CTA loops over rows (row arithmetic as above), folds its
// max into one word with an atomicMax and counts itself, and the CTA that counts last turns the word into the scale and
// returns the scratch to zero.  The second reads x again -- last rows first, of which L2 still has some -- normalises it once
// more with the rstd found, and casts: 9658 x 4096 bf16 are 79 + 79 + 40 MB, where a first launch that writes h and a cast of
// h move 79 + 79 + 79 + 40: 53.9 -> 40.6 us (fp32 85 -> 61).  Those (DENSE, 45.9 with the loops below; bq_rmsnorm_scale and
// bq_cast_act) are what is left where h is wanted anyway.
// ---------------------------------------------------------------------------------------------
// Running max |.| of values of T.
template <typename T>
struct AbsMax {
  float m = 0.0f;
  uint32_t pairs = 0u;      // 16-bit types: two at a time
  __device__ __forceinline__ void add(const Vec4<T>& v) {
    if constexpr (sizeof(T) == 2) {
      const uint2 w = *reinterpret_cast<const uint2*>(&v);
      pairs = absmax2<T>(absmax2<T>(pairs, w.x), w.y);
    } else {
#pragma unroll
      for (int j = 0; j < kVec; ++j) m = nan_max(m, fabsf(widen(v.v[j])));
    }
  }
  __device__ __forceinline__ float value() const {
    if constexpr (sizeof(T) == 2) {
      const float2 f = unpack2<T>(pairs);
      return nan_max(f.x, f.y);
    } else {
      return m;
    }
  }
};

// v <- T(gamma * (rstd * v)), two values rounded at an instruction where T has 16 bits.
template <typename T, int N>
__device__ __forceinline__ void scale_norm(T (&v)[N], const float (&g)[N], float rstd) {
  if constexpr (sizeof(T) == 2) {
    uint32_t* const w = reinterpret_cast<uint32_t*>(v);
#pragma unroll
    for (int i = 0; i < N; i += 2) {
      const float2 y = mul2(make_float2(g[i], g[i + 1]), mul2(make_float2(rstd, rstd), unpack2<T>(w[i / 2])));
      w[i / 2] = pack2<T>(y.x, y.y);
    }
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = __fmul_rn(g[i], __fmul_rn(rstd, v[i]));
  }
}

// DENSE: h is written, and nobody reads rstd.  WHOLE: are rows VPT whole vectors per thread (kAsk: asked here)?  Long rows of fp32 have a
// kernel for either, since both loops in one cost the partial one a CTA per SM (six where they have 80 registers): h of 1776 x 5120
// 18.7 -> 19.8 us.  Held to 80, the partial loop that writes h spills 480 bytes by itself and 16 beside the other one, so that is
// its kernel; whole rows of 8192 want more (1776 x 8192 with 88 registers 31.1, with 80 36.1).
enum Whole { kAsk = -1, kPartial = 0, kWhole = 1 };
template <typename T, int VPT, bool DENSE> constexpr int kPartialKernel = sizeof(T) == 4 && VPT >= 8 && !(DENSE && VPT == 16) ? kPartial : kAsk;
template <typename T, int VPT> constexpr int kWholeKernel = sizeof(T) == 4 && VPT >= 8 ? kWhole : kAsk;
template <typename T, int VPT, int WHOLE> constexpr int kScalePerSm = sizeof(T) == 4 && VPT == 16 && WHOLE != kWhole ? 6 : 0;      // 0: as it comes
template <typename T, int VPT, bool DENSE, int WHOLE>
__global__ void __launch_bounds__(kNormThreads, kScalePerSm<T, VPT, WHOLE>) rmsnorm_scale_kernel(const NormParams p) {
  bq::pdl_launch_dependents();
  __shared__ float s_red_of[2][4];
  __shared__ float s_max[4];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int n_vec = p.cols / kVec;
  // gamma lives in shared memory here, not in registers: a CTA normalises many rows, and 32
  // registers less per thread are three more CTAs per SM to hide the loads behind
  extern __shared__ float4 s_gamma[];
  for (int v = t; v < n_vec; v += kNormThreads) s_gamma[v] = __ldg(reinterpret_cast<const float4*>(p.gamma) + v);
  __syncthreads();
  bq::pdl_wait_prior_grids();
  AbsMax<T> mx;
  // One loop for rows of VPT whole vectors per thread, one for the others.  A third of the instructions of the second are
  // its comparisons, and a launch is bound by its instructions as much as by its bytes.
  auto walk = [&](auto full) {
    constexpr bool kFull = decltype(full)::value;
    auto has = [&](int i) { return kFull || t + i * kNormThreads < n_vec; };
    // where the registers allow it the next row is asked for before this one is summed
    constexpr bool kAhead = VPT * sizeof(T) <= 16;
    const long long step = static_cast<long long>(gridDim.x) * p.ld_x;
    const T* xr = reinterpret_cast<const T*>(p.x) + static_cast<long long>(blockIdx.x) * p.ld_x + t * kVec;
    Vec4<T> buffer[kAhead ? 2 : 1][VPT];
    auto load_row = [&](const T* from, Vec4<T>* to) {
#pragma unroll
      for (int i = 0; i < VPT; ++i)
        if (has(i)) to[i] = load4(from + i * (kNormThreads * kVec));
    };
    auto one_row = [&](int row, Vec4<T>* x, float* r) {
      float s = 0.0f;
#pragma unroll
      for (int i = 0; i < VPT; ++i) {
        if (has(i)) {
#pragma unroll
          for (int j = 0; j < kVec; ++j) {
            const float f = widen(x[i].v[j]);
            s = __fmaf_rn(f, f, s);
          }
        }
      }
      s = warp_tree_sum(s);
      if (lane == 0) r[warp] = s;
      __syncthreads();                       // the other words may still be read
      s = __fadd_rn(__fadd_rn(r[0], r[2]), __fadd_rn(r[1], r[3]));
      s = __fdiv_rn(s, static_cast<float>(p.cols));
      const float rstd = rsqrtf(__fadd_rn(s, p.eps));
      if (!DENSE && t == 0) p.rstd[row] = rstd;
      T* const hr = reinterpret_cast<T*>(p.h_out) + static_cast<long long>(row) * p.ld_h + t * kVec;
#pragma unroll
      for (int i = 0; i < VPT; ++i) {
        if (has(i)) {
          const float4 gv = s_gamma[t + i * kNormThreads];
          const float g[kVec] = {gv.x, gv.y, gv.z, gv.w};
          scale_norm<T, kVec>(x[i].v, g, rstd);
          mx.add(x[i]);
          if constexpr (DENSE) store4(hr + i * (kNormThreads * kVec), x[i]);
        }
      }
    };
    int row = blockIdx.x;
    if (row >= p.rows) return;
    if constexpr (kAhead) {
      load_row(xr, buffer[0]);
      for (;;) {
        xr += step;
        if (row + (int)gridDim.x < p.rows) load_row(xr, buffer[1]);
        one_row(row, buffer[0], s_red_of[0]);
        row += gridDim.x;
        if (row >= p.rows) break;
        xr += step;
        if (row + (int)gridDim.x < p.rows) load_row(xr, buffer[0]);
        one_row(row, buffer[1], s_red_of[1]);
        row += gridDim.x;
        if (row >= p.rows) break;
      }
    } else {
      for (int parity = 0; row < p.rows; row += gridDim.x, xr += step, parity ^= 1) {
        load_row(xr, buffer[0]);
        one_row(row, buffer[0], s_red_of[parity]);
      }
    }
  };
  if constexpr (WHOLE != kAsk) walk(std::integral_constant<bool, WHOLE == kWhole>{});
  else if (n_vec == VPT * kNormThreads) walk(std::true_type{});
  else walk(std::false_type{});
  float m = mx.value();
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) m = nan_max(m, __shfl_xor_sync(0xffffffffu, m, off));
  if (lane == 0) s_max[warp] = m;
  __syncthreads();
  if (t == 0) {
    float w = s_max[0];
    for (int i = 1; i < kNormThreads / 32; ++i) w = nan_max(w, s_max[i]);
    QuantWs* ws = static_cast<QuantWs*>(p.ws);
    // |h| >= 0 or NaN with the sign cleared: bit patterns order like the values, NaN on top
    atomicMax(&ws->amax_bits, __float_as_uint(w));
    __threadfence();
    const unsigned int old = atomicAdd(&ws->arrive, 1u);
    if (old == gridDim.x - 1) {
      __threadfence();
      const unsigned int bits = atomicExch(&ws->amax_bits, 0u);
      p.scale[0] = scale_from_amax(__uint_as_float(bits));
      ws->arrive = 0u;
      __threadfence();
    }
  }
}

// The second launch: a thread keeps gamma of its 8 columns and walks rows, kCastRows of them in flight.  BESIDE: rows of up to
// 128 groups lie p.beside at a time next to one another in a CTA, since one of 64 columns would leave 248 of its threads idle, as
// many as put all rows on the device at once: 9658 x 64 fp32 11.8 -> 9.9 us, 40000 x 64 30.2 -> 21.5, 9658 x 512 bf16 12.5 -> 12.0.
// (In one kernel with the wide rows the registers of two divisions cost those a CTA per SM: 9658 x 4096 fp32 54.5 -> 58.)
constexpr int kCastThreads = 256;
constexpr int kCastRows = 4;
template <typename T, bool BESIDE>
__global__ void __launch_bounds__(kCastThreads) rmsnorm_cast_kernel(const NormParams p) {
  bq::pdl_launch_dependents();
  const int row_groups = p.cols / kGroup;
  const int which = BESIDE ? threadIdx.x / row_groups : 0;
  const int group = BESIDE ? threadIdx.x - which * row_groups : blockIdx.x * blockDim.x + threadIdx.x;
  const int slice = BESIDE ? blockIdx.y * p.beside + which : blockIdx.y;      // of the rows
  const int slices = BESIDE ? gridDim.y * p.beside : gridDim.y;
  const bool live = group < row_groups && (!BESIDE || which < p.beside);
  float g[kGroup];
#pragma unroll
  for (int i = 0; i < kGroup; i += 4) {
    const float4 f = live ? __ldg(reinterpret_cast<const float4*>(p.gamma) + group * 2 + i / 4) : make_float4(0, 0, 0, 0);
    g[i] = f.x; g[i + 1] = f.y; g[i + 2] = f.z; g[i + 3] = f.w;
  }
  bq::pdl_wait_prior_grids();
  const ScaleMul<T> dv(__ldcg(p.scale));
  if (!live) return;
  const T* const x = reinterpret_cast<const T*>(p.x) + group * kGroup;
  by_scale(dv, [&](const auto& scale) {
    for (int top = p.rows - 1 - slice * kCastRows; top >= 0; top -= slices * kCastRows) {
      Pack8<T> v[kCastRows];
      float rstd[kCastRows];
#pragma unroll
      for (int k = 0; k < kCastRows; ++k)
        if (top - k >= 0) {
          v[k] = load8<T>(x + static_cast<long long>(top - k) * p.ld_x);
          rstd[k] = __ldcg(p.rstd + top - k);
        }
#pragma unroll
      for (int k = 0; k < kCastRows; ++k)
        if (top - k >= 0) {
          const int row = top - k;
          scale_norm<T, kGroup>(v[k].v, g, rstd[k]);
          emit8<T, true>(v[k], scale, p.q + static_cast<long long>(row) * p.cols + group * kGroup);
        }
    }
  });
}

// ---------------------------------------------------------------------------------------------
// gated RMSNorm (per 128-wide head) -> quantize.  One CTA per token row, one warp per head
// (warps loop when there are more heads than warps); a lane owns one 4-element vector of a head.
// ---------------------------------------------------------------------------------------------
struct GatedParams {
  const void* y;       // scan output, fp32 or the activation type
  const void* z;       // gate, the activation type
  const float* gamma;  // [128]
  void* h_out;         // looped form: the gated, normalised activation [rows, heads * 128]
  long long ld_h;
  uint8_t* q;
  float* scale;
  void* ws;
  int rows, heads;
  int cta_rows;        // rows per CTA (a grid that is one cluster; else 1)
  long long ld_y, ld_z;
  float eps;
  unsigned long long* phase_ring;   // development builds (BQ_PHASES) only, else nullptr
  int phase_seq;
};

constexpr int kHeadDim = 128;
constexpr int kGatedWarps = 8;
constexpr int kMaxHeadsPerWarp = 8;    // up to 64 heads
constexpr int kWideGatedRows = 256;    // batches whose CTAs have 16 warps

template <typename T, bool Y_F32, int HPW, int WARPS, bool CLUSTER>
__global__ void __launch_bounds__(with_rehearsal(WARPS * 32)) gated_rmsnorm_quant_kernel(const GatedParams p) {
  if (threadIdx.x == 0) { BQ_STAMP(p, 0); BQ_STAMP_META(p, 1); }
  bq::pdl_launch_dependents();
  __shared__ ClusterAmax s_cluster;
  if constexpr (CLUSTER) cluster_amax_begin(s_cluster);
  const RehearsingCta<WARPS * 32> cta{threadIdx.x < WARPS * 32};   // see rmsnorm_quant_kernel
  const bool live = cta.live;
  const int lane = threadIdx.x & 31, warp = cta.warp();
  // head i of this warp: the CTA's rows lie one after the other
  const int first_row = CLUSTER ? blockIdx.x * p.cta_rows : blockIdx.x;
  const int cta_heads = CLUSTER ? (p.rows - first_row < p.cta_rows ? p.rows - first_row : p.cta_rows) * p.heads : p.heads;
  auto place = [&](int at, int& row, int& head) {
    row = CLUSTER ? at / p.heads : 0;
    head = at - row * p.heads;
    row += first_row;
  };
  const float4 gm = __ldg(reinterpret_cast<const float4*>(p.gamma) + lane);
  const float gmv[kVec] = {gm.x, gm.y, gm.z, gm.w};
  Vec4<T> core[HPW];
  Vec4<T> gate[HPW];
  if (live) {
    bq::pdl_wait_prior_grids();
    if (threadIdx.x == 0) BQ_STAMP(p, 2);
  }
#pragma unroll
  for (int i = 0; i < HPW; ++i) {
    core[i] = Vec4<T>{};
    gate[i] = Vec4<T>{};
    if (live && warp + i * WARPS < cta_heads) {
      int row, head;
      place(warp + i * WARPS, row, head);
      const long long off = static_cast<long long>(head) * kHeadDim + lane * kVec;
      if constexpr (Y_F32) {
        // the reference rounds the scan output to the activation type first (gdn.py:383)
        const float4 f = __ldcg(reinterpret_cast<const float4*>(
            reinterpret_cast<const float*>(p.y) + static_cast<long long>(row) * p.ld_y + off));
        core[i].v[0] = narrow<T>(f.x); core[i].v[1] = narrow<T>(f.y);
        core[i].v[2] = narrow<T>(f.z); core[i].v[3] = narrow<T>(f.w);
      } else {
        core[i] = load4(reinterpret_cast<const T*>(p.y) + static_cast<long long>(row) * p.ld_y + off);
      }
      gate[i] = load4(reinterpret_cast<const T*>(p.z) + static_cast<long long>(row) * p.ld_z + off);
    }
  }
  float m = 0.0f;
#pragma unroll
  for (int i = 0; i < HPW; ++i) {
    if (warp + i * WARPS < cta_heads) {   // warp-uniform
      float s = 0.0f;
#pragma unroll
      for (int j = 0; j < kVec; ++j) {
        const float f = widen(core[i].v[j]);
        s = __fmaf_rn(f, f, s);
      }
      s = warp_tree_sum(s);
      s = __shfl_sync(0xffffffffu, s, 0);
      // the three idle warps of the restated kernel contribute exact zeros
      const float sigma2 = __fdiv_rn(s, static_cast<float>(kHeadDim));
      const float rstd = rsqrtf(__fadd_rn(sigma2, p.eps));
#pragma unroll
      for (int j = 0; j < kVec; ++j) {
        const T xn = narrow<T>(__fmul_rn(rstd, widen(core[i].v[j])));
        const float zf = widen(gate[i].v[j]);
        const float silu = __fdiv_rn(zf, 1.0f + expf(-zf));
        const float h = __fmul_rn(__fmul_rn(gmv[j], widen(xn)), silu);
        core[i].v[j] = narrow<T>(h);
        m = nan_max(m, fabsf(widen(core[i].v[j])));
      }
    }
  }
  if (live && threadIdx.x == 0) BQ_STAMP(p, 3);
  float amax;
  unsigned int ticket = 0u;
  if constexpr (CLUSTER) amax = cluster_amax(m, s_cluster, static_cast<QuantWs*>(p.ws), cta);
  else amax = grid_amax(m, static_cast<QuantWs*>(p.ws), ticket, cta);
  const float sc = scale_from_amax(amax);
  if (live && threadIdx.x == 0) BQ_STAMP(p, 4);
  const ScaleDiv dv(sc);
  if (blockIdx.x == 0 && threadIdx.x == 0) p.scale[0] = sc;
  uint8_t* qr = p.q + static_cast<long long>(first_row) * p.heads * kHeadDim;      // codes are contiguous
#pragma unroll
  for (int i = 0; i < HPW; ++i) {
    const int head = warp + i * WARPS;
    if (head < cta_heads) emit4(core[i], dv, qr + head * kHeadDim + lane * kVec, live);
  }
  if constexpr (!CLUSTER) grid_depart(static_cast<QuantWs*>(p.ws), ticket);
  if (threadIdx.x == 0) BQ_STAMP(p, 7);
}

// ---------------------------------------------------------------------------------------------
template <typename Kernel, typename Params>
int launch_rows(Kernel kernel, int rows, int threads, Params p, cudaStream_t stream) {
#ifdef BQ_PHASES
  p.phase_ring = bq::phase_ring_for_launch(&p.phase_seq);
#endif
  if (rows <= kRehearseRows) threads += 32;   // the rehearsing warp
  // every CTA waits for every other: the whole grid must fit on the device at once
  int dev = 0, sms = 0;
  const int per_sm = resident_per_sm(kernel, threads, 0);
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || per_sm < 1) {
    (void)cudaGetLastError();
    return bq::kErrLaunch;
  }
  if (static_cast<long long>(rows) > static_cast<long long>(sms) * per_sm) return bq::kErrTooLarge;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(rows), 1, 1);
  cfg.blockDim = dim3(static_cast<unsigned>(threads), 1, 1);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, p);
  if (e != cudaSuccess) { (void)cudaGetLastError(); return bq::kErrLaunch; }
  return bq::kOk;
}

// Decode batches of up to 64 rows: a grid that is one cluster of up to 16 CTAs, and the exchange goes through its shared
// memory (cluster_amax).  Four graphed layers of hidden 4096, grid-wide exchange -> this, us: norms of 8 rows 240.2 ->
// 225.4, 16 rows 248.3 -> 232.0, 27 rows 259.0 -> 239.1, 48 rows 271.8 -> 257; with the gated norm 8 rows 221.4, 16 rows 225.7,
// 27 rows 237.1.  Eight CTAs at most (what a cluster may be without asking) leave 27 rows at 259.
//
// A CTA takes one row while there are 16 at most: with R rows it has R times the bytes to wait for.  Two groups of 128
// threads to a row from there on: one loses (four rows per CTA, 40 rows 264.4 and 258.0), four give the same up to 4096
// columns and take more of an SM; longer rows need them (hidden 5120, 17 rows, grid-wide 386.4, two groups 390.9, four 366.3).
// Seven rows per CTA lose: 96 rows 296 and 310.  Where values of 4 bytes or long rows leave no room for R rows,
// kErrTooLarge: the grid-wide exchange takes them.
constexpr int kClusterRows = 64;
template <typename T, int VPT>
int launch_rmsnorm_cluster(const NormParams& p, cudaStream_t stream) {
  constexpr int kOne = VPT == 2 ? 2 : 4;              // groups of one row
  constexpr int kRow = VPT * (int)sizeof(T);          // registers of a row, were it one group's
  const int ctas = kMaxCluster;
  if (p.rows <= ctas)
    return launch_cluster(rmsnorm_quant_kernel<T, VPT, kOne, 1, true>, p.rows, with_rehearsal(kOne * kNormThreads), stream, p);
  if constexpr (VPT == 16 && kRow <= 32) {
    if (p.rows <= 2 * ctas)
      return launch_cluster(rmsnorm_quant_kernel<T, VPT, 4, 2, true>, (p.rows + 1) / 2, with_rehearsal(8 * kNormThreads), stream, p);
  } else if constexpr (kRow <= 32) {
    if (p.rows <= 2 * ctas)
      return launch_cluster(rmsnorm_quant_kernel<T, VPT, 2, 2, true>, (p.rows + 1) / 2, with_rehearsal(4 * kNormThreads), stream, p);
  }
  if constexpr (kRow <= 16) {
    if (p.rows <= 3 * ctas)
      return launch_cluster(rmsnorm_quant_kernel<T, VPT, 2, 3, true>, (p.rows + 2) / 3, with_rehearsal(6 * kNormThreads), stream, p);
    if (p.rows <= 4 * ctas)
      return launch_cluster(rmsnorm_quant_kernel<T, VPT, 2, 4, true>, (p.rows + 3) / 4, with_rehearsal(8 * kNormThreads), stream, p);
  }
  return bq::kErrTooLarge;
}

// The gated norm: 16 warps for a row; two rows take 32, so that no warp has more heads than it would have of one (27
// rows 239.1 -> 237.1; with 16 warps 242).  Three rows lose (40 rows 264 and 267).
template <typename T, bool Y_F32>
int launch_gated_cluster(GatedParams p, cudaStream_t stream) {
  constexpr int kWarps = 2 * kGatedWarps;
  p.cta_rows = p.rows <= kMaxCluster ? 1 : 2;
  const int ctas = (p.rows + p.cta_rows - 1) / p.cta_rows, heads = p.cta_rows * p.heads;
  if (ctas > kMaxCluster) return bq::kErrTooLarge;
  if (p.cta_rows == 1) {
    if (heads <= kWarps) return launch_cluster(gated_rmsnorm_quant_kernel<T, Y_F32, 1, kWarps, true>, ctas, with_rehearsal(kWarps * 32), stream, p);
    if (heads <= 2 * kWarps) return launch_cluster(gated_rmsnorm_quant_kernel<T, Y_F32, 2, kWarps, true>, ctas, with_rehearsal(kWarps * 32), stream, p);
    if (heads <= 4 * kWarps) return launch_cluster(gated_rmsnorm_quant_kernel<T, Y_F32, 4, kWarps, true>, ctas, with_rehearsal(kWarps * 32), stream, p);
  } else {
    if (heads <= 2 * kWarps)
      return launch_cluster(gated_rmsnorm_quant_kernel<T, Y_F32, 1, 2 * kWarps, true>, ctas, with_rehearsal(2 * kWarps * 32), stream, p);
    if (heads <= 4 * kWarps)
      return launch_cluster(gated_rmsnorm_quant_kernel<T, Y_F32, 2, 2 * kWarps, true>, ctas, with_rehearsal(2 * kWarps * 32), stream, p);
    if (heads <= 8 * kWarps)
      return launch_cluster(gated_rmsnorm_quant_kernel<T, Y_F32, 4, 2 * kWarps, true>, ctas, with_rehearsal(2 * kWarps * 32), stream, p);
  }
  return bq::kErrTooLarge;
}

// kErrTooLarge where the grid is not resident at once.  launch_row_groups: the most registers and the fewest rows per CTA
// whose grid is.
template <typename T, int VPT, int R, int PER_SM>
int launch_row_groups_of(const NormParams& p, cudaStream_t stream) {
  int dev = 0, sms = 0;
  const size_t smem = static_cast<size_t>(p.cols) * sizeof(float);     // gamma
  const int threads = kRowGroups * kNormThreads;
  const int per_sm = resident_per_sm(rmsnorm_rows_quant_kernel<T, VPT, R, PER_SM>, threads, smem);
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || per_sm < 1) {
    (void)cudaGetLastError();
    return bq::kErrTooLarge;
  }
  const int grid = (p.rows + kRowGroups * R - 1) / (kRowGroups * R);
  if (static_cast<long long>(grid) > static_cast<long long>(sms) * per_sm) return bq::kErrTooLarge;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(grid), 1, 1);
  cfg.blockDim = dim3(static_cast<unsigned>(threads), 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, rmsnorm_rows_quant_kernel<T, VPT, R, PER_SM>, p);
  if (e != cudaSuccess) { (void)cudaGetLastError(); return bq::kErrLaunch; }
  return bq::kOk;
}
template <typename T, int VPT>
int launch_row_groups(const NormParams& p, cudaStream_t stream) {
  if (static_cast<size_t>(p.cols) * sizeof(float) > 40 * 1024) return bq::kErrTooLarge;
  int rc = bq::kErrTooLarge;
  if constexpr (kOneRowPerGroup<T, VPT>) rc = launch_row_groups_of<T, VPT, 1, 2>(p, stream);
  if constexpr (kTwoRowsPerGroup<T, VPT>) {
    if (rc == bq::kErrTooLarge) rc = launch_row_groups_of<T, VPT, 1, 3>(p, stream);
    if (rc == bq::kErrTooLarge) rc = launch_row_groups_of<T, VPT, 2, VPT * sizeof(T) <= 8 ? 3 : 2>(p, stream);
  }
  return rc;
}

template <typename T>
int launch_rmsnorm(const NormParams& p, cudaStream_t stream) {
  const int per_thread = (p.cols / kVec + kNormThreads - 1) / kNormThreads;
  // Decode batches: four times the threads, a quarter of the chain each (see the kernel).  Larger ones need
  // the CTAs resident at once.
  if (p.rows > 1 && p.rows <= kClusterRows && g_cluster_exchange) {
    int rc = bq::kErrTooLarge;
    if (per_thread <= 2) rc = launch_rmsnorm_cluster<T, 2>(p, stream);
    else if (per_thread <= 4) rc = launch_rmsnorm_cluster<T, 4>(p, stream);
    else if (per_thread <= 8) rc = launch_rmsnorm_cluster<T, 8>(p, stream);
    else if (per_thread <= 16) rc = launch_rmsnorm_cluster<T, 16>(p, stream);
    if (rc != bq::kErrTooLarge) return rc;
  }
  if (p.rows <= kWideRows) {
    if (per_thread <= 2) return launch_rows(rmsnorm_quant_kernel<T, 2, 2, 1, false>, p.rows, 2 * kNormThreads, p, stream);
    if (per_thread <= 4) return launch_rows(rmsnorm_quant_kernel<T, 4, 4, 1, false>, p.rows, 4 * kNormThreads, p, stream);
    if (per_thread <= 8) return launch_rows(rmsnorm_quant_kernel<T, 8, 4, 1, false>, p.rows, 4 * kNormThreads, p, stream);
    if (per_thread <= 16) return launch_rows(rmsnorm_quant_kernel<T, 16, 4, 1, false>, p.rows, 4 * kNormThreads, p, stream);
  }
  int rc = bq::kErrTooLarge;
  if (p.rows <= grouped_rows(per_thread)) {}
  else if (per_thread <= 2) rc = launch_row_groups<T, 2>(p, stream);
  else if (per_thread <= 4) rc = launch_row_groups<T, 4>(p, stream);
  else if (per_thread <= 8) rc = launch_row_groups<T, 8>(p, stream);
  else if (per_thread <= 16) rc = launch_row_groups<T, 16>(p, stream);
  if (rc != bq::kErrTooLarge) return rc;
  if (per_thread <= 2) return launch_rows(rmsnorm_quant_kernel<T, 2, 1, 1, false>, p.rows, kNormThreads, p, stream);
  if (per_thread <= 4) return launch_rows(rmsnorm_quant_kernel<T, 4, 1, 1, false>, p.rows, kNormThreads, p, stream);
  if (per_thread <= 8) return launch_rows(rmsnorm_quant_kernel<T, 8, 1, 1, false>, p.rows, kNormThreads, p, stream);
  if (per_thread <= 16) return launch_rows(rmsnorm_quant_kernel<T, 16, 1, 1, false>, p.rows, kNormThreads, p, stream);
  return bq::kErrUnsupported;
}

template <typename T, bool Y_F32>
int launch_gated(const GatedParams& p, cudaStream_t stream) {
  // Decode batches: two heads per warp, 16 warps, so that the chain of a head -- sum, square root,
  // exponentials, divisions -- is walked at most twice one after the other.  Larger batches need the
  // CTAs resident at once.
  if (p.rows > 1 && p.rows <= 2 * kMaxCluster && g_cluster_exchange) {
    const int rc = launch_gated_cluster<T, Y_F32>(p, stream);
    if (rc != bq::kErrTooLarge) return rc;
  }
  if (p.rows <= kWideGatedRows && p.heads > kGatedWarps) {
    constexpr int kWarps = 2 * kGatedWarps;
    if (p.heads <= kWarps) return launch_rows(gated_rmsnorm_quant_kernel<T, Y_F32, 1, kWarps, false>, p.rows, kWarps * 32, p, stream);
    if (p.heads <= 2 * kWarps)
      return launch_rows(gated_rmsnorm_quant_kernel<T, Y_F32, 2, kWarps, false>, p.rows, kWarps * 32, p, stream);
  }
  const int hpw = (p.heads + kGatedWarps - 1) / kGatedWarps;
  const int threads = kGatedWarps * 32;
  if (hpw <= 1) return launch_rows(gated_rmsnorm_quant_kernel<T, Y_F32, 1, kGatedWarps, false>, p.rows, threads, p, stream);
  if (hpw <= 2) return launch_rows(gated_rmsnorm_quant_kernel<T, Y_F32, 2, kGatedWarps, false>, p.rows, threads, p, stream);
  if (hpw <= 4) return launch_rows(gated_rmsnorm_quant_kernel<T, Y_F32, 4, kGatedWarps, false>, p.rows, threads, p, stream);
  if (hpw <= kMaxHeadsPerWarp)
    return launch_rows(gated_rmsnorm_quant_kernel<T, Y_F32, kMaxHeadsPerWarp, kGatedWarps, false>, p.rows, threads, p, stream);
  return bq::kErrUnsupported;
}

inline bool aligned_to(const void* p, size_t a) { return (reinterpret_cast<uintptr_t>(p) % a) == 0; }
inline size_t elem_size(int dtype) { return dtype == BQ_DTYPE_F32 ? 4 : 2; }
inline bool known_dtype(int d) { return d == BQ_DTYPE_F32 || d == BQ_DTYPE_BF16 || d == BQ_DTYPE_F16; }

}  // namespace

// The gated norm for more rows than one co-resident grid has CTAs (prefill): a warp owns four
// heads of one row at a time (head arithmetic exactly as above; no CTA-wide step in it), the
// warps of the grid stride over all (row, quad of heads) units, write the gated activation and fold
// max |h| into one word as rmsnorm_scale_kernel does; the cast pass follows in stream order.
//
// Four heads, because a lone head costs a warp 5 shuffles, a broadcast, a division and a square root for
// 4 elements per lane: the four trees share theirs (quad_tree_sum), and four times the bytes are in
// flight per warp.  With the cast pass, 9658 x 32 heads, fp32 scan output: 121 -> 95 us; 4096 rows 57 -> 44.
constexpr int kQuad = 4;

// The shuffle-down tree sums of four values at once.  Every step halves the lanes of a value and hands
// the other half's lanes to another value, so that 6 shuffles do the work of 20; what is added to
// what is the tree of warp_tree_sum (operands in either order: addition commutes).  Lane l
// returns the sum of s[l / 8].
__device__ __forceinline__ float quad_tree_sum(const float (&s)[kQuad], int lane) {
  const bool hi16 = (lane & 16) != 0, hi8 = (lane & 8) != 0;
  float a0 = hi16 ? s[2] : s[0], a1 = hi16 ? s[3] : s[1];
  const float b0 = hi16 ? s[0] : s[2], b1 = hi16 ? s[1] : s[3];
  a0 = __fadd_rn(a0, __shfl_xor_sync(0xffffffffu, b0, 16));
  a1 = __fadd_rn(a1, __shfl_xor_sync(0xffffffffu, b1, 16));
  float c = hi8 ? a1 : a0;
  c = __fadd_rn(c, __shfl_xor_sync(0xffffffffu, hi8 ? a0 : a1, 8));
#pragma unroll
  for (int off = 4; off > 0; off >>= 1) c = __fadd_rn(c, __shfl_xor_sync(0xffffffffu, c, off));
  return c;
}

template <typename T, bool Y_F32>
__global__ void __launch_bounds__(kGatedWarps * 32) gated_rmsnorm_scale_kernel(const GatedParams p) {
  bq::pdl_launch_dependents();
  __shared__ float s_max[kGatedWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float4 gm = __ldg(reinterpret_cast<const float4*>(p.gamma) + lane);
  const float gmv[kVec] = {gm.x, gm.y, gm.z, gm.w};
  bq::pdl_wait_prior_grids();
  // position of this warp's unit, carried along: (row, quad of heads)
  const int quads = (p.heads + kQuad - 1) / kQuad;
  const long long first = static_cast<long long>(blockIdx.x) * kGatedWarps + warp;
  const long long stride = static_cast<long long>(gridDim.x) * kGatedWarps;
  const long long row_step = stride / quads;
  const int quad_step = static_cast<int>(stride - row_step * quads);
  long long row = first / quads;
  int quad = static_cast<int>(first - row * quads);
  AbsMax<T> mx;
  while (row < p.rows) {
    const int live = p.heads - quad * kQuad < kQuad ? p.heads - quad * kQuad : kQuad;     // heads of this unit
    const long long off = static_cast<long long>(quad) * kQuad * kHeadDim + lane * kVec;
    Vec4<T> core[kQuad], gate[kQuad];
#pragma unroll
    for (int h = 0; h < kQuad; ++h) {
      core[h] = Vec4<T>{};
      gate[h] = Vec4<T>{};
      if (h < live) {
        if constexpr (Y_F32) {
          const float4 f = __ldcg(reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p.y) + row * p.ld_y +
                                                                  off + h * kHeadDim));
          *reinterpret_cast<uint2*>(&core[h]) = make_uint2(pack2<T>(f.x, f.y), pack2<T>(f.z, f.w));
        } else {
          core[h] = load4(reinterpret_cast<const T*>(p.y) + row * p.ld_y + off + h * kHeadDim);
        }
        gate[h] = load4(reinterpret_cast<const T*>(p.z) + row * p.ld_z + off + h * kHeadDim);
      }
    }
    float s[kQuad];
#pragma unroll
    for (int h = 0; h < kQuad; ++h) {
      s[h] = 0.0f;
#pragma unroll
      for (int j = 0; j < kVec; ++j) {
        const float f = widen(core[h].v[j]);
        s[h] = __fmaf_rn(f, f, s[h]);
      }
    }
    const float total = quad_tree_sum(s, lane);      // head lane / 8
    // division by 128: the product with its reciprocal has the same bits
    const float rstd8 = rsqrtf(__fadd_rn(__fmul_rn(total, 1.0f / kHeadDim), p.eps));
#pragma unroll
    for (int h = 0; h < kQuad; ++h) {
      const float rstd = __shfl_sync(0xffffffffu, rstd8, h * 8);
      float silu[kVec] = {widen(gate[h].v[0]), widen(gate[h].v[1]), widen(gate[h].v[2]), widen(gate[h].v[3])};
      gate_group<T, kSilu, kVec>(silu);
      if constexpr (sizeof(T) == 2) {
        uint32_t* const w = reinterpret_cast<uint32_t*>(&core[h]);
#pragma unroll
        for (int j = 0; j < kVec; j += 2) {
          const float2 r = mul2(make_float2(rstd, rstd), unpack2<T>(w[j / 2]));
          const float2 xn = unpack2<T>(pack2<T>(r.x, r.y));
          const float2 y = mul2(mul2(make_float2(gmv[j], gmv[j + 1]), xn), make_float2(silu[j], silu[j + 1]));
          w[j / 2] = pack2<T>(y.x, y.y);
        }
      } else {
#pragma unroll
        for (int j = 0; j < kVec; ++j)
          core[h].v[j] = __fmul_rn(__fmul_rn(gmv[j], __fmul_rn(rstd, core[h].v[j])), silu[j]);
      }
      if (h < live) {
        mx.add(core[h]);
        store4(reinterpret_cast<T*>(p.h_out) + row * p.ld_h + off + h * kHeadDim, core[h]);
      }
    }
    row += row_step;
    quad += quad_step;
    if (quad >= quads) { quad -= quads; ++row; }
  }
  float m = mx.value();
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) m = nan_max(m, __shfl_xor_sync(0xffffffffu, m, off));
  if (lane == 0) s_max[warp] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    float w = s_max[0];
    for (int i = 1; i < kGatedWarps; ++i) w = nan_max(w, s_max[i]);
    QuantWs* ws = static_cast<QuantWs*>(p.ws);
    atomicMax(&ws->amax_bits, __float_as_uint(w));
    __threadfence();
    const unsigned int old = atomicAdd(&ws->arrive, 1u);
    if (old == gridDim.x - 1) {
      __threadfence();
      const unsigned int bits = atomicExch(&ws->amax_bits, 0u);
      p.scale[0] = scale_from_amax(__uint_as_float(bits));
      ws->arrive = 0u;
      __threadfence();
    }
  }
}

namespace {
template <typename T, int VPT, bool DENSE>
cudaError_t launch_rmsnorm_scale_of(const NormParams& p, int sms, size_t smem, cudaStream_t stream) {
  auto launch = [&](auto whole) {
    return launch_resident_smem(rmsnorm_scale_kernel<T, VPT, DENSE, decltype(whole)::value>, p.rows, kNormThreads, sms, true, smem, stream, p);
  };
  if (p.cols == VPT * kNormThreads * kVec) return launch(std::integral_constant<int, kWholeKernel<T, VPT>>{});
  return launch(std::integral_constant<int, kPartialKernel<T, VPT, DENSE>>{});
}
template <typename T, bool DENSE>
int launch_rmsnorm_scale(const NormParams& p, cudaStream_t stream) {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    (void)cudaGetLastError();
    return bq::kErrLaunch;
  }
  const int per_thread = (p.cols / kVec + kNormThreads - 1) / kNormThreads;
  const size_t smem = static_cast<size_t>(p.cols) * sizeof(float);     // gamma
  if (smem > 48 * 1024) return bq::kErrUnsupported;
  cudaError_t e;
  if (per_thread <= 2) e = launch_rmsnorm_scale_of<T, 2, DENSE>(p, sms, smem, stream);
  else if (per_thread <= 4) e = launch_rmsnorm_scale_of<T, 4, DENSE>(p, sms, smem, stream);
  else if (per_thread <= 8) e = launch_rmsnorm_scale_of<T, 8, DENSE>(p, sms, smem, stream);
  else if (per_thread <= 16) e = launch_rmsnorm_scale_of<T, 16, DENSE>(p, sms, smem, stream);
  else return bq::kErrUnsupported;
  if (e != cudaSuccess) { (void)cudaGetLastError(); return bq::kErrLaunch; }
  return bq::kOk;
}

// CTAs that are resident at once, the rows dealt out among those of one column block.
template <typename T, bool BESIDE>
int launch_rmsnorm_cast_of(NormParams p, cudaStream_t stream) {
  int dev = 0, sms = 0;
  const int row_groups = p.cols / kGroup, columns = (row_groups + kCastThreads - 1) / kCastThreads;
  // Wide rows: as many threads as their column blocks need, in whole warps; with 256 always, 2112 columns left half of them idle.
  // us, 256 / so many: fp32 1776 x 2112 12.7 / 10.6, 9658 x 2560 41.7 / 35.3, bf16 9658 x 2560 35.9 / 30.1, 4000 x 4608 23.6 / 21.3.
  const int threads = BESIDE ? kCastThreads : ((row_groups + columns - 1) / columns + 31) / 32 * 32;
  const int per_sm = resident_per_sm(rmsnorm_cast_kernel<T, BESIDE>, threads, 0);
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || per_sm < 1) {
    (void)cudaGetLastError();
    return bq::kErrLaunch;
  }
  p.beside = 1;
  if (BESIDE) {
    const int once = (p.rows - 1) / (kCastRows * per_sm * sms) + 1;
    p.beside = kCastThreads / row_groups < once ? kCastThreads / row_groups : once;
  }
  const int most = (p.rows - 1) / (kCastRows * p.beside) + 1;
  int slices = per_sm * sms / columns;
  if (slices > most) slices = most;
  if (slices < 1) slices = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(columns), static_cast<unsigned>(slices), 1);
  cfg.blockDim = dim3(static_cast<unsigned>(threads), 1, 1);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, rmsnorm_cast_kernel<T, BESIDE>, p);
  if (e != cudaSuccess) { (void)cudaGetLastError(); return bq::kErrLaunch; }
  return bq::kOk;
}
template <typename T>
int launch_rmsnorm_cast(const NormParams& p, cudaStream_t stream) {
  return p.cols / kGroup <= kCastThreads / 2 ? launch_rmsnorm_cast_of<T, true>(p, stream) : launch_rmsnorm_cast_of<T, false>(p, stream);
}
}  // namespace

extern "C" int bq_rmsnorm_scale(const void* x, int dtype, int64_t rows, int64_t cols, int64_t ld_x,
                                const float* gamma, float eps, void* h_out, int64_t ld_h,
                                float* scale_out, void* ws, size_t ws_bytes, void* stream) {
  if (!x || !gamma || !h_out || !scale_out || rows <= 0 || cols <= 0) return bq::kErrBadArg;
  if (!known_dtype(dtype)) return bq::kErrBadArg;
  if (ws == nullptr || ws_bytes < sizeof(QuantWs) || !aligned_to(ws, 16)) return bq::kErrWorkspace;
  const size_t es = elem_size(dtype);
  const size_t vec_bytes = kVec * es;
  if (cols % kVec || ld_x < cols || (ld_x * es) % vec_bytes || !aligned_to(x, vec_bytes) ||
      !aligned_to(gamma, 16) || ld_h < cols || (ld_h * es) % vec_bytes || !aligned_to(h_out, vec_bytes))
    return bq::kErrUnsupported;
  if (rows > 0x7fffffffLL || cols > 0x7fffffffLL) return bq::kErrTooLarge;
  NormParams p{};
  p.x = x; p.gamma = gamma; p.h_out = h_out;
  p.scale = scale_out; p.ws = ws;
  p.rows = static_cast<int>(rows); p.cols = static_cast<int>(cols);
  p.ld_x = ld_x; p.ld_h = ld_h; p.eps = eps;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case BQ_DTYPE_F32: return launch_rmsnorm_scale<float, true>(p, s);
    case BQ_DTYPE_BF16: return launch_rmsnorm_scale<__nv_bfloat16, true>(p, s);
    default: return launch_rmsnorm_scale<__half, true>(p, s);
  }
}

extern "C" int bq_rmsnorm_quant_rows(const void* x, int dtype, int64_t rows, int64_t cols, int64_t ld_x, const float* gamma,
                                     float eps, void* q_out, float* scale_out, float* rstd, void* ws, size_t ws_bytes, void* stream) {
  if (!x || !gamma || !q_out || !scale_out || !rstd || rows <= 0 || cols <= 0) return bq::kErrBadArg;
  if (!known_dtype(dtype)) return bq::kErrBadArg;
  if (ws == nullptr || ws_bytes < sizeof(QuantWs) || !aligned_to(ws, 16)) return bq::kErrWorkspace;
  const size_t es = elem_size(dtype);
  if (cols % kGroup || ld_x < cols || (ld_x * es) % 16 || !aligned_to(x, 16) || !aligned_to(gamma, 16) ||
      !aligned_to(q_out, 8) || !aligned_to(rstd, 4))
    return bq::kErrUnsupported;
  if (rows > 0x7fffffffLL || cols > 0x7fffffffLL) return bq::kErrTooLarge;
  NormParams p{};
  p.x = x; p.gamma = gamma;
  p.q = static_cast<uint8_t*>(q_out); p.scale = scale_out; p.rstd = rstd; p.ws = ws;
  p.rows = static_cast<int>(rows); p.cols = static_cast<int>(cols);
  p.ld_x = ld_x; p.eps = eps;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int rc;
  switch (dtype) {
    case BQ_DTYPE_F32: rc = launch_rmsnorm_scale<float, false>(p, s); break;
    case BQ_DTYPE_BF16: rc = launch_rmsnorm_scale<__nv_bfloat16, false>(p, s); break;
    default: rc = launch_rmsnorm_scale<__half, false>(p, s);
  }
  if (rc != bq::kOk) return rc;
  switch (dtype) {
    case BQ_DTYPE_F32: return launch_rmsnorm_cast<float>(p, s);
    case BQ_DTYPE_BF16: return launch_rmsnorm_cast<__nv_bfloat16>(p, s);
    default: return launch_rmsnorm_cast<__half>(p, s);
  }
}

extern "C" int bq_rmsnorm_quant(const void* x, int dtype, int64_t rows, int64_t cols, int64_t ld_x,
                                const float* gamma, float eps, void* h_out, int64_t ld_h, void* q_out,
                                float* scale_out, void* ws, size_t ws_bytes, void* stream) {
  if (!x || !gamma || !q_out || !scale_out || rows <= 0 || cols <= 0) return bq::kErrBadArg;
  if (!known_dtype(dtype)) return bq::kErrBadArg;
  if (ws == nullptr || ws_bytes < sizeof(QuantWs) || !aligned_to(ws, 16)) return bq::kErrWorkspace;
  const size_t es = elem_size(dtype);
  const size_t vec_bytes = kVec * es;
  if (cols % kVec || ld_x < cols || (ld_x * es) % vec_bytes || !aligned_to(x, vec_bytes) ||
      !aligned_to(gamma, 16) || !aligned_to(q_out, 4))
    return bq::kErrUnsupported;
  if (h_out != nullptr && (ld_h < cols || (ld_h * es) % vec_bytes || !aligned_to(h_out, vec_bytes)))
    return bq::kErrUnsupported;
  if (rows > 0x7fffffffLL || cols > 0x7fffffffLL) return bq::kErrTooLarge;
  NormParams p{};
  p.x = x; p.gamma = gamma; p.h_out = h_out;
  p.q = static_cast<uint8_t*>(q_out); p.scale = scale_out; p.ws = ws;
  p.rows = static_cast<int>(rows); p.cols = static_cast<int>(cols);
  p.ld_x = ld_x; p.ld_h = ld_h; p.eps = eps;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (dtype) {
    case BQ_DTYPE_F32: return launch_rmsnorm<float>(p, s);
    case BQ_DTYPE_BF16: return launch_rmsnorm<__nv_bfloat16>(p, s);
    default: return launch_rmsnorm<__half>(p, s);
  }
}

extern "C" int bq_gated_rmsnorm_quant(const void* y, int y_dtype, int64_t ld_y, const void* z, int dtype,
                                      int64_t ld_z, const float* gamma, float eps, int64_t rows,
                                      int64_t heads, int64_t head_dim, void* q_out, float* scale_out,
                                      void* ws, size_t ws_bytes, void* stream) {
  if (!y || !z || !gamma || !q_out || !scale_out || rows <= 0 || heads <= 0) return bq::kErrBadArg;
  if (!known_dtype(dtype) || (y_dtype != dtype && y_dtype != BQ_DTYPE_F32)) return bq::kErrBadArg;
  if (ws == nullptr || ws_bytes < sizeof(QuantWs) || !aligned_to(ws, 16)) return bq::kErrWorkspace;
  if (head_dim != kHeadDim || heads > kGatedWarps * kMaxHeadsPerWarp) return bq::kErrUnsupported;
  const size_t es = elem_size(dtype), ys = elem_size(y_dtype);
  const int64_t width = heads * head_dim;
  if (ld_y < width || ld_z < width || (ld_y * ys) % (kVec * ys) || (ld_z * es) % (kVec * es) ||
      !aligned_to(y, kVec * ys) || !aligned_to(z, kVec * es) || !aligned_to(gamma, 16) ||
      !aligned_to(q_out, 4))
    return bq::kErrUnsupported;
  if (rows > 0x7fffffffLL) return bq::kErrTooLarge;
  GatedParams p{};
  p.y = y; p.z = z; p.gamma = gamma;
  p.q = static_cast<uint8_t*>(q_out); p.scale = scale_out; p.ws = ws;
  p.rows = static_cast<int>(rows); p.heads = static_cast<int>(heads);
  p.ld_y = ld_y; p.ld_z = ld_z; p.eps = eps;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const bool yf32 = (y_dtype == BQ_DTYPE_F32) && (dtype != BQ_DTYPE_F32);
  switch (dtype) {
    case BQ_DTYPE_F32: return launch_gated<float, false>(p, s);
    case BQ_DTYPE_BF16:
      return yf32 ? launch_gated<__nv_bfloat16, true>(p, s) : launch_gated<__nv_bfloat16, false>(p, s);
    default:
      return yf32 ? launch_gated<__half, true>(p, s) : launch_gated<__half, false>(p, s);
  }
}

extern "C" int bq_gated_rmsnorm_scale(const void* y, int y_dtype, int64_t ld_y, const void* z, int dtype,
                                      int64_t ld_z, const float* gamma, float eps, int64_t rows,
                                      int64_t heads, int64_t head_dim, void* h_out, int64_t ld_h,
                                      float* scale_out, void* ws, size_t ws_bytes, void* stream) {
  if (!y || !z || !gamma || !h_out || !scale_out || rows <= 0 || heads <= 0) return bq::kErrBadArg;
  if (!known_dtype(dtype) || (y_dtype != dtype && y_dtype != BQ_DTYPE_F32)) return bq::kErrBadArg;
  if (ws == nullptr || ws_bytes < sizeof(QuantWs) || !aligned_to(ws, 16)) return bq::kErrWorkspace;
  if (head_dim != kHeadDim) return bq::kErrUnsupported;
  const size_t es = elem_size(dtype), ys = elem_size(y_dtype);
  const int64_t width = heads * head_dim;
  if (ld_y < width || ld_z < width || ld_h < width || (ld_y * ys) % (kVec * ys) ||
      (ld_z * es) % (kVec * es) || (ld_h * es) % (kVec * es) || !aligned_to(y, kVec * ys) ||
      !aligned_to(z, kVec * es) || !aligned_to(h_out, kVec * es) || !aligned_to(gamma, 16))
    return bq::kErrUnsupported;
  if (rows > 0x7fffffffLL || heads > 0x7fffLL) return bq::kErrTooLarge;
  GatedParams p{};
  p.y = y; p.z = z; p.gamma = gamma; p.h_out = h_out; p.ld_h = ld_h;
  p.scale = scale_out; p.ws = ws;
  p.rows = static_cast<int>(rows); p.heads = static_cast<int>(heads);
  p.ld_y = ld_y; p.ld_z = ld_z; p.eps = eps;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    (void)cudaGetLastError();
    return bq::kErrLaunch;
  }
  const long long want = (rows * heads + kGatedWarps - 1) / kGatedWarps;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int threads = kGatedWarps * 32;
  const bool yf32 = (y_dtype == BQ_DTYPE_F32) && (dtype != BQ_DTYPE_F32);
  cudaError_t e;
  switch (dtype) {
    case BQ_DTYPE_F32:
      e = launch_resident(gated_rmsnorm_scale_kernel<float, false>, want, threads, sms, true, st, p);
      break;
    case BQ_DTYPE_BF16:
      e = yf32 ? launch_resident(gated_rmsnorm_scale_kernel<__nv_bfloat16, true>, want, threads, sms, true, st, p)
               : launch_resident(gated_rmsnorm_scale_kernel<__nv_bfloat16, false>, want, threads, sms, true, st, p);
      break;
    default:
      e = yf32 ? launch_resident(gated_rmsnorm_scale_kernel<__half, true>, want, threads, sms, true, st, p)
               : launch_resident(gated_rmsnorm_scale_kernel<__half, false>, want, threads, sms, true, st, p);
  }
  if (e != cudaSuccess) { (void)cudaGetLastError(); return bq::kErrLaunch; }
  return bq::kOk;
}
