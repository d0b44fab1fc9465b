// Per-tensor FP8 W8A8 GEMM for sm_100a:  Y[M,N] = (Xq[M,K] . Wq[N,K]^T) * sx * sw.
//
// Stands in for the `torch._scaled_mm(xq, w.data.t(), scale_a=sx, scale_b=w.scale)`
// call of the reference engine (braid/model/quant.py:232-241).  Both operands are
// K-major, so 128-byte-swizzled TMA tiles feed tcgen05 shared-memory descriptors
// directly; accumulation is fp32 in tensor memory; the dequant scales and the
// output cast are applied in the epilogue.
//
// Two kernels, chosen by M:
//
//  * gemm_stream_kernel (M <= 256, the decode regime; HBM-bound, measured in GB/s).
//    Operands are swapped: 128 WEIGHT rows sit on the MMA M side and the (padded)
//    batch on the MMA N side, so a tile streams 128 x K weight bytes whatever the
//    batch is.  One CTA per (row tile, K slice); the K slices of a tile form a
//    thread-block cluster and are summed through distributed shared memory in a
//    fixed order -- no float atomics, so results are run-to-run identical and a
//    graph replay equals the eager run bit for bit.  Several weights that share
//    one activation (q/k/v, qkv/z, gate/up) go in one launch, each segment with
//    its own scale.
//
//  * gemm_pair_kernel (M > 256, the prefill regime; tensor-bound, measured in
//    TFLOP/s).  Persistent, warp-specialised CTA pairs (cta_group::2): one TMA
//    producer warp, one MMA issuer warp, four epilogue warps; 256x256 output
//    tiles; two 256-column accumulators in tensor memory so a tile's epilogue
//    overlaps the next tile's main loop; the epilogue stages 128-byte row
//    pieces in shared memory and hands them to TMA stores.
//
// Every mbarrier wait is bounded (ptx.cuh); a wait that runs out sets the sticky
// status word and the CTA unwinds through the normal teardown.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include "../../include/braid_b200.h"
#include "ptx.cuh"
#include "quant_device.cuh"
#include "grid_amax.cuh"

namespace {

using namespace bq;

constexpr int kBK = 128;         // K bytes per pipeline stage: one swizzle span
constexpr int kUmmaK = 32;       // K elements one f8 MMA consumes
constexpr int kRowTile = 128;    // MMA M
constexpr int kATileBytes = kRowTile * kBK;   // 16 KiB
constexpr int kMaxSmem = 232448;              // 227 KiB opt-in limit per CTA
#ifndef BQ_STREAM_THREADS
#define BQ_STREAM_THREADS 384
#endif
constexpr int kStreamThreads = BQ_STREAM_THREADS;   // weight-streaming kernel: warps 0 / 1 load and
constexpr int kStreamWarps = kStreamThreads / 32;   // issue MMAs, ALL warps run the epilogue
constexpr int kBarrierBytes = 1024;           // mbarriers + tmem slot + flags
constexpr int kNoIndex = 0x7fffffff;          // greedy pick: "nothing yet", loses against any real column

struct Segment {
  const float* sw;     // device: weight dequant scale
  void* y;             // device: output base of this segment
  long long ldy;       // row stride of y, elements
  const void* res;     // stream kernel: optional residual [M, n] of the output type, added after
                       // the output has been rounded to that type (two roundings, as the separate
                       // GEMM and add kernels give)
  long long ld_res;
  int dense;           // stream kernel: 1 = a 16-bit (bf16 / fp16) weight multiplied with the
                       // unquantized activation (kind::f16 MMA, no scales), 0 = e4m3 weight
  int y_tma;           // pair kernel: the output can be described to TMA (16-byte aligned base and pitch)
  int n;               // weight rows (output columns) of this segment
  int tile_begin;      // tile kernel: index of the segment's first tile
  int split;           // stream kernel: K slices of this weight (1, 2, 4 or 8)
  int split_forced;    // stream kernel: non-zero = use this split instead of the shape rule
  int cluster_begin;   // stream kernel: index of the segment's first cluster
  int un;              // wide kernel: weight rows per unit (gate/up form: output columns per unit);
                       // pair kernel, plain form: output columns per tile
  int unit_begin;      // wide kernel: index of the segment's first unit
  int wide;            // wide kernel: output (and residual) rows are 16-byte aligned
};

// SiLU(gate)*up and the quantization of the product, done in the epilogue of ONE GEMM whose
// 128-row MMA tiles are put together from 64 gate rows and the 64 up rows of the same output
// columns -- two TMA boxes per pipeline stage, read from the two weights where they lie (the
// reference keeps gate_proj and up_proj as two tensors, braid/model/mlp.py:27-29; nothing is
// repacked or copied).
struct PairSilu {
  int on;
  int prefill;             // M > 256: the CTA-pair kernel writes h itself ([M, I], activation type)
                           // and the scale of h; the codes are a separate cast pass
  const void* wq_up;       // device: the up weight [I, K] (segment 0's weight pointer is the gate weight)
  const float* sw_up;      // device: dequant scale of the up half (seg.sw is the gate half's)
  void* h;                 // decode: h itself goes here ([M, I], activation type) and its max to words[0]; the
                           // product that follows casts it.  nullptr: codes and scale, behind a grid-wide exchange
  uint8_t* hq;             // device: e4m3 codes of h, [M, ld_hq]
  long long ld_hq;
  float* sh;               // device: the scale of h
  unsigned int* words;     // [0] amax bits [1] arrivals [2] departures ([3] is the sticky status)
  unsigned int expected;   // CTAs that take part in the exchange (the active ones)
  const uint8_t* next;     // device: what the launch behind this one streams first, next_bytes of it (0: nothing)
  unsigned int next_bytes;
  int next_warp;           // the warp of a CTA that asks for it
};

// Behind the last load of a gate/up launch HBM idles for its tail: the exchange, the cast, the start of the down projection.  One
// warp of every CTA asks its share of the first megabytes of the down weight into L2 meanwhile; behind the exchange, whose trips
// to L2 a saturated memory would delay, and not more than the tail brings in.  Four graphed layers of hidden 4096, none / 8 MB
// / 16 MB / 32 MB: 1 row 198.5 / 196.5 / 196.5 / 203.5 us, 8 rows 217.7 / 214.1 / 213.7 / 220.3, 16 rows 223.7 / 220.3 /
// 219.9 / 225.8, 48 rows 251.2 / 249.0 / 250.6 / 255.0; before the exchange 8 MB give 217.1 at 8 rows and nothing at 27.  In pieces of
// less than 1 KB, so that every CTA of the down projection gets its share, the instructions cost more than that (8 rows
// 220 to 225), and the kernel for wider batches loses (64 rows 274.6 -> 278.3).
// It takes a down weight of 12 MB.  us of one MLP over cold weights, 16 rows, none / asked by warp 0 / by the last warp: 1792 x 5376 (9.6
// MB) 13.1 / 14.7 / 13.6; 2048 x 6144 (12 MB) 14.7 / 15.6 / 15.1, but in graphed layers 127.0 / 125.7 / 124.1; 2304 x 6912 (15) 17.0 / 16.8 /
// 16.6; 2560 x 7680 (19) 20.0 / 18.8 / 18.6; 3072 x 9216 (27) 23.4 / 22.2 / 22.3; 4096 x 12288 (48) 33.5 / 31.8 / 32.1.  The last warp has no
// row to write where rows are few, which a short launch notices; a long one gains more by the first, which asks sooner.
constexpr unsigned int kNextBytes = 8u << 20, kNextPiece = 4096;
constexpr int64_t kNextFrom = 12 << 20, kNextFirstWarpFrom = 32 << 20;
__device__ __forceinline__ void prefetch_next(const PairSilu& pr) {
  for (unsigned int at = (blockIdx.x * 32u + (threadIdx.x & 31u)) * kNextPiece; at < pr.next_bytes; at += gridDim.x * 32u * kNextPiece)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(pr.next + at), "n"(kNextPiece) : "memory");
}

// Greedy pick fused into the lm_head GEMM: every CTA (one 128-row tile of the vocabulary, K not
// split) reduces, per batch row, the largest of ITS 128 logits -- taken after the rounding to the
// output type the logits tensor would have had, lowest index winning ties, NaN winning over
// everything, which is `logits.argmax(-1)` as torch evaluates it -- and writes one (value,
// index) pair per row; a second, tiny kernel reduces the pairs of all tiles.
struct ArgmaxOut {
  int on;
  int store_logits;          // 0 = the logits themselves are not written at all
  uint2* partial;            // device: [tiles][M] pairs {value as fp32 bits, vocabulary index}
};

// a beats b: NaN first, then the larger value, then the lower index
__device__ __forceinline__ bool argmax_beats(float av, int ai, float bv, int bi) {
  const bool an = av != av, bn = bv != bv;
  if (an || bn) return an && (!bn || ai < bi);
  return av > bv || (av == bv && ai < bi);
}

// Column-parallel form: the output tile (or, in the paired form, h) is stored straight into the
// gathered buffer of every rank of the node -- plain stores through peer-mapped pointers, this
// rank's own buffer included.  The CTAs of the launch count themselves on a local word; the last
// one to finish adds 1 to a counter on each rank with a system-scope release (one arrival per
// rank and exchange).  No collective call, no multicast.  The pointers already carry this rank's
// column offset.
constexpr int kMaxPeers = 8;
struct PushParams {
  int n;                          // destinations (0 = not a push launch)
  void* dst[kMaxPeers];
  long long ld;                   // row stride of every destination, elements
  unsigned int* flag[kMaxPeers];  // one arrival counter per destination rank
  unsigned int* done;             // local: CTAs of this launch that have stored their share
  unsigned int expected;          // CTAs that store (the active ones)
  // prefill SiLU form: where this rank's max |h| (float bits) goes on every rank, written by
  // the last CTA before the arrivals; nullptr = not wanted
  unsigned int* amax_dst[kMaxPeers];
  unsigned int* amax_local;       // local running max of the launch (zero between launches)
};

// The activation unquantized, for the few rows that every CTA quantizes for itself (stream kernel).
struct QuantIn {
  const void* x;       // [M, K] contiguous, 16-byte aligned; nullptr = codes and scale are given
  int dtype;
  int n8;              // groups of 8 values
  unsigned int* words; // nullptr, or scratch: [0] bits of max |x|, which need not be looked for then, [1] CTAs that have
                       // read it; the last one returns both to zero
  unsigned int expected;
};

struct GemmParams {
  Segment seg[BQ_MAX_SEGMENTS];
  int n_seg;
  const float* sx;     // device: activation dequant scale
  int M;               // activation rows
  int mma_n;           // stream kernel: padded batch = MMA N (multiple of 16)
  int k_blocks;        // ceil(K / 128)
  int quant_k;         // K, where the activation arrives unquantized
  int k_blocks_dense;  // stream kernel: 128-byte K blocks of a 16-bit row, ceil(2K / 128)
  int dense_fmt;       // stream kernel: tcgen05 operand format of the 16-bit segments (0 f16, 1 bf16)
  int cluster;         // stream kernel: CTAs per cluster = largest split of the launch
  int handover;        // stream kernel: slices are handed to the CTA that sums them (see handover_bytes)
  int stages;          // stream kernel: depth of the weight ring; pair kernel: pipeline depth
  int b_stages;        // stream kernel: depth of the activation ring
  int out_dtype;
  int m_tiles;         // tile kernel: ceil(M / 128)
  int total_tiles;     // tile kernel
  unsigned int* status;
  ArgmaxOut argmax;
  unsigned long long* phase_ring;   // development builds (BQ_PHASES) only, else nullptr
  int phase_seq;
  PairSilu pair;
  PushParams push;
  QuantIn quant;
};

// What a launch's epilogue does and the type it writes, as template parameters of the kernels.  A decode
// launch runs its epilogue once per CTA, on the critical path and through an instruction cache that
// other kernels have used since, and a prefill launch's MMA and epilogue loops should carry no branch that
// the launch cannot take: one kernel with every form in it was 285 KB of code (the K-sliced one), of
// which a launch runs a tenth (35 to 52 KB now).  Four graphed decoder layers, one kernel -> these: hidden
// 4096, 1 row 252 -> 246 us, 128 rows 339 -> 334; hidden 2560, 16 rows 231 -> 224; hidden 5120, 64 rows
// 449 -> 435; hidden 1024, 8 rows 157 -> 149.  At prefill sizes the residual and 16-bit forms in the one
// kernel had cost every launch 8 %.  kAny, with the type taken at run time, is the column-parallel
// forms, and launches whose segments differ in their form.
enum Epi { kAny = -1, kPlain = 0, kResidual = 1, kGateUp = 2, kMixed = 3, kGateUpDense = 4, kArgmax = 5 };
// The greedy pick has kernels of its own too; in the general ones, a vocabulary of 248320 x 4096 with its logits, repeated: 16
// rows 169 -> 163 us, 64 rows 212 -> 198, 128 rows 231 -> 205.
constexpr int kAnyType = -1;

struct alignas(64) WeightMaps {
  CUtensorMap w[BQ_MAX_SEGMENTS];
};

__device__ __forceinline__ int find_segment(const GemmParams& p, int tile) {
  int s = 0;
#pragma unroll
  for (int i = 1; i < BQ_MAX_SEGMENTS; ++i)
    if (i < p.n_seg && tile >= p.seg[i].tile_begin) s = i;
  return s;
}

__device__ __forceinline__ void store_out4(void* y, long long idx, int out_dtype, float4 v) {
  if (out_dtype == BQ_DTYPE_BF16) {
    const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y);
    const __nv_bfloat162 hi = __floats2bfloat162_rn(v.z, v.w);
    uint2 w;
    w.x = *reinterpret_cast<const uint32_t*>(&lo);
    w.y = *reinterpret_cast<const uint32_t*>(&hi);
    *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(y) + idx) = w;
  } else if (out_dtype == BQ_DTYPE_F16) {
    const __half2 lo = __floats2half2_rn(v.x, v.y);
    const __half2 hi = __floats2half2_rn(v.z, v.w);
    uint2 w;
    w.x = *reinterpret_cast<const uint32_t*>(&lo);
    w.y = *reinterpret_cast<const uint32_t*>(&hi);
    *reinterpret_cast<uint2*>(static_cast<__half*>(y) + idx) = w;
  } else {
    *reinterpret_cast<float4*>(static_cast<float*>(y) + idx) = v;
  }
}

struct EpilogueArgs {
  const float* part;       // this CTA's staging buffer [mma_n][128] fp32
  uint32_t part_addr;      // its shared-memory address
  int peer0;               // cluster rank of K slice 0 of this tile
  int slice_rows;          // > 0: the partials were handed over, slice r of row m lies here at (r * slice_rows + m - m_begin)
  int m_begin, m_end;      // output rows this CTA reduces and writes
  int warp, lane;
  int row0;                // first weight row (output column) of the tile
  float scale;
  bool col_ok;
  void* y;
  long long ldy;
  int out_dtype;
  const void* res;
  long long ld_res;
  const PushParams* push;
};

// Four residual values of the output type, as raw bits (16 bytes cover the widest case).  The residual
// and the activation scale come from kernels this one runs ahead of: no `__ldg` (see ld_coherent4).
__device__ __forceinline__ uint4 load_res4(const void* res, long long idx, int out_dtype) {
  uint4 r = make_uint4(0u, 0u, 0u, 0u);
  if (out_dtype == BQ_DTYPE_F32) {
    r = ld_coherent16(static_cast<const float*>(res) + idx);
  } else {
    const uint2 h = ld_coherent8(static_cast<const uint16_t*>(res) + idx);
    r.x = h.x; r.y = h.y;
  }
  return r;
}

// out = T(float(T(v)) + float(res)): the GEMM's own rounding, then the add's.
__device__ __forceinline__ float4 add_res4(float4 v, uint4 raw, int out_dtype) {
  if (out_dtype == BQ_DTYPE_BF16) {
    const __nv_bfloat162 r0 = *reinterpret_cast<const __nv_bfloat162*>(&raw.x);
    const __nv_bfloat162 r1 = *reinterpret_cast<const __nv_bfloat162*>(&raw.y);
    v.x = __bfloat162float(__float2bfloat16_rn(v.x)) + __bfloat162float(r0.x);
    v.y = __bfloat162float(__float2bfloat16_rn(v.y)) + __bfloat162float(r0.y);
    v.z = __bfloat162float(__float2bfloat16_rn(v.z)) + __bfloat162float(r1.x);
    v.w = __bfloat162float(__float2bfloat16_rn(v.w)) + __bfloat162float(r1.y);
  } else if (out_dtype == BQ_DTYPE_F16) {
    const __half2 r0 = *reinterpret_cast<const __half2*>(&raw.x);
    const __half2 r1 = *reinterpret_cast<const __half2*>(&raw.y);
    v.x = __half2float(__float2half_rn(v.x)) + __half2float(r0.x);
    v.y = __half2float(__float2half_rn(v.y)) + __half2float(r0.y);
    v.z = __half2float(__float2half_rn(v.z)) + __half2float(r1.x);
    v.w = __half2float(__float2half_rn(v.w)) + __half2float(r1.y);
  } else {
    // intrinsics: a plain + would be contracted with the scaling multiply into one fma
    v.x = __fadd_rn(v.x, __uint_as_float(raw.x)); v.y = __fadd_rn(v.y, __uint_as_float(raw.y));
    v.z = __fadd_rn(v.z, __uint_as_float(raw.z)); v.w = __fadd_rn(v.w, __uint_as_float(raw.w));
  }
  return v;
}

// The SPLIT partial sums of four columns of a row, from this CTA's memory or from its peers'.
template <int SPLIT>
__device__ __forceinline__ void load_slices(const EpilogueArgs& e, int m, int n4, float4 (&v)[SPLIT]) {
  if constexpr (SPLIT == 1) {
    v[0] = *reinterpret_cast<const float4*>(e.part + m * kRowTile + n4);
  } else if (e.slice_rows > 0) {
#pragma unroll
    for (int r = 0; r < SPLIT; ++r)
      v[r] = *reinterpret_cast<const float4*>(e.part + (r * e.slice_rows + m - e.m_begin) * kRowTile + n4);
  } else {
    const uint32_t off = e.part_addr + static_cast<uint32_t>(m * kRowTile + n4) * 4u;
#pragma unroll
    for (int r = 0; r < SPLIT; ++r) v[r] = ld_cluster_f4(map_to_cta(off, e.peer0 + r));
  }
}

// Sums the SPLIT partial tiles of this CTA's rows in rank order (fixed order:
// the result does not depend on timing) and stores them.  Every thread asks
// for all the partials of a batch of rows before it uses any of them, so the
// remote shared-memory latency is paid once per batch, not once per load.
template <int SPLIT, bool RES>
__device__ __forceinline__ void reduce_store(const EpilogueArgs& e) {
  // rows in flight per thread (half as many when residual values are held as well)
  constexpr int kRows = ((RES && SPLIT < 8) ? 8 / SPLIT : 16 / SPLIT) > (kStreamWarps > 8 ? 2 : 1)
                            ? ((RES && SPLIT < 8) ? 8 / SPLIT : 16 / SPLIT) / (kStreamWarps > 8 ? 2 : 1)
                            : 1;
  constexpr int kWarps = kStreamWarps;
  const int n4 = e.lane * 4;                 // 4 consecutive output columns
  for (int m0 = e.m_begin + e.warp; m0 < e.m_end; m0 += kWarps * kRows) {
    // the residual first: these loads keep their place before the others'
    uint4 rraw[RES ? kRows : 1];
    if constexpr (RES) {
#pragma unroll
      for (int i = 0; i < kRows; ++i) {
        const int m = m0 + i * kWarps;
        if (m < e.m_end && e.col_ok)
          rraw[i] = load_res4(e.res, (long long)m * e.ld_res + e.row0 + n4, e.out_dtype);
      }
    }
    float4 v[kRows][SPLIT];
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      const int m = m0 + i * kWarps;
      if (m < e.m_end) load_slices<SPLIT>(e, m, n4, v[i]);
    }
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      const int m = m0 + i * kWarps;
      if (m < e.m_end) {
        float4 acc = v[i][0];
#pragma unroll
        for (int r = 1; r < SPLIT; ++r) {
          acc.x += v[i][r].x; acc.y += v[i][r].y; acc.z += v[i][r].z; acc.w += v[i][r].w;
        }
        acc.x *= e.scale; acc.y *= e.scale; acc.z *= e.scale; acc.w *= e.scale;
        if constexpr (RES) {
          if (e.col_ok) acc = add_res4(acc, rraw[i], e.out_dtype);
        }
        if (e.col_ok) {
          if (e.push == nullptr) {
            store_out4(e.y, (long long)m * e.ldy + e.row0 + n4, e.out_dtype, acc);
          } else {
            for (int d = 0; d < e.push->n; ++d)
              store_out4(e.push->dst[d], (long long)m * e.push->ld + e.row0 + n4, e.out_dtype, acc);
          }
        }
      }
    }
  }
}

// The order of the greedy pick as one unsigned comparison: NaN on top, -0 and 0 alike.
__device__ __forceinline__ uint32_t argmax_key(float v) {
  const uint32_t b = __float_as_uint(__fadd_rn(v, 0.0f));
  return v != v ? 0xFFFFFFFFu : ((b >> 31) != 0u ? ~b : b | 0x80000000u);
}
__device__ __forceinline__ uint32_t argmax_bits(uint32_t key) {      // the fp32 bits of its value
  return key == 0xFFFFFFFFu ? 0x7FFFFFFFu : ((key >> 31) != 0u ? key & 0x7FFFFFFFu : ~key);
}

// Per batch row of this CTA's share: the best of the tile's 128 logits (see ArgmaxOut), and the logits themselves where
// they are wanted.  K is not split in an argmax launch, so the staged tile is final.  A lane's four, then the warp's 32 in two
// reductions (the largest key, the lowest index that has it); four rows at a time, since a row by itself is one chain.
template <typename T>
__device__ __forceinline__ void argmax_rows(const EpilogueArgs& e, uint2* partial_tile, bool store) {
  using namespace bq::qd;
  constexpr int kRows = 4;
  const int n4 = e.lane * 4;
  for (int m0 = e.m_begin + e.warp; m0 < e.m_end; m0 += kStreamWarps * kRows) {
    float4 v[kRows];
#pragma unroll
    for (int i = 0; i < kRows; ++i)
      if (m0 + i * kStreamWarps < e.m_end)
        v[i] = *reinterpret_cast<const float4*>(e.part + (m0 + i * kStreamWarps) * kRowTile + n4);
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      const int m = m0 + i * kStreamWarps;            // warp-uniform
      if (m < e.m_end) {
        v[i].x *= e.scale; v[i].y *= e.scale; v[i].z *= e.scale; v[i].w *= e.scale;
        if (store && e.col_ok) store_out4(e.y, (long long)m * e.ldy + e.row0 + n4, e.out_dtype, v[i]);
        uint32_t key = 0u;                            // below every value's
        int at = 0;
        if (e.col_ok) {                               // n is a multiple of 16: four columns are in or out
          key = argmax_key(widen(narrow<T>(v[i].x)));
          const uint32_t k1 = argmax_key(widen(narrow<T>(v[i].y))), k2 = argmax_key(widen(narrow<T>(v[i].z)));
          const uint32_t k3 = argmax_key(widen(narrow<T>(v[i].w)));
          if (k1 > key) { key = k1; at = 1; }
          if (k2 > key) { key = k2; at = 2; }
          if (k3 > key) { key = k3; at = 3; }
        }
        const uint32_t best = __reduce_max_sync(0xffffffffu, key);
        const int first = __reduce_min_sync(0xffffffffu, key == best && e.col_ok ? e.row0 + n4 + at : kNoIndex);
        if (e.lane == 0) partial_tile[m] = make_uint2(argmax_bits(best), static_cast<unsigned int>(first));
      }
    }
  }
}

// Second stage of the greedy pick: one CTA per batch row reduces the pairs of all tiles.
__global__ void __launch_bounds__(128) argmax_finish_kernel(const uint2* partial, int tiles, int M,
                                                            long long* idx_out) {
  pdl_wait_prior_grids();
  const int m = blockIdx.x;
  float bv = 0.0f;
  int bi = kNoIndex;
  for (int t = threadIdx.x; t < tiles; t += blockDim.x) {
    const uint2 pr = __ldcg(partial + static_cast<size_t>(t) * M + m);
    const float ov = __uint_as_float(pr.x);
    const int oi = static_cast<int>(pr.y);
    if (oi != kNoIndex && (bi == kNoIndex || argmax_beats(ov, oi, bv, bi))) { bv = ov; bi = oi; }
  }
  __shared__ float s_v[4];
  __shared__ int s_i[4];
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, bv, off);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, off);
    if (oi != kNoIndex && (bi == kNoIndex || argmax_beats(ov, oi, bv, bi))) { bv = ov; bi = oi; }
  }
  if ((threadIdx.x & 31) == 0) { s_v[threadIdx.x >> 5] = bv; s_i[threadIdx.x >> 5] = bi; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 4; ++w)
      if (s_i[w] != kNoIndex && (bi == kNoIndex || argmax_beats(s_v[w], s_i[w], bv, bi))) {
        bv = s_v[w];
        bi = s_i[w];
      }
    idx_out[m] = bi;
  }
}

// Interleaved gate/up tile: columns 0..63 of the tile are gate rows, 64..127 the up rows of the
// same 64 output columns.  Sums the K slices like reduce_store, rounds both halves to the
// activation type T exactly as the plain GEMM would have stored them, forms
// h = T(T(silu(gate)) * up) (the two roundings of the separate torch kernels,
// braid/model/mlp.py:48), and puts h (64 values of T per row) at `park`, row m at m * pitch: the start of
// the row's staging slot in THIS CTA's buffer -- rows of this CTA's share are read by no peer -- or
// the h of the whole batch.
// Lane L < 16 ends up with columns 4L, 4L+1; lane L+16 with 4L+2, 4L+3.  Returns max |h|.
template <int SPLIT, typename T>
__device__ __forceinline__ float silu_pair_rows(const EpilogueArgs& e, float scale_up, T* park, long long pitch) {
  using namespace bq::qd;
  constexpr int kRows = ((SPLIT < 8) ? 8 / SPLIT : 1) > (kStreamWarps > 8 ? 2 : 1)
                            ? ((SPLIT < 8) ? 8 / SPLIT : 1) / (kStreamWarps > 8 ? 2 : 1)
                            : 1;
  constexpr int kWarps = kStreamWarps;
  const int n4 = e.lane * 4;
  const bool up_half = e.lane >= 16;
  const float sc = up_half ? scale_up : e.scale;
  const int hcol = (e.lane & 15) * 4 + (up_half ? 2 : 0);
  float mx = 0.0f;
  for (int m0 = e.m_begin + e.warp; m0 < e.m_end; m0 += kWarps * kRows) {
    float4 v[kRows][SPLIT];
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      const int m = m0 + i * kWarps;
      if (m < e.m_end) load_slices<SPLIT>(e, m, n4, v[i]);
    }
    __syncwarp();   // every lane has its slice of the rows before any lane overwrites them
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      const int m = m0 + i * kWarps;    // warp-uniform
      if (m < e.m_end) {
        float4 acc = v[i][0];
#pragma unroll
        for (int r = 1; r < SPLIT; ++r) {
          acc.x += v[i][r].x; acc.y += v[i][r].y; acc.z += v[i][r].z; acc.w += v[i][r].w;
        }
        // the value the plain GEMM would have stored: one rounding to T
        const float r0 = widen(narrow<T>(acc.x * sc)), r1 = widen(narrow<T>(acc.y * sc));
        const float r2 = widen(narrow<T>(acc.z * sc)), r3 = widen(narrow<T>(acc.w * sc));
        const float got0 = __shfl_xor_sync(0xffffffffu, up_half ? r0 : r2, 16);
        const float got1 = __shfl_xor_sync(0xffffffffu, up_half ? r1 : r3, 16);
        const float g0 = up_half ? got0 : r0, g1 = up_half ? got1 : r1;
        const float u0 = up_half ? r2 : got0, u1 = up_half ? r3 : got1;
        const T s0 = silu_to<T>(g0);
        const T s1 = silu_to<T>(g1);
        const T h0 = narrow<T>(widen(s0) * u0);
        const T h1 = narrow<T>(widen(s1) * u1);
        mx = nan_max(mx, fabsf(widen(h0)));
        mx = nan_max(mx, fabsf(widen(h1)));
        struct alignas(2 * sizeof(T)) Two { T a, b; };
        *reinterpret_cast<Two*>(park + m * pitch + hcol) = Two{h0, h1};
      }
    }
  }
  return mx;
}

// After the grid-wide scale is known: cast the parked h of this CTA's rows and write the codes.
template <typename T>
__device__ __forceinline__ void silu_pair_emit(const EpilogueArgs& e, const float* part, float scale,
                                               uint8_t* hq, long long ld_hq, int col0) {
  using namespace bq::qd;
  const ScaleDiv sc(scale);
  const int hcol = (e.lane & 15) * 4 + (e.lane >= 16 ? 2 : 0);
  for (int m = e.m_begin + e.warp; m < e.m_end; m += kStreamWarps) {
    const T* hrow = reinterpret_cast<const T*>(part + m * kRowTile);
    float f[2] = {widen(hrow[hcol]), widen(hrow[hcol + 1])};
    divide_group<T, 2, true>(sc, f);   // the scale is that of these very values
    const uint32_t pair = __nv_cvt_float2_to_fp8x2(make_float2(f[0], f[1]), __NV_SATFINITE, __NV_E4M3);
    *reinterpret_cast<uint16_t*>(hq + static_cast<long long>(m) * ld_hq + col0 + hcol) =
        static_cast<uint16_t>(pair & 0xFFFFu);
  }
}

// ---------------------------------------------------------------------------
// Weight-streaming kernel (swap-AB, cluster split-K)
// ---------------------------------------------------------------------------
// Shared memory, after aligning the dynamic base to 1024 bytes:
//   [stages x 16 KiB weight tiles][b_stages x (mma_n*128) activation tiles] ... [barrier block][slices]
// Two rings with their own barriers and their own producer thread.  The weight ring is as deep
// as the shared memory allows: its tiles come from HBM, and the bytes in flight per SM are what
// sets the streaming rate.  The activation ring is shallow (2 to 4 tiles at wide batches): its
// tiles are L2 hits shared by every row tile, and a wide batch tile is as large as a weight
// tile, so every activation slot given up is a weight tile more in flight.
// The tile area is reused after the main loop as the fp32 staging buffer
// part[m][128] that the cluster reduction reads.  Up to 48 rows of a sliced weight (handover_bytes) the reduction
// reads the slices instead, [split][rows that this CTA sums][128] fp32 behind the barriers: every CTA of the cluster
// writes its own there from its accumulator, and nothing is staged.
//
// QUANT (fewer rows still): the activation arrives unquantized, and every CTA quantizes it for itself: the
// warps that have nothing to do until the accumulator is complete read the whole activation (a few
// dozen KB, from L2) for its max |x|, then cast this CTA's K slice into the activation tiles.  The same
// values in the same arithmetic everywhere, so every CTA finds the same scale and nothing is
// exchanged (SliceMax is the other form); the quantizer's launch and its hand-over through memory are gone.  Two launches ->
// one, us in a graph and eager: 1 row of 4096 x 4096 6.3 -> 6.5 and 8.5 -> 6.7, 4 rows of 1024 x 4096 5.3 -> 5.0 and 8.4 ->
// 5.5, 8 rows of 2048 x 2048 4.9 -> 5.0 and 8.7 -> 5.4.  Where it stops paying: quantize_inside_pays.
constexpr int kQuantWarps = kStreamWarps - 2;           // all but the weight loads' and the MMAs'
constexpr int kQuantThreads = kQuantWarps * 32;
constexpr int kQuantAhead = 8;                          // groups of 8 a thread asks for at once
// Chunks of 16 that a thread asks for at once where it casts: behind a weight stream a round trip to L2 takes 2 to 3 us.
template <typename T, bool GIVEN> constexpr int kChunksAhead = !GIVEN ? 1 : (sizeof(T) == 2 ? 4 : 2);

// Where a weight is sliced, the slices of a tile are whole x between them: every CTA finds the maximum of its own slice, which it
// keeps in registers for the cast if it is not too long, and the CTAs of the tile exchange four bytes each (see ClusterAmax):
// a quarter of the reads and one pass fewer for one trip inside the cluster.  8 rows of 4096 x 4096 eager 7.9 -> 7.1 us, in
// a graph 8.1 -> 7.2; 16 rows 10.4 -> 8.2.  Where it is taken: own_slices_pay.
struct SliceMax {
  uint32_t bar, slots;     // shared-memory addresses: the barrier that counts the words, one word per slice
  int split, krank, peer0; // slices of the tile, this one, the cluster rank of the first
};
template <typename T> constexpr int kHeldChunks = 8 / (int)sizeof(T);      // 32 registers

// 16 codes where TMA would have put them: 16-byte chunk c of row m at c ^ (m & 7).
template <typename T>
__device__ __forceinline__ void emit_chunk(const uint4 (&raw)[sizeof(T)], const bq::qd::ScaleDiv& dv, uint8_t* dst) {
  using namespace bq::qd;
  constexpr int kWords = sizeof(T);
  Pack8<T> lo, hi;
#pragma unroll
  for (int q = 0; q < kWords; ++q) reinterpret_cast<uint4*>(q < kWords / 2 ? &lo : &hi)[q % (kWords / 2)] = raw[q];
  const uint2 a = codes8<T, true>(lo, dv), b = codes8<T, true>(hi, dv);
  *reinterpret_cast<uint4*>(dst) = make_uint4(a.x, a.y, b.x, b.y);
}

template <typename T>
__device__ __forceinline__ float quantize_own_slice(const QuantIn& in, int M, int K, int kx0, int kb_count, uint8_t* b_tiles,
                                                    int b_tile_bytes, float* s_red, const SliceMax& sm, unsigned int* status) {
  using namespace bq::qd;
  constexpr int kWords = sizeof(T), kHeld = kHeldChunks<T>;
  const int t = threadIdx.x - (kStreamThreads - kQuantThreads), lane = threadIdx.x & 31, warp = t >> 5;
  const T* const x = static_cast<const T*>(in.x);
  const int chunks = kb_count * (kBK / 16), total = M * chunks;     // of a row in this slice, of the slice
  auto load = [&](int i, uint4 (&raw)[kWords]) {                     // K is a multiple of 16; beyond K: zeros
    const int row = i / chunks, k = kx0 + (i - row * chunks) * 16;
    const uint4* const src = reinterpret_cast<const uint4*>(x + static_cast<size_t>(row) * K + k);
#pragma unroll
    for (int q = 0; q < kWords; ++q) raw[q] = k < K ? __ldcg(src + q) : make_uint4(0u, 0u, 0u, 0u);
  };
  auto largest = [&](const uint4 (&raw)[kWords], float m) {
#pragma unroll
    for (int q = 0; q < kWords; q += kWords / 2) m = absmax8(*reinterpret_cast<const Pack8<T>*>(&raw[q]), m);
    return m;
  };
  auto at = [&](int i) {
    const int row = i / chunks, c = i - row * chunks;
    return b_tiles + (c >> 3) * b_tile_bytes + row * kBK + (((c & 7) ^ (row & 7)) << 4);
  };
  uint4 held[kHeld][kWords];
  float m = 0.0f;
#pragma unroll
  for (int u = 0; u < kHeld; ++u)
    if (t + u * kQuantThreads < total) load(t + u * kQuantThreads, held[u]);
#pragma unroll
  for (int u = 0; u < kHeld; ++u)
    if (t + u * kQuantThreads < total) m = largest(held[u], m);
  for (int i = t + kHeld * kQuantThreads; i < total; i += kQuantThreads) {
    uint4 raw[kWords];
    load(i, raw);
    m = largest(raw, m);
  }
  uint32_t bits = __reduce_max_sync(0xffffffffu, __float_as_uint(m));      // bit patterns order like the values, NaN on top
  if (lane == 0) s_red[warp] = __uint_as_float(bits);
  asm volatile("bar.sync 2, %0;" ::"n"(kQuantThreads) : "memory");
  if (warp == 0) {
    bits = __reduce_max_sync(0xffffffffu, lane < kQuantWarps ? __float_as_uint(s_red[lane]) : 0u);
    if (lane < sm.split)
      st_async_cluster(map_to_cta(sm.slots + 4u * sm.krank, sm.peer0 + lane), bits, map_to_cta(sm.bar, sm.peer0 + lane));
  }
  if (!mbar_wait_cluster(sm.bar, 0) && t == 0) atomicExch(status, (unsigned int)kErrDeviceWait);
  bits = 0u;
  if (lane < sm.split) asm volatile("ld.shared.u32 %0, [%1];" : "=r"(bits) : "r"(sm.slots + 4u * lane) : "memory");
  const float scale = scale_from_amax(__uint_as_float(__reduce_max_sync(0xffffffffu, bits)));
  const ScaleDiv dv(scale);
#pragma unroll
  for (int u = 0; u < kHeld; ++u)
    if (t + u * kQuantThreads < total) emit_chunk<T>(held[u], dv, at(t + u * kQuantThreads));
  for (int i = t + kHeld * kQuantThreads; i < total; i += kQuantThreads) {
    uint4 raw[kWords];
    load(i, raw);
    emit_chunk<T>(raw, dv, at(i));
  }
  fence_proxy_async_smem();                             // the MMAs read through the async proxy
  asm volatile("bar.sync 2, %0;" ::"n"(kQuantThreads) : "memory");
  return scale;
}

// Returns the scale.  Called by warps 2.. with all lanes.  GIVEN: max |x| is in `in.words`.
template <typename T, bool GIVEN>
__device__ __forceinline__ float quantize_slice(const QuantIn& in, int M, int K, int kx0, int kb_count, uint8_t* b_tiles,
                                                int b_tile_bytes, float* s_red) {
  using namespace bq::qd;
  const int t = threadIdx.x - (kStreamThreads - kQuantThreads), lane = threadIdx.x & 31, warp = t >> 5;
  const T* const x = static_cast<const T*>(in.x);
  float m = 0.0f;
  if constexpr (GIVEN) m = __uint_as_float(__ldcg(in.words));
  for (int g0 = t; !GIVEN && g0 < in.n8; g0 += kQuantThreads * kQuantAhead / (sizeof(T) / 2)) {
    Pack8<T> v[kQuantAhead / (sizeof(T) / 2)];
#pragma unroll
    for (int u = 0; u < kQuantAhead / (int)(sizeof(T) / 2); ++u)
      if (g0 + u * kQuantThreads < in.n8) v[u] = load8<T>(x + static_cast<size_t>(g0 + u * kQuantThreads) * kGroup);
#pragma unroll
    for (int u = 0; u < kQuantAhead / (int)(sizeof(T) / 2); ++u)
      if (g0 + u * kQuantThreads < in.n8) m = absmax8(v[u], m);
  }
  if constexpr (!GIVEN) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) m = nan_max(m, __shfl_xor_sync(0xffffffffu, m, off));
    if (lane == 0) s_red[warp] = m;
    asm volatile("bar.sync 2, %0;" ::"n"(kQuantThreads) : "memory");
    m = s_red[0];
#pragma unroll
    for (int i = 1; i < kQuantWarps; ++i) m = nan_max(m, s_red[i]);
  }
  const float scale = scale_from_amax(m);
  const ScaleDiv dv(scale);
  // 16 codes at a time, where TMA would have put them: 16-byte chunk c of row m at c ^ (m & 7).  K is a
  // multiple of 16.
  constexpr int kAhead = kChunksAhead<T, GIVEN>;
  const int chunks = kb_count * (kBK / 16), total = M * chunks;     // of a row in this slice, of the slice
  for (int i0 = t; i0 < total; i0 += kQuantThreads * kAhead) {
    constexpr int kWords = sizeof(T);                   // 16-byte words of a chunk
    uint4 raw[kAhead][kWords];
    int at[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      at[u] = -1;
      if (u > 0 && i0 - t + u * kQuantThreads >= total) continue;       // the same for all threads
      const int i = i0 + u * kQuantThreads, row = i / chunks, c = i - row * chunks, k = kx0 + c * 16;
      at[u] = i < total ? (c >> 3) * b_tile_bytes + row * kBK + (((c & 7) ^ (row & 7)) << 4) : -1;
      const bool in = i < total && k < K;               // what a last K block has beyond K casts to zeros
      const uint4* const src = reinterpret_cast<const uint4*>(x + (in ? static_cast<size_t>(row) * K + k : 0));
#pragma unroll
      for (int q = 0; q < kWords; ++q) {
        raw[u][q] = __ldcg(src + q);                    // coherent (see load8)
        if (!in) raw[u][q] = make_uint4(0u, 0u, 0u, 0u);
      }
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      if (at[u] < 0) continue;
      Pack8<T> lo, hi;
#pragma unroll
      for (int q = 0; q < kWords; ++q) reinterpret_cast<uint4*>(q < kWords / 2 ? &lo : &hi)[q % (kWords / 2)] = raw[u][q];
      const uint2 a = codes8<T, true>(lo, dv), b = codes8<T, true>(hi, dv);
      *reinterpret_cast<uint4*>(b_tiles + at[u]) = make_uint4(a.x, a.y, b.x, b.y);
    }
  }
  fence_proxy_async_smem();                             // the MMAs read through the async proxy
  asm volatile("bar.sync 2, %0;" ::"n"(kQuantThreads) : "memory");
  if (GIVEN && t == 0 && atomicAdd(&in.words[1], 1u) == in.expected - 1u) {
    in.words[0] = 0u;
    in.words[1] = 0u;
  }
  return scale;
}

#ifndef BQ_STREAM_MIN_CTAS
#define BQ_STREAM_MIN_CTAS 2
#endif
template <int EPI, int DT, int QUANT>      // QUANT: 1 the activation's maximum is looked for, 2 it is given, 3 each slice looks for its own
__global__ void __launch_bounds__(kStreamThreads, BQ_STREAM_MIN_CTAS)
gemm_stream_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_xd,
                   const __grid_constant__ WeightMaps tm_w, const __grid_constant__ GemmParams p,
                   const int smem_tile_bytes) {
  extern __shared__ uint8_t smem_dyn[];
  const bool pair_on = EPI == kAny ? p.pair.on != 0 : (EPI == kGateUp || EPI == kGateUpDense);
  const PushParams* const push = EPI == kAny && p.push.n > 0 ? &p.push : nullptr;
  const int out_dtype = DT == kAnyType ? p.out_dtype : DT;
  const uint32_t base = (smem_u32(smem_dyn) + 1023u) & ~1023u;
  uint8_t* const base_ptr = smem_dyn + (base - smem_u32(smem_dyn));
  const int b_tile_bytes = p.mma_n * kBK;
  const uint32_t a_base = base;
  const uint32_t b_base = base + p.stages * kATileBytes;
  const uint32_t bar_base = base + smem_tile_bytes;          // 8-byte aligned
  // barrier block: weight ring full / empty, activation ring full, accumulator.  One
  // tcgen05.commit per K block: it arrives on the weight slot's "empty" barrier, and the
  // activation producer watches the same barrier for the block whose activation slot it wants
  // to refill.
  const int n_bars = 2 * p.stages + p.b_stages;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (p.stages + s); };
  auto full_bar_b = [&](int s) { return bar_base + 8u * (2 * p.stages + s); };
  const uint32_t accum_bar = bar_base + 8u * n_bars;
  volatile uint32_t* const tmem_slot =
      reinterpret_cast<volatile uint32_t*>(base_ptr + smem_tile_bytes + 8 * (n_bars + 1));
  volatile uint32_t* const abort_flag = tmem_slot + 1;
  float* const s_quant = reinterpret_cast<float*>(const_cast<uint32_t*>(tmem_slot) + 2);   // one float per warp
  const uint32_t slice_bar = bar_base + 896u;       // QUANT: SliceMax, behind whatever the others need
  volatile float* const s_scale = reinterpret_cast<volatile float*>(base_ptr + smem_tile_bytes + kBarrierBytes - 8);

  if (threadIdx.x == 0) { BQ_STAMP(p, 0); BQ_STAMP_META(p, 0); }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // A cluster of p.cluster CTAs works on p.cluster / split row tiles of one weight
  // at a time: CTAs [g*split, (g+1)*split) of the cluster hold the K slices of
  // tile g and reduce among themselves.
  const int crank = (p.cluster > 1) ? static_cast<int>(cluster_ctarank()) : 0;
  const int cluster_id = blockIdx.x / p.cluster;
  int sg = 0;
#pragma unroll
  for (int i = 1; i < BQ_MAX_SEGMENTS; ++i)
    if (i < p.n_seg && cluster_id >= p.seg[i].cluster_begin) sg = i;
  const Segment seg = p.seg[sg];
  const int split = seg.split;
  const int group = crank / split;              // which tile of the cluster
  const int krank = crank - group * split;      // which K slice of that tile
  const int tile_in_seg = (cluster_id - seg.cluster_begin) * (p.cluster / split) + group;
  const int row0 = tile_in_seg * kRowTile;
  const bool active = row0 < seg.n;             // padding CTAs only keep the cluster barriers

  // this CTA's K slice, balanced to within one block
  // a 16-bit segment (a weight the reference keeps unquantized) walks 128-byte K blocks of
  // 64 elements over the dense activation; everything else about the pipeline is the same
  const bool dense = seg.dense != 0;
  const int seg_k_blocks = dense ? p.k_blocks_dense : p.k_blocks;
  const CUtensorMap* const x_map = dense ? &tm_xd : &tm_x;
  const int kb_base = seg_k_blocks / split, kb_rem = seg_k_blocks % split;
  const int kb_count = active ? kb_base + (krank < kb_rem ? 1 : 0) : 0;
  const int kb_begin = krank * kb_base + (krank < kb_rem ? krank : kb_rem);

  uint32_t tmem_cols = 32;
  while (tmem_cols < static_cast<uint32_t>(p.mma_n)) tmem_cols <<= 1;

  if (threadIdx.x == 0) {
    if (!QUANT) tma_prefetch_desc(x_map);
    tma_prefetch_desc(&tm_w.w[sg]);
    if (pair_on) tma_prefetch_desc(&tm_w.w[1]);
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int s = 0; s < p.b_stages; ++s) mbar_init(full_bar_b(s), 1);
    mbar_init(accum_bar, 1);
    if (QUANT == 3) mbar_init(slice_bar, 1);
    *abort_flag = 0;
    fence_mbar_init();
    if (QUANT == 3) mbar_expect_tx(slice_bar, 4u * split);
  }
  if (warp == 1 && active) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), tmem_cols);
    tmem_relinquish();
  }
  // The next kernel may start its own set-up -- only now: a CTA of it that shares this SM takes tensor memory too and
  // keeps it until this kernel is done.
  if (warp == 1) pdl_launch_dependents();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (threadIdx.x == 0) BQ_STAMP(p, 1);

  // slices (and maxima) are written into a peer's memory: once it has started, which this says
  if (QUANT == 3 || p.handover) cluster_arrive_relaxed();
  if (!active) {
    // nothing to multiply: it only matches the cluster barriers of the working CTAs
    if (QUANT == 3 && !p.handover) cluster_wait();
    if (p.handover) { cluster_wait(); cluster_sync_all(); }
    else if (p.cluster > 1) { cluster_sync_all(); cluster_sync_all(); }
    return;
  }

  if (warp == 0) {
    // Weights do not depend on any earlier kernel: this warp never waits for the kernel that produces the
    // activation, it only follows the MMAs through the weight ring.  See ptx.cuh for why the whole warp
    // walks the loop.  Weights are read once: evict first.
    const uint32_t issue = elect_one() ? 1u : 0u;
    const uint64_t pol_w = policy_evict_first();
    // one 128-row box, or (paired gate/up) two 64-row boxes from the two weights
    const bool paired = pair_on;
    const int half_row0 = tile_in_seg * (kRowTile / 2);
    // slot and phase are carried along: an integer division by a run-time depth costs a
    // single issuing thread more than the loads it issues
    int s = 0;
    uint32_t phase = 1;                      // parity of the completion that frees slot s
    for (int i = 0; i < kb_count; ++i) {
      if (i >= p.stages && !mbar_wait(empty_bar(s), phase)) {
        *abort_flag = 1;
        break;
      }
      mbar_expect_tx(issue, full_bar(s), kATileBytes);
      const int kx = (kb_begin + i) * kBK;
      const uint32_t dst = a_base + s * kATileBytes;
      if (paired) {
        tma_load_2d(issue, dst, &tm_w.w[0], full_bar(s), kx, half_row0, pol_w);
        tma_load_2d(issue, dst + kATileBytes / 2, &tm_w.w[1], full_bar(s), kx, half_row0, pol_w);
      } else {
        tma_load_2d(issue, dst, &tm_w.w[sg], full_bar(s), kx, row0, pol_w);
      }
      if (++s == p.stages) { s = 0; phase ^= 1u; }
    }
    if (EPI == kGateUpDense) prefetch_next(p.pair);      // no exchange to wait for
    __syncwarp();
  } else if (QUANT && warp >= 2) {
    if constexpr (QUANT) {
      pdl_wait_prior_grids();   // the kernel that produces the activation has completed
      const int kx0 = kb_begin * kBK;
      uint8_t* const tiles = base_ptr + (b_base - base);
      using T = typename std::conditional<DT == BQ_DTYPE_F32, float,
                                          typename std::conditional<DT == BQ_DTYPE_F16, __half, __nv_bfloat16>::type>::type;
      float sc;
      if constexpr (QUANT == 3) {
        cluster_wait();
        sc = quantize_own_slice<T>(p.quant, p.M, p.quant_k, kx0, kb_count, tiles, b_tile_bytes, s_quant,
                                   SliceMax{slice_bar, slice_bar + 8u, split, krank, group * split}, p.status);
      } else {
        sc = quantize_slice<T, QUANT == 2>(p.quant, p.M, p.quant_k, kx0, kb_count, tiles, b_tile_bytes, s_quant);
      }
      if (threadIdx.x == kStreamThreads - kQuantThreads) {
        *s_scale = sc;
        mbar_arrive(full_bar_b(0));
      }
    }
    __syncwarp();
  } else if (warp == 2) {
    // the activation tile is shared by every row tile: keep it in L2
    const uint32_t issue = elect_one() ? 1u : 0u;
    const uint64_t pol_x = policy_evict_last();
    pdl_wait_prior_grids();   // the kernel that produces the activation has completed
    if (issue) BQ_STAMP(p, 2);
    // Activation slot s was last read by the MMAs of block j = i - b_stages, whose completion
    // is completion number j / stages of weight slot j % stages.  That barrier cannot complete
    // a second time before this thread has looked: block j + stages >= i needs THIS load first
    // (the host keeps b_stages <= stages).
    int s = 0, js = 0;                       // activation slot of block i, weight slot of block j
    uint32_t jphase = 0;                     // parity of completion j / stages
    for (int i = 0; i < kb_count; ++i) {
      if (i >= p.b_stages) {
        if (!mbar_wait(empty_bar(js), jphase)) {
          *abort_flag = 1;
          break;
        }
        if (++js == p.stages) { js = 0; jphase ^= 1u; }
      }
      mbar_expect_tx(issue, full_bar_b(s), b_tile_bytes);
      tma_load_2d(issue, b_base + s * b_tile_bytes, x_map, full_bar_b(s), (kb_begin + i) * kBK, 0, pol_x);
      if (++s == p.b_stages) s = 0;
    }
    __syncwarp();
  } else if (warp == 1) {
    const uint32_t issue = elect_one() ? 1u : 0u;
    const uint32_t idesc = dense ? idesc_f16(kRowTile, p.mma_n, p.dense_fmt)
                                 : idesc_e4m3(kRowTile, p.mma_n);
    auto multiply = [&](auto is_dense) {
      // A commit per block tells the loading warps that its slots are free; where none is filled twice nobody asks (four
      // graphed layers of hidden 4096, 1 row 199.9 -> 197.7 us, 48 rows 250.9 -> 249.9).  (Copies of the activation that bring 2
      // or 4 blocks save its warp 100 clocks a block, 0.3 % of those layers, and counting boxes in this loop costs 2 %.)
      // Where this kernel casts the activation itself the test costs more than it saves: linear of 8 rows 7.93 and 8.13.
      const bool reuse = kb_count > p.stages || kb_count > p.b_stages;
      int s = 0, sb = 0;
      uint32_t phase = 0, phase_b = 0;
      bool ready = false, ready_b = false;
      for (int i = 0; i < kb_count; ++i) {
        if ((!ready && !mbar_wait(full_bar(s), phase)) ||
            ((!QUANT || i == 0) && !ready_b && !mbar_wait(full_bar_b(sb), phase_b))) {
          *abort_flag = 1;
          break;
        }
        const uint32_t a_tile = a_base + s * kATileBytes, b_tile = b_base + sb * b_tile_bytes, empty = empty_bar(s);
        if (++s == p.stages) { s = 0; phase ^= 1u; }
        if (++sb == p.b_stages) { sb = 0; phase_b ^= 1u; }
        // look at the next block's barriers now: the answers arrive while this block's MMAs are issued
        ready = mbar_test(full_bar(s), phase);
        if (!QUANT) ready_b = mbar_test(full_bar_b(sb), phase_b);
        tc_fence_after();
        if (issue && i == 0) BQ_STAMP(p, 3);
        const uint64_t da = smem_desc_sw128(a_tile), db = smem_desc_sw128(b_tile);
#pragma unroll
        for (int j = 0; j < kBK / kUmmaK; ++j) {
          // +32 bytes along K inside the swizzle span = +2 in descriptor units (32 e4m3 or 16
          // 16-bit elements: one MMA's K either way)
          if constexpr (is_dense.value) mma_f16(issue, tmem_base, da + 2u * j, db + 2u * j, idesc, (i | j) != 0 ? 1u : 0u);
          else mma_f8(issue, tmem_base, da + 2u * j, db + 2u * j, idesc, (i | j) != 0 ? 1u : 0u);
        }
        if (QUANT || reuse) mma_commit(issue, empty);   // both slots are free once these MMAs retire
      }
    };
    if (dense) multiply(std::true_type{});
    else multiply(std::false_type{});
    mma_commit(issue, accum_bar);     // accumulator complete
    __syncwarp();
  }

  // ---- epilogue: TMEM -> fp32 staging in shared memory ----------------------
  pdl_wait_prior_grids();   // scales are read and outputs written only after this
  // the epilogue warps get here at once and have the scale ready long before
  // the accumulator is
  const float sw = dense ? 1.0f : __ldg(seg.sw);
  float sx_ready = 1.0f;
  if (!QUANT && !dense) sx_ready = ld_coherent4(p.sx);
  bool ok = mbar_wait(accum_bar, 0);
  tc_fence_after();
  if (threadIdx.x == 0) BQ_STAMP(p, 4);
  if (!ok) *abort_flag = 1;
  __syncthreads();
  if (QUANT) sx_ready = *s_scale;
  ok = (*abort_flag == 0);
  const float scale = sx_ready * sw;
  float* const part = reinterpret_cast<float*>(base_ptr);   // [mma_n][128]
  float* const slices = reinterpret_cast<float*>(base_ptr + smem_tile_bytes + kBarrierBytes);   // [split][per][128]
  const int per = (p.M + split - 1) / split;               // rows that a CTA sums
  const bool handover = p.handover && split > 1;
  if (QUANT == 3 ? warp < 2 : p.handover) cluster_wait();      // QUANT == 3: the others have waited
  if (ok && handover) {
    const int quad = warp & 3;
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
    const uint32_t mine = smem_u32(slices) + static_cast<uint32_t>(krank * per * kRowTile + quad * 32 + lane) * 4u;
    for (int c = (warp >> 2) * 16; c < p.M; c += 4 * kStreamWarps) {
      uint32_t r[16];
      tmem_ld16(lane_addr + c, r);
      tmem_ld_wait();
      int owner = c / per, row = c - owner * per;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        if (c + j < p.M)
          st_cluster_f1(map_to_cta(mine + row * (kRowTile * 4), group * split + owner), __uint_as_float(r[j]));
        if (++row == per) { row = 0; ++owner; }
      }
    }
  } else if (ok) {
    // 8 warps: warp w reads TMEM lanes 32*(w%4).. (the only ones it may touch)
    // and every other 16-column chunk, starting at chunk w/4
    const int quad = warp & 3;
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
    const int n_local = quad * 32 + lane;
    for (int c = (warp >> 2) * 16; c < p.mma_n; c += 4 * kStreamWarps) {
      uint32_t r[16];
      tmem_ld16(lane_addr + c, r);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 16; ++j) part[(c + j) * kRowTile + n_local] = __uint_as_float(r[j]);
    }
  } else if (threadIdx.x == 0) {
    atomicExch(p.status, (unsigned int)kErrDeviceWait);
  }
  tc_fence_before();
  if (p.cluster > 1) cluster_sync_all(); else __syncthreads();
  if (threadIdx.x == 0) BQ_STAMP(p, 5);

  // ---- reduce the K slices in rank order and write this CTA's share of rows --
  float pair_max = 0.0f;
  const int m_begin = krank * per;
  const int m_end = (m_begin + per < p.M) ? (m_begin + per) : p.M;
  if (ok) {
    const bool col_ok = (row0 + lane * 4) < seg.n;      // n is a multiple of 4
    const uint32_t part_addr = smem_u32(part);
    const int peer0 = group * split;
    const EpilogueArgs ea{handover ? slices : part, part_addr, peer0, handover ? per : 0, m_begin, m_end, warp, lane, row0,
                          scale, col_ok, seg.y, seg.ldy, out_dtype, seg.res, seg.ld_res, push};
    if (pair_on) {
      const float scale_up = sx_ready * __ldg(p.pair.sw_up);
      float mx;
#define BQ_PAIR_ROWS(TT)                                                                           \
      constexpr bool dense_h = EPI == kGateUpDense;                                                 \
      TT* const park = dense_h ? static_cast<TT*>(p.pair.h) + tile_in_seg * (kRowTile / 2)          \
                               : reinterpret_cast<TT*>(part);                                       \
      const long long pitch = dense_h ? seg.n / 2 : kRowTile * 4 / (int)sizeof(TT);                 \
      switch (split) {                                                                              \
        case 1: mx = silu_pair_rows<1, TT>(ea, scale_up, park, pitch); break;                       \
        case 2: mx = silu_pair_rows<2, TT>(ea, scale_up, park, pitch); break;                       \
        case 4: mx = silu_pair_rows<4, TT>(ea, scale_up, park, pitch); break;                       \
        default: mx = silu_pair_rows<8, TT>(ea, scale_up, park, pitch); break;                      \
      }
      if (out_dtype == BQ_DTYPE_BF16) { BQ_PAIR_ROWS(__nv_bfloat16) }
      else if (out_dtype == BQ_DTYPE_F16) { BQ_PAIR_ROWS(__half) }
      else { BQ_PAIR_ROWS(float) }
#undef BQ_PAIR_ROWS
      pair_max = mx;
      if (EPI == kGateUpDense) {
        // nobody waits for anybody: the bits of |h| order like the values, NaN on top, and whoever reads the word
        // does so behind the end of this launch
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) mx = bq::qd::nan_max(mx, __shfl_xor_sync(0xffffffffu, mx, off));
        if (lane == 0) s_quant[warp] = mx;
        __syncthreads();
        if (threadIdx.x == 0) {
#pragma unroll
          for (int i = 1; i < kStreamWarps; ++i) mx = bq::qd::nan_max(mx, s_quant[i]);
          atomicMax(&p.pair.words[0], __float_as_uint(mx));
        }
      }
    } else if (EPI == kArgmax) {
      uint2* const mine = p.argmax.partial + static_cast<size_t>(tile_in_seg) * p.M;
      const bool store = p.argmax.store_logits != 0;
      if (out_dtype == BQ_DTYPE_BF16) argmax_rows<__nv_bfloat16>(ea, mine, store);
      else if (out_dtype == BQ_DTYPE_F16) argmax_rows<__half>(ea, mine, store);
      else argmax_rows<float>(ea, mine, store);
    } else if (EPI == kPlain || (EPI == kAny && seg.res == nullptr)) {
      switch (split) {
        case 1: reduce_store<1, false>(ea); break;
        case 2: reduce_store<2, false>(ea); break;
        case 4: reduce_store<4, false>(ea); break;
        default: reduce_store<8, false>(ea); break;
      }
    } else {
      switch (split) {
        case 1: reduce_store<1, true>(ea); break;
        case 2: reduce_store<2, true>(ea); break;
        case 4: reduce_store<4, true>(ea); break;
        default: reduce_store<8, true>(ea); break;
      }
    }
  }
  if (threadIdx.x == 0) BQ_STAMP(p, 6);
  // nobody leaves while a peer may still read its staging buffer
  if (p.cluster > 1 && !p.handover) cluster_sync_all(); else __syncthreads();
  if (pair_on && push != nullptr) {
    // ---- column-parallel form: h itself goes to every rank's gathered buffer; the amax needs
    // all ranks' shards and is taken by the quantizer that follows the exchange ----
    __syncthreads();   // parked rows are complete
    if (ok) {
      const int col0 = tile_in_seg * (kRowTile / 2);
      const int hcol = (lane & 15) * 4 + (lane >= 16 ? 2 : 0);
      for (int m = m_begin + warp; m < m_end; m += kStreamWarps) {
        const long long at = static_cast<long long>(m) * p.push.ld + col0 + hcol;
        if (out_dtype == BQ_DTYPE_F32) {
          const float2 v = *reinterpret_cast<const float2*>(part + m * kRowTile + hcol);
          for (int d = 0; d < p.push.n; ++d)
            *reinterpret_cast<float2*>(static_cast<float*>(p.push.dst[d]) + at) = v;
        } else {
          const uint32_t v = *reinterpret_cast<const uint32_t*>(
              reinterpret_cast<const uint16_t*>(part + m * kRowTile) + hcol);
          for (int d = 0; d < p.push.n; ++d)
            *reinterpret_cast<uint32_t*>(static_cast<uint16_t*>(p.push.dst[d]) + at) = v;
        }
      }
    }
  } else if (pair_on && EPI != kGateUpDense) {
    // ---- grid-wide max |h| -> scale -> codes of this CTA's rows (h is parked in `part`) ----
    using namespace bq::qd;
    pair_max = bq::qd::warp_amax(pair_max);
    if (lane == 0) s_quant[warp] = pair_max;
    __syncthreads();
    if (warp == 0) {
      float w = warp_amax(lane < kStreamWarps ? s_quant[lane] : 0.0f);
      __syncwarp();
      if (lane == 0) {
        // an aborted CTA still arrives (with 0), so the others are not left waiting
        if (p.pair.expected > 1) w = exchange_max(w, p.pair.words, p.pair.expected, p.status);
        const float sc = scale_from_amax(w);
        if (blockIdx.x == 0) p.pair.sh[0] = sc;
        s_quant[0] = sc;
      }
    }
    __syncthreads();
    if (EPI == kGateUp && warp == p.pair.next_warp) prefetch_next(p.pair);
    const float sc = s_quant[0];
    if (ok) {
      const EpilogueArgs ea{part, smem_u32(part), 0, 0, m_begin, m_end, warp, lane, row0, 0.0f, true,
                            nullptr, 0, out_dtype, nullptr, 0, push};
      const int col0 = tile_in_seg * (kRowTile / 2);
      if (out_dtype == BQ_DTYPE_BF16)
        silu_pair_emit<__nv_bfloat16>(ea, part, sc, p.pair.hq, p.pair.ld_hq, col0);
      else if (out_dtype == BQ_DTYPE_F16)
        silu_pair_emit<__half>(ea, part, sc, p.pair.hq, p.pair.ld_hq, col0);
      else
        silu_pair_emit<float>(ea, part, sc, p.pair.hq, p.pair.ld_hq, col0);
    }
    if (threadIdx.x == 0 && p.pair.expected > 1) exchange_end(p.pair.words, p.pair.expected, exchange_leave(p.pair.words));
  }
  if (push != nullptr) {
    // The stores of all threads of this CTA are ordered before thread 0's fence by the barrier
    // (fences are cumulative); the fence orders them before this CTA's count; the last CTA sees
    // every count, fences again and only then signals the ranks: every store of the launch
    // happens before every arrival.
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence_system();
      const unsigned int old = atomicAdd(p.push.done, 1u);
      if (old == p.push.expected - 1u) {
        *p.push.done = 0u;                       // ready for the next launch on this scratch
        __threadfence_system();
        for (int d = 0; d < p.push.n; ++d)
          asm volatile("red.release.sys.global.add.u32 [%0], 1;" ::"l"(p.push.flag[d]) : "memory");
      }
    }
  }
  if (warp == 1) tmem_dealloc(tmem_base, tmem_cols);
  if (threadIdx.x == 0) BQ_STAMP(p, 7);
}

// Waits (bounded) until `flag` has counted `count` more arrivals than at the end of the
// previous wait, i.e. until every CTA of every rank's push launch has stored its share into
// this rank's gathered buffer.  One thread; the arrival total is kept in `seen`.
__global__ void wait_flag_kernel(const unsigned int* flag, unsigned int* seen, unsigned int count,
                                 unsigned int* status) {
  const unsigned int target = *seen + count;
  const long long t0 = clock64();
  for (;;) {
    unsigned int v;
    asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
    if (static_cast<int>(v - target) >= 0) break;
    if (clock64() - t0 > kSpinLimitCycles) {
      atomicExch(status, (unsigned int)kErrDeviceWait);
      break;
    }
  }
  *seen = target;
  __threadfence();
}

// The same wait, then the quantization scale of the gathered h from the ranks' max |h| words
// (each written by its rank ahead of that rank's arrival): scale = max over ranks, turned into
// the scale as the quantizer does it.  The maximum of the shards' maxima is the maximum of the
// whole tensor, so this is the scale the unsharded quantizer computes, bit for bit.
__global__ void wait_flag_scale_kernel(const unsigned int* flag, unsigned int* seen, unsigned int count,
                                       unsigned int* status, const unsigned int* amax_slots, int n,
                                       int slots_hold_scales, float* scale_out) {
  const unsigned int target = *seen + count;
  const long long t0 = clock64();
  for (;;) {
    unsigned int v;
    asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
    if (static_cast<int>(v - target) >= 0) break;
    if (clock64() - t0 > kSpinLimitCycles) {
      atomicExch(status, (unsigned int)kErrDeviceWait);
      break;
    }
  }
  unsigned int best = 0u;
  for (int i = 0; i < n; ++i) {
    unsigned int b;
    asm volatile("ld.relaxed.sys.global.u32 %0, [%1];" : "=r"(b) : "l"(amax_slots + i) : "memory");
    best = b > best ? b : best;      // |h| bit patterns order like the values, NaN on top
  }
  // the scale is a monotone function of the amax (and its lower clamp commutes with max), so
  // the maximum of the ranks' scales is the scale of the maximum
  *scale_out = slots_hold_scales ? __uint_as_float(best) : bq::qd::scale_from_amax(__uint_as_float(best));
  *seen = target;
  __threadfence();
}

// ---------------------------------------------------------------------------
// Persistent tile kernel on CTA pairs (prefill regime, cta_group::2)
// ---------------------------------------------------------------------------
// Two CTAs on neighbouring SMs share one 256 x 256 output tile: each loads 128
// activation rows and 128 weight rows per K block (32 KB instead of the 48 KB a
// lone CTA needs for 128 x 256), the leader issues one MMA that spans both SMs,
// and each CTA keeps the accumulator of its own 128 rows in its tensor memory.
// Shared-memory traffic per flop drops by a third, which is what limits the
// a lone CTA with a 128 x 256 tile.  Warp roles per CTA: 0 = TMA producer, 1 = MMA issuer
// (leader CTA only), 2..5 = epilogue.
//
// Epilogue: eight warps; a warp owns 32 rows (its TMEM lane quarter) and one half of the
// columns of the CTA's 128 x 256 accumulator.  It walks them in pieces of 128 bytes of output
// per row (64 columns of a 16-bit type, 32 of fp32): tcgen05.ld -> scale -> cast -> one 32-row x
// 128-byte box in shared memory, written in the 128-byte swizzle pattern so that neither the
// lane-per-row writes nor the reader meet bank conflicts -> one TMA store of the box (clipped
// at M and N by the tensor map); the next piece waits until the store has read the box.  Outputs whose base or row pitch is not 16-byte aligned
// cannot be described to TMA: the same staged box is then written with coalesced 128-byte
// row segments by the warp itself.
// Ring: six stages of 16 KB of activation rows and 16 KB of weight rows, or, where no tile of the launch is wider than
// 128 columns, eight of 16 + 8 KB: a launch of one round waits for its copies, not for its MMAs.  us at 333 rows, six
// stages -> eight: 4096 x 12288 28.3 -> 24.2, 4096 x 4096 13.7 -> 12.5.
constexpr int kPairRingBytes = 6 * 2 * kATileBytes;
constexpr int kPairMaxStages = 8;
constexpr int kPairTile = 256;
constexpr int kPairEpiWarps = 8;                    // two per TMEM lane quarter
constexpr int kTileThreads = 64 + 32 * kPairEpiWarps;
constexpr int kStoreBoxBytes = 32 * 128;            // 32 rows x 128 bytes
constexpr int kPairStagingBytes = kPairEpiWarps * kStoreBoxBytes;   // one box per epilogue warp

// Order in which a weight's 256 x 256 tiles are visited: bands of kRasterM tile rows, inside a
// band the row index runs fastest.  The ~74 tiles in flight at a time then cover about
// 8 x 9 tiles -- (8 + 9) x 256 x K operand bytes, which stay in L2 for every K of the model --
// instead of all tile rows of two or three tile columns (M x K activation bytes per wave:
// 100 MB at M = 8192, K = 12288, more than L2 holds).
constexpr int kRasterM = 8;
__device__ __forceinline__ void pair_tile_coords(int local, int m_tiles, int n_tiles, int& m_idx,
                                                 int& n_idx) {
  const int band_tiles = kRasterM * n_tiles;      // every band but the last is full
  const int band = local / band_tiles;
  const int r = local - band * band_tiles;
  const int m_begin = band * kRasterM;
  const int height = (m_tiles - m_begin) < kRasterM ? (m_tiles - m_begin) : kRasterM;
  n_idx = r / height;
  m_idx = m_begin + (r - n_idx * height);
}

struct alignas(64) OutMaps {
  CUtensorMap y[BQ_MAX_SEGMENTS];
};

// 16 accumulator values -> scaled, cast to the output type, as 16-byte pieces.
template <int ES>
__device__ __forceinline__ void cast16(const uint32_t (&r)[16], float scale, int out_dtype,
                                       uint4 (&out)[ES == 4 ? 4 : 2]) {
  if constexpr (ES == 4) {
#pragma unroll
    for (int q = 0; q < 4; ++q)
      out[q] = make_uint4(__float_as_uint(__uint_as_float(r[4 * q]) * scale),
                          __float_as_uint(__uint_as_float(r[4 * q + 1]) * scale),
                          __float_as_uint(__uint_as_float(r[4 * q + 2]) * scale),
                          __float_as_uint(__uint_as_float(r[4 * q + 3]) * scale));
  } else {
    uint32_t w[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const float a = __uint_as_float(r[2 * q]) * scale, b = __uint_as_float(r[2 * q + 1]) * scale;
      if (out_dtype == BQ_DTYPE_BF16) {
        const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
        w[q] = *reinterpret_cast<const uint32_t*>(&v);
      } else {
        const __half2 v = __floats2half2_rn(a, b);
        w[q] = *reinterpret_cast<const uint32_t*>(&v);
      }
    }
    out[0] = make_uint4(w[0], w[1], w[2], w[3]);
    out[1] = make_uint4(w[4], w[5], w[6], w[7]);
  }
}

// h = T(T(silu(gate)) * up) of 16 columns from the 16 gate and the 16 up accumulator values of
// the same columns, each first rounded to T as the plain GEMM would have stored it
// (braid/model/mlp.py:46-48), as 16-byte pieces; returns max |h| folded into `mx`.
template <typename T>
__device__ __forceinline__ void silu16(const uint32_t (&g)[16], const uint32_t (&u)[16], float sg,
                                       float su, uint4 (&out)[sizeof(T) == 4 ? 4 : 2], float& mx) {
  using namespace bq::qd;
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    float gg[8], uu[8];
    if constexpr (sizeof(T) == 2) {
#pragma unroll
      for (int i = 0; i < 8; i += 2) {
        const int j = half * 8 + i;
        const float2 a = unpack2<T>(pack2<T>(__uint_as_float(g[j]) * sg, __uint_as_float(g[j + 1]) * sg));
        const float2 b = unpack2<T>(pack2<T>(__uint_as_float(u[j]) * su, __uint_as_float(u[j + 1]) * su));
        gg[i] = a.x; gg[i + 1] = a.y;
        uu[i] = b.x; uu[i + 1] = b.y;
      }
      gated_product<T, kSilu, 8>(gg, uu);
      uint32_t w[4], m = 0u;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        w[i] = pack2<T>(gg[2 * i], gg[2 * i + 1]);
        m = absmax2<T>(m, w[i]);
      }
      const float2 mm = unpack2<T>(m);
      mx = nan_max(mx, mm.x);
      mx = nan_max(mx, mm.y);
      out[half] = make_uint4(w[0], w[1], w[2], w[3]);
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        gg[i] = __uint_as_float(g[half * 8 + i]) * sg;
        uu[i] = __uint_as_float(u[half * 8 + i]) * su;
      }
      gated_product<T, kSilu, 8>(gg, uu);
#pragma unroll
      for (int i = 0; i < 8; ++i) mx = nan_max(mx, fabsf(gg[i]));
#pragma unroll
      for (int q = 0; q < 2; ++q)
        out[half * 2 + q] = make_uint4(__float_as_uint(gg[4 * q]), __float_as_uint(gg[4 * q + 1]),
                                       __float_as_uint(gg[4 * q + 2]), __float_as_uint(gg[4 * q + 3]));
    }
  }
}

// 16 bytes of the output type, already rounded to it, plus 16 residual bytes, rounded again.
template <int ES>
__device__ __forceinline__ uint4 add_res_piece(const uint4& v, const uint4& r, int out_dtype) {
  using namespace bq::qd;
  const uint32_t a[4] = {v.x, v.y, v.z, v.w}, b[4] = {r.x, r.y, r.z, r.w};
  uint32_t o[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if constexpr (ES == 4) {
      o[i] = __float_as_uint(__fadd_rn(__uint_as_float(a[i]), __uint_as_float(b[i])));
    } else if (out_dtype == BQ_DTYPE_BF16) {
      const float2 x = unpack2<__nv_bfloat16>(a[i]), y = unpack2<__nv_bfloat16>(b[i]);
      o[i] = pack2<__nv_bfloat16>(__fadd_rn(x.x, y.x), __fadd_rn(x.y, y.y));
    } else {
      const float2 x = unpack2<__half>(a[i]), y = unpack2<__half>(b[i]);
      o[i] = pack2<__half>(__fadd_rn(x.x, y.x), __fadd_rn(x.y, y.y));
    }
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}

// The epilogue of one warp for one tile: 32 rows x 256 accumulator columns.  SILU: the tile's
// columns [0,128) are gate and [128,256) up of the same 128 output columns, and the output is
// h = silu(gate) * up (128 columns); max |h| is folded into `mx`.
// RES: the residual's rows come in as coalesced 128-byte pieces (asked for before the box is free), go
// through the box into the lane-per-row order of the accumulator, and the sums replace them there.  The
// reads hide behind the next tile's MMAs; a separate add moved three times the bytes (38 us at 9658 x
// 4096, and a launch).
template <int ES, bool SILU, bool RES, bool PUSH>
__device__ __forceinline__ void pair_epilogue_rows(const GemmParams& p, const Segment& seg,
                                                   const CUtensorMap* ymap, bool use_tma,
                                                   uint32_t taddr, float scale, float scale_up,
                                                   int out_dtype, int m_row0, int n0, uint8_t* box,
                                                   uint32_t box_addr, int lane, int col_half,
                                                   float& mx) {
  constexpr int kCols = 128 / ES;              // output columns per 128-byte piece
  constexpr int kPieces = ES == 4 ? 4 : 2;     // 16-byte pieces per 16 accumulator columns
  const int out_cols = SILU ? kPairTile / 2 : seg.un;
  const int half_cols = (out_cols / 2 + kCols - 1) / kCols * kCols;   // whole pieces: 16-bit weights may be narrow
  const int c_end = (col_half + 1) * half_cols < out_cols ? (col_half + 1) * half_cols : out_cols;   // of this tile
  for (int c = col_half * half_cols; c < c_end; c += kCols) {
    // pieces beyond this weight's rows are never stored (warp-uniform)
    if ((n0 + c) >= seg.n) break;
    uint4 rv[RES ? 8 : 1];
    if constexpr (RES) {
      const int col = n0 + c + (lane & 7) * (16 / ES);
#pragma unroll
      for (int pass = 0; pass < 8; ++pass) {
        const int m = m_row0 + pass * 4 + (lane >> 3);
        rv[pass] = make_uint4(0u, 0u, 0u, 0u);
        if (m < p.M && col < seg.n) {
          const uint8_t* src = static_cast<const uint8_t*>(seg.res) + ((long long)m * seg.ld_res + col) * ES;
          if (seg.wide) {
            rv[pass] = ld_coherent16(src);
          } else {                              // rows are 8-byte aligned at least (checked by the host)
            const uint2 lo = ld_coherent8(src), hi = ld_coherent8(src + 8);
            rv[pass] = make_uint4(lo.x, lo.y, hi.x, hi.y);
          }
        }
      }
    }
    // the TMA store of the previous piece must have finished reading the box
    if (use_tma && lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    __syncwarp();
    if constexpr (RES) {
#pragma unroll
      for (int pass = 0; pass < 8; ++pass) {
        const int row = pass * 4 + (lane >> 3);
        *reinterpret_cast<uint4*>(box + row * 128 + (((lane & 7) ^ (row & 7)) << 4)) = rv[pass];
      }
      __syncwarp();
    }
#pragma unroll
    for (int j = 0; j < kCols; j += 16) {
      uint32_t r[16];
      tmem_ld16(taddr + c + j, r);          // warp-collective: no divergence before it
      uint4 v[kPieces];
      if constexpr (SILU) {
        uint32_t up[16];
        tmem_ld16(taddr + kPairTile / 2 + c + j, up);
        tmem_ld_wait();
        if constexpr (ES == 4) silu16<float>(r, up, scale, scale_up, v, mx);
        else if (out_dtype == BQ_DTYPE_BF16) silu16<__nv_bfloat16>(r, up, scale, scale_up, v, mx);
        else silu16<__half>(r, up, scale, scale_up, v, mx);
      } else {
        tmem_ld_wait();
        cast16<ES>(r, scale, out_dtype, v);
      }
#pragma unroll
      for (int q = 0; q < kPieces; ++q) {
        const int piece = (j * ES) / 16 + q;                  // 0..7 along the 128-byte row
        uint4* const at = reinterpret_cast<uint4*>(box + lane * 128 + ((piece ^ (lane & 7)) << 4));
        if constexpr (RES) *at = add_res_piece<ES>(v[q], *at, out_dtype);
        else *at = v[q];
      }
    }
    if (use_tma) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        // column-parallel form: the same box into every rank's gathered buffer (ymap[d] then
        // describes rank d's buffer at this rank's columns; peers' buffers are reached through
        // peer-mapped addresses by plain, non-multicast bulk stores)
        const int n_dst = PUSH && p.push.n > 0 ? p.push.n : 1;
        for (int d = 0; d < n_dst; ++d) tma_store_2d(ymap + d, box_addr, n0 + c, m_row0);
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      }
    } else {
      __syncwarp();
      // 8 lanes cover one 128-byte row segment, 4 rows per pass
      const int piece = lane & 7;
      const int col = n0 + c + piece * (16 / ES);
#pragma unroll
      for (int pass = 0; pass < 8; ++pass) {
        const int row = pass * 4 + (lane >> 3);
        const int m = m_row0 + row;
        const uint4 v = *reinterpret_cast<const uint4*>(box + row * 128 + ((piece ^ (row & 7)) << 4));
        if (m < p.M && col < seg.n) {
          // rows are 8-byte aligned at least (checked by the host); n is a multiple of 16, or of 4 for a 16-bit weight,
          // whose last piece may be in by half
          if (!PUSH || p.push.n == 0) {
            uint8_t* dst = static_cast<uint8_t*>(seg.y) + ((long long)m * seg.ldy + col) * ES;
            *reinterpret_cast<uint2*>(dst) = make_uint2(v.x, v.y);
            if (ES == 4 || col + 4 < seg.n) *reinterpret_cast<uint2*>(dst + 8) = make_uint2(v.z, v.w);
          } else {
            // column-parallel form: the same piece into every rank's gathered buffer (plain
            // stores through peer-mapped pointers, this rank's own buffer included)
            // 16-byte stores (destinations and row pitch are 16-byte aligned, checked by the
            // host): 8 lanes write one whole 128-byte line, which is what the link moves well --
            // halves of 32-byte sectors, as the 8-byte stores above produce, reached 0.3 TB/s
            const long long at = ((long long)m * p.push.ld + col) * ES;
            for (int d = 0; d < p.push.n; ++d)
              *reinterpret_cast<uint4*>(static_cast<uint8_t*>(p.push.dst[d]) + at) = v;
          }
        }
      }
      __syncwarp();
    }
  }
}

template <int EPI, int DT>
__global__ void __launch_bounds__(kTileThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_xd,
                 const __grid_constant__ WeightMaps tm_w, const __grid_constant__ OutMaps tm_y,
                 const __grid_constant__ GemmParams p) {
  extern __shared__ uint8_t smem_dyn[];
  const int out_dtype = DT == kAnyType ? p.out_dtype : DT;
  const int push_n = EPI == kAny ? p.push.n : 0;
  const uint32_t base = (smem_u32(smem_dyn) + 1023u) & ~1023u;
  uint8_t* const base_ptr = smem_dyn + (base - smem_u32(smem_dyn));
  const uint32_t bar_base = base + kPairRingBytes;
  const int stages = p.stages;
  const uint32_t stage_bytes = stages == kPairMaxStages ? kPairRingBytes / kPairMaxStages : 2 * kATileBytes;
  auto a_tile = [&](int s) { return base + s * stage_bytes; };
  auto b_tile = [&](int s) { return base + s * stage_bytes + kATileBytes; };
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (kPairMaxStages + s); };
  auto acc_full = [&](int b) { return bar_base + 8u * (2 * kPairMaxStages + b); };
  auto acc_empty = [&](int b) { return bar_base + 8u * (2 * kPairMaxStages + 2 + b); };
  volatile uint32_t* const tmem_slot = reinterpret_cast<volatile uint32_t*>(
      base_ptr + kPairRingBytes + 8 * (2 * kPairMaxStages + 4));
  volatile uint32_t* const abort_flag = tmem_slot + 1;
  // store boxes of the epilogue warps, after the barrier block (1024-byte aligned: the swizzle
  // pattern of a box is a function of its address bits)
  uint8_t* const staging = base_ptr + kPairRingBytes + kBarrierBytes;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_ctarank());     // 0 = leader of the pair
  const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
  const int m_tiles = (p.M + kPairTile - 1) / kPairTile;
  const bool silu = EPI == kAny ? p.pair.on != 0 : EPI == kGateUp;                       // gate/up tiles, h = silu(gate) * up out
  // output columns per tile: 128 of h in the SiLU form, in the plain form what the host chose for the
  // segment (the sums are the same either way)
  auto tile_cols = [&](const Segment& g) { return silu ? kPairTile / 2 : g.un; };
  float* const s_amax = reinterpret_cast<float*>(base_ptr + kPairRingBytes + 512);

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tm_x);
    for (int i = 0; i < p.n_seg; ++i) tma_prefetch_desc(&tm_w.w[i]);
    for (int s = 0; s < stages; ++s) {
      mbar_init(full_bar(s), 1);     // the leader's producer arrives, bytes of both CTAs expected
      mbar_init(empty_bar(s), 1);    // one MMA commit per use
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(acc_full(b), 1);
      mbar_init(acc_empty(b), 2 * kPairEpiWarps);    // the epilogue warps of both CTAs of the pair
    }
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(smem_u32(const_cast<uint32_t*>(tmem_slot)), 512);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  cluster_sync_all();     // the peer's barriers exist before anything signals them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents();
  pdl_wait_prior_grids();

  if (warp == 0) {
    const uint32_t issue = elect_one() ? 1u : 0u, expect = rank == 0 ? issue : 0u;
    const uint64_t pol = policy_evict_last();
    int s = 0;
    uint32_t phase = 1;                          // a fresh barrier counts as completed
    bool ok = true;
    for (int t = pair; t < p.total_tiles && ok; t += n_pairs) {
      const int sg = find_segment(p, t);
      const int local = t - p.seg[sg].tile_begin;
      const bool dense = EPI == kMixed && p.seg[sg].dense != 0;
      int m_idx, n_idx;
      const int n_step = tile_cols(p.seg[sg]);
      pair_tile_coords(local, m_tiles, (p.seg[sg].n + n_step - 1) / n_step, m_idx, n_idx);
      const int m0 = m_idx * kPairTile + rank * kRowTile;
      // plain: this CTA's half of the tile's weight rows; SiLU form: the leader loads 128
      // gate rows, its peer the 128 up rows of the same output columns
      const int rows = silu ? kRowTile : n_step / 2;
      const int n0 = silu ? n_idx * kRowTile : n_idx * n_step + rank * rows;
      const CUtensorMap* const w_map = silu ? &tm_w.w[rank] : &tm_w.w[sg];
      const CUtensorMap* const x_map = dense ? &tm_xd : &tm_x;
      const int blocks = dense ? p.k_blocks_dense : p.k_blocks;
      const uint32_t bytes = 2u * (kATileBytes + (uint32_t)rows * kBK);
      for (int kb = 0; kb < blocks; ++kb) {
        if (!mbar_wait(empty_bar(s), phase)) { ok = false; break; }
        mbar_expect_tx(expect, full_bar(s), bytes);
        tma_load_2d_pair(issue, a_tile(s), x_map, full_bar(s), kb * kBK, m0, pol);
        tma_load_2d_pair(issue, b_tile(s), w_map, full_bar(s), kb * kBK, n0, pol);
        if (++s == stages) { s = 0; phase ^= 1u; }
      }
    }
    if (!ok) *abort_flag = 1;
    __syncwarp();
  } else if (warp == 1) {
    if (rank == 0) {
      const uint32_t issue = elect_one() ? 1u : 0u;
      int s = 0, tile_iter = 0;
      uint32_t phase = 0;
      bool ok = true, ready = false;
      for (int t = pair; t < p.total_tiles && ok; t += n_pairs, ++tile_iter) {
        const int b = tile_iter & 1, use_b = tile_iter >> 1;
        if (use_b > 0 && !mbar_wait(acc_empty(b), (use_b - 1) & 1)) { ok = false; break; }
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + b * kPairTile;
        const Segment& seg = p.seg[find_segment(p, t)];
        const bool dense = EPI == kMixed && seg.dense != 0;
        const uint32_t idesc = dense ? idesc_f16(kPairTile, seg.un, p.dense_fmt)
                                     : idesc_e4m3(kPairTile, silu ? kPairTile : seg.un);
        const int blocks = dense ? p.k_blocks_dense : p.k_blocks;
        // one loop per operand kind: a choice inside it cost every tile of a mixed launch 8 %
        auto multiply = [&](auto is_dense) {
          for (int kb = 0; kb < blocks; ++kb) {
            if (!ready && !mbar_wait(full_bar(s), phase)) { ok = false; break; }
            const uint64_t da = smem_desc_sw128(a_tile(s)), db = smem_desc_sw128(b_tile(s));
            const uint32_t empty = empty_bar(s);
            if (++s == stages) { s = 0; phase ^= 1u; }
            // look at the next stage's barrier now: the answer arrives while this one's MMAs are issued
            ready = mbar_test(full_bar(s), phase);
            tc_fence_after();
#pragma unroll
            for (int j = 0; j < kBK / kUmmaK; ++j) {
              if constexpr (is_dense.value)
                mma_f16_pair(issue, tmem_d, da + 2u * j, db + 2u * j, idesc, (kb | j) != 0 ? 1u : 0u);
              else
                mma_f8_pair(issue, tmem_d, da + 2u * j, db + 2u * j, idesc, (kb | j) != 0 ? 1u : 0u);
            }
            mma_commit_pair(issue, empty);   // the stage is free in BOTH CTAs once these MMAs retire
          }
        };
        if (EPI == kMixed && dense) multiply(std::true_type{});
        else multiply(std::false_type{});
        if (ok) mma_commit_pair(issue, acc_full(b));
      }
      if (!ok) *abort_flag = 1;
    }
    __syncwarp();
  } else {
    const int quad = warp & 3;                   // TMEM lanes [32 * quad, +32): rows of the tile
    const int col_half = (warp - 2) >> 2;        // which half of the columns this warp stores
    int tile_iter = 0;
    bool ok = true;
    float h_max = 0.0f;                          // SiLU form: max |h| over everything this thread wrote
    uint8_t* const stage = staging + (warp - 2) * kStoreBoxBytes;
    const uint32_t stage_addr = smem_u32(stage);
    const uint32_t leader_acc_empty0 = map_to_cta(acc_empty(0), 0);
    const uint32_t leader_acc_empty1 = map_to_cta(acc_empty(1), 0);
    for (int t = pair; t < p.total_tiles && ok; t += n_pairs, ++tile_iter) {
      const int b = tile_iter & 1, use_b = tile_iter >> 1;
      const int sg = find_segment(p, t);
      const Segment seg = p.seg[sg];
      const int local = t - seg.tile_begin;
      int m_idx, n_idx;
      const int n_step = tile_cols(seg);
      pair_tile_coords(local, m_tiles, (seg.n + n_step - 1) / n_step, m_idx, n_idx);
      const int m0 = m_idx * kPairTile + rank * kRowTile;
      const int n0 = n_idx * n_step;
      if (!mbar_wait(acc_full(b), use_b & 1)) { ok = false; break; }
      tc_fence_after();
      const float sx = ld_coherent4(p.sx);
      const float scale = EPI == kMixed && seg.dense ? 1.0f : sx * __ldg(seg.sw);
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + b * kPairTile;
      const bool use_tma = seg.y_tma != 0;
      const CUtensorMap* const ymap = &tm_y.y[push_n > 0 ? 0 : sg];
      const float scale_up = silu ? sx * __ldg(p.pair.sw_up) : 0.0f;
#define BQ_ROWS(ES, SILU, RES)                                                                                          \
  pair_epilogue_rows<ES, SILU, RES, EPI == kAny>(p, seg, ymap, use_tma, taddr, scale, scale_up, out_dtype, m0 + quad * 32, \
                                                 n0, stage, stage_addr, lane, col_half, h_max)
      if constexpr (DT == BQ_DTYPE_F32) {
        BQ_ROWS(4, EPI == kGateUp, EPI == kResidual);
      } else if constexpr (DT != kAnyType) {
        BQ_ROWS(2, EPI == kGateUp, EPI == kResidual);
      } else if (out_dtype == BQ_DTYPE_F32) {
        if (silu) BQ_ROWS(4, true, false); else BQ_ROWS(4, false, false);
      } else {
        if (silu) BQ_ROWS(2, true, false); else BQ_ROWS(2, false, false);
      }
#undef BQ_ROWS
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(b == 0 ? leader_acc_empty0 : leader_acc_empty1);
    }
    // the boxes must stay valid until the last stores have read them; for the column-parallel
    // form the wait also means the stores have been written, before anybody is told to look
    if (lane == 0) {
      asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
      if (push_n > 0) asm volatile("fence.proxy.async;" ::: "memory");
    }
    __syncwarp();
    if (!ok) *abort_flag = 1;
    if (push_n > 0) {
      // The stores of all epilogue threads are ordered before the elected thread's fence by the
      // barrier (fences are cumulative); the fence orders them before this CTA's count; the
      // last CTA sees every count, fences again and only then signals the ranks: every store of
      // the launch happens before every arrival.
      const bool want_amax = silu && p.push.amax_local != nullptr;
      if (want_amax) {
        using namespace bq::qd;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
          h_max = nan_max(h_max, __shfl_xor_sync(0xffffffffu, h_max, off));
        if (lane == 0) s_amax[warp - 2] = h_max;
      }
      asm volatile("bar.sync 1, %0;" ::"n"(32 * kPairEpiWarps) : "memory");
      if (warp == 2 && lane == 0) {
        if (want_amax) {
          using namespace bq::qd;
          float w = s_amax[0];
#pragma unroll
          for (int i = 1; i < kPairEpiWarps; ++i) w = nan_max(w, s_amax[i]);
          // bit patterns of |h| order like the values, NaN on top: exact and order-free
          atomicMax(p.push.amax_local, __float_as_uint(w));
        }
        __threadfence_system();
        const unsigned int old = atomicAdd(p.push.done, 1u);
        if (old == p.push.expected - 1u) {
          *p.push.done = 0u;                     // ready for the next launch on this scratch
          if (want_amax) {
            // every CTA's max is in (its atomicMax precedes its count): hand this rank's
            // max |h| to every rank, ahead of the arrival that tells them to look
            const unsigned int bits = atomicExch(p.push.amax_local, 0u);
            for (int d = 0; d < p.push.n; ++d)
              if (p.push.amax_dst[d] != nullptr)
                asm volatile("st.relaxed.sys.global.u32 [%0], %1;" ::"l"(p.push.amax_dst[d]), "r"(bits) : "memory");
          }
          __threadfence_system();
          for (int d = 0; d < p.push.n; ++d)
            asm volatile("red.release.sys.global.add.u32 [%0], 1;" ::"l"(p.push.flag[d]) : "memory");
        }
      }
    } else if (silu) {
      // max |h| of the launch: warps -> CTA -> one atomicMax per CTA on the bit pattern (exact
      // and order-free; NaN patterns sort on top); the CTA that arrives last turns the result into
      // the scale of h and returns the scratch words to zero
      using namespace bq::qd;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1)
        h_max = nan_max(h_max, __shfl_xor_sync(0xffffffffu, h_max, off));
      if (lane == 0) s_amax[warp - 2] = h_max;
      asm volatile("bar.sync 1, %0;" ::"n"(32 * kPairEpiWarps) : "memory");      // the epilogue warps
      if (warp == 2 && lane == 0) {
        float w = s_amax[0];
#pragma unroll
        for (int i = 1; i < kPairEpiWarps; ++i) w = nan_max(w, s_amax[i]);
        unsigned int* const words = p.pair.words;
        atomicMax(&words[0], __float_as_uint(w));
        __threadfence();
        const unsigned int old = atomicAdd(&words[1], 1u);
        if (old == gridDim.x - 1) {
          __threadfence();
          const unsigned int bits = atomicMax(&words[0], 0u);
          p.pair.sh[0] = scale_from_amax(__uint_as_float(bits));
          words[0] = 0u;
          words[1] = 0u;
          __threadfence();
        }
      }
    }
  }

  tc_fence_before();
  cluster_sync_all();     // nobody frees tensor memory while the peer may still use the pair
  if (threadIdx.x == 0 && *abort_flag != 0) atomicExch(p.status, (unsigned int)kErrDeviceWait);
  if (warp == 1) tmem_dealloc_pair(tmem_base, 512);
}

#include "gemm_wide.cuh"

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(sym);
  }
  return fn;
}

// [rows, K] uint8 row-major tensor, box = 128 K-bytes x box_rows, 128-byte swizzle,
// out-of-range rows/columns read as zero.
int make_map(CUtensorMap* out, const void* ptr, long long rows, long long K, int box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) return kErrNoDriver;
  const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)K};
  const cuuint32_t box[2] = {(cuuint32_t)kBK, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult rc = fn(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(ptr), dims,
                         strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return rc == CUDA_SUCCESS ? kOk : kErrUnsupported;
}

// The same tensor seen as [K / 128][rows][128 bytes], so that one box brings `kb` K blocks of
// box_rows rows (blocks beyond K read as zero): a box costs the copy engine 62 clocks however
// few rows it has, which is more than the MMAs of one K block.  `flat` (K not a multiple of 128):
// one K block per box, addressed by x.
int make_map_kb(CUtensorMap* out, const void* ptr, long long rows, long long K, int box_rows, int kb, bool flat) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) return kErrNoDriver;
  const cuuint64_t dims[3] = {flat ? (cuuint64_t)K : (cuuint64_t)kBK, (cuuint64_t)rows,
                              flat ? 1 : (cuuint64_t)(K / kBK)};
  const cuuint64_t strides[2] = {(cuuint64_t)K, flat ? (cuuint64_t)K : (cuuint64_t)kBK};
  const cuuint32_t box[3] = {(cuuint32_t)kBK, (cuuint32_t)box_rows, (cuuint32_t)kb};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult rc = fn(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(ptr), dims,
                         strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return rc == CUDA_SUCCESS ? kOk : kErrUnsupported;
}

// [M, N] output of the prefill kernel, row pitch ldy elements: boxes of 32 rows x 128 bytes,
// 128-byte swizzle; rows beyond M and columns beyond N are clipped by the store.
int make_out_map(CUtensorMap* out, void* ptr, long long M, long long N, long long ldy, int out_dtype) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) return kErrNoDriver;
  const cuuint64_t es = out_dtype == BQ_DTYPE_F32 ? 4 : 2;
  const CUtensorMapDataType dt = out_dtype == BQ_DTYPE_F32   ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                 : out_dtype == BQ_DTYPE_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                                                              : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  const cuuint64_t dims[2] = {(cuuint64_t)N, (cuuint64_t)M};
  const cuuint64_t strides[1] = {(cuuint64_t)ldy * es};
  const cuuint32_t box[2] = {(cuuint32_t)(128 / es), 32};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult rc = fn(out, dt, 2, ptr, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return rc == CUDA_SUCCESS ? kOk : kErrUnsupported;
}

int device_sms() {
  static int sms[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  if (sms[dev] == 0) {
    int v = 0;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    sms[dev] = v;
  }
  return sms[dev];
}

long long g_opt_split = 0, g_opt_stages = 0, g_opt_stream_max_m = 256, g_opt_cta_target = 160;
long long g_opt_wide = -1;   // decode: CTA-pair kernel (-1 by batch, 0 never, 1 always)
long long g_opt_push_tma = 1;   // prefill push epilogue: bulk tensor stores (0: 16-byte plain stores)
long long g_opt_pair_narrow = -1;   // prefill: columns of a plain launch's tiles (-1 by rule, 0: 256, 1: 128, else so many)
long long g_opt_pdl = 1;   // programmatic dependent launch on by default
long long g_opt_b_stages = 0;   // activation ring depth: 0 = heuristic, -1 = as deep as the weight ring
long long g_opt_quant_inside = -1;   // bytes of an activation that every CTA quantizes for itself (-1 by rule)
long long g_opt_smem_cap = 0;   // 0 = no cap on pipeline bytes per CTA
thread_local long long g_fail_in = 0;   // tests: so many weight-streaming launches from now, one is not made
thread_local int g_argmax_slots = 0;     // pairs per batch row the last launch wrote (greedy pick)
thread_local long long g_last_launch[6] = {0, 0, 0, 0, 0, 0};
thread_local int g_last_quantizes = 0;     // its CTAs cast the activation for themselves

inline bool aligned_to(const void* p, size_t a) { return (reinterpret_cast<uintptr_t>(p) % a) == 0; }

using StreamKernel = decltype(&gemm_stream_kernel<kAny, kAnyType, 0>);
using WideKernel = decltype(&gemm_wide_kernel<1, kAny, kAnyType>);
using PairKernel = decltype(&gemm_pair_kernel<kAny, kAnyType>);

// The kernels by [epilogue][type]; the types are BQ_DTYPE_F32, BF16, F16 = 0, 1, 2.
const StreamKernel kStream[3][3] = {
    {gemm_stream_kernel<kPlain, 0, 0>, gemm_stream_kernel<kPlain, 1, 0>, gemm_stream_kernel<kPlain, 2, 0>},
    {gemm_stream_kernel<kResidual, 0, 0>, gemm_stream_kernel<kResidual, 1, 0>, gemm_stream_kernel<kResidual, 2, 0>},
    {gemm_stream_kernel<kGateUp, 0, 0>, gemm_stream_kernel<kGateUp, 1, 0>, gemm_stream_kernel<kGateUp, 2, 0>}};
const StreamKernel kStreamGateUpDense[3] = {gemm_stream_kernel<kGateUpDense, 0, 0>, gemm_stream_kernel<kGateUpDense, 1, 0>,
                                           gemm_stream_kernel<kGateUpDense, 2, 0>};
#define BQ_QUANT_KERNELS(Q)                                                                                       \
  {{gemm_stream_kernel<kPlain, 0, Q>, gemm_stream_kernel<kPlain, 1, Q>, gemm_stream_kernel<kPlain, 2, Q>},        \
   {gemm_stream_kernel<kResidual, 0, Q>, gemm_stream_kernel<kResidual, 1, Q>, gemm_stream_kernel<kResidual, 2, Q>}}
const StreamKernel kStreamQuant[3][2][3] = {BQ_QUANT_KERNELS(1), BQ_QUANT_KERNELS(2), BQ_QUANT_KERNELS(3)};
#undef BQ_QUANT_KERNELS
const StreamKernel kStreamArgmax[3] = {gemm_stream_kernel<kArgmax, 0, 0>, gemm_stream_kernel<kArgmax, 1, 0>,
                                      gemm_stream_kernel<kArgmax, 2, 0>};
const StreamKernel kStreamAny = gemm_stream_kernel<kAny, kAnyType, 0>;
template <int MODE>
struct WideKernels {
  static constexpr WideKernel any = gemm_wide_kernel<MODE, kAny, kAnyType>;
  static constexpr WideKernel of[3][3] = {
      {gemm_wide_kernel<MODE, kPlain, 0>, gemm_wide_kernel<MODE, kPlain, 1>, gemm_wide_kernel<MODE, kPlain, 2>},
      {gemm_wide_kernel<MODE, kResidual, 0>, gemm_wide_kernel<MODE, kResidual, 1>, gemm_wide_kernel<MODE, kResidual, 2>},
      {gemm_wide_kernel<MODE, kGateUp, 0>, gemm_wide_kernel<MODE, kGateUp, 1>, gemm_wide_kernel<MODE, kGateUp, 2>}};
  static constexpr WideKernel argmax[3] = {gemm_wide_kernel<MODE, kArgmax, 0>, gemm_wide_kernel<MODE, kArgmax, 1>,
                                           gemm_wide_kernel<MODE, kArgmax, 2>};
};
const PairKernel kPair[4][3] = {
    {gemm_pair_kernel<kPlain, 0>, gemm_pair_kernel<kPlain, 1>, gemm_pair_kernel<kPlain, 2>},
    {gemm_pair_kernel<kResidual, 0>, gemm_pair_kernel<kResidual, 1>, gemm_pair_kernel<kResidual, 2>},
    {gemm_pair_kernel<kGateUp, 0>, gemm_pair_kernel<kGateUp, 1>, gemm_pair_kernel<kGateUp, 2>},
    {nullptr, gemm_pair_kernel<kMixed, 1>, gemm_pair_kernel<kMixed, 2>}};
const PairKernel kPairAny = gemm_pair_kernel<kAny, kAnyType>;

// The form all segments of a launch share, or kAny.  `mixed`: does the kernel have a form for 16-bit
// segments (elsewhere they are a matter of a segment)?
int epilogue_of(const GemmParams& p, bool mixed) {
  if (p.argmax.on) return kArgmax;
  if (p.push.n > 0) return kAny;
  if (p.pair.on) return p.pair.h != nullptr ? kGateUpDense : kGateUp;
  int with = 0, dense = 0;
  for (int i = 0; i < p.n_seg; ++i) {
    with += p.seg[i].res != nullptr;
    dense += p.seg[i].dense != 0;
  }
  if (mixed && dense > 0) return kMixed;               // never with a residual
  return with == 0 ? kPlain : (with == p.n_seg ? kResidual : kAny);
}

int configure_once() {
  static int rc = -1;
  if (rc < 0) {
    bool ok = true;
    auto set = [&](const void* kernel) {
      ok = ok && cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem) == cudaSuccess;
    };
    set((const void*)kStreamAny);
    set((const void*)WideKernels<1>::any);
    set((const void*)WideKernels<2>::any);
    set((const void*)kPairAny);
    for (int d = 0; d < 3; ++d) {
      set((const void*)kStreamGateUpDense[d]);
      set((const void*)kStreamArgmax[d]);
      set((const void*)WideKernels<1>::argmax[d]);
      set((const void*)WideKernels<2>::argmax[d]);
    }
    for (int e = 0; e < 4; ++e)
      for (int d = 0; d < 3; ++d) {
        if (kPair[e][d] != nullptr) set((const void*)kPair[e][d]);
        if (e == 3) continue;
        set((const void*)kStream[e][d]);
        for (int g = 0; e < 2 && g < 3; ++g) set((const void*)kStreamQuant[g][e][d]);
        set((const void*)WideKernels<1>::of[e][d]);
        set((const void*)WideKernels<2>::of[e][d]);
      }
    rc = ok ? kOk : kErrLaunch;
    if (rc != kOk) (void)cudaGetLastError();
  }
  return rc;
}

// Largest grid of the stream kernel that is resident at once with this cluster
// size and shared-memory footprint (the paired gate/up epilogue has a grid-wide wait).
int max_resident_ctas(StreamKernel kernel, int cluster, int smem) {
  struct Entry { StreamKernel kernel; int cluster, smem, cap; };
  static Entry cache[64];
  static int n_cached = 0;
  for (int i = 0; i < n_cached; ++i)
    if (cache[i].kernel == kernel && cache[i].cluster == cluster && cache[i].smem == smem) return cache[i].cap;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)(cluster * 64), 1, 1);
  cfg.blockDim = dim3(kStreamThreads, 1, 1);
  cfg.dynamicSmemBytes = (size_t)smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int clusters = 0;
  if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    clusters = 0;
  }
  // The occupancy calculator reports one CTA per SM for this kernel even where two
  // demonstrably run side by side (all 256 CTAs of a 100 KB launch start within 1.3 us of
  // each other), so the per-SM count is derived from the resources themselves: shared
  // memory (1 KB reserved per CTA), registers, and the two-CTA cap of the launch bounds.
  cudaFuncAttributes fa;
  memset(&fa, 0, sizeof(fa));
  int regs = 128;
  if (cudaFuncGetAttributes(&fa, kernel) == cudaSuccess && fa.numRegs > 0)
    regs = fa.numRegs;
  else
    (void)cudaGetLastError();
  int per_sm = 233472 / (smem + 1024);
  const int by_regs = 65536 / (((regs + 7) / 8) * 8 * kStreamThreads);
  if (per_sm > by_regs) per_sm = by_regs;
  if (per_sm > 2) per_sm = 2;
  if (per_sm < 1) per_sm = 1;
  int cap = clusters * cluster * per_sm > 0 ? clusters * cluster * per_sm : -1;
  if (getenv("BQ_DEBUG"))
    fprintf(stderr, "[bq] residency: cluster %d smem %d regs %d -> %d clusters x %d per SM = %d CTAs\n",
            cluster, smem, regs, clusters, per_sm, cap);
  if (n_cached < 64) cache[n_cached++] = Entry{kernel, cluster, smem, cap};
  return cap;
}

// K slices of one weight.  A function of the weight's own shape only -- never of
// what else shares the launch or of the batch -- so an output element is summed
// in the same order whether its weight is multiplied alone or grouped with
// others (`project` stays bit-identical to per-weight calls).  Small weights
// are sliced so that their tiles x slices cover most of the SMs.
int split_for_weight(long long n_rows, int k_blocks) {
  const long long tiles = (n_rows + kRowTile - 1) / kRowTile;
  // at most 4: clusters of 8 leave a fifth of the SMs unusable (15 clusters of 8 fit on the
  // 148 SMs, against 33 clusters of 4)
  int s = 1;
  while (s < 4 && tiles * (s * 2) <= g_opt_cta_target && (s * 2) * 2 <= k_blocks) s *= 2;
  if (g_opt_split > 0) {
    s = 1;
    while (s * 2 <= g_opt_split && s < 8) s *= 2;
    while (s > 1 && s > k_blocks) s /= 2;
  }
  return s;
}

// Few rows: is the launch whose CTAs quantize the activation for themselves the faster form?  It saves a launch;
// every CTA reads all of the activation and casts its K slice, and its weights wait for that.  So what counts is
// the bytes a CTA reads plus those it casts.  us of an eager call, one launch and two, at the bytes of the activation and
// the K slices of the weight: 8 KB in 4 (1 row of 4096 x 4096) 6.7 and 8.5, 64 KB in 4 (8 rows) 7.4 and 8.4; 64 KB in 4 (8
// rows of 1024 x 4096) 5.9 and 8.5; 32 KB in 1 (8 rows of 12288 x 2048) 8.4 and 8.6, 64 KB in 1 (16 rows) 10.7 and 8.5.  In a graph
// the second launch costs no host, and since its quantizer exchanges inside a cluster it costs less on the device too:
// 6.5 and 6.3, 7.2 and 6.6, 5.6 and 5.3, 8.2 and 7.0, 10.6 and 7.2.  The line of a captured call, 60 KB of both, is where
// the two were equal before that; what it gives up below is 0 to 1.2 us, against one scratch slot and launch less.
constexpr int64_t kInsideBytes = 65536, kInsideWork = 61440, kInsideWorkEager = 92160;

bool quantize_inside_pays(int64_t M, int64_t K, int element_size, int n_seg, const int64_t* N, cudaStream_t stream) {
  const int64_t bytes = M * K * element_size;
  if (g_opt_quant_inside >= 0) return bytes <= g_opt_quant_inside;
  const int k_blocks = (int)((K + kBK - 1) / kBK);
  int64_t cast = 0, ctas = 0;
  for (int i = 0; i < n_seg; ++i) {
    const int split = split_for_weight(N[i], k_blocks);
    if (bytes / split > cast) cast = bytes / split;
    ctas += (N[i] + kRowTile - 1) / kRowTile * split;
  }
  if (bytes > kInsideBytes || bytes + cast > kInsideWorkEager) return false;
  if (bytes + cast <= kInsideWork || ctas <= 64) return true;
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &status) != cudaSuccess) (void)cudaGetLastError();
  return status == cudaStreamCaptureStatusNone;
}

// The same question where such a launch has no room beside the slices handed over (handover_bytes below), and would
// fetch them: the longest slices that fit, one or two rows, on 82 to 160 CTAs.  us, one launch and two: 1 row of
// 9600 x 5760 eager 13.8 and 15.2, in a graph 13.7 and 13.9; 1 row of 9472 x 14336 eager 25.0 and 26.9, 25.4 and 26.1; 5248 x
// 14336 17.6 and 19.0, 17.6 and 17.6; 2 rows of 5120 x 11520 (45 KB) eager 15.2 and 15.6, 14.7 and 14.4; beyond
// kInsideWork two launches win eager as well: 5 rows of 9600 x 5760 16.3 and 15.8, 2 rows of 5248 x 14336 19.4 and 18.7,
// 1 row of 2048 x 28672 17.4 and 17.0.
constexpr int64_t kInsideFetched = 32768;

bool fetched_inside_pays(const GemmParams& p, int split, cudaStream_t stream) {
  const int64_t bytes = (int64_t)p.M * p.quant_k * (p.out_dtype == BQ_DTYPE_F32 ? 4 : 2);
  if (g_opt_quant_inside >= 0) return true;           // the caller has chosen
  if (bytes + bytes / split > kInsideWork) return false;
  if (bytes <= kInsideFetched) return true;
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &status) != cudaSuccess) (void)cudaGetLastError();
  return status == cudaStreamCaptureStatusNone;
}

// Where every weight is sliced the CTAs may look at their own slices alone (quantize_own_slice) instead of at all of x.  In a
// graph, the time with all of x over that with own slices, 13 weights of 512 to 10240 rows by 9 of 1024 to 12288 columns, by KB of x:
// 16 bits, halves: 31 to 41 KB 0.98, to 46 KB 1.04, to 60 KB 1.05; quarters 1.00, 1.085, 1.10; where two CTAs share an SM 1.04 to
// 1.06, 1.11 to 1.13, 1.14; fp32 1.09 to 1.14, 1.19 to 1.24, 1.15 to 1.24.  So the line lies at 32 KB, and for 16 bits with an SM
// per CTA at 40 KB (between them 5 rows of 8192 x 4096 8.2 and 8.5 us, 2 rows of 5760 x 9728 10.2 and 11.0).
constexpr int64_t kOwnSliceBytes = 32768, kOwnSliceBytes16 = 40960;
bool own_slices_pay(const GemmParams& p, int min_split, int per_sm) {
  const bool fp32 = p.out_dtype == BQ_DTYPE_F32;
  return min_split > 1 && (int64_t)p.M * p.quant_k * (fp32 ? 4 : 2) > (fp32 || per_sm > 1 ? kOwnSliceBytes : kOwnSliceBytes16);
}

// Where the K slices of a tile are summed.  Up to 48 rows every CTA writes its share of a tile straight from its
// accumulator into the memory of the CTA that sums those rows, and one cluster barrier ends the exchange; more
// rows would take the memory of too many weight tiles, and are staged and fetched between two barriers.
// us, fetched -> handed over: linear of 8 rows of 4096 x 4096 8.8 -> 7.9; four graphed layers of hidden 4096, 16 rows
// 249.2 -> 246.6, 27 rows 263 -> 257.5, 48 rows 274 -> 273, 1 row the same; hidden 1024, 16 rows 147 -> 145.8.
// Two CTAs per SM have room for three stages beside it from 45 rows on, which the long slices of halves pay for: 48 rows of
// 9728 x 5760 14.4 fetched, 14.8 with three stages (13.9 fetched with the present loops), four layers of hidden 3072 250.4 and
// 245.0 so; slices of quarters gain all the same (48 rows of 5120 x 2560 6.7 and 6.3, 5120 x 7680 11.4 and 11.0).
constexpr int kHandoverStages = 4;
int handover_bytes(int64_t M, int split) {
  return split > 1 && M <= 48 ? (int)((M + split - 1) / split) * split * kRowTile * 4 : 0;
}

// Shared memory that three CTAs of an SM cannot have (228 KB, of which 1 KB per CTA is reserved).
constexpr int kThirdOfSmem = (233472 / 3 - 1024) / 128 * 128 + 128;

// Shared memory of a CTA for rings: what lets the whole grid be resident at once (up to 2 CTAs per SM), so that one
// CTA's epilogue overlaps its neighbour's loads.
int stream_budget(long long grid, int sms, int* per_sm_out = nullptr) {
  int per_sm = (int)((grid + sms - 1) / sms);
  if (per_sm < 1) per_sm = 1;
  if (per_sm > 2) per_sm = 2;
  if (per_sm_out != nullptr) *per_sm_out = per_sm;
  return kMaxSmem / per_sm - 1024 - kBarrierBytes - 1024;
}

// Rings of a launch whose CTAs cast the activation for themselves: a slice's activation tiles all stay, the weight
// ring gets the rest.  0: no room.
int cast_stages(int budget, int b_tile, int kb_max) {
  int stages = (budget - kb_max * b_tile) / kATileBytes;
  if (stages > kb_max) stages = kb_max;
  if (stages > 24) stages = 24;
  // long slices of few rows: tiles padded to 16 rows would crowd out the weights (1 row of 8192 x 20480: 33 -> 36 us)
  if (2 * kb_max * b_tile > budget) return 0;
  return stages < (kb_max < 4 ? kb_max : 4) || 2 * stages + kb_max + 1 > 100 ? 0 : stages;
}

int launch_stream(const CUtensorMap& tm_x, const CUtensorMap& tm_xd, const WeightMaps& maps,
                  GemmParams& p, cudaStream_t stream) {
  const int sms = device_sms();
  if (sms <= 0) return kErrLaunch;
  p.mma_n = ((p.M + 15) / 16) * 16;
  const int b_tile = p.mma_n * kBK;
  const int stage_bytes = kATileBytes + b_tile;
  int cluster = 1, min_split = 8;
  for (int i = 0; i < p.n_seg; ++i) {
    p.seg[i].split = p.seg[i].split_forced > 0 ? p.seg[i].split_forced
                                               : split_for_weight(p.seg[i].n, p.seg[i].dense ? p.k_blocks_dense
                                                                                             : p.k_blocks);
    if (p.seg[i].split > cluster) cluster = p.seg[i].split;
    if (p.seg[i].split < min_split) min_split = p.seg[i].split;
  }
  p.cluster = cluster;
  int clusters = 0;
  for (int i = 0; i < p.n_seg; ++i) {
    const int tiles = (p.seg[i].n + kRowTile - 1) / kRowTile;
    const int per_cluster = cluster / p.seg[i].split;
    p.seg[i].cluster_begin = clusters;
    clusters += (tiles + per_cluster - 1) / per_cluster;
  }
  const long long grid = (long long)clusters * cluster;
  if (grid > 0x7fffffffLL) return kErrTooLarge;
  int kb_max = (p.k_blocks + min_split - 1) / min_split;
  for (int i = 0; i < p.n_seg; ++i)
    if (p.seg[i].dense) {
      const int kb = (p.k_blocks_dense + p.seg[i].split - 1) / p.seg[i].split;
      if (kb > kb_max) kb_max = kb;
    }
  const int staging = p.mma_n * kRowTile * 4;
  int per_sm = 1, handover = 0;
  for (int i = 0; i < p.n_seg; ++i) {
    const int bytes = handover_bytes(p.M, p.seg[i].split);
    if (bytes > handover) handover = bytes;
  }
  const bool quant = p.quant.x != nullptr;
  int whole = stream_budget(grid, sms, &per_sm);
  const int beside = (whole - handover) / stage_bytes;      // stages that the handed-over slices leave
  if (!quant && min_split == 2 && beside < kHandoverStages && beside < kb_max) handover = 0;
  p.handover = handover > 0 ? 1 : 0;
  int budget = whole - handover;
  // Leave room for the NEXT kernel's CTAs: with programmatic dependent launch they
  // become resident while this kernel still runs and pre-load their weights.
  if (g_opt_smem_cap > 0 && whole > g_opt_smem_cap) whole = (int)g_opt_smem_cap;
  if (budget > whole) budget = whole;
  int stages = budget / stage_bytes;            // both rings equally deep: the starting point
  if (stages > kb_max) stages = kb_max;
  if (stages > 24) stages = 24;
  if (stages < 2) stages = kb_max < 2 ? kb_max : 2;
  if (g_opt_stages > 0 && g_opt_stages < stages) stages = (int)g_opt_stages;
  int b_stages = stages;
  // Wide batch tiles: a shallow activation ring (its tiles are L2 hits), the rest goes to
  // weight tiles in flight.  Two slots cover the L2 latency at the rate one CTA of a two-per-SM
  // launch consumes tiles; a CTA that has the SM to itself consumes twice as fast.
  long long want_b = g_opt_b_stages;
  if (want_b == 0) want_b = b_tile >= 8192 ? (per_sm == 2 ? 2 : 4) : -1;
  if (want_b > 0 && want_b < b_stages && !(g_opt_stages > 0)) {
    b_stages = (int)want_b;
    stages = (budget - b_stages * b_tile) / kATileBytes;
    if (stages > kb_max) stages = kb_max;
    if (stages > 24) stages = 24;
    if (b_stages > stages) b_stages = stages;
  }
  if (quant) {
    b_stages = kb_max;
    stages = cast_stages(budget, b_tile, kb_max);
    if (stages == 0 && handover > 0 && p.quant.words == nullptr && fetched_inside_pays(p, min_split, stream)) {
      handover = p.handover = 0;
      stages = cast_stages(whole, b_tile, kb_max);
    }
    if (stages == 0) return kErrUnsupported;
  }
  p.stages = stages;
  p.b_stages = b_stages;
  int tile_bytes = stages * kATileBytes + b_stages * b_tile;
  if (tile_bytes < staging) tile_bytes = staging;
  int smem = tile_bytes + kBarrierBytes + handover + 1024;
  // More than 128 rows take half of an SM's tensor memory: a third CTA there would wait for it until one of the two
  // is done, and where they wait for the whole grid's maximum that is never.  So no third one gets in.
  if (p.mma_n > 128 && smem < kThirdOfSmem) smem = kThirdOfSmem;
  if (smem > kMaxSmem) return kErrUnsupported;
  const int epi = epilogue_of(p, false);
  if (quant && epi != kPlain && epi != kResidual) return kErrUnsupported;
  const StreamKernel kernel =
      quant ? kStreamQuant[p.quant.words != nullptr ? 1 : (own_slices_pay(p, min_split, per_sm) ? 2 : 0)][epi][p.out_dtype]
            : (epi == kAny ? kStreamAny : epi == kArgmax ? kStreamArgmax[p.out_dtype] : (epi == kGateUpDense ? kStreamGateUpDense[p.out_dtype] : kStream[epi][p.out_dtype]));
  if (p.pair.on) p.pair.expected = (unsigned)((p.seg[0].n / kRowTile) * p.seg[0].split);
  if (p.push.n > 0)
    p.push.expected = (unsigned)(((p.seg[0].n + kRowTile - 1) / kRowTile) * p.seg[0].split);
  if (quant) p.quant.expected = (unsigned)(((p.seg[0].n + kRowTile - 1) / kRowTile) * p.seg[0].split);
  if (p.pair.on && p.push.n == 0 && p.pair.h == nullptr) {
    // the epilogue's amax exchange waits on the whole grid: every CTA must be resident
    const int cap = max_resident_ctas(kernel, cluster, smem);
    if (getenv("BQ_DEBUG"))
      fprintf(stderr, "[bq] paired launch: grid %lld cluster %d smem %d resident cap %d\n", grid,
              cluster, smem, cap);
    if (cap <= 0 || grid > cap) return kErrUnsupported;
  }

  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)grid, 1, 1);
  cfg.blockDim = dim3(kStreamThreads, 1, 1);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = g_opt_pdl ? 2 : 1;
  g_last_quantizes = quant ? 1 : 0;
  g_last_launch[0] = 0; g_last_launch[1] = grid; g_last_launch[2] = cluster;
  g_last_launch[3] = stages; g_last_launch[4] = smem; g_last_launch[5] = p.mma_n;
  g_argmax_slots = (p.seg[0].n + kRowTile - 1) / kRowTile;   // one pair per row tile
#ifdef BQ_PHASES
  p.phase_ring = bq::phase_ring_for_launch(&p.phase_seq);
#endif
  if (g_fail_in > 0 && --g_fail_in == 0) return kErrLaunch;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, tm_x, tm_xd, maps, p, tile_bytes);
  if (e != cudaSuccess) { (void)cudaGetLastError(); return kErrLaunch; }
  return kOk;
}

// CTA pairs of the wide kernel that are resident at once (one CTA per SM).
int max_pairs() {
  static int cached[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  if (cached[dev] == 0) {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(2, 1, 1);
    cfg.blockDim = dim3(kWideThreads, 1, 1);
    cfg.dynamicSmemBytes = kMaxSmem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, WideKernels<2>::any, &cfg) != cudaSuccess || clusters < 1) {
      (void)cudaGetLastError();
      clusters = device_sms() / 2;
    }
    cached[dev] = clusters;
  }
  return cached[dev];
}

// How a launch of the wide kernel is laid out; the sums do not depend on any of it.
// kErrUnsupported: no one-round layout of a form that needs one, or a shape that leaves no room for
// the rings; the K-sliced kernel takes those.
int plan_wide(GemmParams& p, WideShape& sh, bool flat) {
  memset(&sh, 0, sizeof(sh));
  const bool silu = p.pair.on != 0;
  sh.mode = p.M > 128 ? 2 : 1;
  constexpr int cg = 2;
  sh.nm = silu ? 2 : 1;
  sh.m_half = ((p.M + cg - 1) / cg + 7) / 8 * 8;
  constexpr int step = 32;                               // MMA N granularity
  const int max_units = max_pairs();
  if (max_units < 1) return kErrLaunch;
  auto round_up = [&](int n) { return (n + step - 1) / step * step; };
  // tensor-memory columns per weight row: a pair of 128 keeps half of a unit's columns in each half
  // of the lanes
  const int row_cols_x2 = sh.mode == 1 ? 1 : 2;
  int buffers = 1;
  for (int i = 0; i < p.n_seg; ++i)
    p.seg[i].split =    // the greedy pick: K in one piece, as on the K-sliced kernel
        p.argmax.on ? 1 : split_for_weight(p.seg[i].n, p.seg[i].dense ? p.k_blocks_dense : p.k_blocks);
  auto seg_un = [&](const Segment& s, int un) {
    int most = 1024 / (row_cols_x2 * buffers * sh.nm * s.split) / step * step;
    if (most > 256) most = 256;
    if (s.dense && round_up(s.n) < most) most = round_up(s.n);
    return un < most ? un : most;
  };
  auto count = [&](int un) {
    long long units = 0;
    for (int i = 0; i < p.n_seg; ++i) units += (p.seg[i].n + seg_un(p.seg[i], un) - 1) / seg_un(p.seg[i], un);
    return units;
  };
  // rows per unit: the fewest that make the launch one round; where one MMA (N <= 256) or tensor
  // memory does not reach that far, two accumulators and the rows with the least padding
  int un = 0;
  for (int u = step; u <= 256; u += step)
    if (count(u) <= max_units) { un = u; break; }
  if (un == 0) {
    if (silu) return kErrUnsupported;                    // h waits for a grid-wide exchange inside its CTA
    buffers = 2;
    long long best = 0;
    for (int u = 256; u >= 64; u -= step) {
      const long long cost = (count(u) + max_units - 1) / max_units * (u + 8);   // 8: what a round costs by itself
      if (un == 0 || cost < best) { un = u; best = cost; }
    }
  }
  const long long units = count(un);
  if (units > 0x3fffffffLL) return kErrTooLarge;
  sh.units = (int)units;
  sh.rounds = (int)((units + max_units - 1) / max_units);
  sh.grid = (int)(units < max_units ? units : max_units) * cg;
  int at = 0, k_blocks[2] = {0, 0}, w_rows[2] = {0, 0};
  for (int i = 0; i < p.n_seg; ++i) {
    Segment& s = p.seg[i];
    s.un = seg_un(s, un);
    s.unit_begin = at;
    at += (s.n + s.un - 1) / s.un;
    const int d = s.dense && sh.rounds == 1 ? 1 : 0;
    const int kb = s.dense ? p.k_blocks_dense : p.k_blocks;
    if (kb > k_blocks[d]) k_blocks[d] = kb;
    if (s.un > w_rows[d]) w_rows[d] = s.un;
    const int cols = s.un * row_cols_x2 / 2 * sh.nm * s.split;
    if (cols > sh.acc_cols) sh.acc_cols = cols;
  }
  sh.tmem_cols = 32;
  while (sh.tmem_cols < sh.acc_cols * buffers) sh.tmem_cols *= 2;
  if (sh.tmem_cols > 512) return kErrUnsupported;
  sh.flat = flat;
  const int budget = g_opt_smem_cap > 0 && g_opt_smem_cap < kMaxSmem - 1024 - kBarrierBytes
                         ? (int)g_opt_smem_cap : kMaxSmem - 1024 - kBarrierBytes;
  for (int d = 0; d < 2; ++d) {
    if (w_rows[d] == 0) continue;
    RingShape& r = sh.ring[d];
    r.a_block = sh.m_half * kBK;
    r.w_block = sh.nm * (w_rows[d] / cg) * kBK;
    // a stage holds 16 KB of weights or more: what the issuing threads spend per stage is fixed
    r.kb_stage = r.w_block >= 16384 || flat ? 1 : (r.w_block >= 8192 ? 2 : 4);
    while (r.kb_stage > 1 && (r.kb_stage > k_blocks[d] || r.kb_stage * r.a_block > 32768)) r.kb_stage /= 2;
    const int a_bytes = r.kb_stage * r.a_block, w_bytes = r.kb_stage * r.w_block;
    const int want = (k_blocks[d] + r.kb_stage - 1) / r.kb_stage * sh.rounds;   // stages of a CTA's work
    // 96 KB of activation tiles in flight, four stages at least: once the previous kernel is done every
    // CTA walks the same tiles of L2 at the same time, and that latency under load is what a wide
    // batch waits for (128 rows, 4096 x 12288: 16.9 / 14.3 / 13.4 us with 2 / 3 / 4 stages of 32 KB).
    // The weight ring gets the rest; it streams at full rate from about 100 KB on.
    int a_stages = 98304 / a_bytes;
    if (a_stages < 4) a_stages = 4;
    if (a_stages > 16) a_stages = 16;
    if (g_opt_b_stages > 0) a_stages = g_opt_b_stages < kWideMaxA ? (int)g_opt_b_stages : kWideMaxA;
    if (a_stages > want) a_stages = want;
    int w_stages = (budget - a_stages * a_bytes) / w_bytes;
    if (w_stages > kWideMaxW) w_stages = kWideMaxW;
    if (w_stages > want) w_stages = want;
    if (g_opt_stages > 0 && w_stages > g_opt_stages) w_stages = (int)g_opt_stages;
    if (w_stages < 1) return kErrUnsupported;
    if (a_stages > w_stages) a_stages = w_stages;
    r.a_stages = a_stages;
    r.w_stages = w_stages;
    // an MMA reads 64 or 128 rows from the start of any batch tile, whatever the batch
    const int reach = (a_stages * r.kb_stage - 1) * r.a_block + (sh.mode == 2 ? 128 : 64) * kBK;
    const int bytes = a_stages * a_bytes + w_stages * w_bytes;
    if (bytes > sh.ring_bytes) sh.ring_bytes = bytes;
    if (reach > sh.ring_bytes) sh.ring_bytes = reach;
  }
  if (w_rows[1] == 0) sh.ring[1] = sh.ring[0];
  const int es = p.out_dtype == BQ_DTYPE_F32 ? 4 : 2;
  if (silu && sh.ring_bytes < sh.m_half * (2 * un * es + 16)) sh.ring_bytes = sh.m_half * (2 * un * es + 16);
  sh.ring_bytes = (sh.ring_bytes + 127) / 128 * 128;
  if (sh.ring_bytes + kBarrierBytes + 1024 > kMaxSmem) return kErrUnsupported;
  return kOk;
}

// (value, index) pairs per batch row that the greedy pick of a launch leaves: one per unit walker and
// column group (a pair of 128 holds a row's columns in two lane quarters).
int argmax_slots(const WideShape& sh) {
  return sh.grid / 2 * (sh.mode == 1 ? 2 : 1) * (sh.rounds > 1 ? (kWideWarps - 4) / 4 : kWideWarps / 4);
}

int launch_wide(const CUtensorMap& tm_x, const CUtensorMap& tm_xd, const WeightMaps& maps,
                  GemmParams& p, const WideShape& sh, cudaStream_t stream) {
  const int smem = sh.ring_bytes + kBarrierBytes + 1024;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)sh.grid, 1, 1);
  cfg.blockDim = dim3(kWideThreads, 1, 1);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = g_opt_pdl ? 2 : 1;
  g_last_quantizes = 0;
  g_last_launch[0] = 1; g_last_launch[1] = sh.grid; g_last_launch[2] = p.seg[0].split;
  g_last_launch[3] = sh.ring[0].w_stages; g_last_launch[4] = smem; g_last_launch[5] = 64 << sh.mode;
  g_argmax_slots = argmax_slots(sh);
#ifdef BQ_PHASES
  p.phase_ring = bq::phase_ring_for_launch(&p.phase_seq);
#endif
  const int epi = epilogue_of(p, false);
  const WideKernel kernel =
      sh.mode == 1 ? (epi == kAny ? WideKernels<1>::any : epi == kArgmax ? WideKernels<1>::argmax[p.out_dtype]
                                                                         : WideKernels<1>::of[epi][p.out_dtype])
                   : (epi == kAny ? WideKernels<2>::any : epi == kArgmax ? WideKernels<2>::argmax[p.out_dtype]
                                                                         : WideKernels<2>::of[epi][p.out_dtype]);
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, tm_x, tm_xd, maps, p, sh);
  if (e != cudaSuccess) { (void)cudaGetLastError(); return kErrLaunch; }
  return kOk;
}

int launch_pair(const CUtensorMap& tm_x, const CUtensorMap& tm_xd, const WeightMaps& maps, const OutMaps& ymaps, GemmParams& p,
                cudaStream_t stream) {
  const int sms = device_sms();
  if (sms <= 0) return kErrLaunch;
  const int smem = kPairRingBytes + kBarrierBytes + kPairStagingBytes + 1024;
  static_assert(kPairRingBytes + kBarrierBytes + kPairStagingBytes + 1024 <= kMaxSmem,
                "pair kernel: pipeline + store boxes exceed the shared memory of an SM");
  int pairs = p.total_tiles < sms / 2 ? p.total_tiles : sms / 2;
  if (pairs < 1) pairs = 1;
  const int epi = epilogue_of(p, true);
  // the general form of this kernel is the column-parallel one's: it adds no residual
  if (epi == kAny && p.push.n == 0) return kErrUnsupported;
  if (p.push.n > 0) p.push.expected = (unsigned)(2 * pairs);   // every CTA has a tile and stores
  g_last_quantizes = 0;
  g_last_launch[0] = 2; g_last_launch[1] = 2 * pairs; g_last_launch[2] = 2;
  p.stages = kPairMaxStages;
  for (int i = 0; i < p.n_seg; ++i)
    if (p.pair.on || p.seg[i].un > kPairTile / 2) p.stages = 6;
  g_last_launch[3] = p.stages; g_last_launch[4] = smem; g_last_launch[5] = p.pair.on ? kPairTile : p.seg[0].un;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)(2 * pairs), 1, 1);
  cfg.blockDim = dim3(kTileThreads, 1, 1);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = g_opt_pdl ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, epi == kAny ? kPairAny : kPair[epi][p.out_dtype], tm_x, tm_xd, maps, ymaps, p);
  if (e != cudaSuccess) { (void)cudaGetLastError(); return kErrLaunch; }
  return kOk;
}

}  // namespace

namespace bq {
int gemm_set_option(const char* key, long long value);
}
int bq::gemm_set_option(const char* key, long long value) {
  if (strcmp(key, "decode_split_k") == 0) { g_opt_split = value; return kOk; }
  if (strcmp(key, "decode_stages") == 0) { g_opt_stages = value; return kOk; }
  if (strcmp(key, "decode_b_stages") == 0) { g_opt_b_stages = value; return kOk; }
  if (strcmp(key, "gemm_pdl") == 0) { g_opt_pdl = value ? 1 : 0; return kOk; }
  if (strcmp(key, "push_tma") == 0) { g_opt_push_tma = value ? 1 : 0; return kOk; }
  if (strcmp(key, "pair_narrow") == 0) {
    if (value > 1 && (value % 64 || value > kPairTile)) return kErrBadArg;
    g_opt_pair_narrow = value < 0 ? -1 : value;
    return kOk;
  }
  if (strcmp(key, "decode_quant_inside") == 0) {
    if (value > 262144) return kErrBadArg;
    g_opt_quant_inside = value < 0 ? -1 : value;
    return kOk;
  }
  if (strcmp(key, "fail_stream_launch") == 0) { g_fail_in = value; return kOk; }
  if (strcmp(key, "decode_smem_cap") == 0) { g_opt_smem_cap = value; return kOk; }
  if (strcmp(key, "decode_wide") == 0) { g_opt_wide = value < 0 ? -1 : (value ? 1 : 0); return kOk; }
  if (strcmp(key, "decode_cta_target") == 0) {
    if (value < 1) return kErrBadArg;
    g_opt_cta_target = value;
    return kOk;
  }
  if (strcmp(key, "stream_max_m") == 0) {
    if (value < 1 || value > 256) return kErrBadArg;
    g_opt_stream_max_m = value;
    return kOk;
  }
  return kErrBadArg;
}

extern "C" size_t bq_gemm_workspace_bytes(int64_t, int64_t, int64_t) {
  // the status word and the counters of the paired / push epilogues; partial sums never leave the chip
  return 16;
}

namespace {

// Weights of a mixed launch that are NOT quantized: kind[i] != 0 marks segment i as a 16-bit
// weight [N_i, K] of type `dtype`, multiplied with the unquantized activation `x` [M, K].
struct DenseArgs {
  const void* x;
  int dtype;
  const int* kind;
};

// Which launches the wide kernel takes: batches that fill its MMA shape (128 rows, or 256) well enough.
// All figures are the K-sliced kernel's time over this one's, graphed, weights from HBM (banks larger
// than L2); where a line says nothing, it lies between 1.0 and 1.4, beyond 208 rows up to 2.5.
//
// One round.  Four decoder layers of hidden 1024 / 2048 / 2560 / 4096 / 5120: 33 to 48 rows 1.03 / 1.00 / 0.99 /
// 1.00 / 1.04, 49 rows 1.09 / 1.03 / 1.01 / 1.06 / 1.07, 128 rows 1.21 / 1.13 / 1.09 / 1.10 / 1.09, 129 rows
// 1.15 / 1.04 / 1.00 / 0.98 / 0.99, 161 rows 1.20 / 1.11 / 1.07 / 1.09 / 1.14: 49 rows on, without 129 to 160.
// (Gate/up of 16384 columns alone measures 0.96 at 49 rows, but in the chain of a layer it is the
// faster one: hidden 4096, 312 us here, 324 with that launch on the K-sliced kernel.)
// Within that, what the K-sliced kernel does better:
//  * short K in units that leave no pair of SMs free: up to 64 rows (9472 x 1024 behind a norm: 49 rows
//    0.83, 80 rows 1.05), and in the longest units from 177 rows on (18944 x 1024: 176 rows 1.00,
//    192 rows 0.97, 256 rows 0.96);
//  * few rows and long K beyond 160 rows: one thread's chain of MMAs against a quarter of it
//    (4096 x 12288: 161 rows 0.93, 224 rows 0.99, 240 rows 1.03, and four layers of hidden 4096 393 -> 390 us
//    at 161 rows; 2560 x 7680: 0.96 alone, but the layers 324 -> 328 us: the line lies between).
//
// Several rounds (a vocabulary) pay an epilogue per round.  Where K is long it is hidden (60016 x 4096:
// 129 rows 1.09).  Up to 48 rows the two are within 4 % of one another at full clock there (248320 x 4096 with the greedy pick, 48
// rows 167 us on the K-sliced kernel and 163 here), but a stream of that length runs into the power limit when it is
// repeated, and this kernel multiplies 128 rows whatever the batch: 176 to 180 and 186 to 195 us; 64 rows 197 and 185 to 205, 195
// and 170 at full clock.  With fewer tiles than one and a half times what the K-sliced kernel holds it has a nearly
// empty last wave (40000 x 4096, 33 rows 1.05).  Where K is short the batch has to be larger (60016 x 1024: 65 rows 1.14,
// 129 rows 1.06).  The K-sliced kernel holds up to two CTAs per SM at once; while its tiles fit and fill
// three quarters of that room, only its wide accumulators (more than 96 rows, and again more than 160) are
// slower (32000 x 4096: 49 rows 0.95, 97 rows 1.01, 129 rows 0.88, 161 rows 1.06; 24576 x 4096: 1.08,
// 1.12, 0.97, 1.24), and with K below 1536 only those that no longer fit twice (20480 x 1024: 65 rows
// 0.80, 192 rows 0.95, 256 rows 1.62).
bool wide_applies(const GemmParams& p, const WideShape& sh) {
  if (g_opt_wide >= 0) return g_opt_wide != 0;
  const int sms = device_sms();
  long long ctas = 0;                                  // of the K-sliced kernel
  for (int i = 0; i < p.n_seg; ++i)
    ctas += (long long)((p.seg[i].n + kRowTile - 1) / kRowTile) * p.seg[i].split;
  const bool between = p.M > 128 && p.M <= 160;
  const bool short_k = p.k_blocks < 12;
  if (sh.rounds > 1) {
    if (ctas <= 2 * sms && short_k) return p.M > 208;
    if (ctas <= 2 * sms && 2 * ctas > 3 * sms && p.k_blocks >= 16) return p.M > 96 && !between;
    if (p.k_blocks >= 16) return p.M > (ctas >= 3 * sms ? 48 : 32);
    return p.M > 64 && !between;
  }
  if (p.M <= 48 || between) return false;
  if (p.pair.on) return true;
  if (short_k && sh.units >= max_pairs() && (p.seg[0].un > 224 ? p.M > 176 : p.M <= 64)) return false;
  if (p.seg[0].split == 4 && ctas <= sms && p.k_blocks > 64 && p.M > 160) return p.M > 224;
  return true;
}

// The launch on the wide kernel; kErrUnsupported where it has no layout for it or the K-sliced one is
// the faster.  `p` holds everything but
// the segments.
int run_wide(GemmParams p, const void* xq, int64_t K, const void* const* wq, const float* const* sw,
             void* const* y, const int64_t* N, const int64_t* ldy, const void* const* res,
             const int64_t* ld_res, const DenseArgs* dn, cudaStream_t stream) {
  const bool silu = p.pair.on != 0, flat = K % kBK != 0;
  const bool no_y = silu || p.push.n > 0 || (p.argmax.on && !p.argmax.store_logits);
  const long long es = p.out_dtype == BQ_DTYPE_F32 ? 4 : 2;
  for (int i = 0; i < p.n_seg; ++i) {
    Segment& s = p.seg[i];
    s.sw = sw[i];
    s.n = (int)(silu ? N[i] / 2 : N[i]);      // the gate/up form's N counts gate and up rows
    s.dense = (dn != nullptr && dn->kind[i] != 0) ? 1 : 0;
    s.y = no_y ? nullptr : y[i];
    s.ldy = no_y ? 0 : ldy[i];
    s.res = res ? res[i] : nullptr;
    s.ld_res = res ? ld_res[i] : 0;
    bool wide = true;
    if (p.push.n > 0) {
      wide = (p.push.ld * es) % 16 == 0;
      for (int d = 0; d < p.push.n; ++d) wide = wide && aligned_to(p.push.dst[d], 16);
    } else if (!no_y) {
      wide = aligned_to(y[i], 16) && (ldy[i] * es) % 16 == 0;
    }
    if (s.res) wide = wide && aligned_to(s.res, 16) && (s.ld_res * es) % 16 == 0;
    s.wide = wide ? 1 : 0;
  }
  WideShape sh;
  if (int rc = plan_wide(p, sh, flat)) return rc;
  if (!wide_applies(p, sh)) return kErrUnsupported;
  // the caller's scratch for the greedy pick has a pair per row and 128 vocabulary rows
  if (p.argmax.on && argmax_slots(sh) > (p.seg[0].n + kRowTile - 1) / kRowTile) return kErrUnsupported;
  auto map = [&](CUtensorMap* m, const void* ptr, long long rows, bool dense, int box_rows) {
    // a 16-bit operand is described by its bytes: [rows, 2K]
    return make_map_kb(m, ptr, rows, dense ? 2 * K : K, box_rows, sh.ring[dense ? 1 : 0].kb_stage, flat);
  };
  WeightMaps maps;
  memset(&maps, 0, sizeof(maps));
  CUtensorMap tm_x;
  for (int i = 0; i < p.n_seg; ++i)
    if (int rc = map(&maps.w[i], wq[i], p.seg[i].n, p.seg[i].dense != 0, p.seg[i].un / 2)) return rc;
  if (silu)
    if (int rc = map(&maps.w[1], p.pair.wq_up, p.seg[0].n, false, p.seg[0].un / 2)) return rc;
  if (int rc = map(&tm_x, xq, p.M, false, sh.m_half)) return rc;
  CUtensorMap tm_xd = tm_x;
  if (dn != nullptr)
    if (int rc = map(&tm_xd, dn->x, p.M, true, sh.m_half)) return rc;
  return launch_wide(tm_x, tm_xd, maps, p, sh, stream);
}

// Tiles of a plain prefill launch: 256, 192, 128 or 64 columns (the sums are the same, tile by tile; whole
// 128-byte pieces of 16-bit output), and the last columns of its widest weight as 128-column tiles that
// are visited last, where that evens out the last round.  A launch takes as long as its busiest CTA pair
// (tiles are dealt out in turn), a tile its columns plus a part that does not shrink with them: the
// activation rows' loads and MMA passes, the epilogue.  Measured, us with tiles of 256 / 192 / 128 columns:
// 4096 x 12288 at 300 rows 34.3 / 28.5 / 21.9, at 600 35.6 / 30.5 / 36.9, at 1100 64.0 / 53.9 / 56.3, at 1500
// 66.4 / 60.2 / 62.8, at 3000 115.9 / 121.5 / 127.4: one round of n columns costs n + 128 within 6 % (128 columns alone,
// with their deeper ring, n + 114).  Of 13 weights at 16 batches of 257 to 4000 rows, the choices timed in turn, the rule's is
// more than 3 % behind the best at 7 of 208 (2560 x 7680 at 2600 rows 43.9 where 128 columns take 41.5, 15360 x 5120
// at 1100 rows 78.8 with a split and 76.4 without; the others below 0.7 us).
// 64 columns where half of the pairs hold such tiles: a K block's turn is shorter by more than its share of the round, us with 128
// and with 64: 1024 x 4096 at 413 rows fp32 9.8 / 8.6, 16-bit 9.1 / 8.2, 1024 x 12288 18.3 / 16.5, 256 x 1024 at 2000
// rows 5.6 / 5.1; at more tiles the gain goes, 48 tiles of 1024 x 4096 9.1 / 8.7, 64 tiles 9.3 / 9.0 (2048 x 1024 5.6 / 5.6).  Of K
// below 8 blocks 512 x 512 at 512 rows takes 5.1 / 4.5; those stay at 128, as above.  Split: q, k and v of 8192 + 1024 + 1024 columns at 1500 rows
// 58.0 -> 54.8, 2560 x 7680 at 4096 rows 76.8 -> 69.7 (both before the issue loops were walked by whole warps).
struct TilePlan {
  int cols;            // columns of a tile
  int split;           // weight whose end becomes a segment of 128-column tiles, -1: none
  int64_t split_at;    // its first column there
};
constexpr int kTileFixedCols = 128;

TilePlan plan_tiles(const int64_t* N, const int* dense, int n_seg, int m_tiles, int k_blocks, bool may_split) {
  TilePlan best{kPairTile, -1, 0};
  if (g_opt_pair_narrow >= 0) {
    best.cols = g_opt_pair_narrow == 0 ? kPairTile : (g_opt_pair_narrow == 1 ? kPairTile / 2 : (int)g_opt_pair_narrow);
    return best;
  }
  const long long pairs = device_sms() / 2 > 0 ? device_sms() / 2 : 1;
  int widest = -1;
  for (int i = 0; i < n_seg; ++i)
    if ((dense == nullptr || dense[i] == 0) && (widest < 0 || N[i] > N[widest])) widest = i;
  if (widest < 0) return best;
  // cost of `wide` tiles of n columns, then `small` ones of 128, dealt out in turn
  auto cost_of = [&](long long wide, int n, long long small) {
    const long long cw = n + kTileFixedCols, cs = kPairTile / 2 + kTileFixedCols;
    const long long full = wide / pairs, r = wide % pairs;
    const long long first = pairs - r;                   // small tiles that level the pairs out
    if (small <= first) {
      const long long a = (full + (r > 0 ? 1 : 0)) * cw, b = full * cw + (small > 0 ? cs : 0);
      return a > b ? a : b;
    }
    const long long extra = small - first;
    const long long a = r > 0 ? (full + 1) * cw + (extra + pairs - 1) / pairs * cs : 0;
    const long long b = full * cw + cs + (extra > r ? (extra - r + pairs - 1) / pairs * cs : 0);
    return a > b ? a : b;
  };
  auto tiles_of = [&](int n, int64_t less) {
    long long tiles = 0;
    for (int i = 0; i < n_seg; ++i)
      if (dense == nullptr || dense[i] == 0) tiles += ((i == widest ? N[i] - less : N[i]) + n - 1) / n * m_tiles;
    return tiles;
  };
  long long best_cost = 0;
  for (int n = kPairTile; n >= 128; n -= 64) {
    if (n == 192 && k_blocks < 8) continue;              // so short a tile is mostly the fixed part
    const long long cost = cost_of(tiles_of(n, 0), n, 0);
    if (best_cost == 0 || cost < best_cost) { best = TilePlan{n, -1, 0}; best_cost = cost; }
  }
  if (k_blocks >= 8 && 2 * tiles_of(64, 0) <= pairs) return TilePlan{64, -1, 0};
  if (!may_split || n_seg == BQ_MAX_SEGMENTS || k_blocks < 8) return best;
  const int64_t columns = (N[widest] + kPairTile - 1) / kPairTile;
  for (int j = 1; j <= 6 && j < columns; ++j) {
    const int64_t at = (columns - j) * kPairTile, tail = N[widest] - at;
    const long long small = (tail + kPairTile / 2 - 1) / (kPairTile / 2) * m_tiles;
    const long long cost = cost_of(tiles_of(kPairTile, tail), kPairTile, small);
    // a split has to give something: one tile's fixed part at least
    if (cost + kTileFixedCols < best_cost) { best = TilePlan{kPairTile, widest, at}; best_cost = cost; }
  }
  return best;
}

int run_grouped(const void* xq, const float* sx, int64_t M, int64_t K, int n_seg,
                const void* const* wq, const float* const* sw, void* const* y, const int64_t* N,
                const int64_t* ldy, int out_dtype, void* ws, size_t ws_bytes, void* stream_v,
                const void* const* res = nullptr,
                const int64_t* ld_res = nullptr, const PairSilu* pair = nullptr,
                int split_forced = 0, const PushParams* push = nullptr,
                const DenseArgs* dn = nullptr, const ArgmaxOut* am = nullptr, const QuantIn* qi = nullptr) {
  if ((qi == nullptr && (!xq || !sx)) || (qi != nullptr && !qi->x) || !wq || !sw || !y || !N || !ldy || M <= 0 || K <= 0) return kErrBadArg;
  if (n_seg < 1 || n_seg > BQ_MAX_SEGMENTS) return kErrBadArg;
  if (out_dtype != BQ_DTYPE_F32 && out_dtype != BQ_DTYPE_BF16 && out_dtype != BQ_DTYPE_F16)
    return kErrBadArg;
  if (ws == nullptr || ws_bytes < 16u || !aligned_to(ws, 16)) return kErrWorkspace;
  if (K % 16 || !aligned_to(qi != nullptr ? qi->x : xq, 16)) return kErrUnsupported;
  if (M > 0x7fffff00LL || K > 0x7fffff00LL) return kErrTooLarge;
  const int out_align = out_dtype == BQ_DTYPE_F32 ? 16 : 8;
  for (int i = 0; i < n_seg; ++i) {   // argument checks first: no CUDA call before they pass
    const bool is_dense = dn != nullptr && dn->kind[i] != 0;
    if (!wq[i] || (!sw[i] && !is_dense) || N[i] <= 0) return kErrBadArg;
    if (N[i] % (is_dense ? 4 : 16) || !aligned_to(wq[i], 16)) return kErrUnsupported;
    if ((pair == nullptr || pair->prefill) && push == nullptr &&
        !(am != nullptr && !am->store_logits)) {   // forms that write y
      if (!y[i]) return kErrBadArg;
      if (ldy[i] < N[i] || ldy[i] % 4 || !aligned_to(y[i], out_align)) return kErrUnsupported;
    }
    if (N[i] > 0x7fffff00LL) return kErrTooLarge;
  }
  const bool stream_path = M <= g_opt_stream_max_m;
  if (qi != nullptr) {
    // the weight-streaming kernel alone has this form: the others read codes and scale, which are not given.  Its
    // rings are cut to the activation, so forced depths are left to the two launches.
    if (!stream_path || dn || push || am || pair || g_opt_wide > 0 || g_opt_stages > 0 || g_opt_b_stages != 0 ||
        M > BQ_LINEAR_MAX_ROWS || (qi->words != nullptr && n_seg != 1) ||
        (qi->words == nullptr &&
         !quantize_inside_pays(M, K, qi->dtype == BQ_DTYPE_F32 ? 4 : 2, n_seg, N, static_cast<cudaStream_t>(stream_v))))
      return kErrUnsupported;
  }
  if (dn != nullptr) {
    if (pair || push || res) return kErrUnsupported;
    // prefill sizes: 16-bit weights of one tile column (gates); wider ones are a library GEMM's business
    for (int i = 0; i < n_seg && !stream_path; ++i)
      if (dn->kind[i] != 0 && N[i] > kPairTile) return kErrUnsupported;
    if (!dn->x || (dn->dtype != BQ_DTYPE_BF16 && dn->dtype != BQ_DTYPE_F16)) return kErrBadArg;
    if (!aligned_to(dn->x, 16)) return kErrUnsupported;
  }
  if (pair && stream_path == (pair->prefill != 0)) return kErrUnsupported;   // each form has its regime
  if (pair && (res || n_seg != 1)) return kErrBadArg;
  if (push) {
    if (res || n_seg != 1) return kErrBadArg;
    // the prefill kernel stores 16-byte pieces
    if (!stream_path) {
      const long long es = out_dtype == BQ_DTYPE_F32 ? 4 : 2;
      if ((push->ld * es) % 16) return kErrUnsupported;
      for (int d = 0; d < push->n; ++d)
        if (!aligned_to(push->dst[d], 16)) return kErrUnsupported;
    }
  }
  if (res != nullptr) {
    if (ld_res == nullptr) return kErrUnsupported;
    for (int i = 0; i < n_seg; ++i)
      if (res[i] && (ld_res[i] < N[i] || ld_res[i] % 4 || !aligned_to(res[i], out_align)))
        return kErrUnsupported;
  }
  if (int rc = configure_once()) return rc;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_v);

  GemmParams p;
  memset(&p, 0, sizeof(p));
  WeightMaps maps;
  memset(&maps, 0, sizeof(maps));
  p.n_seg = n_seg;
  p.sx = sx;
  p.M = (int)M;
  p.k_blocks = (int)((K + kBK - 1) / kBK);
  p.k_blocks_dense = (int)((2 * K + kBK - 1) / kBK);
  p.dense_fmt = (dn != nullptr && dn->dtype == BQ_DTYPE_BF16) ? 1 : 0;
  p.out_dtype = out_dtype;
  if (qi != nullptr) {
    p.quant = *qi;
    p.quant.n8 = (int)(M * K / 8);
    p.quant_k = (int)K;
  }
  // the sticky status word is the 4th word of the scratch, as in the quantizer
  p.status = static_cast<unsigned int*>(ws) + 3;
  if (pair) {
    p.pair = *pair;
    p.pair.on = 1;
    p.pair.words = static_cast<unsigned int*>(ws);
  }
  if (am) {
    if (!stream_path || pair || push || res || dn || n_seg != 1) return kErrUnsupported;
    p.argmax = *am;
    p.argmax.on = 1;
  }
  if (push) {
    p.push = *push;
    p.push.done = static_cast<unsigned int*>(ws);   // first scratch word: zero between launches
    // second scratch word: the launch's running max |h| where the ranks want it
    p.push.amax_local = (push->amax_dst[0] != nullptr) ? static_cast<unsigned int*>(ws) + 1 : nullptr;
  }

  if (stream_path && qi == nullptr && (p.M > 32 || g_opt_wide > 0)) {
    const int rc = run_wide(p, xq, K, wq, sw, y, N, ldy, res, ld_res, dn, stream);
    if (rc != kErrUnsupported) return rc;
  }
  const bool pair_path = !stream_path;
  p.m_tiles = pair_path ? (int)((M + kPairTile - 1) / kPairTile) : (int)((M + kRowTile - 1) / kRowTile);
  // plain prefill form: the tiles' columns, and perhaps the end of a weight as a segment of its own
  const void* part_w[BQ_MAX_SEGMENTS];
  const float* part_sw[BQ_MAX_SEGMENTS];
  void* part_y[BQ_MAX_SEGMENTS];
  const void* part_res[BQ_MAX_SEGMENTS];
  int64_t part_n[BQ_MAX_SEGMENTS], part_ld[BQ_MAX_SEGMENTS], part_ld_res[BQ_MAX_SEGMENTS];
  int part_kind[BQ_MAX_SEGMENTS];
  DenseArgs part_dn;
  TilePlan plan{kPairTile, -1, 0};
  if (pair_path && pair == nullptr) {
    plan = plan_tiles(N, dn != nullptr ? dn->kind : nullptr, n_seg, p.m_tiles, p.k_blocks, push == nullptr);
    if (plan.split >= 0) {
      const size_t es = out_dtype == BQ_DTYPE_F32 ? 4 : 2;
      for (int i = 0; i <= n_seg; ++i) {
        const int from = i < n_seg ? i : plan.split;
        const int64_t at = i < n_seg ? 0 : plan.split_at;
        part_w[i] = static_cast<const uint8_t*>(wq[from]) + at * K;
        part_sw[i] = sw[from];
        part_y[i] = static_cast<uint8_t*>(y[from]) + at * es;
        part_n[i] = i == plan.split ? plan.split_at : N[from] - at;
        part_ld[i] = ldy[from];
        part_res[i] = res != nullptr && res[from] != nullptr ? static_cast<const uint8_t*>(res[from]) + at * es : nullptr;
        part_ld_res[i] = res != nullptr ? ld_res[from] : 0;
        part_kind[i] = i < n_seg && dn != nullptr ? dn->kind[i] : 0;
      }
      wq = part_w; sw = part_sw; y = part_y; N = part_n; ldy = part_ld;
      if (res != nullptr) { res = part_res; ld_res = part_ld_res; }
      if (dn != nullptr) { part_dn = DenseArgs{dn->x, dn->dtype, part_kind}; dn = &part_dn; }
      p.n_seg = ++n_seg;
    }
  }
  const bool plain_pair = pair_path && pair == nullptr;
  OutMaps ymaps;
  memset(&ymaps, 0, sizeof(ymaps));
  int tiles = 0;
  for (int i = 0; i < n_seg; ++i) {
    p.seg[i].sw = sw[i];
    const bool no_y = (pair && !pair->prefill) || push || (am != nullptr && !am->store_logits);
    p.seg[i].y = no_y ? nullptr : y[i];
    p.seg[i].ldy = no_y ? 0 : ldy[i];
    p.seg[i].split_forced = split_forced;
    p.seg[i].res = res ? res[i] : nullptr;
    p.seg[i].ld_res = res ? ld_res[i] : 0;
    p.seg[i].n = (int)N[i];
    p.seg[i].dense = (dn != nullptr && dn->kind[i] != 0) ? 1 : 0;
    p.seg[i].tile_begin = tiles;
    if (plain_pair)     // a 16-bit weight is one tile column, in the MMA N granularity of a pair
      p.seg[i].un = p.seg[i].dense ? (int)((N[i] + 31) / 32 * 32)
                                   : (plan.split >= 0 && i == n_seg - 1 ? kPairTile / 2 : plan.cols);
    const int tile_n = plain_pair ? p.seg[i].un : (pair_path ? kPairTile / 2 : kRowTile);
    if (pair_path && res != nullptr && res[i] != nullptr) {
      const size_t es = out_dtype == BQ_DTYPE_F32 ? 4 : 2;
      p.seg[i].wide = aligned_to(res[i], 16) && (ld_res[i] * es) % 16 == 0 ? 1 : 0;
    }
    const long long nt = (N[i] + tile_n - 1) / tile_n;
    const long long add = stream_path ? nt : nt * p.m_tiles;
    if (tiles + add > 0x3fffffffLL) return kErrTooLarge;
    tiles += (int)add;
    if (pair_path && !no_y) {
      const size_t es = out_dtype == BQ_DTYPE_F32 ? 4 : 2;
      p.seg[i].y_tma = aligned_to(y[i], 16) && (ldy[i] * es) % 16 == 0 &&
                       make_out_map(&ymaps.y[i], y[i], M, N[i], ldy[i], out_dtype) == kOk;
    }
    if (pair_path && push && g_opt_push_tma) {
      // one map per destination rank over its [M, N shard] window (n_seg is 1 for a push)
      bool ok = true;
      for (int d = 0; d < push->n && ok; ++d)
        ok = make_out_map(&ymaps.y[d], push->dst[d], M, N[i], push->ld, out_dtype) == kOk;
      p.seg[i].y_tma = ok ? 1 : 0;
    }
    if (pair && pair->prefill) {
      // two maps over the two weights, 128-row boxes: one CTA of a pair loads gate rows, the other
      // the up rows of the same output columns
      if (int rc = make_map(&maps.w[0], wq[0], N[0], K, kRowTile)) return rc;
      if (int rc = make_map(&maps.w[1], pair->wq_up, N[0], K, kRowTile)) return rc;
    } else if (pair) {
      // two maps over the two weights, 64-row boxes: the kernel puts a tile together from both
      if (int rc = make_map(&maps.w[0], wq[0], N[0] / 2, K, kRowTile / 2)) return rc;
      if (int rc = make_map(&maps.w[1], pair->wq_up, N[0] / 2, K, kRowTile / 2)) return rc;
    } else {
      // a 16-bit weight is described by its bytes: [N, 2K]
      const int box_rows = plain_pair ? p.seg[i].un / 2 : kRowTile;
      if (int rc = make_map(&maps.w[i], wq[i], N[i], p.seg[i].dense ? 2 * K : K, box_rows)) return rc;
    }
  }
  p.total_tiles = tiles;
  CUtensorMap tm_x;
  if (stream_path) {
    const int mma_n = (int)(((M + 15) / 16) * 16);
    if (qi != nullptr) return launch_stream(maps.w[0], maps.w[0], maps, p, stream);   // no map of the activation
    if (int rc = make_map(&tm_x, xq, M, K, mma_n)) return rc;
    CUtensorMap tm_xd = tm_x;
    if (dn != nullptr)
      if (int rc = make_map(&tm_xd, dn->x, M, 2 * K, mma_n)) return rc;
    return launch_stream(tm_x, tm_xd, maps, p, stream);
  }
  if (int rc = make_map(&tm_x, xq, M, K, kRowTile)) return rc;
  CUtensorMap tm_xd = tm_x;
  if (dn != nullptr)
    if (int rc = make_map(&tm_xd, dn->x, M, 2 * K, kRowTile)) return rc;
  return launch_pair(tm_x, tm_xd, maps, ymaps, p, stream);
}

}  // namespace

extern "C" int bq_gemm_w8a8_grouped(const void* xq, const float* sx, int64_t M, int64_t K, int n_seg,
                                    const void* const* wq, const float* const* sw, void* const* y,
                                    const int64_t* N, const int64_t* ldy, int out_dtype, void* ws,
                                    size_t ws_bytes, void* stream_v) {
  return run_grouped(xq, sx, M, K, n_seg, wq, sw, y, N, ldy, out_dtype, ws, ws_bytes, stream_v);
}

extern "C" int bq_linear_w8a8(const void* x, int dtype, int64_t M, int64_t K, int n_seg, const void* const* wq,
                              const float* const* sw, const void* residual, int64_t ld_res, void* const* y,
                              const int64_t* N, const int64_t* ldy, void* ws, size_t ws_bytes, void* stream) {
  if (x == nullptr || (residual != nullptr && n_seg != 1)) return kErrBadArg;
  const QuantIn qi{x, dtype, 0, nullptr, 0};
  const void* rs[1] = {residual};
  const int64_t ldrs[1] = {ld_res};
  return run_grouped(nullptr, nullptr, M, K, n_seg, wq, sw, y, N, ldy, dtype, ws, ws_bytes, stream,
                     residual != nullptr ? rs : nullptr, residual != nullptr ? ldrs : nullptr, nullptr, 0, nullptr, nullptr,
                     nullptr, &qi);
}

extern "C" int bq_project_mixed(const void* xq, const float* sx, const void* x_dense, int dense_dtype,
                                int64_t M, int64_t K, int n_seg, const void* const* w,
                                const float* const* sw, const int* kind, void* const* y,
                                const int64_t* N, const int64_t* ldy, int out_dtype, void* ws,
                                size_t ws_bytes, void* stream_v) {
  if (kind == nullptr) return kErrBadArg;
  bool any_dense = false;
  for (int i = 0; i < n_seg && i < BQ_MAX_SEGMENTS; ++i) any_dense = any_dense || kind[i] != 0;
  if (!any_dense)
    return run_grouped(xq, sx, M, K, n_seg, w, sw, y, N, ldy, out_dtype, ws, ws_bytes, stream_v);
  if (out_dtype != dense_dtype) return kErrUnsupported;   // F.linear returns the activation's type
  const DenseArgs dn{x_dense, dense_dtype, kind};
  return run_grouped(xq, sx, M, K, n_seg, w, sw, y, N, ldy, out_dtype, ws, ws_bytes, stream_v,
                     nullptr, nullptr, nullptr, 0, nullptr, &dn);
}

extern "C" int bq_gemm_w8a8(const void* xq, const void* wq, const float* sx, const float* sw,
                            void* y, int out_dtype, int64_t M, int64_t N, int64_t K, int64_t ldy,
                            void* ws, size_t ws_bytes, void* stream) {
  const void* wqs[1] = {wq};
  const float* sws[1] = {sw};
  void* ys[1] = {y};
  const int64_t Ns[1] = {N};
  const int64_t ldys[1] = {ldy};
  return bq_gemm_w8a8_grouped(xq, sx, M, K, 1, wqs, sws, ys, Ns, ldys, out_dtype, ws, ws_bytes,
                              stream);
}

extern "C" size_t bq_lm_head_argmax_workspace_bytes(int64_t M, int64_t N) {
  if (M <= 0 || N <= 0) return 0;
  return static_cast<size_t>((N + kRowTile - 1) / kRowTile) * static_cast<size_t>(M) * sizeof(uint2);
}

extern "C" int bq_lm_head_argmax(const void* xq, const void* wq, const float* sx, const float* sw,
                                 int out_dtype, int64_t M, int64_t N, int64_t K, void* logits_or_null,
                                 int64_t ldy, int64_t* idx_out, void* partial, size_t partial_bytes,
                                 void* ws, size_t ws_bytes, void* stream) {
  if (!idx_out || !partial || M <= 0 || N <= 0) return kErrBadArg;
  if (M > g_opt_stream_max_m) return kErrUnsupported;
  if (partial_bytes < bq_lm_head_argmax_workspace_bytes(M, N) || !aligned_to(partial, 8) ||
      !aligned_to(idx_out, 8))
    return kErrWorkspace;
  ArgmaxOut am;
  memset(&am, 0, sizeof(am));
  am.store_logits = logits_or_null != nullptr ? 1 : 0;
  am.partial = static_cast<uint2*>(partial);
  const void* wqs[1] = {wq};
  const float* sws[1] = {sw};
  void* ys[1] = {logits_or_null};
  const int64_t Ns[1] = {N};
  const int64_t ldys[1] = {ldy};
  // K is not split: every tile's logits are final inside one CTA
  if (int rc = run_grouped(xq, sx, M, K, 1, wqs, sws, ys, Ns, ldys, out_dtype, ws, ws_bytes, stream,
                           nullptr, nullptr, nullptr, 1, nullptr, nullptr, &am))
    return rc;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((unsigned)M, 1, 1);
  cfg.blockDim = dim3(128, 1, 1);
  cfg.stream = static_cast<cudaStream_t>(stream);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = g_opt_pdl ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, argmax_finish_kernel, am.partial, g_argmax_slots, (int)M,
                                           reinterpret_cast<long long*>(idx_out));
  if (e != cudaSuccess) { (void)cudaGetLastError(); return kErrLaunch; }
  return kOk;
}

namespace {
void set_next(PairSilu* pair, const void* next, int64_t bytes) {
  pair->next = static_cast<const uint8_t*>(next);
  pair->next_bytes = next != nullptr && bytes >= kNextFrom ? kNextBytes : 0u;
  pair->next_warp = bytes >= kNextFirstWarpFrom ? 0 : kStreamWarps - 1;
}
}  // namespace

extern "C" int bq_gate_up_silu_quant_w8a8(const void* xq, const float* sx, const void* wq_gate, const void* wq_up,
                                          const float* sw_gate, const float* sw_up, int64_t M, int64_t I, int64_t K,
                                          int act_dtype, void* hq_out, float* sh_out, void* ws, size_t ws_bytes,
                                          void* stream) {
  return bq_gate_up_silu_quant_next_w8a8(xq, sx, wq_gate, wq_up, sw_gate, sw_up, M, I, K, act_dtype, hq_out, sh_out, nullptr, 0,
                                         ws, ws_bytes, stream);
}

extern "C" int bq_gate_up_silu_quant_next_w8a8(const void* xq, const float* sx, const void* wq_gate, const void* wq_up,
                                               const float* sw_gate, const float* sw_up, int64_t M, int64_t I, int64_t K,
                                               int act_dtype, void* hq_out, float* sh_out, const void* next,
                                               int64_t next_bytes, void* ws, size_t ws_bytes, void* stream) {
  if (!aligned_to(next, 16)) return kErrUnsupported;
  if (!wq_gate || !wq_up || !sw_gate || !sw_up || !hq_out || !sh_out || I <= 0) return kErrBadArg;
  if (I % (kRowTile / 2) || !aligned_to(hq_out, 2) || !aligned_to(wq_up, 16)) return kErrUnsupported;
  PairSilu pair;
  memset(&pair, 0, sizeof(pair));
  pair.wq_up = wq_up;
  pair.sw_up = sw_up;
  pair.hq = static_cast<uint8_t*>(hq_out);
  pair.ld_hq = I;
  pair.sh = sh_out;
  set_next(&pair, next, next_bytes);
  const void* wqs[1] = {wq_gate};
  const float* sws[1] = {sw_gate};
  void* ys[1] = {nullptr};
  const int64_t Ns[1] = {2 * I};
  const int64_t ldys[1] = {0};
  // K slices as the gate weight alone would get them: every dot product is then summed in the
  // order of the separate gate and up GEMMs
  const int k_blocks = (int)((K + kBK - 1) / kBK);
  const int split = (K > 0 && K <= 0x7fffff00LL) ? split_for_weight((int)I, k_blocks) : 1;
  return run_grouped(xq, sx, M, K, 1, wqs, sws, ys, Ns, ldys, act_dtype, ws, ws_bytes, stream,
                     nullptr, nullptr, &pair, split);
}

// Few rows: where the CTAs of the down projection cast h for themselves.  It takes the grid-wide exchange and the
// cast out of the gate/up launch, behind whose stream HBM idles for them; down's CTAs do the cast while their first
// weights arrive, 4 chunks of 16 values a thread and round of loads (5 spill), a round 2 to 3 us.
//
// Rows: us of one MLP in a graph, separate launches -> this.  One round, 4096 x 12288: 1 row 34.4 -> 30.9, 4 rows 34.8 ->
// 32.9, 6 rows 35.5 -> 33.8.  Two: 6 rows of 4096 x 14336 39.5 -> 38.4, of 3584 x 18944 43.8 -> 42.0; of 8192 x 12288
// 4 rows 58.9 -> 58.2, 6 rows 58.9 and 59.9.  Three: 6 rows of 6144 x 14080 52.2 and 54.1, 1 row 51.7 -> 49.6.  The last
// two lose less than what a call made outside a graph saves where gate/up has more CTAs than are resident at once and
// would go through a [M, 2I] buffer: 6 rows of 4096 x 28160 66.5 and 68.3 in a graph, 87.8 -> 68.2 eager.  Four layers
// of hidden 4096, before slices were handed over: 8 rows 240.5 and 238.3, 16 rows 249 and 257.
// Weights: a smaller down weight has arrived before the cast is done.  Hidden 2560 (20 MB), four layers: 4 rows 241.8 and
// 241.3, 8 rows 312.3 and 313.8; hidden 2048 (13 MB), 1 row 123.7 and 124.5.
// Width: the slice of h, in tiles padded to 16 rows, may take half of the rings' memory (see cast_stages) and has to leave
// four weight tiles.
namespace {
bool mlp_sizes_go(int64_t M, int64_t I, int64_t N, int act_dtype) {
  return M > 0 && I > 0 && N > 0 && I <= 0x3fffff00LL && N <= 0x7fffff00LL && I % (kRowTile / 2) == 0 && N % 16 == 0 &&
         M <= (act_dtype == BQ_DTYPE_F32 ? BQ_MLP_MAX_ROWS / 2 : BQ_MLP_MAX_ROWS) && I * N >= BQ_MLP_MIN_WEIGHT &&
         M <= g_opt_stream_max_m && g_opt_wide <= 0 && g_opt_stages <= 0 && g_opt_b_stages == 0 && g_opt_smem_cap <= 0 &&
         g_opt_quant_inside < 0;
}
bool mlp_slice_fits(int64_t M, int64_t I, int64_t N, int sms) {
  const int blocks = (int)((I + kBK - 1) / kBK), split = split_for_weight(N, blocks);
  const int budget = stream_budget((N + kRowTile - 1) / kRowTile * split, sms) - handover_bytes(M, split);
  return cast_stages(budget, (int)((M + 15) / 16 * 16) * kBK, (blocks + split - 1) / split) > 0;
}
}  // namespace

extern "C" int bq_mlp_w8a8_takes(int64_t M, int64_t I, int64_t N, int act_dtype) {
  if (!mlp_sizes_go(M, I, N, act_dtype)) return 0;
  const int sms = device_sms();
  return sms > 0 && mlp_slice_fits(M, I, N, sms) ? 1 : 0;
}

extern "C" int bq_mlp_w8a8(const void* xq, const float* sx, const void* wq_gate, const void* wq_up, const void* wq_down,
                           const float* sw_gate, const float* sw_up, const float* sw_down, const void* residual,
                           int64_t ld_res, int64_t M, int64_t K, int64_t I, int64_t N, int act_dtype, void* h, void* y,
                           int64_t ldy, void* ws, size_t ws_bytes, void* stream) {
  if (!xq || !sx || !wq_gate || !wq_up || !wq_down || !sw_gate || !sw_up || !sw_down || !h || !y || M <= 0 || K <= 0 ||
      I <= 0 || N <= 0)
    return kErrBadArg;
  if (act_dtype != BQ_DTYPE_F32 && act_dtype != BQ_DTYPE_BF16 && act_dtype != BQ_DTYPE_F16) return kErrBadArg;
  // Everything the second launch would refuse is refused before the first one runs.
  const int out_align = act_dtype == BQ_DTYPE_F32 ? 16 : 8;
  if (!aligned_to(wq_up, 16) || !aligned_to(wq_down, 16) || !aligned_to(h, 16) || ldy < N || ldy % 4 ||
      !aligned_to(y, out_align))
    return kErrUnsupported;
  if (residual != nullptr && (ld_res < N || ld_res % 4 || !aligned_to(residual, out_align))) return kErrUnsupported;
  if (!mlp_sizes_go(M, I, N, act_dtype)) return kErrUnsupported;
  const int sms = device_sms();
  if (sms <= 0) return kErrLaunch;
  if (!mlp_slice_fits(M, I, N, sms)) return kErrUnsupported;
  PairSilu pair;
  memset(&pair, 0, sizeof(pair));
  pair.wq_up = wq_up;
  pair.sw_up = sw_up;
  pair.h = h;
  set_next(&pair, wq_down, I * N);
  const void* wqs[1] = {wq_gate};
  const float* sws[1] = {sw_gate};
  void* none[1] = {nullptr};
  const int64_t Ns[1] = {2 * I}, zero[1] = {0};
  const int k_blocks = (int)((K + kBK - 1) / kBK);
  if (int rc = run_grouped(xq, sx, M, K, 1, wqs, sws, none, Ns, zero, act_dtype, ws, ws_bytes, stream, nullptr, nullptr,
                           &pair, K <= 0x7fffff00LL ? split_for_weight(I, k_blocks) : 1))
    return rc;
  const QuantIn qi{h, act_dtype, 0, static_cast<unsigned int*>(ws), 0};
  const void* wds[1] = {wq_down};
  const float* sds[1] = {sw_down};
  void* ys[1] = {y};
  const int64_t Nd[1] = {N}, ldys[1] = {ldy}, ldrs[1] = {ld_res};
  const void* rs[1] = {residual};
  const int rc = run_grouped(nullptr, nullptr, M, I, 1, wds, sds, ys, Nd, ldys, act_dtype, ws, ws_bytes, stream,
                             residual != nullptr ? rs : nullptr, residual != nullptr ? ldrs : nullptr, nullptr, 0, nullptr,
                             nullptr, nullptr, &qi);
  if (rc == kOk) return kOk;
  // The first launch leaves max |h| in the scratch and only the second returns it to zero; whoever takes the scratch next
  // would start from it.
  if (cudaMemsetAsync(ws, 0, 8, static_cast<cudaStream_t>(stream)) != cudaSuccess) (void)cudaGetLastError();
  return rc == kErrUnsupported ? kErrLaunch : rc;      // unsupported cannot be: checked above
}

extern "C" int bq_gate_up_silu_w8a8(const void* xq, const float* sx, const void* wq_gate,
                                    const void* wq_up, const float* sw_gate, const float* sw_up,
                                    int64_t M, int64_t I, int64_t K, int act_dtype, void* h_out,
                                    int64_t ld_h, float* sh_out, void* ws, size_t ws_bytes,
                                    void* stream) {
  if (!wq_gate || !wq_up || !sw_gate || !sw_up || !h_out || !sh_out || I <= 0) return kErrBadArg;
  if (I % 16 || !aligned_to(wq_up, 16)) return kErrUnsupported;
  PairSilu pair;
  memset(&pair, 0, sizeof(pair));
  pair.prefill = 1;
  pair.wq_up = wq_up;
  pair.sw_up = sw_up;
  pair.sh = sh_out;
  const void* wqs[1] = {wq_gate};
  const float* sws[1] = {sw_gate};
  void* ys[1] = {h_out};
  const int64_t Ns[1] = {I};
  const int64_t ldys[1] = {ld_h};
  return run_grouped(xq, sx, M, K, 1, wqs, sws, ys, Ns, ldys, act_dtype, ws, ws_bytes, stream,
                     nullptr, nullptr, &pair);
}

namespace {
int fill_push(PushParams* pp, int n_peers, void* const* dst, int64_t ld, void* const* flags,
              int64_t width, size_t align, void* const* amax_slots = nullptr) {
  if (n_peers < 1 || n_peers > kMaxPeers || !dst || !flags) return kErrBadArg;
  if (ld < width || ld % 4) return kErrUnsupported;
  memset(pp, 0, sizeof(*pp));
  pp->n = n_peers;
  pp->ld = ld;
  for (int i = 0; i < n_peers; ++i) {
    if (!dst[i] || !flags[i]) return kErrBadArg;
    if (!aligned_to(dst[i], align) || !aligned_to(flags[i], 4)) return kErrUnsupported;
    pp->dst[i] = dst[i];
    pp->flag[i] = static_cast<unsigned int*>(flags[i]);
    if (amax_slots != nullptr) {
      if (!amax_slots[i]) return kErrBadArg;
      if (!aligned_to(amax_slots[i], 4)) return kErrUnsupported;
      pp->amax_dst[i] = static_cast<unsigned int*>(amax_slots[i]);
    }
  }
  return kOk;
}
}  // namespace

extern "C" int bq_gemm_w8a8_push(const void* xq, const void* wq, const float* sx, const float* sw,
                                 int out_dtype, int64_t M, int64_t N, int64_t K, int n_peers,
                                 void* const* y_dst, int64_t ldy, void* const* flags, void* ws,
                                 size_t ws_bytes, void* stream) {
  PushParams push;
  if (int rc = fill_push(&push, n_peers, y_dst, ldy, flags, N, out_dtype == BQ_DTYPE_F32 ? 16 : 8))
    return rc;
  const void* wqs[1] = {wq};
  const float* sws[1] = {sw};
  void* ys[1] = {nullptr};
  const int64_t Ns[1] = {N};
  const int64_t ldys[1] = {0};
  return run_grouped(xq, sx, M, K, 1, wqs, sws, ys, Ns, ldys, out_dtype, ws, ws_bytes, stream,
                     nullptr, nullptr, nullptr, 0, &push);
}

extern "C" int bq_gate_up_silu_push_w8a8(const void* xq, const float* sx, const void* wq_gate,
                                         const void* wq_up, const float* sw_gate,
                                         const float* sw_up, int64_t M,
                                         int64_t I, int64_t K, int act_dtype, int n_peers,
                                         void* const* h_dst, int64_t ld_h, void* const* flags,
                                         void* const* amax_slots, void* ws, size_t ws_bytes,
                                         void* stream) {
  if (!wq_gate || !wq_up || !sw_gate || !sw_up || I <= 0) return kErrBadArg;
  if (I % (kRowTile / 2) || !aligned_to(wq_up, 16)) return kErrUnsupported;
  // the max |h| of the shard travels with the prefill form only (decode sizes re-quantize the
  // gathered h in the kernel that waits for it)
  if (amax_slots != nullptr && M <= g_opt_stream_max_m) amax_slots = nullptr;
  PushParams push;
  if (int rc = fill_push(&push, n_peers, h_dst, ld_h, flags, I, act_dtype == BQ_DTYPE_F32 ? 8 : 4,
                         amax_slots))
    return rc;
  PairSilu pair;
  memset(&pair, 0, sizeof(pair));
  pair.wq_up = wq_up;
  pair.sw_up = sw_up;
  const void* wqs[1] = {wq_gate};
  const float* sws[1] = {sw_gate};
  void* ys[1] = {nullptr};
  const int64_t ldys[1] = {0};
  if (M > g_opt_stream_max_m) {
    // prefill sizes: the CTA-pair kernel, SiLU*mul in its epilogue, h pieces to every rank
    pair.prefill = 1;
    const int64_t Ns[1] = {I};
    return run_grouped(xq, sx, M, K, 1, wqs, sws, ys, Ns, ldys, act_dtype, ws, ws_bytes, stream,
                       nullptr, nullptr, &pair, 0, &push);
  }
  const int64_t Ns[1] = {2 * I};
  const int k_blocks = (int)((K + kBK - 1) / kBK);
  const int split = (K > 0 && K <= 0x7fffff00LL) ? split_for_weight(I, k_blocks) : 1;
  return run_grouped(xq, sx, M, K, 1, wqs, sws, ys, Ns, ldys, act_dtype, ws, ws_bytes, stream,
                     nullptr, nullptr, &pair, split, &push);
}

extern "C" int bq_wait_flag(const void* flag, void* seen, unsigned int count, void* status_word,
                            void* stream) {
  if (!flag || !seen || !status_word || count == 0) return kErrBadArg;
  if (!aligned_to(flag, 4) || !aligned_to(seen, 4) || !aligned_to(status_word, 4)) return kErrUnsupported;
  wait_flag_kernel<<<1, 1, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const unsigned int*>(flag), static_cast<unsigned int*>(seen), count,
      static_cast<unsigned int*>(status_word));
  if (cudaGetLastError() != cudaSuccess) return kErrLaunch;
  return kOk;
}

// One warp, lane d for rank d: the 4-byte word at `word` (a scale, a max) into `dst_words[d]`,
// then one arrival on that rank's counter, the word first (system-scope release on the
// counter).  One lane per rank so that the round trips to the ranks run side by side (a single
// thread walking four ranks took 12 us).
__global__ void word_push_kernel(const unsigned int* word, int n, PushParams dst) {
  const int d = threadIdx.x;
  if (d >= n) return;
  const unsigned int v = __ldcg(word);
  asm volatile("st.relaxed.sys.global.u32 [%0], %1;" ::"l"(dst.amax_dst[d]), "r"(v) : "memory");
  __threadfence_system();
  asm volatile("red.release.sys.global.add.u32 [%0], 1;" ::"l"(dst.flag[d]) : "memory");
}

extern "C" int bq_word_push(const void* word, int n_peers, void* const* dst_words, void* const* flags,
                            void* stream) {
  if (!word || !dst_words || !flags || n_peers < 1 || n_peers > kMaxPeers) return kErrBadArg;
  if (!aligned_to(word, 4)) return kErrUnsupported;
  PushParams pp;
  memset(&pp, 0, sizeof(pp));
  for (int i = 0; i < n_peers; ++i) {
    if (!dst_words[i] || !flags[i]) return kErrBadArg;
    if (!aligned_to(dst_words[i], 4) || !aligned_to(flags[i], 4)) return kErrUnsupported;
    pp.amax_dst[i] = static_cast<unsigned int*>(dst_words[i]);
    pp.flag[i] = static_cast<unsigned int*>(flags[i]);
  }
  word_push_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const unsigned int*>(word),
                                                                   n_peers, pp);
  if (cudaGetLastError() != cudaSuccess) return kErrLaunch;
  return kOk;
}

extern "C" int bq_wait_flag_scale(const void* flag, void* seen, unsigned int count, void* status_word,
                                  const void* amax_slots, int n_slots, int slots_hold_scales,
                                  float* scale_out, void* stream) {
  if (!flag || !seen || !status_word || !amax_slots || !scale_out || count == 0) return kErrBadArg;
  if (n_slots < 1 || n_slots > kMaxPeers) return kErrBadArg;
  if (!aligned_to(flag, 4) || !aligned_to(seen, 4) || !aligned_to(status_word, 4) ||
      !aligned_to(amax_slots, 4) || !aligned_to(scale_out, 4))
    return kErrUnsupported;
  wait_flag_scale_kernel<<<1, 1, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const unsigned int*>(flag), static_cast<unsigned int*>(seen), count,
      static_cast<unsigned int*>(status_word), static_cast<const unsigned int*>(amax_slots), n_slots,
      slots_hold_scales, scale_out);
  if (cudaGetLastError() != cudaSuccess) return kErrLaunch;
  return kOk;
}

extern "C" int bq_gemm_w8a8_residual(const void* xq, const void* wq, const float* sx, const float* sw,
                                     const void* residual, int64_t ld_res, void* y, int out_dtype,
                                     int64_t M, int64_t N, int64_t K, int64_t ldy, void* ws,
                                     size_t ws_bytes, void* stream) {
  if (residual == nullptr) return kErrBadArg;
  const void* wqs[1] = {wq};
  const float* sws[1] = {sw};
  void* ys[1] = {y};
  const int64_t Ns[1] = {N};
  const int64_t ldys[1] = {ldy};
  const void* rs[1] = {residual};
  const int64_t ldrs[1] = {ld_res};
  return run_grouped(xq, sx, M, K, 1, wqs, sws, ys, Ns, ldys, out_dtype, ws, ws_bytes, stream,
                     rs, ldrs);
}


extern "C" int bq_last_gemm_quantizes(void) { return g_last_quantizes; }

extern "C" int bq_last_gemm_launch(int64_t out[6]) {
  if (!out) return kErrBadArg;
  for (int i = 0; i < 6; ++i) out[i] = g_last_launch[i];
  return kOk;
}
