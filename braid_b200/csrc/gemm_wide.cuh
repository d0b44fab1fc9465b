// Weight-streaming GEMM on CTA pairs (the wide half of the decode regime, up to M = 256; HBM-bound,
// measured in GB/s).
//
// The batch sits on the MMA M side (lane = batch row of the accumulator in tensor memory) and a
// unit's weight rows on the N side.  A unit is a CTA pair (cta_group::2) and owns `un` weight rows
// over the WHOLE of K, `un` chosen so that the launch is one round of at most one CTA per SM.  That
// is what sets the speed of a short launch: nothing is summed across CTAs, so after the last MMA an
// accumulator goes from tensor memory to registers to the output, without staging, cluster
// barriers or a reduction.  Each CTA loads half of the batch and half of the unit's weight rows.
// Batch tiles are stored with the rows they have, not with those the MMA reads: rows beyond the
// batch are whatever follows in shared memory and only reach accumulator rows nobody reads.
//
// Two MMA shapes by batch: 128 and 256 rows (64 and 128 per CTA).  An MMA whose N is small costs
// what loading its M rows costs (measured 22 and 40 clocks for N <= 32 x K = 32), and a CTA issues
// K / 32 of them one after another.  That chain is why small batches stay on the K-sliced kernel
// (gemm_w8a8.cu): a 64-row form of this one took 3.6 us instead of 2.5 from the activation's arrival
// to the last MMA of a 4096 x 4096 weight; four graphed decoder layers were 4 % slower with it at
// 1 row and 1 % at 27, and it was not kept.  At 128 rows those layers (hidden 4096, bf16) take 341 us
// here and 376 on the K-sliced kernel (before both had kernels of their own per epilogue; 298 now).  Norm + greedy pick with logits
// over a 248320 x 4096 vocabulary, eager and repeated: 200 to 203 us at 64 rows, 205 at 128, at the clock that the power
// cap leaves.
//
// Sums.  Weights of few rows are summed in 2 or 4 K slices, each with an accumulator of its own,
// added in order at the end: the order of summation is a function of the weight's shape alone and
// that of the K-sliced kernel, so `project` equals per-weight calls bit for bit and results do not
// depend on the layout of a launch.
//
// Two rings with their own barriers and producer threads.  The weight ring takes what shared
// memory is left (bytes in flight per SM set the streaming rate) and starts filling at launch,
// before the previous kernel has finished; the activation ring waits for that kernel.  One
// tcgen05.commit per stage frees both slots: the activation producer watches the weight slot's
// barrier.  Weights too large for one round (a vocabulary) loop over units with two accumulators.
#pragma once

struct RingShape {
  int kb_stage;        // 128-byte K blocks per stage, loaded by one box per operand
  int a_block, w_block;      // bytes of one K block in the two rings
  int a_stages, w_stages;
};
struct WideShape {
  int mode;            // 1 / 2: 128- / 256-row MMA
  int units;           // units of the launch
  int grid;            // CTAs
  int rounds;          // units per pair, rounded up
  int nm;              // MMAs per K step: 2 in the gate/up form, 1 otherwise
  int m_half;          // batch rows per CTA, multiple of 8
  int flat;            // K is not a multiple of 128 bytes: K blocks are x positions, one per stage
  RingShape ring[2];   // of the units of e4m3 weights / of 16-bit weights
  int acc_cols;        // tensor-memory columns of one unit
  int tmem_cols;
  int ring_bytes;      // both rings, or the staging that reuses them
};

constexpr int kWideThreads = 384;     // warps 0 / 1 / 2 load weights, issue MMAs, load activations
constexpr int kWideWarps = kWideThreads / 32;
// Deepest rings: two barriers per weight slot, one per activation slot and four for the accumulators
// lie before the last 128 bytes of the barrier area (tensor-memory slot, abort flag, s_red).
constexpr int kWideMaxW = 40, kWideMaxA = 28;
static_assert(8 * (2 * kWideMaxW + kWideMaxA + 4) <= kBarrierBytes - 128, "the barriers overrun the flags");

// Where the accumulators of a CTA's batch rows lie in tensor memory (lanes x columns):
//   pair of 128   rows 0..63 in lanes 0..63 (columns of CTA 0's weight rows) and again in lanes
//                 64..127 (columns of CTA 1's): half as many columns as weight rows
//   pair of 256   rows 0..127 in lanes 0..127
template <int MODE>
struct LaneMap {
  static constexpr int kMmaM = 64 << MODE;
  static __device__ __forceinline__ int row0(int quad) { return (MODE == 1 ? quad & 1 : quad) * 32; }
  static __host__ __device__ __forceinline__ int cols(int un) { return MODE == 1 ? un / 2 : un; }
  static __device__ __forceinline__ int col0(int quad, int un) { return MODE == 1 ? (quad >> 1) * (un / 2) : 0; }
};

// 16 accumulator columns of this warp's lanes, the K slices added in order.
__device__ __forceinline__ void load_sums(uint32_t taddr, int split, int slice_cols, float (&v)[16]) {
  uint32_t r[16];
  tmem_ld16(taddr, r);
  tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
  for (int k = 1; k < split; ++k) {
    tmem_ld16(taddr + k * slice_cols, r);
    tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] += __uint_as_float(r[i]);
  }
}

// 16 scaled accumulator values -> (+ residual) -> output type -> memory.  `wide`: 16-byte accesses
// are aligned; otherwise 8-byte ones are.
template <typename T>
__device__ __forceinline__ void store16(T* dst, const float (&v)[16], bool wide) {
  using namespace bq::qd;
  if constexpr (sizeof(T) == 4) {
#pragma unroll
    for (int q = 0; q < 4; ++q)
      reinterpret_cast<float4*>(dst)[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
  } else {
    alignas(16) T t[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) t[i] = narrow<T>(v[i]);
    const uint4* w = reinterpret_cast<const uint4*>(t);
    if (wide) {
      reinterpret_cast<uint4*>(dst)[0] = w[0];
      reinterpret_cast<uint4*>(dst)[1] = w[1];
    } else {
      uint2* d = reinterpret_cast<uint2*>(dst);
      d[0] = make_uint2(w[0].x, w[0].y); d[1] = make_uint2(w[0].z, w[0].w);
      d[2] = make_uint2(w[1].x, w[1].y); d[3] = make_uint2(w[1].z, w[1].w);
    }
  }
}

// v <- float(T(v)) + float(res): the GEMM's own rounding, then the add's (the store rounds again).
template <typename T>
__device__ __forceinline__ void add_res16(float (&v)[16], const T* res, bool wide) {
  using namespace bq::qd;
  alignas(16) T r[16];
  if constexpr (sizeof(T) == 4) {
#pragma unroll
    for (int q = 0; q < 4; ++q) reinterpret_cast<uint4*>(r)[q] = ld_coherent16(res + 4 * q);
  } else if (wide) {
    reinterpret_cast<uint4*>(r)[0] = ld_coherent16(res);
    reinterpret_cast<uint4*>(r)[1] = ld_coherent16(res + 8);
  } else {
#pragma unroll
    for (int q = 0; q < 4; ++q) reinterpret_cast<uint2*>(r)[q] = ld_coherent8(res + 4 * q);
  }
  // the intrinsic: a plain + would be contracted with the scaling multiply for fp32 outputs
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __fadd_rn(widen(narrow<T>(v[i])), widen(r[i]));
}

// What an epilogue thread needs to know of its unit.
struct UnitOut {
  const GemmParams& p;
  const Segment& seg;
  int row0;            // weight row (output column) of this thread's first accumulator column
  int m;               // batch row of this thread
  bool row_ok;
};

template <typename T, int EPI>
__device__ __forceinline__ void store_chunk(const UnitOut& o, int c, float (&v)[16]) {
  const int col = o.row0 + c;
  if (!o.row_ok || col >= o.seg.n) return;        // n is a multiple of 16: a chunk is in or out ...
  const bool wide = o.seg.wide != 0;
  if constexpr (sizeof(T) == 2 && EPI != kResidual) {
    if (o.seg.n - col < 16) {                     // ... but a 16-bit weight's is one of 4
      T* const dst = static_cast<T*>(o.seg.y) + (long long)o.m * o.seg.ldy + col;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (col + 4 * q < o.seg.n)
          reinterpret_cast<uint2*>(dst)[q] = make_uint2(bq::qd::pack2<T>(v[4 * q], v[4 * q + 1]), bq::qd::pack2<T>(v[4 * q + 2], v[4 * q + 3]));
      return;
    }
  }
  if (EPI == kResidual || (EPI == kAny && o.seg.res != nullptr))
    add_res16<T>(v, static_cast<const T*>(o.seg.res) + (long long)o.m * o.seg.ld_res + col, wide);
  if (EPI != kAny || o.p.push.n == 0) {
    store16<T>(static_cast<T*>(o.seg.y) + (long long)o.m * o.seg.ldy + col, v, wide);
  } else {
    for (int d = 0; d < o.p.push.n; ++d)
      store16<T>(static_cast<T*>(o.p.push.dst[d]) + (long long)o.m * o.p.push.ld + col, v, wide);
  }
}

// The best of 16 logits after their rounding to the output type (see ArgmaxOut).
template <typename T>
__device__ __forceinline__ void argmax_chunk(const UnitOut& o, int c, const float (&v)[16], float& bv, int& bi) {
  using namespace bq::qd;
  const int col = o.row0 + c;
  if (col >= o.seg.n) return;
  // columns come in ascending order: what is not larger than the best so far loses, by its index if by nothing else
  float r[16];
  bool ordered = true;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    r[i] = widen(narrow<T>(v[i]));
    ordered = ordered && r[i] == r[i];
  }
  if (bi == kNoIndex) { bv = r[0]; bi = col; }
  if (ordered) {
#pragma unroll
    for (int i = 0; i < 16; ++i)
      if (r[i] > bv) { bv = r[i]; bi = col + i; }
  } else {
    for (int i = 0; i < 16; ++i)
      if (argmax_beats(r[i], col + i, bv, bi)) { bv = r[i]; bi = col + i; }
  }
}

// ---- gate/up form ---------------------------------------------------------------------------
// The unit's accumulator columns are `un` gate rows then the `un` up rows of the same output
// columns.  Only the lanes of real batch rows hold values, so the halves first go to shared
// memory -- rounded to the activation type T, as the plain GEMM would have stored them -- and
// every thread of the CTA then takes its share of h = T(T(silu(gate)) * up), the two roundings
// of the separate torch kernels (braid/model/mlp.py:48).  h replaces the gate half.
template <typename T>
struct PairTile {
  T* base;
  int pitch;     // elements per row: 2 un + 16 bytes, so that the lane-per-row writes spread over the banks
  int rows, un;
};

template <typename T>
__device__ __forceinline__ void pair_park(const PairTile<T>& t, uint32_t taddr, int row, bool row_ok, int col0, int cols,
                                          int split, int col_group, int n_groups, float sg, float su) {
  using namespace bq::qd;
  for (int c = col_group * 16; c < 2 * cols; c += 16 * n_groups) {
    float a[16];
    load_sums(taddr + c, split, 2 * cols, a);
    const bool up = c >= cols;
    const float sc = up ? su : sg;
    if (row_ok) {
      alignas(16) T v[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = narrow<T>(a[i] * sc);
      uint4* dst = reinterpret_cast<uint4*>(t.base + row * t.pitch + (up ? t.un + c - cols : c) + col0);
#pragma unroll
      for (int q = 0; q < (int)sizeof(T); ++q) dst[q] = reinterpret_cast<const uint4*>(v)[q];
    }
  }
}

// Which (row, group of 8 columns) a thread takes: the groups of all rows in turn.  (Whole rows per warp left 8 of 32
// lanes idle at 192 columns, and took six rounds instead of four for 64 rows: four graphed layers of 128 rows take 0.9 % less.)
template <typename T, typename F>
__device__ __forceinline__ void for_each_group(const PairTile<T>& t, F f) {
  const int per_row = t.un / 8, rows = kWideThreads / per_row, left = kWideThreads - rows * per_row;   // of one round
  int row = threadIdx.x / per_row, c = threadIdx.x - row * per_row;
  while (row < t.rows) {
    f(row, c * 8);
    row += rows;
    c += left;
    if (c >= per_row) { c -= per_row; ++row; }
  }
}

// h of this thread's elements; returns max |h|.
template <typename T>
__device__ __forceinline__ float pair_silu(const PairTile<T>& t) {
  using namespace bq::qd;
  float mx = 0.0f;
  for_each_group(t, [&](int row, int c) {
    Pack8<T>* const gp = reinterpret_cast<Pack8<T>*>(t.base + row * t.pitch + c);
    Pack8<T> h = *gp;
    apply_prologue<T, kSiluMul, true>(h, *reinterpret_cast<const Pack8<T>*>(t.base + row * t.pitch + t.un + c));
    mx = absmax8(h, mx);
    *gp = h;
  });
  return mx;
}

// Codes of the parked h under the grid-wide scale.
template <typename T>
__device__ __forceinline__ void pair_emit(const PairTile<T>& t, float scale, uint8_t* hq, long long ld, int m0,
                                          int col0, int cols) {
  using namespace bq::qd;
  const ScaleDiv sc(scale);
  for_each_group(t, [&](int row, int c) {
    if (col0 + c >= cols) return;                 // the output width is a multiple of 64
    const uint2 w = codes8<T, true>(*reinterpret_cast<const Pack8<T>*>(t.base + row * t.pitch + c), sc);
    uint8_t* const dst = hq + (long long)(m0 + row) * ld + col0 + c;
    if ((reinterpret_cast<uintptr_t>(dst) & 7) == 0) {
      *reinterpret_cast<uint2*>(dst) = w;
    } else {                                      // the caller's buffer is only known to be 2-byte aligned
      uint16_t* const d = reinterpret_cast<uint16_t*>(dst);
      d[0] = static_cast<uint16_t>(w.x); d[1] = static_cast<uint16_t>(w.x >> 16);
      d[2] = static_cast<uint16_t>(w.y); d[3] = static_cast<uint16_t>(w.y >> 16);
    }
  });
}

// Column-parallel form: the parked h unchanged, into every rank's gathered buffer.
template <typename T>
__device__ __forceinline__ void pair_push(const PairTile<T>& t, const PushParams& push, int m0, int col0, int cols) {
  struct alignas(2 * sizeof(T)) V2 { T v[2]; };
  const int per_row = t.un / 2, total = t.rows * per_row;
  for (int i = threadIdx.x; i < total; i += kWideThreads) {
    const int row = i / per_row, c = (i - row * per_row) * 2;
    if (col0 + c >= cols) continue;
    const V2 h = *reinterpret_cast<const V2*>(t.base + row * t.pitch + c);
    const long long at = (long long)(m0 + row) * push.ld + col0 + c;
    for (int d = 0; d < push.n; ++d) *reinterpret_cast<V2*>(static_cast<T*>(push.dst[d]) + at) = h;
  }
}

// Everything after the accumulator of the gate/up form is complete.  All threads of the CTA.
template <typename T, int MODE, int EPI>
__device__ __forceinline__ void pair_finish(const GemmParams& p, uint8_t* smem, float* s_red, uint32_t taddr, int unit,
                                            int m0, int rows, bool ok, float sg, float su) {
  using namespace bq::qd;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int un = p.seg[0].un;
  PairTile<T> t{reinterpret_cast<T*>(smem), 2 * un + 16 / (int)sizeof(T), rows, un};
  const int quad = warp & 3, row = LaneMap<MODE>::row0(quad) + lane;
  if (ok && LaneMap<MODE>::row0(quad) < rows)
    pair_park(t, taddr, row, row < rows, LaneMap<MODE>::col0(quad, un),
              LaneMap<MODE>::cols(un), p.seg[0].split, warp >> 2, kWideWarps / 4, sg, su);
  __syncthreads();
  if (threadIdx.x == 0) BQ_STAMP(p, 1);
  float mx = ok ? pair_silu(t) : 0.0f;
  const int col0 = unit * un, cols = p.seg[0].n;
  if (EPI == kAny && p.push.n > 0) {
    __syncthreads();
    if (ok) pair_push(t, p.push, m0, col0, cols);
    return;      // the amax needs every rank's shard: the quantizer behind the exchange takes it
  }
  mx = warp_amax(mx);
  if (lane == 0) s_red[warp] = mx;
  __syncthreads();
  unsigned int ticket = 0u;
  if (warp == 0) {
    float w = warp_amax(lane < kWideWarps ? s_red[lane] : 0.0f);
    __syncwarp();
    if (lane == 0) {
      // an aborted CTA still arrives (with 0), so the others are not left waiting
      if (gridDim.x > 1) {
        w = exchange_max(w, p.pair.words, gridDim.x, p.status);
        ticket = exchange_leave(p.pair.words);
      }
      const float sc = scale_from_amax(w);
      if (blockIdx.x == 0) p.pair.sh[0] = sc;
      s_red[0] = sc;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) BQ_STAMP(p, 5);
  if (ok) pair_emit(t, s_red[0], p.pair.hq, p.pair.ld_hq, m0, col0, cols);
  if (threadIdx.x == 0 && gridDim.x > 1) exchange_end(p.pair.words, gridDim.x, ticket);
}

// ---- the kernel -----------------------------------------------------------------------------
// Ring positions of the issuing thread, carried from unit to unit.
struct RingPos {
  int s = 0, sa = 0;
  uint32_t phase = 0, phase_a = 0;
};

// The MMAs of one unit.  One thread issues them and its instructions are on the critical path of
// a launch whose MMAs take 22 to 60 clocks each: the operand kind and the number of MMAs per K step
// are template parameters, descriptors are one 64-bit add.
template <int MODE, bool DENSE, int NM>
__device__ __forceinline__ bool issue_unit(const GemmParams& p, const RingShape& sh, const Segment& seg, RingPos& pos,
                                           uint32_t bar_base, uint32_t a_base, uint32_t w_base, uint32_t d,
                                           uint32_t issue) {
  const uint32_t idesc = DENSE ? idesc_f16(LaneMap<MODE>::kMmaM, seg.un, p.dense_fmt)
                               : idesc_e4m3(LaneMap<MODE>::kMmaM, seg.un);
  const int cols = LaneMap<MODE>::cols(seg.un);
  // descriptor units are 16 bytes
  const uint64_t a_desc = smem_desc_sw128(a_base), w_desc = smem_desc_sw128(w_base);
  const uint32_t a_blk = sh.a_block >> 4, w_blk = (seg.un / 2 * kBK) >> 4, w_up = w_blk * sh.kb_stage;
  const uint32_t a_stage = a_blk * sh.kb_stage, w_stage = (sh.w_block >> 4) * sh.kb_stage;
  const int blocks = DENSE ? p.k_blocks_dense : p.k_blocks;
  const int each = blocks / seg.split;
  int rem = blocks - each * seg.split;
  int left = each + (rem > 0 ? 1 : 0);          // K blocks left in this slice
  uint32_t acc = 0;
  const uint32_t full_a = bar_base + 8u * (2 * sh.w_stages);
  bool w_ready = false, a_ready = false;
  for (int kb = 0; kb < blocks; kb += sh.kb_stage) {
    if (!w_ready && !mbar_wait(bar_base + 8u * pos.s, pos.phase)) return false;
    if (!a_ready && !mbar_wait(full_a + 8u * pos.sa, pos.phase_a)) return false;
    uint64_t da = a_desc + pos.sa * a_stage, dw = w_desc + pos.s * w_stage;
    const uint32_t empty = bar_base + 8u * (sh.w_stages + pos.s);
    if (++pos.s == sh.w_stages) { pos.s = 0; pos.phase ^= 1u; }
    if (++pos.sa == sh.a_stages) { pos.sa = 0; pos.phase_a ^= 1u; }
    // look at the next stage's barriers now: the answers arrive while this stage's MMAs are issued
    w_ready = mbar_test(bar_base + 8u * pos.s, pos.phase);
    a_ready = mbar_test(full_a + 8u * pos.sa, pos.phase_a);
    const int nb = blocks - kb < sh.kb_stage ? blocks - kb : sh.kb_stage;
    for (int j = 0; j < nb; ++j) {
#pragma unroll
      for (int h = 0; h < NM; ++h) {
        const uint64_t dh = dw + (h ? w_up : 0u);
        const uint32_t dst = d + (h ? cols : 0);
#pragma unroll
        for (int q = 0; q < kBK / kUmmaK; ++q) {
          // +32 bytes along K inside the swizzle span = +2 in descriptor units (32 e4m3 or 16
          // 16-bit elements: one MMA's K either way)
          const uint32_t accumulate = q == 0 ? acc : 1u;
          if constexpr (DENSE) mma_f16_pair(issue, dst, da + 2u * q, dh + 2u * q, idesc, accumulate);
          else mma_f8_pair(issue, dst, da + 2u * q, dh + 2u * q, idesc, accumulate);
        }
      }
      da += a_blk;
      dw += w_blk;
      acc = 1;
      if (--left == 0) {                         // next slice, next accumulator
        d += NM * cols;
        left = each + (--rem > 0 ? 1 : 0);
        acc = 0;
      }
    }
    // both slots are free, in both CTAs of a pair, once these MMAs retire
    mma_commit_pair(issue, empty);
  }
  return true;
}

template <int MODE, int EPI, int DT>
__global__ void __launch_bounds__(kWideThreads, 1)
gemm_wide_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_xd,
                   const __grid_constant__ WeightMaps tm_w, const __grid_constant__ GemmParams p,
                   const __grid_constant__ WideShape sh) {
  using Lanes = LaneMap<MODE>;
  const int out_dtype = DT == kAnyType ? p.out_dtype : DT;
  extern __shared__ uint8_t smem_dyn[];
  const uint32_t base = (smem_u32(smem_dyn) + 1023u) & ~1023u;
  uint8_t* const base_ptr = smem_dyn + (base - smem_u32(smem_dyn));
  const int unit0 = blockIdx.x / 2, unit_step = gridDim.x / 2;
  auto segment_of = [&](int unit) {
    int s = 0;
#pragma unroll
    for (int i = 1; i < BQ_MAX_SEGMENTS; ++i)
      if (i < p.n_seg && unit >= p.seg[i].unit_begin) s = i;
    return s;
  };
  // one layout per CTA (where a CTA walks several units the host makes both the same)
  const RingShape rs = sh.ring[p.seg[segment_of(unit0)].dense ? 1 : 0];
  const uint32_t a_bytes = rs.kb_stage * rs.a_block, w_bytes = rs.kb_stage * rs.w_block;
  const uint32_t a_base = base, w_base = base + rs.a_stages * a_bytes;
  // barriers: weight ring full, weight ring empty, activation ring full, accumulators
  const uint32_t bar_base = base + sh.ring_bytes;
  auto full_w = [&](int s) { return bar_base + 8u * s; };
  auto empty_w = [&](int s) { return bar_base + 8u * (rs.w_stages + s); };
  auto full_a = [&](int s) { return bar_base + 8u * (2 * rs.w_stages + s); };
  const int n_ring_bars = 2 * rs.w_stages + rs.a_stages;
  auto acc_full = [&](int b) { return bar_base + 8u * (n_ring_bars + b); };
  auto acc_empty = [&](int b) { return bar_base + 8u * (n_ring_bars + 2 + b); };
  uint8_t* const misc = base_ptr + sh.ring_bytes + kBarrierBytes - 128;
  volatile uint32_t* const tmem_slot = reinterpret_cast<volatile uint32_t*>(misc);
  volatile uint32_t* const abort_flag = tmem_slot + 1;
  float* const s_red = reinterpret_cast<float*>(misc + 16);

  if (threadIdx.x == 0) { BQ_STAMP(p, 0); BQ_STAMP_META(p, 0); }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int crank = static_cast<int>(cluster_ctarank());
  const bool many = sh.rounds > 1;                           // two accumulators, dedicated epilogue warps
  const bool paired = EPI == kAny ? p.pair.on != 0 : EPI == kGateUp;
  const int m0 = crank * sh.m_half;                          // first batch row of this CTA

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tm_w.w[segment_of(unit0)]);
    if (paired) tma_prefetch_desc(&tm_w.w[1]);
    for (int s = 0; s < rs.w_stages; ++s) {
      mbar_init(full_w(s), 1);
      mbar_init(empty_w(s), 1);
    }
    for (int s = 0; s < rs.a_stages; ++s) mbar_init(full_a(s), 1);
    for (int b = 0; b < 2; ++b) {
      mbar_init(acc_full(b), 1);
      mbar_init(acc_empty(b), 2 * (kWideWarps - 4));      // the epilogue warps, where they are dedicated
    }
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(smem_u32(const_cast<uint32_t*>(tmem_slot)), sh.tmem_cols);
    tmem_relinquish_pair();
    // The next kernel may start its own set-up -- only now: a CTA of it that shares this SM takes
    // tensor memory too and keeps it until this kernel is done.
    pdl_launch_dependents();
  }
  __syncwarp();
  tc_fence_before();
  cluster_sync_all();         // the peer's barriers exist before anything signals them
  tc_fence_after();

  if (warp == 0) {
    // Weights do not depend on any earlier kernel: this warp never waits for the kernel that
    // produces the activation, it only follows the MMAs through the ring.  Read once: evict
    // first.  Slot and phase are carried along: an integer division by a run-time depth costs a
    // single issuing thread more than the loads it issues.
    const uint32_t issue = elect_one() ? 1u : 0u, expect = crank == 0 ? issue : 0u;
    const uint64_t pol_w = policy_evict_first();
    int s = 0;
    uint32_t phase = 1;                      // a fresh barrier counts as completed
    bool ok = true;
    for (int unit = unit0; unit < sh.units && ok; unit += unit_step) {
      const int sg = segment_of(unit);
      const Segment& seg = p.seg[sg];
      const int box = seg.un / 2;            // weight rows of one box
      const int row = (unit - seg.unit_begin) * seg.un + crank * box;
      const CUtensorMap* const map = &tm_w.w[sg];
      const uint32_t half = rs.kb_stage * box * kBK;         // bytes of one box
      const int blocks = seg.dense ? p.k_blocks_dense : p.k_blocks;
      for (int kb = 0; kb < blocks; kb += rs.kb_stage) {
        if (!mbar_wait(empty_w(s), phase)) { ok = false; break; }
        mbar_expect_tx(expect, full_w(s), 2 * sh.nm * half);
        const uint32_t dst = w_base + s * w_bytes;
        const int x = sh.flat ? kb * kBK : 0, z = sh.flat ? 0 : kb;
        tma_load_3d_pair(issue, dst, map, full_w(s), x, row, z, pol_w);
        if (paired) tma_load_3d_pair(issue, dst + half, &tm_w.w[1], full_w(s), x, row, z, pol_w);
        if (++s == rs.w_stages) { s = 0; phase ^= 1u; }
      }
    }
    if (!ok) *abort_flag = 1;
    __syncwarp();
  } else if (warp == 2) {
    // the activation is shared by every unit: keep it in L2
    const uint32_t issue = elect_one() ? 1u : 0u, expect = crank == 0 ? issue : 0u;
    const uint64_t pol_x = policy_evict_last();
    pdl_wait_prior_grids();   // the kernel that produces the activation has completed
    if (issue) BQ_STAMP(p, 2);
    // Activation slot s was last read by the MMAs of stage j = i - a_stages, whose completion is
    // completion number j / w_stages of weight slot j % w_stages.  That barrier cannot complete
    // a second time before this thread has looked: stage j + w_stages >= i needs THIS load
    // first (the host keeps a_stages <= w_stages).
    int s = 0, js = 0, i = 0;
    uint32_t jphase = 0;
    bool ok = true;
    for (int unit = unit0; unit < sh.units && ok; unit += unit_step) {
      const Segment& seg = p.seg[segment_of(unit)];
      const CUtensorMap* const map = seg.dense ? &tm_xd : &tm_x;
      const int blocks = seg.dense ? p.k_blocks_dense : p.k_blocks;
      for (int kb = 0; kb < blocks; kb += rs.kb_stage, ++i) {
        if (i >= rs.a_stages) {
          if (!mbar_wait(empty_w(js), jphase)) { ok = false; break; }
          if (++js == rs.w_stages) { js = 0; jphase ^= 1u; }
        }
        mbar_expect_tx(expect, full_a(s), 2 * a_bytes);
        const int x = sh.flat ? kb * kBK : 0, z = sh.flat ? 0 : kb;
        tma_load_3d_pair(issue, a_base + s * a_bytes, map, full_a(s), x, m0, z, pol_x);
        if (++s == rs.a_stages) s = 0;
      }
    }
    if (!ok) *abort_flag = 1;
    __syncwarp();
  } else if (warp == 1) {
    if (crank == 0) {
      const uint32_t issue = elect_one() ? 1u : 0u;
      const uint32_t tmem = *tmem_slot;
      RingPos pos;
      int round = 0;
      bool ok = true;
      for (int unit = unit0; unit < sh.units && ok; unit += unit_step, ++round) {
        const Segment& seg = p.seg[segment_of(unit)];
        const int b = many ? round & 1 : 0;
        if (round >= 2 && !mbar_wait(acc_empty(b), ((round >> 1) - 1) & 1)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d = tmem + b * sh.acc_cols;
        if (paired) ok = issue_unit<MODE, false, 2>(p, rs, seg, pos, bar_base, a_base, w_base, d, issue);
        else if (seg.dense) ok = issue_unit<MODE, true, 1>(p, rs, seg, pos, bar_base, a_base, w_base, d, issue);
        else ok = issue_unit<MODE, false, 1>(p, rs, seg, pos, bar_base, a_base, w_base, d, issue);
        mma_commit_pair(issue, acc_full(b));
      }
      if (!ok) *abort_flag = 1;
    }
    __syncwarp();
  }

  // ---- epilogue: all warps where there is one unit, else the warps without another role -----
  const int first_warp = many ? 4 : 0;
  if (warp >= first_warp) {
    pdl_wait_prior_grids();   // scales are read and outputs written only after this
    const int quad = warp & 3, col_group = (warp - first_warp) >> 2, n_groups = (kWideWarps - first_warp) / 4;
    const int row = Lanes::row0(quad) + lane;                 // batch row of this CTA
    const int rows = p.M - m0 < sh.m_half ? p.M - m0 : sh.m_half;   // may be <= 0 in a pair's second CTA
    const bool row_ok = row < rows;
    const bool warp_ok = Lanes::row0(quad) < rows;            // some lane of the warp holds a real row
    const float sx = ld_coherent4(p.sx);
    float bv = 0.0f;
    int bi = kNoIndex;
    int round = 0;
    for (int unit = unit0; unit < sh.units; unit += unit_step, ++round) {
      const Segment& seg = p.seg[segment_of(unit)];
      const float sw = seg.dense ? 1.0f : __ldg(seg.sw);
      const float sw_up = paired ? __ldg(p.pair.sw_up) : 0.0f;
      const int b = many ? round & 1 : 0;
      if ((EPI == kResidual || (EPI == kAny && seg.res != nullptr)) && row_ok) {
        // the residual's lines on their way while the MMAs run
        const int col = (unit - seg.unit_begin) * seg.un + Lanes::col0(quad, seg.un) + col_group * 16;
        const int es = out_dtype == BQ_DTYPE_F32 ? 4 : 2;
        if (col < seg.n)
          asm volatile("prefetch.global.L1 [%0];" ::"l"(static_cast<const uint8_t*>(seg.res) +
                                                         ((long long)(m0 + row) * seg.ld_res + col) * es));
      }
      bool ok = mbar_wait(acc_full(b), (many ? round >> 1 : 0) & 1);
      tc_fence_after();
      if (threadIdx.x == 0) BQ_STAMP(p, 4);
      if (!ok) *abort_flag = 1;
      if (!many) {
        __syncthreads();
        ok = *abort_flag == 0;
      }
      const uint32_t taddr = *tmem_slot + (static_cast<uint32_t>(quad * 32) << 16) + b * sh.acc_cols;
      const float scale = seg.dense ? 1.0f : sx * sw;
      if (paired) {
        const float su = sx * sw_up;
        if (out_dtype == BQ_DTYPE_BF16)
          pair_finish<__nv_bfloat16, MODE, EPI>(p, base_ptr, s_red, taddr, unit, m0, rows, ok, scale, su);
        else if (out_dtype == BQ_DTYPE_F16)
          pair_finish<__half, MODE, EPI>(p, base_ptr, s_red, taddr, unit, m0, rows, ok, scale, su);
        else
          pair_finish<float, MODE, EPI>(p, base_ptr, s_red, taddr, unit, m0, rows, ok, scale, su);
      } else if (ok && warp_ok) {
        const int cols = Lanes::cols(seg.un);
        const UnitOut o{p, seg, (unit - seg.unit_begin) * seg.un + Lanes::col0(quad, seg.un), m0 + row, row_ok};
        for (int c = col_group * 16; c < cols; c += 16 * n_groups) {
          if (o.row0 + c >= seg.n) break;
          float v[16];
          load_sums(taddr + c, seg.split, cols, v);
#pragma unroll
          for (int q = 0; q < 16; ++q) v[q] *= scale;
          if constexpr (EPI == kArgmax) {
            if (out_dtype == BQ_DTYPE_BF16) argmax_chunk<__nv_bfloat16>(o, c, v, bv, bi);
            else if (out_dtype == BQ_DTYPE_F16) argmax_chunk<__half>(o, c, v, bv, bi);
            else argmax_chunk<float>(o, c, v, bv, bi);
            if (!p.argmax.store_logits) continue;
          }
          if (out_dtype == BQ_DTYPE_BF16) store_chunk<__nv_bfloat16, EPI>(o, c, v);
          else if (out_dtype == BQ_DTYPE_F16) store_chunk<__half, EPI>(o, c, v);
          else store_chunk<float, EPI>(o, c, v);
        }
      }
      if (many) {
        if (!ok) break;
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(map_to_cta(acc_empty(b), 0));
      }
    }
    if (EPI == kArgmax && row_ok) {
      // a pair of 128 holds a row's columns in two lane quarters: two slots per column group
      const int slot = (unit0 * n_groups + col_group) * (MODE == 1 ? 2 : 1) + (MODE == 1 ? quad >> 1 : 0);
      p.argmax.partial[static_cast<size_t>(slot) * p.M + m0 + row] =
          make_uint2(__float_as_uint(bv), static_cast<unsigned int>(bi));
    }
    if (threadIdx.x == 0) BQ_STAMP(p, 6);
  }
  tc_fence_before();
  // Nobody frees tensor memory while the peer may still use the pair.  That wants no order of the outputs' stores, for
  // whose way to L2 (0.5 us) a releasing barrier waits; where a peer counts arrivals here, or the stores are counted, it does.
  if (many || EPI == kAny) cluster_sync_all();
  else { cluster_arrive_relaxed(); cluster_wait(); }
  if (EPI == kAny && p.push.n > 0 && threadIdx.x == 0) {
    // The stores of all threads of this CTA are ordered before thread 0's fence by the barrier
    // (fences are cumulative); the fence orders them before this CTA's count; the last CTA sees
    // every count, fences again and only then signals the ranks: every store of the launch
    // happens before every arrival.
    __threadfence_system();
    const unsigned int old = atomicAdd(p.push.done, 1u);
    if (old == gridDim.x - 1u) {
      *p.push.done = 0u;                       // ready for the next launch on this scratch
      __threadfence_system();
      for (int d = 0; d < p.push.n; ++d)
        asm volatile("red.release.sys.global.add.u32 [%0], 1;" ::"l"(p.push.flag[d]) : "memory");
    }
  }
  if (*abort_flag != 0 && threadIdx.x == 0) {
    atomicExch(p.status, (unsigned int)kErrDeviceWait);
    // copies that were issued get a bounded time to land before the shared memory goes away
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000LL) {}
  }
  if (warp == 1) {
    tmem_dealloc_pair(*tmem_slot, sh.tmem_cols);
  }
  if (threadIdx.x == 0) BQ_STAMP(p, 7);
}
