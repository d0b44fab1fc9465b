// Device-side building blocks of the FP8 activation quantizer, shared by the stand-alone
// quantizer kernels (quant_act.cu, norm_quant.cu) and the paired gate/up epilogue (gemm_w8a8.cu).
// The arithmetic is the reference's torch spelling as a CUDA device evaluates it
// (braid/model/quant.py:108-115, :228-229): reciprocal-multiply scale, IEEE division, clamp to
// +-448 (NaN survives), NaN-propagating max, round-to-nearest-even e4m3 cast; the
// prologues keep the per-operation rounding of the separate torch kernels
// (braid/model/mlp.py:48, braid/model/attention.py:215).
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <type_traits>

namespace bq {
namespace qd {

constexpr float kFp8Max = 448.0f;
// torch divides a tensor by a host scalar as t * (1/scalar) in fp32.
constexpr float kInvFp8Max = 1.0f / 448.0f;
constexpr float kEps = 1e-12f;

constexpr int kGroup = 8;      // elements per group (one 128-bit load of a 16-bit type)

enum Mode { kPlain = 0, kSiluMul = 1, kSigmoidGate = 2 };

// n / d for 32-bit n without a division: floor((n * mul) >> 32 >> shift) with the round-up multiplier of Granlund and
// Montgomery (PLDI 1994), exact for n < 2^31.
struct FastDiv {
  unsigned int d, mul, shift;
  static FastDiv by(unsigned int d) {
    unsigned int l = 0;
    while ((1ull << l) < d) ++l;
    const unsigned long long m = ((1ull << (31 + l)) + d - 1) / d;      // 2^31 <= m < 2^32 unless d is 1
    return l == 0 ? FastDiv{d, 0u, 0u} : FastDiv{d, static_cast<unsigned int>(m), l - 1};
  }
  __device__ __forceinline__ unsigned int operator()(unsigned int n) const {
    return mul == 0u ? n : __umulhi(n, mul) >> shift;
  }
};

struct QParams {
  const void* a;        // x | gate | o
  const void* b;        // - | up   | gate
  uint8_t* q;
  float* scale;
  void* ws;             // kernel-specific scratch words
  float* partial;       // weight quantizer: the CTAs' maxima, from its first launch to its second
  unsigned int n_groups;      // full groups of 8
  unsigned int tail;          // plain mode only: leftover elements (< 8)
  FastDiv groups_per_row;
  long long ld_a, ld_b;       // row strides in elements (prologue modes)
  FastDiv chunk;              // sigmoid gate: head width of the strided gate view
  long long chunk_stride;     // sigmoid gate: distance between heads
  int held;                   // groups each thread keeps (hold kernel)
  // column-parallel form: the input is a gathered buffer other ranks store into; wait until the
  // arrival counter has advanced by wait_count beyond *wait_seen before loading (nullptr = no wait)
  const unsigned int* wait_flag;
  unsigned int* wait_seen;
  unsigned int wait_count;
  unsigned long long* phase_ring;   // development builds (BQ_PHASES) only, else nullptr
  int phase_seq;
};

template <typename T> struct alignas(16) Pack8 { T v[8]; };
template <> struct alignas(16) Pack8<float> { float v[8]; };

__device__ __forceinline__ float widen(float v) { return v; }
__device__ __forceinline__ float widen(__half v) { return __half2float(v); }
__device__ __forceinline__ float widen(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename T> __device__ __forceinline__ T narrow(float v);
template <> __device__ __forceinline__ float narrow<float>(float v) { return v; }
template <> __device__ __forceinline__ __half narrow<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 narrow<__nv_bfloat16>(float v) {
  return __float2bfloat16_rn(v);
}

// NaN-propagating max: once either side is NaN the result is NaN.
__device__ __forceinline__ float nan_max(float m, float v) { return (v != v || v > m) ? v : m; }

// What an earlier kernel writes is read with `ld.global.cg` (volatile to the compiler): the kernels
// run ahead of that kernel, and a load of what the compiler takes for constant memory (`__ldg`)
// may be moved above the wait for it.  For gathered buffers the load also has to see what other
// GPUs stored while this kernel was waiting for their arrival.
template <typename T>
__device__ __forceinline__ Pack8<T> load8(const T* p) {
  Pack8<T> r;
  if constexpr (sizeof(T) == 4) {
    const float4* q = reinterpret_cast<const float4*>(p);
    const float4 lo = __ldcg(q);
    const float4 hi = __ldcg(q + 1);
    r.v[0] = lo.x; r.v[1] = lo.y; r.v[2] = lo.z; r.v[3] = lo.w;
    r.v[4] = hi.x; r.v[5] = hi.y; r.v[6] = hi.z; r.v[7] = hi.w;
  } else {
    const uint4 raw = __ldcg(reinterpret_cast<const uint4*>(p));
    *reinterpret_cast<uint4*>(&r) = raw;
  }
  return r;
}

// two values rounded to a 16-bit T and packed, low half first
template <typename T>
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  if constexpr (std::is_same<T, __half>::value) {
    const __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
  } else {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
  }
}
template <typename T>
__device__ __forceinline__ float2 unpack2(uint32_t w) {
  if constexpr (std::is_same<T, __half>::value) return __half22float2(*reinterpret_cast<const __half2*>(&w));
  else return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w));
}
// Two fp32 products at an instruction, each rounded as by itself.
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  unsigned long long x, y, z;
  float2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "f"(a.x), "f"(a.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(y) : "f"(b.x), "f"(b.y));
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(z) : "l"(x), "l"(y));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(z));
  return r;
}

// max(m, |v[0..7]|), NaN-propagating.  The 16-bit types take the maximum on packed pairs
// (`abs` and `max.NaN` on two values per instruction; the maximum of 16-bit values is one of
// them, so nothing is rounded) and widen once at the end.
template <typename T>
__device__ __forceinline__ float absmax8(const Pack8<T>& v, float m) {
  if constexpr (sizeof(T) == 2) {
    using T2 = typename std::conditional<std::is_same<T, __half>::value, __half2, __nv_bfloat162>::type;
    const T2* w = reinterpret_cast<const T2*>(&v);
    const T2 m01 = __hmax2_nan(__habs2(w[0]), __habs2(w[1]));
    const T2 m23 = __hmax2_nan(__habs2(w[2]), __habs2(w[3]));
    const T2 mm = __hmax2_nan(m01, m23);
    m = nan_max(m, widen(mm.x));
    m = nan_max(m, widen(mm.y));
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) m = nan_max(m, fabsf(widen(v.v[i])));
  }
  return m;
}

// x / sc for a divisor every element of the tensor shares, with the bits of the IEEE division
// the reference spells (`x / scale`): the reciprocal is rounded once (`__frcp_rn`), and every
// element takes a product and two residual corrections.  After the first correction the
// quotient is within one unit in the last place, so the second one rounds correctly
// (Markstein's division step: y = RN(1/b), q faithful, r = a - b*q exact, RN(q + r*y) =
// RN(a/b)).  That holds while nothing leaves the normal range: the scale has to lie in
// [2^-60, 2^60], a quotient that overflows or an operand that is not finite shows as a NaN and
// takes the division instruction instead, and quotients too small for the corrections to be
// exact are far below half of the smallest e4m3 step, where only the sign reaches the code
// (hence the copysign, which also keeps -0).
// Values of a 16-bit type take one correction: over all 2^23 divisor mantissas and all dividend
// mantissas of 8 (bf16) and of 11 bits (fp16), checked one by one, the quotient after the first
// correction is the IEEE one.  Two instructions of about ten per element: the weight loader's cast, a
// 12288 x 4096 weight in all, 48.6 -> 44.5 us; a prompt layer of 9658 rows 2,260 -> 2,235 us, four graphed
// decoder layers of 128 rows 344.9 -> 341.9 us.
struct ScaleDiv {
  float sc, inv;
  bool fast;
  __device__ __forceinline__ explicit ScaleDiv(float s) {
    sc = s;
    inv = __frcp_rn(s);
    fast = s >= 0x1p-60f && s <= 0x1p60f;
  }
  // The quotient by the corrections alone; NaN where the division instruction has to decide.
  template <int CORRECTIONS>
  __device__ __forceinline__ float corrected(float x) const {
    float q = __fmul_rn(x, inv);
#pragma unroll
    for (int i = 0; i < CORRECTIONS; ++i) q = __fmaf_rn(__fmaf_rn(-q, sc, x), inv, q);
    return copysignf(q, x);
  }
};

// x[i] <- x[i] / sc for the N values of one group: one test for the whole group decides
// between the corrected products and N division instructions.  OWN_SCALE says the scale was
// taken from the very values being divided (sc = max|x| / 448, clamped from below): then a
// scale inside the range means every x is finite and no quotient exceeds 448, and the test
// for NaN among the results is left out.  What goes on to the saturating e4m3 conversion is
// the bare quotient: the reference clamps to +-448 before its (non-saturating) cast,
// `cvt.rn.satfinite` does the same clamp itself (finite values and infinities beyond the
// range become +-448, NaN stays NaN).
// T is the type the x are values of.
template <typename T, int N, bool OWN_SCALE = false>
__device__ __forceinline__ void divide_group(const ScaleDiv& d, float (&x)[N]) {
  float q[N];
  bool ok = d.fast;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    q[i] = d.corrected<sizeof(T) == 2 ? 1 : 2>(x[i]);
    if constexpr (!OWN_SCALE) ok = ok && (q[i] == q[i]);
  }
  if (ok) {
#pragma unroll
    for (int i = 0; i < N; ++i) x[i] = q[i];
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) x[i] = __fdiv_rn(x[i], d.sc);
  }
}

__device__ __forceinline__ float quant_one(float x, const ScaleDiv& d) {
  float v[1] = {x};
  divide_group<float, 1>(d, v);
  return v[0];
}

// the 8 e4m3 codes of one group, as two 32-bit words
template <typename T, bool OWN_SCALE = false>
__device__ __forceinline__ uint2 codes8(const Pack8<T>& v, const ScaleDiv& sc) {
  float f[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) f[i] = widen(v.v[i]);
  divide_group<T, 8, OWN_SCALE>(sc, f);
  uint32_t w[2];
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(f[half * 4], f[half * 4 + 1]), __NV_SATFINITE, __NV_E4M3);
    const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(f[half * 4 + 2], f[half * 4 + 3]), __NV_SATFINITE, __NV_E4M3);
    w[half] = (lo & 0xFFFFu) | ((hi & 0xFFFFu) << 16);
  }
  return make_uint2(w[0], w[1]);
}

// The codes of x / scale by ONE product, for x of a 16-bit type T.  A code depends on its quotient only by the side of the
// ties between neighbouring codes that it lies on, and the ties have 16 mantissas, n / 16 with n = 16 .. 31 (those of e4m3's
// subnormal steps among them).  For each of them there is one x of T's mantissa nearest to tie * scale; every other x
// is half a unit of T or more away, 2^-12 of its value, where no rounding reaches.  So a multiplier gives every code if for
// these 16 it puts x * multiplier on the side of the tie (or on it) that the IEEE quotient is on; powers of two do not
// matter (scales in [2^-60, 2^60]: what underflows is below every tie, and both keep the sign of a zero; beyond +-448, in
// infinity and in NaN both saturate alike).  Tried are the rounded reciprocal and its two neighbours: one of them
// does for 99.99 % of all scales of bf16 values, 99.98 % of fp16's, and for 90 % of the scales that are max|x| / 448 of a value
// of the type itself, where x = 3/4 max|x| may lie on a tie exactly.  The others take ScaleDiv's correction, 4 instructions
// an element where this is half of one.  us, quotients / one product, and a scale that takes the quotients: a 12288 x 4096
// weight 43.2 / 38.4 / 44.2, cast of 9658 x 4096 bf16 21.9 / 17.5 / 21.5, of 9658 x 12288 62.3 / 57.9 / 61.5, 9658 x 4096 bf16
// quantized 34.0 / 29.7 / 34.2.  Each has a loop of its own (by_scale): with the choice inside the loop those were 39.7 and
// 44.9, 17.9 and 22.0, 58.9 and 62.1, 31.7 and 35.9.
// For kernels that cast many groups a thread: the proof is a division and two ballots per warp, which a CTA of one row per
// group pays for once and loses by (1500 x 4096 normed 11.6 -> 12.1), and so does a thread of one group: cast of 32768
// values 1.8 -> 2.05, of 1.21 M (one each) 2.85 -> 3.1; 2.46 M (two) 3.6 -> 3.35, 3.16 M (2.6) 4.1 -> 3.6.
constexpr int kProofPays = 2;      // more groups of 8 per thread
template <typename T> struct OneProduct { float mul; };

template <typename T>
struct ScaleMul {
  ScaleDiv div;
  float mul;
  bool one;
  // By whole warps, of one mind about `worth`.
  __device__ __forceinline__ explicit ScaleMul(float s, bool worth = true) : div(s), mul(0.0f), one(false) {
    if constexpr (sizeof(T) == 2) {
      if (!div.fast || !worth) return;
      constexpr int kBits = std::is_same<T, __half>::value ? 11 : 8;
      const unsigned int lane = threadIdx.x & 31u, n = 16u + (lane & 15u);
      const float tie = static_cast<float>(n) * 0.0625f;
      const unsigned int bits = __float_as_uint(s), m = (bits & 0x7FFFFFu) | 0x800000u;
      const float sc = __uint_as_float((bits & 0x7FFFFFu) | 0x3F800000u);       // in [1, 2)
      const unsigned int y = m * n, step = 1u << ((y >> 28 ? 29 : 28) - kBits);    // tie * scale in units of 2^-27
      const float x = static_cast<float>((y + (step >> 1)) & ~(step - 1u)) * 0x1p-27f;
      const float r = __frcp_rn(sc), q = __fdiv_rn(x, sc);
      auto side = [&](float v) { return v > tie ? 1 : (v < tie ? -1 : 0); };
      auto agrees = [&](int ulps) { return side(__fmul_rn(x, __uint_as_float(__float_as_uint(r) + ulps))) == side(q); };
      // lanes 0..15 the reciprocal, lanes 16..31 its upper neighbour; then the lower one
      const unsigned int got = __ballot_sync(0xffffffffu, agrees(lane < 16u ? 0 : 1));
      const unsigned int low = __ballot_sync(0xffffffffu, agrees(-1));
      const int ulps = (got & 0xFFFFu) == 0xFFFFu ? 0 : (got >> 16 == 0xFFFFu ? 1 : -1);
      one = ulps >= 0 || low == 0xffffffffu;
      // r is the reciprocal of the mantissa alone: 2^-exponent goes back in
      mul = __uint_as_float(__float_as_uint(r) + ulps - ((bits & 0x7F800000u) - 0x3F800000u));
    }
  }
};

// four quotients' codes, two products an instruction
template <typename T>
__device__ __forceinline__ uint32_t codes4_mul(uint32_t lo, uint32_t hi, float mul) {
  uint32_t out[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    out[i] = __nv_cvt_float2_to_fp8x2(mul2(unpack2<T>(i == 0 ? lo : hi), make_float2(mul, mul)), __NV_SATFINITE, __NV_E4M3);
  }
  return __byte_perm(out[0], out[1], 0x5410);
}

template <typename T, bool OWN_SCALE = false>
__device__ __forceinline__ uint2 codes8(const Pack8<T>& v, const OneProduct<T>& sc) {
  const uint4 w = *reinterpret_cast<const uint4*>(&v);
  return make_uint2(codes4_mul<T>(w.x, w.y, sc.mul), codes4_mul<T>(w.z, w.w, sc.mul));
}

// f(scale) with what the codes are taken by.
template <typename T, typename F>
__device__ __forceinline__ void by_scale(const ScaleMul<T>& s, F&& f) {
  if constexpr (sizeof(T) == 2) {
    if (s.one) { f(OneProduct<T>{s.mul}); return; }
  }
  f(s.div);
}

template <typename T, bool OWN_SCALE = false, typename Scale>
__device__ __forceinline__ void emit8(const Pack8<T>& v, const Scale& sc, uint8_t* dst) {
  *reinterpret_cast<uint2*>(dst) = codes8<T, OWN_SCALE>(v, sc);
}

__device__ __forceinline__ float scale_from_amax(float amax) {
  const float raw = amax * kInvFp8Max;
  return (raw < kEps) ? kEps : raw;   // NaN compares false and stays NaN
}

// x / (1 + exp(-x)) and 1 / (1 + exp(-x)) rounded to T as torch evaluates F.silu and
// torch.sigmoid of a T tensor on a CUDA device: fp32, expf, an IEEE division, one rounding.
template <typename T> __device__ __forceinline__ T silu_to(float x) {
  return narrow<T>(__fdiv_rn(x, 1.0f + expf(-x)));
}
template <typename T> __device__ __forceinline__ T sigmoid_to(float x) {
  return narrow<T>(__fdiv_rn(1.0f, 1.0f + expf(-x)));
}

// The same two functions of N values, the rounding to T left to the caller.
// For 16-bit T the division is a reciprocal estimate and one residual correction of the quotient
// (q = x y, q + (x - d q) y; Markstein, IBM J. Res. Dev. 34(1), 1990): with |x| <= 80 the divisor lies
// in [1, 2^116] and nothing leaves the normal range, and x takes only 65,536 values: the fp32
// quotients are the IEEE ones, bit for bit (tested for SiLU down to quotients of 2^-120, where its
// fp32 value is used; for the value rounded to T over all inputs of both functions and types).
// (-0 needs the sign put back.)  Values beyond 80, infinities and NaN
// take the division itself, decided once per group of N.  For the kernels that run the arithmetic
// many times over; those of small decode batches run it once from a cold instruction cache, where
// the shorter code of silu_to / sigmoid_to is the faster one (four graphed decoder layers of 27 fp16
// rows: 291.4 us with them, 297.5 with this).
__device__ __forceinline__ float corrected_quotient(float x, float d) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(d));
  const float q = __fmul_rn(x, y);
  return copysignf(__fmaf_rn(__fmaf_rn(-d, q, x), y, q), x);
}

// 1 / d of the same: the first quotient is the estimate itself, and nothing is negative.
__device__ __forceinline__ float corrected_reciprocal(float d) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(d));
  return __fmaf_rn(__fmaf_rn(-d, y, 1.0f), y, y);
}

enum Gate { kSilu, kSigmoid };

template <typename T, Gate G, int N>
__device__ __forceinline__ void gate_group(float (&x)[N]) {
  if constexpr (sizeof(T) == 2) {
    bool ok = true;
#pragma unroll
    for (int i = 0; i < N; ++i) ok = ok && fabsf(x[i]) <= 80.0f;
    if (ok) {
#pragma unroll
      for (int i = 0; i < N; ++i) {
        const float d = 1.0f + expf(-x[i]);
        x[i] = G == kSilu ? corrected_quotient(x[i], d) : corrected_reciprocal(d);
      }
      return;
    }
  }
  // rare for 16-bit types: kept rolled so that it costs little code
#pragma unroll(sizeof(T) == 2 ? 1 : N)
  for (int i = 0; i < N; ++i) x[i] = __fdiv_rn(G == kSilu ? x[i] : 1.0f, 1.0f + expf(-x[i]));
}

// running |.| maximum of packed pairs, NaN-propagating; starts at 0
template <typename T>
__device__ __forceinline__ uint32_t absmax2(uint32_t m, uint32_t w) {
  using T2 = typename std::conditional<std::is_same<T, __half>::value, __half2, __nv_bfloat162>::type;
  const T2 r = __hmax2_nan(*reinterpret_cast<const T2*>(&m), __habs2(*reinterpret_cast<const T2*>(&w)));
  return *reinterpret_cast<const uint32_t*>(&r);
}

// N values of `gated` pass through the gate function, are rounded to T, multiplied by `other` in fp32
// and rounded again (the two roundings of the separate torch kernels).  Results in `gated`, as
// values of T widened.
template <typename T, Gate G, int N>
__device__ __forceinline__ void gated_product(float (&gated)[N], const float (&other)[N]) {
  gate_group<T, G, N>(gated);
  if constexpr (sizeof(T) == 2) {
#pragma unroll
    for (int i = 0; i < N; i += 2) {
      const float2 p = mul2(unpack2<T>(pack2<T>(gated[i], gated[i + 1])), make_float2(other[i], other[i + 1]));
      const float2 h = unpack2<T>(pack2<T>(p.x, p.y));
      gated[i] = h.x;
      gated[i + 1] = h.y;
    }
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) gated[i] = gated[i] * other[i];
  }
}

// Raw operands of one group: one 8-pack for the plain mode, two for the prologues.
template <typename T, int MODE>
__device__ __forceinline__ void load_raw(const QParams& p, unsigned int g, Pack8<T>& a, Pack8<T>& b) {
  if constexpr (MODE == kPlain) {
    a = load8<T>(reinterpret_cast<const T*>(p.a) + static_cast<size_t>(g) * kGroup);
  } else {
    const unsigned int row = p.groups_per_row(g);
    const unsigned int col = (g - row * p.groups_per_row.d) * kGroup;
    const T* pa = reinterpret_cast<const T*>(p.a) + static_cast<long long>(row) * p.ld_a + col;
    const T* pb;
    if constexpr (MODE == kSiluMul) {
      pb = reinterpret_cast<const T*>(p.b) + static_cast<long long>(row) * p.ld_b + col;
    } else {
      const unsigned int head = p.chunk(col);
      pb = reinterpret_cast<const T*>(p.b) + static_cast<long long>(row) * p.ld_b +
           static_cast<long long>(head) * p.chunk_stride + (col - head * p.chunk.d);
    }
    a = load8<T>(pa);
    b = load8<T>(pb);
  }
}

// a <- the activation values (in place); plain mode is the identity.
// LARGE: the kernel runs this many times over (see gate_group).
template <typename T, int MODE, bool LARGE = false>
__device__ __forceinline__ void apply_prologue(Pack8<T>& a, const Pack8<T>& b) {
  if constexpr (MODE != kPlain && LARGE && sizeof(T) == 2) {
    // the operand of the gate function: gate of SiLU(gate) * up, gate of o * sigmoid(gate)
    const uint4 gw = *reinterpret_cast<const uint4*>(MODE == kSiluMul ? &a : &b);
    const uint4 ow = *reinterpret_cast<const uint4*>(MODE == kSiluMul ? &b : &a);
    const uint32_t g[4] = {gw.x, gw.y, gw.z, gw.w}, o[4] = {ow.x, ow.y, ow.z, ow.w};
    float x[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 v = unpack2<T>(g[i]);
      x[2 * i] = v.x;
      x[2 * i + 1] = v.y;
    }
    gate_group<T, MODE == kSiluMul ? kSilu : kSigmoid, 8>(x);
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      // two roundings to T, as of the separate kernels
      const float2 h = mul2(unpack2<T>(pack2<T>(x[2 * i], x[2 * i + 1])), unpack2<T>(o[i]));
      w[i] = pack2<T>(h.x, h.y);
    }
    *reinterpret_cast<uint4*>(&a) = make_uint4(w[0], w[1], w[2], w[3]);
  } else if constexpr (MODE != kPlain && LARGE) {
    float x[8], y[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      x[i] = widen(MODE == kSiluMul ? a.v[i] : b.v[i]);
      y[i] = widen(MODE == kSiluMul ? b.v[i] : a.v[i]);
    }
    gated_product<T, MODE == kSiluMul ? kSilu : kSigmoid, 8>(x, y);
#pragma unroll
    for (int i = 0; i < 8; ++i) a.v[i] = narrow<T>(x[i]);
  } else if constexpr (MODE != kPlain) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if constexpr (MODE == kSiluMul) {
        // silu in fp32, rounded to T; product in fp32, rounded to T
        const float x = widen(a.v[i]);
        const T sl = silu_to<T>(x);
        a.v[i] = narrow<T>(widen(sl) * widen(b.v[i]));
      } else {
        const float gt = widen(b.v[i]);
        const T sg = sigmoid_to<T>(gt);
        a.v[i] = narrow<T>(widen(a.v[i]) * widen(sg));
      }
    }
  }
}


}  // namespace qd
}  // namespace bq
