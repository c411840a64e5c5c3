// Per-group arithmetic of the quantizers.
//
// Results follow baseline/kernels/quantize_w4a4_act_fuse_lora/ref.py:40-48 and
// baseline/kernels/_nvfp4.py:27-41, :82-91 of the reference bit for bit; none of it
// runs a per-element IEEE divide.
//
// Activations (the fused kernels).  Only decisions leave the kernel - a scale byte per group, a code per
// element - so nothing needs the quotients themselves, only the side of each bound they are on.  Inputs
// and smoothing factors have at most 11 significant bits, scales 4 and bounds of codes 3, so a quotient
// x / s that is not exactly on a bound is off it by more than 2^-19.2 of it (a scale's rounding
// bound: 2^-18.5).  One fp32 multiplication by a reciprocal is good to 2^-23, and errs on a known side if
// the reciprocal is nudged: f = x r with r = RN((1 / s)(1 + 2^-22)) is above the exact quotient by
// 2^-24 to 2^-21.4 of it.
//   codes   the E2M1 conversion (nearest, two elements an instruction) of f c, c = rcp(scale)(1 + 2^-21):
//           a quotient on a bound comes out above it, as the definition wants, one below it stays below
//   scales  RN(f RN((1/6)(1 - 2^-22))), rounded to 20 significant bits: a quotient on a rounding bound of
//           E4M3, which has at most 5, is put back on it exactly (so that its tie rule decides), any
//           other stays on its side
// (checked exhaustively over significand pairs on the CPU).  A group costs some 60 instructions, a third of
// the two-step IEEE quotient with a truncation that this replaced, and a smoothing factor's table entry
// is 4 bytes instead of 8; with the same kernel around it 4352 rows of 3840 / 10240 / 15360 columns
// went from 16.4 / 33.5 / 54.9 to 16.2 / 30.4 / 49.8 us.  f = fma(x, r, +0) turns a -0 input into +0, which the reference's sign rule wants.
// Nothing may over- or underflow: the table builder sets a flag when a smooth value lies outside the safe
// range, and the kernels then divide with __fdiv_rn, after which the same steps hold (f exact).
// Groups whose scale byte is 0 (everything non-zero saturates) or the 448 clamp (ratios are unbounded)
// compare against the seven exact products instead.
//
// fp32 values (weights, the next layer's activations in the GEMM's epilogue) have 24 significant bits.  Scales have 4 and
// bounds of codes 3, so every product scale * bound is among the numbers of 12 significant bits, and cutting a value
// down to those (one AND, towards zero, the sign stays) leaves it on its side of all of them.  What is left and not on a
// bound is off it by 2^-12 of it, far more than one multiplication by rcp(scale)(1 + 2^-21) errs, and a value on a bound
// comes out above it: the conversion instruction of the product returns the reference's code.  (Exact floors of 4 v / 2^E,
// rescaled by a second multiplication, took a slow conversion and a multiplication an element more: the next layer's codes of
// 4352 x 1024 -> 3072 bf16, both kernels, 32.8 -> 30.0 us; packing, which memory bounds, takes the same time.)
#pragma once

#include "nvfp4_math.cuh"


namespace svdq {
namespace qmath {

// Widen a pair of 16-bit values.  CANON adds +0 first, which turns -0 into +0 and changes nothing
// else (the reference gives a zero the sign bit only when the value tests < 0).  The smoothing
// does the same by itself (see above), so only calls without it ask for it.
template <typename T, bool CANON> __device__ __forceinline__ float2 unpack2(uint32_t v);
template <> __device__ __forceinline__ float2 unpack2<__half, true>(uint32_t v) {
  return __half22float2(__hadd2(*reinterpret_cast<__half2*>(&v), __float2half2_rn(0.0f)));
}
template <> __device__ __forceinline__ float2 unpack2<__half, false>(uint32_t v) {
  return __half22float2(*reinterpret_cast<__half2*>(&v));
}
template <> __device__ __forceinline__ float2 unpack2<__nv_bfloat16, true>(uint32_t v) {
  const __nv_bfloat162 c = __hadd2(*reinterpret_cast<__nv_bfloat162*>(&v), __float2bfloat162_rn(0.0f));
  const uint32_t u = *reinterpret_cast<const uint32_t*>(&c);
  return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xFFFF0000u));
}
template <> __device__ __forceinline__ float2 unpack2<__nv_bfloat16, false>(uint32_t v) {
  return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xFFFF0000u));
}

template <typename T, bool CANON>
__device__ __forceinline__ void unpack_group(const uint4& lo16, const uint4& hi16, float2 (&f)[8]) {
  const uint32_t w[8] = {lo16.x, lo16.y, lo16.z, lo16.w, hi16.x, hi16.y, hi16.z, hi16.w};
#pragma unroll
  for (int j = 0; j < 8; ++j) f[j] = unpack2<T, CANON>(w[j]);
}

// The smoothing table (svdq_prepare_smooth): K reciprocals, then K smoothing factors, as floats, then the flag
// word.  Inside each 64-column slab the entries lie so that the four lanes of a quad, which work on the slab's
// four 16-column groups, read 64 consecutive bytes at once: chunk j (four columns) of group g at float4 4 j + g.
__host__ __device__ __forceinline__ int smooth_table_slot(int k) {
  return (k & ~63) | ((k & 12) << 2) | ((k & 48) >> 2) | (k & 3);
}
// table entry of one column; float64 keeps the nudged reciprocal to a single rounding
__device__ __forceinline__ float smooth_reciprocal(float s) {
  return static_cast<float>((1.0 / static_cast<double>(s)) * (1.0 + 2.384185791015625e-07));
}

// Near quotients of two rows of the same 16 columns; tb points at the group's chunk 0 of the slab's 64 entries in
// shared memory.  Every entry is loaded once for both rows: a 16-byte shared-memory load costs its wavefronts however
// many lanes share its address, and the load/store unit is what the fused quantizer keeps busiest.
__device__ __forceinline__ void smooth_multiply2(float2 (&f0)[8], float2 (&f1)[8], const float4* tb) {
  const float2 zero = make_float2(0.0f, 0.0f);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float4 t = tb[4 * j];
    const float2 a = make_float2(t.x, t.y), b = make_float2(t.z, t.w);
    f0[2 * j] = __ffma2_rn(f0[2 * j], a, zero); f0[2 * j + 1] = __ffma2_rn(f0[2 * j + 1], b, zero);
    f1[2 * j] = __ffma2_rn(f1[2 * j], a, zero); f1[2 * j + 1] = __ffma2_rn(f1[2 * j + 1], b, zero);
  }
}
// The exact quotients for a launch whose table is flagged: tb points at the smoothing factors themselves.
__device__ __forceinline__ void smooth_divide2(float2 (&f0)[8], float2 (&f1)[8], const float4* tb) {
  auto div = [](float2 v, float2 d) {                              // an underflow to -0 counts as +0
    return make_float2(__fadd_rn(__fdiv_rn(v.x, d.x), 0.0f), __fadd_rn(__fdiv_rn(v.y, d.y), 0.0f));
  };
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float4 t = tb[4 * j];
    const float2 a = make_float2(t.x, t.y), b = make_float2(t.z, t.w);
    f0[2 * j] = div(f0[2 * j], a); f0[2 * j + 1] = div(f0[2 * j + 1], b);
    f1[2 * j] = div(f1[2 * j], a); f1[2 * j + 1] = div(f1[2 * j + 1], b);
  }
}

constexpr int kScaleLutEntries = 128;

__device__ __forceinline__ float max3abs(float a, float b, float c) {
  float r;
  asm("max.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// Four pairs of floats -> eight E2M1 codes in one word (element 2j in bits 8j..8j+3, element 2j+1
// above it), round to nearest, saturating, sign included.
__device__ __forceinline__ uint32_t cvt_e2m1x8(float2 a, float2 b, float2 c, float2 d) {
  uint32_t r;
  asm("{\n\t.reg .b8 q0, q1, q2, q3;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 q0, %2, %1;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 q1, %4, %3;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 q2, %6, %5;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 q3, %8, %7;\n\t"
      "mov.b32 %0, {q0, q1, q2, q3};\n\t}"
      : "=r"(r)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y), "f"(d.x), "f"(d.y));
  return r;
}

// Four or eight floats -> their codes, element i in bits 4 i .. 4 i + 3
template <int N> __device__ __forceinline__ uint32_t cvt_e2m1(const float (&w)[N]);
template <> __device__ __forceinline__ uint32_t cvt_e2m1<8>(const float (&w)[8]) {
  return cvt_e2m1x8(make_float2(w[0], w[1]), make_float2(w[2], w[3]), make_float2(w[4], w[5]), make_float2(w[6], w[7]));
}
template <> __device__ __forceinline__ uint32_t cvt_e2m1<4>(const float (&w)[4]) {
  uint32_t r;
  asm("{\n\t.reg .b8 q0, q1, z;\n\tmov.b16 {z, _}, 0;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 q0, %2, %1;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 q1, %4, %3;\n\t"
      "mov.b32 %0, {q0, q1, z, z};\n\t}"
      : "=r"(r)
      : "f"(w[0]), "f"(w[1]), "f"(w[2]), "f"(w[3]));
  return r;
}

// amax -> scale byte: e4m3(clamp(amax / 6, 1e-12, 448)), the divide correctly rounded (amax is finite and >= 0;
// tiny quotients are clamped away)
__device__ __forceinline__ uint32_t scale_byte(float amax) {
  const float r6 = 0.16666667163372039794921875f;   // RN(1/6)
  const float s0 = amax * r6;
  float s = fmaf(fmaf(-6.0f, s0, amax), r6, s0);
  s = fminf(fmaxf(s, 1e-12f), 448.0f);
  return static_cast<uint32_t>(__nv_cvt_float_to_fp8(s, __NV_SATFINITE, __NV_E4M3));
}

// max |f| of a 16-element group
__device__ __forceinline__ float group_amax(const float2 (&f)[8]) {
  const float m0 = max3abs(f[0].x, f[0].y, f[1].x), m1 = max3abs(f[1].y, f[2].x, f[2].y);
  const float m2 = max3abs(f[3].x, f[3].y, f[4].x), m3 = max3abs(f[4].y, f[5].x, f[5].y);
  const float m4 = max3abs(f[6].x, f[6].y, f[7].x);
  return fmaxf(max3abs(m0, m1, m2), max3abs(m3, m4, f[7].y));
}
// amax of a 16-element group -> scale byte
__device__ __forceinline__ uint32_t group_scale_byte(const float2 (&f)[8]) { return scale_byte(group_amax(f)); }

// Zero scale (everything non-zero saturates) or the 448 clamp (ratios are unbounded): compare path
__device__ __forceinline__ void group_codes_compare(const float2 (&f)[8], uint32_t sb, uint32_t& code_lo, uint32_t& code_hi) {
  float sf = e4m3_to_f32(static_cast<uint8_t>(sb));
  sf = (sf == 0.0f) ? __uint_as_float(4u) : sf;     // 2^-147 * {.25 .. 5}: positive, below any normal number
  GroupBounds gb;
  gb.p[0] = sf * 0.25f; gb.p[1] = sf * 0.75f; gb.p[2] = sf * 1.25f; gb.p[3] = sf * 1.75f;
  gb.p[4] = sf * 2.5f;  gb.p[5] = sf * 3.5f;  gb.p[6] = sf * 5.0f;
  uint32_t lo = 0, hi = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) lo += (e2m1_code(f[j].x, gb) << (8 * j)) + (e2m1_code(f[j].y, gb) << (8 * j + 4));
#pragma unroll
  for (int j = 0; j < 4; ++j) hi += (e2m1_code(f[4 + j].x, gb) << (8 * j)) + (e2m1_code(f[4 + j].y, gb) << (8 * j + 4));
  code_lo = lo; code_hi = hi;
}

// Division by a per-column constant with its reciprocal at hand: q0 = RN(a r), e = a - s q0 (exact in one
// fma), q = RN(q0 + e r).  With r = RN(1 / s) this is the correctly rounded a / s whenever nothing over- or
// underflows on the way (Markstein's correction step; it needs a correctly rounded reciprocal and a divisor
// whose significand is not all ones, which a 16-bit s cannot be).  svdq_selftest_divide checks it against
// __fdiv_rn for every fp32 significand of a and every 11-bit significand of s; powers of two scale through
// all three steps exactly.  Arguments: the pair of dividends, the NEGATED divisors and the reciprocals.
__device__ __forceinline__ float2 divide_by_constant2(float2 a, float2 neg_s, float2 r) {
  const float2 q0 = __fmul2_rn(a, r);
  const float2 e = __ffma2_rn(neg_s, q0, a);
  return __ffma2_rn(e, r, q0);
}

// Scale byte from the largest near quotient of a group (see the head of this file).  Values above 448 saturate in
// the conversion, values below the smallest scale's rounding bound give byte 0: no clamps.
__device__ __forceinline__ uint32_t scale_byte_near(float amax) {
  const float v = amax * 0.16666662693023681640625f;                   // RN((1/6)(1 - 2^-22))
  const float snapped = __uint_as_float((__float_as_uint(v) + 8u) & 0xFFFFFFF0u);
  return static_cast<uint32_t>(__nv_cvt_float_to_fp8(snapped, __NV_SATFINITE, __NV_E4M3));
}
__device__ __forceinline__ float rcp_approx(float v) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}

// Multiplier of the codes of a group with scale byte sb, 1 <= sb < 0x7E
__device__ __forceinline__ float near_multiplier(uint32_t sb) {
  const __half_raw h = __nv_cvt_fp8_to_halfraw(static_cast<__nv_fp8_storage_t>(sb), __NV_E4M3);
  return rcp_approx(__half2float(__half(h))) * 1.000000476837158203125f;     // 1 + 2^-21
}
// The same for every scale byte; 0 for the two that take the compare path
__device__ __forceinline__ void fill_near_lut(float* lut, int tid, int nthreads) {
  for (int i = tid; i < kScaleLutEntries; i += nthreads) lut[i] = static_cast<uint32_t>(i) - 1u < 0x7Du ? near_multiplier(i) : 0.0f;
}

// An fp32 value cut to 12 significant bits (see the head of this file)
__device__ __forceinline__ float cut12(float v) { return __uint_as_float(__float_as_uint(v) & 0xFFFFF000u); }
// Codes of a group of fp32 values, c = near_multiplier of its scale byte (1 <= byte < 0x7E)
__device__ __forceinline__ void group_codes_cut(const float2 (&f)[8], float c, uint32_t& code_lo, uint32_t& code_hi) {
  const float2 cc = make_float2(c, c);
  float2 w[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) w[j] = __fmul2_rn(make_float2(cut12(f[j].x), cut12(f[j].y)), cc);
  code_lo = cvt_e2m1x8(w[0], w[1], w[2], w[3]);
  code_hi = cvt_e2m1x8(w[4], w[5], w[6], w[7]);
}

// One 16-element group of near quotients and its group_amax: scale byte and eight code bytes
__device__ __forceinline__ void quantize_group_near(const float2 (&f)[8], float amax, uint32_t& code_lo, uint32_t& code_hi, uint32_t& sbyte) {
  const uint32_t sb = scale_byte_near(amax);
  sbyte = sb;
  code_lo = code_hi = 0u;
  if (sb - 1u < 0x7Du) {
    const float c = near_multiplier(sb);
    const float2 cc = make_float2(c, c);
    float2 w[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) w[j] = __fmul2_rn(f[j], cc);
    code_lo = cvt_e2m1x8(w[0], w[1], w[2], w[3]);
    code_hi = cvt_e2m1x8(w[4], w[5], w[6], w[7]);
  } else if (amax != 0.0f) {
    // Not for groups of zeros: rows of the padding are nothing else, and with them in this path the warps that hold
    // them took twice the time of the others (any row count that is not a multiple of the padding: 3840 columns,
    // 500 rows 20.4 us against 9.6 us for 512, two K ranks each).
    group_codes_compare(f, sb, code_lo, code_hi);
  }
}

}  // namespace qmath
}  // namespace svdq
