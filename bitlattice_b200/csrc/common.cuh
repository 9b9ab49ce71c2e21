// Device and host helpers shared by the NVFP4 kernels: counter-based RNG, E4M3 scale codec, E2M1 level arithmetic,
// error reporting of the C ABI.
//
// Arithmetic contract: every kernel that produces codes, scale bytes or phase bytes reproduces the reference's fp32
// operation order bit for bit (bitlattice/reference.py; csrc/common.cuh of the reference). The translation units that
// include this header for such kernels are compiled with --fmad=false, so a*b+c is two roundings unless fmaf is
// written out.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdint>
#include <cstdio>

#include "../../include/bitlattice_b200.h"

namespace blb {

// ---------------------------------------------------------------------------------------------- host: errors

void set_error(const char* fmt, ...);

#define BL_REQUIRE(cond, ...)            \
  do {                                   \
    if (!(cond)) {                       \
      ::blb::set_error(__VA_ARGS__);     \
      return 1;                          \
    }                                    \
  } while (0)

#define BL_CUDA(expr)                                                                      \
  do {                                                                                     \
    cudaError_t err__ = (expr);                                                            \
    if (err__ != cudaSuccess) {                                                            \
      ::blb::set_error("%s failed: %s (%s:%d)", #expr, cudaGetErrorString(err__), __FILE__, __LINE__); \
      return 2;                                                                            \
    }                                                                                      \
  } while (0)

// Makes `device` current for the lifetime of the object and restores the previous device afterwards.
struct DeviceGuard {
  int prev = -1;
  bool changed = false;
  cudaError_t status = cudaSuccess;
  explicit DeviceGuard(int device) {
    status = cudaGetDevice(&prev);
    if (status == cudaSuccess && prev != device) {
      status = cudaSetDevice(device);
      changed = status == cudaSuccess;
    }
  }
  ~DeviceGuard() {
    if (changed) cudaSetDevice(prev);
  }
};

#define BL_DEVICE(device)                                                          \
  ::blb::DeviceGuard guard__(device);                                              \
  if (guard__.status != cudaSuccess) {                                             \
    ::blb::set_error("cannot select CUDA device %d: %s", device, cudaGetErrorString(guard__.status)); \
    return 2;                                                                      \
  }

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

int sm_count(int device);

// ---------------------------------------------------------------------------------------------- device: RNG

// u in [0, 1) from (element index, seed, step): bitlattice/reference.py:22-30. idx is truncated to 32 bits.
__device__ __forceinline__ float hash_uniform(uint32_t idx, uint32_t key) {
  uint32_t x = idx * 0x27D4EB2Fu + key;
  x = (x ^ (x >> 16)) * 0x7FEB352Du;
  x = (x ^ (x >> 15)) * 0x846CA68Bu;
  x ^= x >> 16;
  return static_cast<float>(x >> 8) * 5.9604644775390625e-08f;
}

__host__ __device__ __forceinline__ uint32_t hash_key(uint32_t seed, uint32_t step) {
  return seed * 0x9E3779B1u + step * 0x85EBCA77u;
}

// Rounding draw of the lattice projection (bitlattice/reference.py:41-51). For 'strat' key is hash_key(seed, 0).
struct RoundParams {
  int mode;        // BL_ROUND_*
  uint32_t key;
  float strat_j;
  float strat_k;
};

__device__ __forceinline__ float rounding_u(const RoundParams& rp, uint32_t idx) {
  if (rp.mode == BL_ROUND_SR) return hash_uniform(idx, rp.key);
  if (rp.mode == BL_ROUND_STRAT) {
    const float v = (rp.strat_j + hash_uniform(idx, rp.key)) / rp.strat_k;
    return v - truncf(v);
  }
  return 0.5f;
}

// ---------------------------------------------------------------------------------------------- device: E4M3

__device__ __forceinline__ float e4m3_decode(uint32_t byte) {
  __nv_fp8_e4m3 v;
  v.__x = static_cast<__nv_fp8_storage_t>(byte);
  return static_cast<float>(v);
}

// clamp to [2^-9, 448], round to nearest even (bitlattice/reference.py:71-72)
__device__ __forceinline__ uint32_t e4m3_encode(float s) {
  const __nv_fp8_e4m3 v(fminf(fmaxf(s, 0.001953125f), 448.0f));
  return v.__x;
}

// ---------------------------------------------------------------------------------------------- device: E2M1 levels
// The 15 levels of NVFP4 in ascending order have rank 0..14 (-6 ... 0 ... 6); rank 7 is zero.
// bitlattice/formats.py:151-170: code c < 8 -> rank 7 + c; code 8 (-0) reads as rank 7; code c > 8 -> rank 15 - c.

__device__ __forceinline__ int rank_of_code(uint32_t c) { return c < 8u ? 7 + static_cast<int>(c) : (c == 8u ? 7 : 15 - static_cast<int>(c)); }
__device__ __forceinline__ uint32_t code_of_rank(int r) { return r >= 7 ? static_cast<uint32_t>(r - 7) : static_cast<uint32_t>(15 - r); }

// magnitude of E2M1 index k in 0..7: {0, .5, 1, 1.5, 2, 3, 4, 6}, built from two byte tables with PRMT (no memory)
__device__ __forceinline__ float mag_of(uint32_t k) {
  const uint32_t hi = __byte_perm(0x3F3F3F00u, 0x40404040u, k << 12);
  const uint32_t lo = __byte_perm(0xC0800000u, 0xC0804000u, k << 8);
  return __uint_as_float(hi | lo);
}

__device__ __forceinline__ float level_of_rank(int r) {
  const int d = r - 7;
  const float m = mag_of(static_cast<uint32_t>(d < 0 ? -d : d));
  return d < 0 ? -m : m;
}

// rank of the nearest level, ties to the lower level: the number of midpoints strictly below x
// (bitlattice/reference.py:130-135)
__device__ __forceinline__ int nearest_rank(float x) {
  return (x > -5.0f) + (x > -3.5f) + (x > -2.5f) + (x > -1.75f) + (x > -1.25f) + (x > -0.75f) + (x > -0.25f) +
         (x > 0.25f) + (x > 0.75f) + (x > 1.25f) + (x > 1.75f) + (x > 2.5f) + (x > 3.5f) + (x > 5.0f);
}

// E2M1 code of the level nearest to v, ties to the lower value: rank -> canonical code
__device__ __forceinline__ uint32_t e2m1_code_nearest(float v) { return code_of_rank(nearest_rank(v)); }

// stochastic rounding between the two E2M1 neighbours of v (bitlattice/fp4ref.py:71-78)
__device__ __forceinline__ uint32_t e2m1_code_sr(float v, float u) {
  const float a = fminf(fabsf(v), 6.0f);
  uint32_t m = (a >= 0.5f) + (a >= 1.0f) + (a >= 1.5f) + (a >= 2.0f) + (a >= 3.0f) + (a >= 4.0f) + (a >= 6.0f);
  if (m < 7u) {
    const float lo = mag_of(m), hi = mag_of(m + 1u);
    m += u * (hi - lo) < a - lo;
  }
  return (v < 0.0f && m ? 8u : 0u) | m;
}

// ---------------------------------------------------------------------------------------------- device: division
// x / y rounded to nearest from ry = RN(1 / y), which the caller shares between the many quotients by one divisor:
// Markstein's correction ("Computation of elementary functions on the IBM RISC System/6000 processor", IBM Journal of
// Research and Development 34, 1990; the case of a divisor known in advance: Brisebarre, Muller and Raina, "Accelerating
// correctly rounded floating-point division when the divisor is known in advance", IEEE Transactions on Computers 53,
// 2004): the product q = RN(x ry) is off by less than two units in the last place, its residual r = x - y q is formed by
// one fused multiply-add, and RN(q + r ry) is the correctly rounded quotient. The theorems leave the divisors open for which
// q is not a neighbour of the quotient, so every pair of fp32 significands is compared with the plain division
// (bl_selftest_division_slice; 2^46 pairs, none differs on a B200). Exponents only scale the three operations while
// nothing leaves the normal range and the residual, a multiple of 2^-48 x or less, is a float: |x| > 2^-100, a normal ry, a
// quotient far from either end. The callers of div2p establish that; div_rn checks it.
static __device__ __noinline__ float div_general(float x, float y) { return x / y; }

__device__ __forceinline__ float div_rn(float x, float y, float ry) {
  const float q0 = x * ry;
  const float q = fmaf(fmaf(-y, q0, x), ry, q0);
  const float aq = fabsf(q0);
  // zero, tiny, huge or non-finite: the general path, kept out of line so that it costs nothing when not taken
  const bool in_range = aq > 1e-30f && aq < 1e30f && fabsf(x) > 7.8886091e-31f && fabsf(ry) >= 1.1754943508222875e-38f;
  if (__builtin_expect(!in_range, 0)) return div_general(x, y);
  return q;
}

// The two divisions of a block scale, amax / 6 and the quotient by the per-tensor scale g, checked by their quotients alone:
// the first's bounds its dividend (6e-30 > 2^-100), and rg = scale_rcp(g) is a NaN, which fails every check, unless g is
// large enough (1e-12, the least that is ever computed) for the second's to do so. With the dividends checked themselves the
// row quantizers took 1 to 2 % longer.
constexpr float kInv6 = 0.16666667163372039794921875f;   // the float nearest to 1/6
constexpr float kScaleQuotient = 8.6736174e-19f;         // 2^-60: 2^-60 * 1e-12 > 2^-100; a block 2^69 below the maximum

__device__ __forceinline__ float scale_rcp(float g) {
  return g >= 1e-12f && g < 8.507059e37f ? __frcp_rn(g) : __int_as_float(0x7FFFFFFF);
}
__device__ __forceinline__ float div_checked(float x, float y, float ry, float lo, bool& ok) {
  const float q0 = x * ry, aq = fabsf(q0);
  ok = ok && aq > lo && aq < 1e30f;
  return fmaf(fmaf(-y, q0, x), ry, q0);
}
// div_rn for callers whose dividend is above 2^-100, or the quotient immaterial
__device__ __forceinline__ float div_quotient(float x, float y, float ry) {
  bool ok = true;
  const float q = div_checked(x, y, ry, 1e-30f, ok);
  return __builtin_expect(ok, 1) ? q : div_general(x, y);
}
__device__ __forceinline__ float div_six(float x) { return div_quotient(x, 6.0f, kInv6); }
__device__ __forceinline__ float div_scale(float x, float g, float rg) {
  bool ok = true;
  const float q = div_checked(x, g, rg, kScaleQuotient, ok);
  return __builtin_expect(ok, 1) ? q : div_general(x, g);
}
// amax / 6 / g; ok: both quotients are exact (amax is neither zero nor tiny beside g, infinite nor a NaN)
__device__ __forceinline__ float div_block_scale(float amax, float g, float rg, bool& ok) {
  return div_checked(div_checked(amax, 6.0f, kInv6, 1e-30f, ok), g, rg, kScaleQuotient, ok);
}

// 1 / x to within an ulp or so: a start for a correction, or a bracket
__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// ---------------------------------------------------------------------------------------------- device: fp32 pairs
// Two independent fp32 operations per instruction, each lane rounded to nearest like the scalar operation (the fused
// multiply-add is written out only where a single rounding is wanted: the residuals of the divisions).

using f32x2 = unsigned long long;

__device__ __forceinline__ f32x2 pk(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void upk(f32x2 p, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(p)); }
__device__ __forceinline__ f32x2 mul2p(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 add2p(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 add2p_up(f32x2 a, f32x2 b) {       // rounded toward +infinity
  f32x2 r;
  asm("add.rp.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 sub2p(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 fma2p(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// a * b per lane, rounded once, for products that FEED A SUM: written as a fused multiply-add with a +0 addend, which
// the assembler can neither merge with the following add (it would have to fuse two roundings) nor turn back into a
// plain multiply (the +0 turns a product of -0 into +0). Only for uses where the sign of a zero product cannot matter.
__device__ __forceinline__ f32x2 prod2p(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(0ull));
  return r;
}
// x / y per lane from ny = -y and ry = rcp_rn(y): div_rn without its range check (the caller establishes the range)
__device__ __forceinline__ f32x2 div2p(f32x2 x, f32x2 ny, f32x2 ry) {
  const f32x2 q = mul2p(x, ry);
  return fma2p(fma2p(ny, q, x), ry, q);
}

// ---------------------------------------------------------------------------------------------- device: fast E2M1
// The hardware conversion cvt.rn.satfinite.e2m1x2.f32 rounds two floats to E2M1 nibbles (ties to even, -0 kept).
// It gives the reference's code (ties to the lower level, +0 only) whenever its input is not at, or within rounding
// error of, a midpoint between two levels; the callers below establish that by converting a lower and an upper bound
// of the exact quotient and comparing, and take the exact ladder otherwise.

// byte with the code of `hi` in the upper and of `lo` in the lower nibble
__device__ __forceinline__ uint32_t cvt_e2m1x2(float hi, float lo) {
  uint32_t r;
  asm("{\n\t.reg .b8 t;\n\tcvt.rn.satfinite.e2m1x2.f32 t, %1, %2;\n\tcvt.u32.u8 %0, t;\n\t}" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

// 8 floats -> 8 nibbles (element i in nibble i)
__device__ __forceinline__ uint32_t cvt_e2m1x8(const float v[8]) {
  return cvt_e2m1x2(v[1], v[0]) | (cvt_e2m1x2(v[3], v[2]) << 8) | (cvt_e2m1x2(v[5], v[4]) << 16) |
         (cvt_e2m1x2(v[7], v[6]) << 24);
}

// clear the sign bit of every nibble whose magnitude is zero (-0 -> +0: the reference never writes code 8)
__device__ __forceinline__ uint32_t e2m1_drop_negative_zero(uint32_t w) {
  const uint32_t m = w & 0x77777777u;
  const uint32_t nz = (m | (m >> 1) | (m >> 2)) & 0x11111111u;
  return m | (w & (nz << 3));
}

// Round-to-nearest codes (ties to the lower level) of v[i] / se for 8 values, se > 0.
// inv_lo / inv_hi: (1/se) scaled by (1 - 2^-20) and (1 + 2^-20): v*inv_lo and v*inv_hi bracket the exact quotient
// (the two roundings of each product are below 2^-22 relative), E2M1 rounding is monotone, so equal conversions of
// the two bounds equal the conversion of the quotient, which then is no tie.
// the exact ladder for 8 values: kept out of line so the common path stays small
static __device__ __noinline__ uint32_t e2m1_nearest_x8_exact(float v0, float v1, float v2, float v3, float v4, float v5,
                                                       float v6, float v7, float se) {
  return e2m1_code_nearest(v0 / se) | (e2m1_code_nearest(v1 / se) << 4) | (e2m1_code_nearest(v2 / se) << 8) |
         (e2m1_code_nearest(v3 / se) << 12) | (e2m1_code_nearest(v4 / se) << 16) | (e2m1_code_nearest(v5 / se) << 20) |
         (e2m1_code_nearest(v6 / se) << 24) | (e2m1_code_nearest(v7 / se) << 28);
}

__device__ __forceinline__ uint32_t e2m1_nearest_x8(const float v[8], float se, float inv_lo, float inv_hi) {
  float a[8], b[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    a[i] = v[i] * inv_lo;
    b[i] = v[i] * inv_hi;
  }
  const uint32_t wa = cvt_e2m1x8(a), wb = cvt_e2m1x8(b);
  if (__builtin_expect(wa == wb, 1)) return e2m1_drop_negative_zero(wa);
  return e2m1_nearest_x8_exact(v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], se);   // at or next to a midpoint
}

// Stochastic-rounding codes of x[i] = v[i] * inv (bitlattice/fp4ref.py:71-78) for 8 values; u from hash(idx0 + i).
// lo = largest level <= min(|x|, 6) (the float truncated to one mantissa bit, or 0 / 0.5 below 1), gap to the next.
__device__ __forceinline__ uint32_t e2m1_sr_x8(const float v[8], float inv, uint32_t key, uint32_t idx0) {
  float r[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float x = v[i] * inv;
    const float a = fminf(fabsf(x), 6.0f);
    const uint32_t ab = __float_as_uint(a);
    const float lo = a >= 1.0f ? __uint_as_float(ab & 0xFFC00000u) : (a >= 0.5f ? 0.5f : 0.0f);
    const float gap = a >= 2.0f ? __uint_as_float((ab & 0x7F800000u) - 0x00800000u) : 0.5f;
    const float u = hash_uniform(idx0 + i, key);
    const bool up = lo < 6.0f && u * gap < a - lo;
    r[i] = copysignf(up ? lo + gap : lo, x);
  }
  return e2m1_drop_negative_zero(cvt_e2m1x8(r));
}

// ---------------------------------------------------------------------------------------------- device: blocks of 16
// Whole 16-element blocks in one thread, written for few issue slots per element: packed fp32x2 multiplies, four
// conversions merged into one register, and stochastic rounding decided in 2^-25 fixed point.

// {a * s, b * s}: one packed multiply, each lane rounded to nearest like a scalar multiply
__device__ __forceinline__ void mul2(float a, float b, float s, float& ra, float& rb) {
  asm("{\n\t.reg .b64 p, q;\n\t"
      "mov.b64 p, {%2, %3};\n\t"
      "mov.b64 q, {%4, %4};\n\t"
      "mul.rn.f32x2 p, p, q;\n\t"
      "mov.b64 {%0, %1}, p;\n\t}"
      : "=f"(ra), "=f"(rb)
      : "f"(a), "f"(b), "f"(s));
}

// 8 floats -> 8 nibbles in one register (element i in nibble i), hardware rounding (nearest, ties to even)
__device__ __forceinline__ uint32_t cvt_e2m1x8_merged(const float v[8]) {
  uint32_t w;
  asm("{\n\t.reg .b8 t0, t1, t2, t3;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 t0, %2, %1;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 t1, %4, %3;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 t2, %6, %5;\n\t"
      "cvt.rn.satfinite.e2m1x2.f32 t3, %8, %7;\n\t"
      "mov.b32 %0, {t0, t1, t2, t3};\n\t}"
      : "=r"(w)
      : "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]));
  return w;
}

// Round-to-nearest codes (ties to the lower level) of (v[i] * pre) / se for 16 values, se > 0; pre is 1 or a power of
// two folded into the bracket. inv approximates 1 / se to a few ulps; the bracket (1 -+ 2^-19) around it contains the
// exact quotient, so equal conversions of both ends are the conversion of the quotient, which then is no tie;
// otherwise (at or next to a midpoint) the exact ladder decides.
// exact code of one value, out of line: the per-element repair of e2m1_rtn16
static __device__ __noinline__ uint32_t e2m1_nearest_exact(float v, float se) { return e2m1_code_nearest(v / se); }

__device__ __forceinline__ uint2 e2m1_rtn16(const float v[16], float pre, float se, float inv) {
  const float lo = inv * pre * 0.99999809265136718750f, hi = inv * pre * 1.00000190734863281250f;
  float a[16], b[16];
#pragma unroll
  for (int i = 0; i < 16; i += 2) {
    mul2(v[i], v[i + 1], lo, a[i], a[i + 1]);
    mul2(v[i], v[i + 1], hi, b[i], b[i + 1]);
  }
  uint32_t w[2] = {cvt_e2m1x8_merged(a), cvt_e2m1x8_merged(a + 8)};
  uint32_t d[2] = {w[0] ^ cvt_e2m1x8_merged(b), w[1] ^ cvt_e2m1x8_merged(b + 8)};
  // (the reciprocal is only trusted for scales well inside the normal range)
  if (!(se > 1e-30f && se < 1e30f)) d[0] = d[1] = 0xFFFFFFFFu;
  if (__builtin_expect((d[0] | d[1]) != 0u, 0)) {
    // Values at a midpoint between two levels are common with 8-bit inputs and few-bit scales: repair only the
    // elements whose two conversions differ.
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const uint32_t m = 0xFu << (4 * (i & 7));
      if (d[i >> 3] & m) w[i >> 3] = (w[i >> 3] & ~m) | (e2m1_nearest_exact(v[i] * pre, se) << (4 * (i & 7)));
    }
  }
  return make_uint2(e2m1_drop_negative_zero(w[0]), e2m1_drop_negative_zero(w[1]));
}

// the same for two blocks at once, one in each lane of the pairs (pre = 1)
__device__ __forceinline__ void e2m1_rtn16x2(const f32x2 v[16], float se_a, float se_b, float inv_a, float inv_b, uint32_t ca[2],
                                             uint32_t cb[2]) {
  constexpr float kLo = 0.99999809265136718750f, kHi = 1.00000190734863281250f;
  const f32x2 lo = pk(inv_a * kLo, inv_b * kLo), hi = pk(inv_a * kHi, inv_b * kHi);
  const bool sane = se_a > 1e-30f && se_a < 1e30f && se_b > 1e-30f && se_b < 1e30f;
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const f32x2* p = v + 8 * half;
    float xa[8], xb[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) upk(mul2p(p[i], lo), xa[i], xb[i]);
    uint32_t wa = cvt_e2m1x8_merged(xa), wb = cvt_e2m1x8_merged(xb);
#pragma unroll
    for (int i = 0; i < 8; ++i) upk(mul2p(p[i], hi), xa[i], xb[i]);
    uint32_t da = wa ^ cvt_e2m1x8_merged(xa), db = wb ^ cvt_e2m1x8_merged(xb);
    if (__builtin_expect((da | db) != 0u || !sane, 0)) {
      if (!sane) da = db = 0xFFFFFFFFu;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint32_t m = 0xFu << (4 * i);
        float a, b;
        upk(p[i], a, b);
        if (da & m) wa = (wa & ~m) | (e2m1_nearest_exact(a, se_a) << (4 * i));
        if (db & m) wb = (wb & ~m) | (e2m1_nearest_exact(b, se_b) << (4 * i));
      }
    }
    ca[half] = e2m1_drop_negative_zero(wa);
    cb[half] = e2m1_drop_negative_zero(wb);
  }
}

// Stochastic-rounding codes of x[i] = v[i] * inv for 16 values (bitlattice/fp4ref.py:71-78), u from hash(idx0 + i), every
// draw decided on all of its 24 bits. With a = min(|x|, 6) and A = ceil(a * 2^25) (exact for a >= 0.5), shifting A right by
// t = [a >= 2] + [a >= 4] puts the level index below a in the bits above 24 and the position between the two neighbouring
// levels, as a fraction of 2^24, in the bits below. The draw n = hash >> 8 rounds up iff n < that fraction, which is the
// carry of adding (2^24 - 1 - n): so the code is ((A >> t) + (~hash >> 8) >> 24) + 2 t. Identical to comparing
// u * gap < a - lo in real numbers, which is what the reference's fp32 expression evaluates without rounding.
// Out of line, for eight elements x = v * inv among which sr_pair cannot decide one on 16 bits.
static __device__ __noinline__ uint32_t e2m1_sr8_exact(float4 x0, float4 x1, uint32_t h0) {
  const float x[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
  uint32_t w = 0u;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float a = fminf(fabsf(x[i]), 6.0f);
    const uint32_t A = __float2uint_ru(a * 33554432.0f);
    const uint32_t t = __byte_perm(0x02020100u, 0u, A >> 26);
    uint32_t h = h0 + static_cast<uint32_t>(i) * 0x27D4EB2Fu;
    h = (h ^ (h >> 16)) * 0x7FEB352Du;
    h = (h ^ (h >> 15)) * 0x846CA68Bu;
    h = ~(h ^ (h >> 16));
    const uint32_t k = (((A >> t) + (h >> 8)) >> 24) + 2u * t;
    w |= (k | ((__float_as_uint(x[i]) >> 28) & 8u)) << (4 * i);
  }
  return e2m1_drop_negative_zero(w);
}

// Two elements x (already times inv) with the first hash words ha, hb of their draws -> the levels they round to.
//
// E2M1 is a float with one mantissa bit and subnormals below 1, so x * 2^-126, whose subnormals begin at the same place,
// carries the level index in bits 22 and up of its bit pattern and the position between the two neighbouring levels
// in the 22 bits below (truncated, for |x| < 1; the sign stays in bit 31). The draw rounds up iff it is below that
// fraction: the carry of adding its complement. The hash ends with x ^= x >> 16, which leaves the upper 16 bits as they
// are, so the draw's upper 16 bits decide unless they equal the fraction's; the last step and the low bits are left
// out here. z collects the minimum of ((sum's bits 6 .. 21) + 1 mod 2^16) << 16 plus lower bits: below 2^17 for every
// element that needs its low bits (2 of 2^16 sums, its eight elements then take e2m1_sr8_exact). A carry out of the last level
// gives 8, which the conversion to E2M1 saturates to 6, as it does everything above 6.
//
// The loop is bound by issue (83 % of the slots in the row quantizer) beside the ALU pipe (shifts, bit operations, selects; 64
// lanes per SM and clock; 77 %), which alone bound it before: 8 such instructions per element against 20 -- no clamp, no float-to-integer conversion, no level look-up, no sign and nibble merging --
// with the additions that can be multiply-adds on the other pipe. At 65536 x 4096 bf16 on a B200: 310 -> 187 us for the row
// quantizer, 468 -> 331 us for the transposed one. (The rounding conversion cvt.rs of this architecture draws from 8 bits per
// element and cannot give the reference's codes.)
static __device__ __constant__ uint32_t kPipeMul[1] = {1u << 10};   // from constant memory, so that the product stays a product

__device__ __forceinline__ f32x2 mul2p_down(f32x2 a, f32x2 b) {            // rounded toward zero
  f32x2 r;
  asm("mul.rz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

__device__ __forceinline__ void sr_pair(f32x2 x, uint32_t ha, uint32_t hb, float& la, float& lb, uint32_t& z) {
  constexpr float kDown = 1.1754943508222875e-38f, kUp = 8.507059173023462e+37f;     // 2^-126, 2^126
  float ba, bb;
  upk(mul2p_down(x, pk(kDown, kDown)), ba, bb);
  const uint32_t ya = ((ha ^ (ha >> 16)) * 0x7FEB352Du), yb = ((hb ^ (hb >> 16)) * 0x7FEB352Du);
  const uint32_t na = (ya ^ (ya >> 15)) * (0u - 0x846CA68Bu) - 1u;                   // ~(product): -x - 1
  const uint32_t nb = (yb ^ (yb >> 15)) * (0u - 0x846CA68Bu) - 1u;
  const uint32_t sa = __float_as_uint(ba) + (na >> 10), sb = __float_as_uint(bb) + (nb >> 10);
  const uint32_t shl10 = kPipeMul[0];
  z = __vimin3_u32(z, sa * shl10 + 0x10000u, sb * shl10 + 0x10000u);
  upk(mul2p(pk(__uint_as_float(sa & 0xFFC00000u), __uint_as_float(sb & 0xFFC00000u)), pk(kUp, kUp)), la, lb);
}

constexpr uint32_t kSrUndecided = 0x20000u;

// one block, elements (2 j, 2 j + 1) in the pairs; special: a product can be a NaN
__device__ __forceinline__ uint2 e2m1_sr16(const float v[16], float inv, uint32_t key, uint32_t idx0, bool special = false) {
  const uint32_t h0 = idx0 * 0x27D4EB2Fu + key;
  const f32x2 inv2 = pk(inv, inv);
  uint32_t w[2];
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const float* p = v + 8 * half;
    const uint32_t h = h0 + static_cast<uint32_t>(8 * half) * 0x27D4EB2Fu;
    float l[8];
    uint32_t z = special ? 0u : 0xFFFFFFFFu;
#pragma unroll
    for (int i = 0; i < 8; i += 2)
      sr_pair(mul2p(pk(p[i], p[i + 1]), inv2), h + static_cast<uint32_t>(i) * 0x27D4EB2Fu,
              h + static_cast<uint32_t>(i + 1) * 0x27D4EB2Fu, l[i], l[i + 1], z);
    w[half] = e2m1_drop_negative_zero(cvt_e2m1x8_merged(l));
    if (__builtin_expect(z < kSrUndecided, 0))
      w[half] = e2m1_sr8_exact(make_float4(p[0] * inv, p[1] * inv, p[2] * inv, p[3] * inv),
                               make_float4(p[4] * inv, p[5] * inv, p[6] * inv, p[7] * inv), h);
  }
  return make_uint2(w[0], w[1]);
}

// two blocks at once, one in each lane of the pairs; h0a, h0b: first hash words of their first elements
__device__ __forceinline__ void e2m1_sr16x2(const f32x2 v[16], float inv_a, float inv_b, uint32_t h0a, uint32_t h0b,
                                            uint32_t ca[2], uint32_t cb[2]) {
  const f32x2 inv2 = pk(inv_a, inv_b);
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const f32x2* p = v + 8 * half;
    const uint32_t ha = h0a + static_cast<uint32_t>(8 * half) * 0x27D4EB2Fu, hb = h0b + static_cast<uint32_t>(8 * half) * 0x27D4EB2Fu;
    float la[8], lb[8];
    uint32_t z = 0xFFFFFFFFu;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      sr_pair(mul2p(p[i], inv2), ha + static_cast<uint32_t>(i) * 0x27D4EB2Fu, hb + static_cast<uint32_t>(i) * 0x27D4EB2Fu,
              la[i], lb[i], z);
    ca[half] = e2m1_drop_negative_zero(cvt_e2m1x8_merged(la));
    cb[half] = e2m1_drop_negative_zero(cvt_e2m1x8_merged(lb));
    if (__builtin_expect(z < kSrUndecided, 0)) {
      float xa[8], xb[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) upk(mul2p(p[i], inv2), xa[i], xb[i]);
      ca[half] = e2m1_sr8_exact(make_float4(xa[0], xa[1], xa[2], xa[3]), make_float4(xa[4], xa[5], xa[6], xa[7]), ha);
      cb[half] = e2m1_sr8_exact(make_float4(xb[0], xb[1], xb[2], xb[3]), make_float4(xb[4], xb[5], xb[6], xb[7]), hb);
    }
  }
}

// max |v[i]| of 16 values (three-input maximum of this architecture): a NaN is ignored, unless all are (0)
__device__ __forceinline__ float max_abs3(float a, float b, float c) {
  float r;
  asm("max.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float max_abs16(const float v[16]) {
  const float a = max_abs3(v[0], v[1], v[2]), b = max_abs3(v[3], v[4], v[5]), c = max_abs3(v[6], v[7], v[8]),
              d = max_abs3(v[9], v[10], v[11]), e = max_abs3(v[12], v[13], v[14]);
  return max_abs3(max_abs3(a, b, c), max_abs3(d, e, v[15]), 0.0f);
}
// the same with NaN kept
__device__ __forceinline__ float max_abs3_nan(float a, float b, float c) {
  float r;
  asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float max_abs16_nan(const float v[16]) {
  const float a = max_abs3_nan(v[0], v[1], v[2]), b = max_abs3_nan(v[3], v[4], v[5]), c = max_abs3_nan(v[6], v[7], v[8]),
              d = max_abs3_nan(v[9], v[10], v[11]), e = max_abs3_nan(v[12], v[13], v[14]);
  return max_abs3_nan(max_abs3_nan(a, b, c), max_abs3_nan(d, e, v[15]), 0.0f);
}

// sr_pair must not see a NaN: the sum with the draw would carry its bit pattern into a zero. Here a block that can hold one is
// decided on 24 bits, where it takes the largest level, as in the plain expressions: no product is a NaN if the largest
// (NaN kept) is finite.
__device__ __forceinline__ uint2 e2m1_sr16_any(const float v[16], float inv, uint32_t key, uint32_t idx0) {
  return e2m1_sr16(v, inv, key, idx0, !(max_abs16_nan(v) * inv < __int_as_float(0x7F800000)));
}

// Stochastic codes and scale byte of a block for which div_block_scale is not exact: its maximum is zero, tiny, infinite or
// (NaN kept) unknown, or the per-tensor scale is out of range. The scale ignores a NaN, which takes the largest level.
struct SrBlock {
  uint2 codes;
  uint32_t scale;
};
static __device__ __noinline__ SrBlock sr_block_general(float4 v0, float4 v1, float4 v2, float4 v3, float g, uint32_t h0) {
  const float v[16] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w, v2.x, v2.y, v2.z, v2.w, v3.x, v3.y, v3.z, v3.w};
  SrBlock out;
  out.scale = e4m3_encode(max_abs16(v) / 6.0f / g);
  const float t = e4m3_decode(out.scale) * g;
  const float inv = t > 0.0f ? __frcp_rn(t) : 0.0f;
  out.codes = make_uint2(0u, 0u);
  if (max_abs16_nan(v) * inv != 0.0f) {                         // else nothing but zeros
    out.codes.x = e2m1_sr8_exact(make_float4(v[0] * inv, v[1] * inv, v[2] * inv, v[3] * inv),
                                 make_float4(v[4] * inv, v[5] * inv, v[6] * inv, v[7] * inv), h0);
    out.codes.y = e2m1_sr8_exact(make_float4(v[8] * inv, v[9] * inv, v[10] * inv, v[11] * inv),
                                 make_float4(v[12] * inv, v[13] * inv, v[14] * inv, v[15] * inv), h0 + 8u * 0x27D4EB2Fu);
  }
  return out;
}
__device__ __forceinline__ SrBlock sr_block_general(const float v[16], float g, uint32_t h0) {
  return sr_block_general(make_float4(v[0], v[1], v[2], v[3]), make_float4(v[4], v[5], v[6], v[7]),
                          make_float4(v[8], v[9], v[10], v[11]), make_float4(v[12], v[13], v[14], v[15]), g, h0);
}

// ---------------------------------------------------------------------------------------------- device: dense loads

template <typename T> __device__ __forceinline__ float to_f(T v);
template <> __device__ __forceinline__ float to_f<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <> __device__ __forceinline__ float to_f<__half>(__half v) { return __half2float(v); }

template <typename T> __device__ __forceinline__ T from_f(float v);
template <> __device__ __forceinline__ float from_f<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <> __device__ __forceinline__ __half from_f<__half>(float v) { return __float2half_rn(v); }

// 8 consecutive elements starting at a multiple of 8 (16-byte aligned for 2-byte types, 32 for fp32)
template <typename T>
__device__ __forceinline__ void load8(const T* p, float v[8]) {
  if constexpr (sizeof(T) == 4) {
    const float4 a = reinterpret_cast<const float4*>(p)[0];
    const float4 b = reinterpret_cast<const float4*>(p)[1];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else {
    const uint4 raw = *reinterpret_cast<const uint4*>(p);
    const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = to_f<T>(e[i]);
  }
}

}  // namespace blb
