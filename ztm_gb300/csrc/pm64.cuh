// pm64.cuh - the double point-mass sums (pointmass.cu: forward, pm_adjoint.cu:
// transposed) with the kernel's r^-3 in integer instructions.
//
// GB300 issues two FP64 results a clock per SM; a pair of the double sums took
// 12.7 of them (6.4 clocks), most in 1/r^3.  Both sums are arranged so that a
// pair needs one FP64 instruction, the multiply-add.  A call sums one level's
// nodes at a time: X^2 + Y^2 is an integer of the fine grid (lengths in its
// spacing) and z^2 is shared by a level, so r^2 is formed in 64-bit fixed point
// (PmFixed) and r^-3 from that on the integer and FP32 pipes beside the FP64
// one, to 1.0e-16 rms (three products of the library's rsqrt: 2.1e-16).  Pairs
// much closer than the farthest, whose r^2 would have fewer than 53 bits, add
// r^2 in double and take its bits (pm_cube_rsqrt).
//
// Bound by issue and the ALU pipe (85 instructions a pair, the FP64 pipe 60%
// busy): a 61x61x33-node grid, 41x41 stations, 1.05 -> 0.80 ms a sum with r^2
// in fixed point instead of a second FP64 instruction.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "ztm_internal.cuh"

// Selected nodes in node order (k, j, i), and the first of every row (k, j).
struct __align__(16) Pm64Node {
  double w;  // weight (forward)
  int i;     // fine-grid i
  int n;     // node index
};
struct Pm64List {
  Pm64Node* node;  // up to N
  int* row;        // kk*jj + 1 offsets
};
size_t ztm_pm64_list_ws(const PmParams& p);
// adj: select by the adjoint's rule (pma_sel), else by the forward's weights.
void ztm_pm64_list(ztm_ctx* c, const PmParams& p, const double* d_drho, const int* d_mult, bool adj,
                   WsCarver& wc, Pm64List* list);

// Largest fine-grid row the forward's table of squares holds, and the largest
// offsets whose squares add up within 31 bits (adjoint).
constexpr int PM64_MAX_II = 4096;
constexpr int PM64_MAX_OFF = 32767;

#ifdef __CUDACC__

// r2^(-3/2) to about half a unit in the last place, for r2 in the middle of
// double's range; elsewhere (zero, subnormal, huge, not finite) by the library's
// rsqrt.  r2 = m 4^q, m in [1, 4): y a 24-bit float estimate of m^(-1/2) (its
// residual below 2^-22.4), P = y^2 exactly in 48 bits, g = 1 - m P from the
// middle words of the exact product, m^(-3/2) = y P (1 + 1.5 (g + 1.25 g^2)).
__device__ __forceinline__ double pm_cube_rsqrt(double r2) {
  const uint32_t hi = (uint32_t)__double2hiint(r2), lo = (uint32_t)__double2loint(r2);
  if (hi - 0x1a800000u >= 0x4b000000u) {  // outside 2^-600 .. 2^600
    const double rs = rsqrt(r2);
    return rs * rs * rs;
  }
  const int e = (int)(hi >> 20) - 1023, k = e & 1, q = e >> 1;
  const uint32_t m1 = (hi & 0x000fffffu) | 0x00100000u, m0 = lo;
  // m to 24 bits, rounded
  const float mf = __uint_as_float(((127u + k) << 23) + (((hi & 0x000fffffu) << 3) | (lo >> 29)) +
                                   ((lo >> 28) & 1u));
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(mf));
  y = fmaf(0.5f * y, fmaf(-__fmul_rn(mf, y), y, 1.f), y);
  const uint32_t Y = (__float_as_uint(fminf(y, 0.99999994f)) & 0x007fffffu) | 0x00800000u;  // y 2^24
  const uint64_t P = (uint64_t)Y * Y;
  const uint32_t p0 = (uint32_t)P, p1 = (uint32_t)(P >> 32);
  uint64_t acc = (uint64_t)m1 * p0 + __umulhi(m0, p0);
  acc += (uint64_t)m0 * p1;
  acc += (uint64_t)(m1 * p1) << 32;
  const int64_t g = -(int64_t)(acc << k);  // g 2^68 (the leading one drops out modulo 2^64)
  const int gs = (int)(g >> 30);
  const int c = (int)((g + (1 << 14)) >> 15) +
                (int)((((uint32_t)(gs * gs) >> 8) * 5u + (1u << 16)) >> 17);  // (g + 1.25 g^2) 2^53
  const uint64_t Q = (((uint64_t)Y * p1) << 23) + (((uint64_t)Y * p0) >> 9);  // y^3 2^63
  const int64_t pr = (int64_t)(int)((Q + (1ull << 31)) >> 32) * c;
  const uint64_t K = Q + ((pr + (pr >> 1) + (1 << 20)) >> 21);
  const int z = __clzll((long long)K);  // 0 .. 3
  const uint64_t x = K << z;
  const uint64_t r = (x >> 11) + ((x >> 10) & 1u);  // bit 52 adds one to the exponent
  return __longlong_as_double((long long)(((uint64_t)(uint32_t)(1022 - z - 3 * q) << 52) + r));
}

// r^2 = z2 + n in fixed point for integers n <= nmax: F 2^-sh, sh even, the
// largest one filling 61 bits and more.  A pair with at least 53 (PM_FIXED_MIN in the high
// word) is as accurate as the sum in double.
constexpr uint32_t PM_FIXED_MIN = 1u << 20;
struct __align__(16) PmFixed {
  uint64_t z;         // z2 2^sh, rounded
  uint32_t mul;       // n 2^sh = (n << a) mul
  short a, sh;
  __device__ __forceinline__ void set(double z2, uint32_t nmax, bool ok) {
    const double r2max = z2 + (double)nmax;
    const int e = (int)(((uint32_t)__double2hiint(r2max) >> 20) & 2047u) - 1023;  // log2, rounded down
    z = 0;  // F = 0, never fixed point: for NaN, infinite, huge and tiny
    mul = 0;
    a = sh = 0;
    if (!ok || !(r2max < 1099511627776.0) || e < -600) return;
    sh = (short)((62 - e) & ~1);
    const int s = min(__clz((int)max(nmax, 1u)), (int)sh);
    a = (short)s;
    mul = sh - s < 32 ? 1u << (sh - s) : 0u;  // 0: nmax = 0
    z = __double2ull_rn(z2 * __hiloint2double((1023 + sh) << 20, 0));
  }
  __device__ __forceinline__ uint64_t r2(uint32_t n) const { return z + (uint64_t)(n << a) * mul; }
};

// (F 2^-sh)^(-3/2), 2^52 <= F < 2^63, sh even, as pm_cube_rsqrt: r2 = m 4^q, m
// in [1, 4) in 64 bits, its float from the high word; factors scaled to full
// words, so that high words of products need no shifts.
__device__ __forceinline__ double pm_cube_rsqrt_fixed(uint64_t F, int sh) {
  const int z0 = __clz((int)(uint32_t)(F >> 32));
  const uint64_t M = F << (z0 & 30);  // m 2^62
  const int q = (31 - (sh >> 1)) - (z0 >> 1);
  const uint32_t m1 = (uint32_t)(M >> 32), m0 = (uint32_t)M;
  const float mf = __uint2float_rn(m1);  // m 2^30
  float y;                               // m^(-1/2) 2^-15
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(mf));
  y = fmaf(0.5f * y, fmaf(-__fmul_rn(mf, y), y, 1.f), y);
  const uint32_t Y = (__float_as_uint(fminf(y, 0.99999994f / 32768.f)) << 8) | 0x80000000u;  // 2^32
  const uint64_t P = (uint64_t)Y * Y;  // y^2 2^64
  const uint32_t p0 = (uint32_t)P, p1 = (uint32_t)(P >> 32);
  const uint64_t mp = (uint64_t)m1 * p1 + __umulhi(m0, p1) + __umulhi(m1, p0);  // m y^2 2^62
  // g = 1 - m y^2 in units of 2^-62; half a unit of c for its rounding and half
  // for the second term's
  const uint64_t g = (1ull << 62) + (1ull << 9) - mp;
  int c = (int)(uint32_t)(g >> 9);
  const uint32_t gs = (uint32_t)(c >> 15);
  c += (int)__umulhi(gs * gs, 640u);  // (g + 1.25 g^2) 2^53
  // y^3 2^63, and half a unit of its high word
  const uint64_t Q = (uint64_t)(Y >> 1) * p1 + (__umulhi(Y >> 1, p0) + 0x80000000u);
  const uint32_t Qh = (uint32_t)(Q >> 32);
  int64_t pr = (int64_t)(int)Qh * c;
  pr += (pr >> 1) + ((1ll << 20) - (1ll << 52));
  const uint64_t K = Q + (uint64_t)(pr >> 21);
  const int z = __clz((int)(uint32_t)(K >> 32));  // 0 .. 3
  const uint64_t x = K << z;
  const uint64_t r = (x >> 11) + ((x >> 10) & 1u);  // bit 52 adds one to the exponent
  return __longlong_as_double((long long)(((uint64_t)(uint32_t)(1022 - z - 3 * q) << 52) + r));
}

// A non-negative integer below 2^31 as a double, by its bits.
__device__ __forceinline__ double pm_int_double(uint32_t v) {
  const int z = __clz((int)v);
  const uint32_t x = v << z;  // bit 31 set
  const double d = __hiloint2double((int)(((uint32_t)(1053 - z) << 20) + (x >> 11)), (int)(x << 21));
  return v ? d : 0.0;
}
#endif
