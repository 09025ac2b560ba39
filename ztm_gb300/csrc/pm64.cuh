// pm64.cuh - the double point-mass sums (pointmass.cu: forward, pm_adjoint.cu:
// transposed) with the kernel's r^-3 in integer instructions.
//
// GB300 issues two FP64 results a clock per SM; a pair of the double sums took
// 12.7 of them (6.4 clocks), most in 1/r^3.  Both sums are arranged so that a
// pair needs two FP64 instructions, r^2 = z^2 + (X^2 + Y^2) and the
// multiply-add; r^-3 is formed from r^2's bits by pm_cube_rsqrt on the integer
// and FP32 pipes beside them, to 1.2e-16 rms (three products of the library's
// rsqrt: 2.1e-16).  A call sums one level's nodes at a time: X^2 + Y^2 is an
// integer of the fine grid (lengths in its spacing), z^2 is shared by a level.
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

// A non-negative integer below 2^31 as a double, by its bits.
__device__ __forceinline__ double pm_int_double(uint32_t v) {
  const int z = __clz((int)v);
  const uint32_t x = v << z;  // bit 31 set
  const double d = __hiloint2double((int)(((uint32_t)(1053 - z) << 20) + (x >> 11)), (int)(x << 21));
  return v ? d : 0.0;
}
#endif
