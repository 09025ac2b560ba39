// lm.cu - the damped Gauss-Newton step of ZTM's optimiser on the GPU.
//
// LMA::fit (TFM.cpp:155-167) forms, per iteration, JJ = MTM(J) = J^T J
// (zmath.cpp:260-262, one host thread per column), M = diag(diag(JJ)),
// A = diag(1/sig^2), and for every damping pair d of its grid the trial
// B = b + inv(JJ + d0 M + d1 A) J^T r (TFM.cpp:160), the inverse by
// Gauss-Jordan elimination with partial pivoting (zmath.cpp:129-140), one
// host thread per damping pair.
//
// Both parts are matrix products, and GB300's FP64 pipe issues two results a
// clock per SM: J^T J of 12000 x 2700 alone took it 84 ms at 99% busy.  Here the
// products run on the tensor cores in exact integer arithmetic (the splitting
// of Ozaki, Ogita, Oishi and Rump, Numer. Algorithms 59, 2012): every column of
// J (row of a panel) is scaled by a power of two and cut into seven signed
// 8-bit digits, 56 bits; a digit is exact in bf16, a product of two below 2^14,
// and sums of at most 2^10 products exact in the FP32 accumulator.  The digit
// products with p + q <= 6 are summed by level p + q in TMEM, read back before
// they can exceed 2^24, and gathered in 64-bit integers: 28 bf16 products in
// place of one in double, with less rounding than the FP64 sum (one, at the
// end; the digits left out are below 2^-56 of the product of the two columns'
// largest entries).  See oz_kernel.
//   lm_colstat / lm_colfinish  largest entry of every column, and J^T r
//   lm_slice                   digits of J in the tensor core's operand layout
//   oz_kernel<0>, lm_reduce    J^T J: upper tiles, row slices, then mirrored
//   lm_assemble                per damping pair the lower half of
//                              JJ + d0 M + d1 A with J^T r as a further row
//   lm_potrf, lm_trsm,         Cholesky by panels of 64 columns, all pairs at
//   oz_kernel<1>               once: diagonal block and panel in double, the
//                              trailing update on the tensor cores.  The further
//                              row comes out as the forward substitution.
//   lm_backstep                L^T x = y, 64 unknowns a launch
//   lm_finish                  B = b + x
//   lm_lu_all                  the systems that are not positive definite (a
//                              pivot that is zero, negative or not a number:
//                              a parameter without data or damping, negative
//                              damping): blocked LU with the reference's pivot
//                              rule, one launch that ends at once when there
//                              are none; singular ones keep B = b, as the
//                              reference's inv returns zeros there
// A positive definite system needs no pivoting, and the step is the
// reference's up to rounding.
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>

#include "tc_tf32.cuh"
#include "ztm_internal.cuh"

namespace {

__device__ __forceinline__ double lm_pow2(int e) {  // 2^e, e clamped to doubles' range
  return __hiloint2double((1023 + max(-1022, min(1023, e))) << 20, 0);
}

// ---- exact products on the tensor cores -------------------------------------
constexpr int OZ_S = 7;         // digits
constexpr int OZ_M = 128;       // rows of a tile (operand A)
constexpr int OZ_N = 64;        // columns of a tile (operand B): 7 levels x 64
                                // columns fill 448 of TMEM's 512
constexpr int OZ_KC = 32;       // K of a shared-memory stage
constexpr int OZ_T = 320;       // 8 warps read back, one copies, one issues MMAs
constexpr int OZ_SLICE_A = OZ_M * OZ_KC * 2;          // bytes of a digit's stage tile
constexpr int OZ_SLICE_B = OZ_N * OZ_KC * 2;
constexpr int OZ_CHUNK = OZ_S * OZ_SLICE_A;           // 57,344 bytes in global memory
constexpr int OZ_STAGE = OZ_CHUNK + OZ_S * OZ_SLICE_B;  // 86,016 bytes
constexpr size_t OZ_SMEM = 1024 + 2 * (size_t)OZ_STAGE;
constexpr int OZ_COLS = 512;    // TMEM columns (all: one block per SM)

// Digits of a block of 128 indices and 32 values of K, as lm_slice and lm_trsm
// write them: [digit][k / 8][index / 8][index % 8][k % 8] in bf16, K-major core
// matrices of 8 x 16 bytes without swizzle.
__host__ __device__ constexpr uint32_t oz_off(int digit, int k8, int i) {
  return (uint32_t)(digit * OZ_SLICE_A + k8 * (OZ_M * 16) + i * 16);
}

// Instruction descriptor (kind::f16): D F32 (bits 4-5 = 1), A and B BF16 (bits
// 7-9, 10-12 = 1), both K-major, N >> 3 in bits 17-22, M >> 4 in bits 24-28.
constexpr uint32_t OZ_IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(OZ_N >> 3) << 17) |
                              ((uint32_t)(OZ_M >> 4) << 24);

__device__ __forceinline__ void oz_mma(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                       uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(OZ_IDESC), "r"(accumulate)
      : "memory");
}

// Levels read back after stage t of n: level l takes l + 1 products of 2^14 at
// most per K, so it may hold 32/(l+1) stages of 32; all levels after the last.
__device__ __forceinline__ unsigned oz_flush(int t, int n) {
  if (t + 1 == n) return (1u << OZ_S) - 1u;
  unsigned m = 0;
#pragma unroll
  for (int l = 0; l < OZ_S; l++)
    if ((t + 1) % (32 / (l + 1)) == 0) m |= 1u << l;
  return m;
}

struct OzArgs {
  const unsigned char* dig;  // [rowblock][chunk][OZ_CHUNK]
  int nkc;                   // chunks per row block
  int n;                     // indices (rows and columns of the result)
  const int* exps;           // scale exponents of the indices
  int* err;
  // <0>: JJ partial sums, one matrix per row slice
  int tiles_j;               // column tiles
  int per;                   // chunks per slice
  double* out;               // [slice][n][n]
  // <1>: trailing update of the systems' lower halves
  size_t dig_stride;         // bytes per system
  int exp_stride;
  double* S;                 // [pair][(rows)][ld]
  size_t s_stride;
  int ld, r0;                // the trailing block starts at row and column r0
  const int* bad;            // per pair: not positive definite
};

struct OzShared {
  uint64_t full[2], empty[2], ready, flushed, fin;
  uint32_t tmem;
  int fail;
};

// One 128 x 64 tile: 8 warps of read-back (thread: one row, 32 columns), a
// thread that copies stages of operand digits (two, 84 KB each), a thread that
// issues the 56 MMAs of a stage.  The digits of both operands stay in shared
// memory for all 28 products, so a stage feeds 2,700 clocks of MMA from 84 KB.
// After a read-back the levels it covers are issued last in the next stage,
// so that the tensor core works on the others meanwhile.
// MODE 0: result rows and columns are columns of J (upper tiles).
// MODE 1: S -= L L^T over the panel's 64 columns (lower tiles).
template <int MODE>
__global__ void __launch_bounds__(OZ_T, 1) oz_kernel(const __grid_constant__ OzArgs a) {
  extern __shared__ __align__(1024) unsigned char oz_smem[];
  OzShared& sh = *reinterpret_cast<OzShared*>(oz_smem);
  unsigned char* stage = oz_smem + 1024;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int pair = MODE == 1 ? blockIdx.y : 0;
  if (MODE == 1 && a.bad[pair]) return;  // uniform: before any barrier or TMEM
  // the tile's row block and column tile
  int ib = 0, jt = blockIdx.x;
  if (MODE == 0) {
    while (jt >= a.tiles_j - 2 * ib) jt -= a.tiles_j - 2 * ib++;
    jt += 2 * ib;
  } else {
    while (jt >= 2 * ib + 2) jt -= 2 * ib++ + 2;
  }
  const int c0 = MODE == 0 ? blockIdx.y * a.per : 0;
  const int T = min(a.per, a.nkc - c0);
  const unsigned char* dig = a.dig + pair * a.dig_stride;
  if (warp == 0) {
    tmem_alloc(&sh.tmem, OZ_COLS);
    tmem_relinquish();
  }
  if (threadIdx.x == 32) {
    for (int q = 0; q < 2; q++) {
      mbar_init(&sh.full[q], 1);
      mbar_init(&sh.empty[q], 1);
    }
    mbar_init(&sh.ready, 1);
    mbar_init(&sh.flushed, 256);
    mbar_init(&sh.fin, 1);
    sh.fail = 0;
    fence_mbar_init();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh.tmem;
  volatile int* fail = &sh.fail;
  long long hi[32], lo[32];
  if (warp < 8) {
#pragma unroll
    for (int j = 0; j < 32; j++) hi[j] = lo[j] = 0;
    int ph = 0;
    for (int t = 0; t < T; t++) {
      const unsigned m = oz_flush(t, T);
      if (!m) continue;
      // one verdict per warp: the TMEM reads below take whole warps
      if (!__all_sync(0xffffffffu, mbar_wait(&sh.ready, ph & 1))) {
        *fail = 1;
        break;
      }
      ph++;
      tc_fence_after();
#pragma unroll
      for (int l = 0; l < OZ_S; l++) {
        if (!((m >> l) & 1u)) continue;
#pragma unroll
        for (int h = 0; h < 2; h++) {
          uint32_t v[16];
          tmem_ld16(tmem + ((uint32_t)(32 * (warp & 3)) << 16) + 64 * l + 32 * (warp >> 2) + 16 * h, v);
          tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 16; j++) {
            const long long x = __float2int_rn(__uint_as_float(v[j]));
            if (l < 3)
              hi[16 * h + j] += x * (1ll << (l < 3 ? 8 * (2 - l) : 0));
            else
              lo[16 * h + j] += x * (1ll << (8 * (6 - l)));
          }
        }
      }
      tc_fence_before();
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&sh.flushed)) : "memory");
    }
  } else if (warp == 8 && lane == 0) {
    const unsigned char* A = dig + ((size_t)ib * a.nkc + c0) * OZ_CHUNK;
    const unsigned char* B = dig + ((size_t)(jt >> 1) * a.nkc + c0) * OZ_CHUNK + (jt & 1) * 1024;
    for (int t = 0; t < T; t++) {
      const int b = t & 1;
      if (t >= 2 && !mbar_wait(&sh.empty[b], ((t >> 1) - 1) & 1)) {
        *fail = 1;
        break;
      }
      unsigned char* d = stage + b * OZ_STAGE;
      mbar_expect_tx(&sh.full[b], OZ_STAGE);
      bulk_g2s(d, A + (size_t)t * OZ_CHUNK, OZ_CHUNK, &sh.full[b]);
      for (int q = 0; q < 4 * OZ_S; q++)  // 64 of a chunk's 128 indices, per digit and k/8
        bulk_g2s(d + OZ_CHUNK + q * 1024, B + (size_t)t * OZ_CHUNK + q * 2048, 1024, &sh.full[b]);
    }
  } else if (warp == 9 && lane == 0) {
    unsigned fresh = (1u << OZ_S) - 1u, prev = 0;
    int waits = 0;
    for (int t = 0; t < T; t++) {
      const int b = t & 1;
      if (!mbar_wait(&sh.full[b], (t >> 1) & 1)) {
        *fail = 1;
        break;
      }
      tc_fence_after();
      const uint32_t sa = smem_u32(stage + b * OZ_STAGE), sb = sa + OZ_CHUNK;
      auto level = [&](int l) {
        for (int ks = 0; ks < 2; ks++)
          for (int p = 0; p <= l; p++) {
            const uint64_t da = tc_smem_desc(sa + p * OZ_SLICE_A + ks * 4096, 2048, 128);
            const uint64_t db = tc_smem_desc(sb + (l - p) * OZ_SLICE_B + ks * 2048, 1024, 128);
            oz_mma(tmem + 64 * l, da, db, (fresh >> l) & 1u ? 0u : 1u);
            fresh &= ~(1u << l);
          }
      };
      for (int l = 0; l < OZ_S; l++)
        if (!((prev >> l) & 1u)) level(l);
      if (prev) {
        if (!mbar_wait(&sh.flushed, waits & 1)) {
          *fail = 1;
          break;
        }
        waits++;
        tc_fence_after();
        for (int l = 0; l < OZ_S; l++)
          if ((prev >> l) & 1u) level(l);
      }
      tc_commit(&sh.empty[b]);
      prev = oz_flush(t, T);
      if (prev) {
        tc_commit(&sh.ready);
        fresh |= prev;
      }
    }
    // every MMA complete before the block frees TMEM and its stages
    tc_commit(&sh.fin);
    if (!mbar_wait(&sh.fin, 0)) *fail = 1;
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (*fail) {
    // copies that nobody waited for land before the block's shared memory goes
    if (threadIdx.x == 0) {
      atomicOr(a.err, ZTM_DEVERR_TIMEOUT);
      for (int q = 0; q < 2; q++)
        for (int ph = 0; ph < 2; ph++) mbar_wait(&sh.full[q], ph, 1u << 12);
    }
    __syncthreads();
  }
  if (warp == 0) tmem_dealloc(tmem, OZ_COLS);
  if (warp >= 8 || *fail) return;
  // hi 2^32 + lo, scaled by 2^(e_i + e_j - 64)
  const int i = ib * OZ_M + 32 * (warp & 3) + lane, j0 = jt * OZ_N + 32 * (warp >> 2);
  const int* ex = a.exps + pair * a.exp_stride;
  if (i >= a.n) return;
  const int ei = ex[i];
  double* out = MODE == 0 ? a.out + ((size_t)blockIdx.y * a.n + i) * a.n
                          : a.S + pair * a.s_stride + (size_t)(a.r0 + i) * a.ld + a.r0;
#pragma unroll
  for (int j = 0; j < 32; j++) {
    const int jj = j0 + j;
    if (MODE == 0 ? (jj < i || jj >= a.n) : (jj > i)) continue;
    // integers to double by their bits: |h| < 2^51, 0 <= l < 2^32
    const long long h = hi[j] + (lo[j] >> 32);
    const double hd = __longlong_as_double(h + 0x4338000000000000ll) - 6755399441055744.0;
    const double ld = __hiloint2double(0x43300000, (int)lo[j]) - 4503599627370496.0;
    const int e = ei + ex[jj] - 64, e1 = e >> 1;
    const double v = fma(hd, 4294967296.0, ld) * lm_pow2(e1) * lm_pow2(e - e1);
    if (MODE == 0)
      out[jj] = v;
    else
      out[jj] -= v;
  }
}

// The seven digits of x scaled by 2^-e (|x| < 2^(e-1)): x 2^-e = sum of
// d_p 2^(-8(p+1)), d_p in [-128, 128], most significant first; as bf16 bits.
__device__ __forceinline__ void oz_digits(double x, double sc, unsigned (&d)[OZ_S]) {
  long long X = __double2ll_rn(x * sc);  // sc = 2^(56 - e)
#pragma unroll
  for (int p = OZ_S - 1; p >= 0; p--) {
    const int v = p ? (int)(signed char)(X & 255) : (int)X;
    X = (X - v) >> 8;
    d[p] = __float_as_uint(__int_as_float(0x4B400000 + v) - 12582912.f) >> 16;
  }
}

// Digits of eight K values x(0..7) of one index: one core-matrix row per digit.
template <class F>
__device__ __forceinline__ void oz_put8(unsigned char* chunk, int k8, int i, double sc, F&& x) {
  uint32_t w[OZ_S][4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    unsigned a[OZ_S], b[OZ_S];
    oz_digits(x(2 * q), sc, a);
    oz_digits(x(2 * q + 1), sc, b);
#pragma unroll
    for (int p = 0; p < OZ_S; p++) w[p][q] = a[p] | (b[p] << 16);
  }
#pragma unroll
  for (int p = 0; p < OZ_S; p++)
    *reinterpret_cast<uint4*>(chunk + oz_off(p, k8, i)) = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
}

// Scale exponent of values whose largest |x| has high word hw: |x| < 2^(e-1).
// Columns below 2^-902 count as 2^-902: their products underflow anyway.
__device__ __forceinline__ int oz_exp(unsigned hw) { return max((int)(hw >> 20) - 1021, -900); }

// ---- J ----------------------------------------------------------------------
constexpr int LM_STAT_ROWS = 128;  // rows of J per block of lm_colstat

// Per column the largest |J| (high word) and J^T r over LM_STAT_ROWS rows.
__global__ void __launch_bounds__(128)
    lm_colstat(const double* __restrict__ J, int nrows, int ncols, const double* __restrict__ r,
               unsigned* __restrict__ pmax, double* __restrict__ pdot) {
  const int i = blockIdx.x * 128 + threadIdx.x;
  if (i >= ncols) return;
  const int k0 = blockIdx.y * LM_STAT_ROWS, k1 = min(nrows, k0 + LM_STAT_ROWS);
  unsigned m = 0;
  double s = 0.0;
#pragma unroll 8
  for (int k = k0; k < k1; k++) {
    const double x = J[(long long)k * ncols + i];
    m = max(m, (unsigned)__double2hiint(x) & 0x7fffffffu);
    s = fma(x, r[k], s);
  }
  pmax[(size_t)blockIdx.y * ncols + i] = m;
  pdot[(size_t)blockIdx.y * ncols + i] = s;
}

__global__ void lm_colfinish(int ncols, int nb, const unsigned* __restrict__ pmax,
                             const double* __restrict__ pdot, int* __restrict__ ex,
                             int* __restrict__ odd, double* __restrict__ g) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ncols) return;
  unsigned m = 0;
  double s = 0.0;
  for (int q = 0; q < nb; q++) {
    m = max(m, pmax[(size_t)q * ncols + i]);
    s += pdot[(size_t)q * ncols + i];
  }
  odd[i] = (m >> 20) >= 2047u;  // an infinity or NaN: the column's products are NaN
  ex[i] = odd[i] ? 0 : oz_exp(m);
  g[i] = s;
}

// Digits of 32 rows of J (blockIdx.y, from row k0) for 128 columns.
__global__ void __launch_bounds__(256)
    lm_slice(const double* __restrict__ J, int k0, int nrows, int ncols,
             const int* __restrict__ ex, const int* __restrict__ odd,
             unsigned char* __restrict__ dig) {
  __shared__ double t[OZ_KC][OZ_M + 1];
  const int i0 = blockIdx.x * OZ_M, r0 = k0 + blockIdx.y * OZ_KC;
  for (int q = threadIdx.x; q < OZ_KC * OZ_M; q += 256) {
    const int k = q / OZ_M, i = q % OZ_M;
    t[k][i] = (r0 + k < nrows && i0 + i < ncols) ? J[(long long)(r0 + k) * ncols + i0 + i] : 0.0;
  }
  __syncthreads();
  unsigned char* chunk = dig + ((size_t)blockIdx.x * gridDim.y + blockIdx.y) * OZ_CHUNK;
  for (int u = threadIdx.x; u < OZ_M * 4; u += 256) {
    const int i = u & (OZ_M - 1), k8 = u / OZ_M;
    const bool ok = i0 + i < ncols && !odd[i0 + i];
    const double sc = ok ? lm_pow2(56 - ex[i0 + i]) : 0.0;
    oz_put8(chunk, k8, i, sc, [&](int k) { return ok ? t[8 * k8 + k][i] : 0.0; });
  }
}

// JJ (both halves) = [JJ +] the sum of the row slices' upper tiles.
__global__ void __launch_bounds__(256)
    lm_reduce(int n, int slices, const double* __restrict__ part, const int* __restrict__ odd,
              int add, double* __restrict__ JJ) {
  if (blockIdx.x < blockIdx.y) return;
  __shared__ double t[32][33];
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
  const int j = blockIdx.x * 32 + x;
  for (int q = y; q < 32; q += 8) {
    const int i = blockIdx.y * 32 + q;
    double v = 0.0;
    if (i < n && j < n && j >= i) {
      const size_t o = (size_t)i * n + j;
      for (int s = 0; s < slices; s++) v += part[(size_t)s * n * n + o];
      if (add) v += JJ[o];
      if (odd[i] || odd[j]) v = __longlong_as_double(0x7ff8000000000000ll);
      JJ[o] = v;
    }
    t[q][x] = v;
  }
  __syncthreads();
  for (int q = y; q < 32; q += 8) {  // the mirrored tile: row j, column i
    const int jj = blockIdx.x * 32 + q, ii = blockIdx.y * 32 + x;
    if (jj < n && ii < n && jj > ii) JJ[(size_t)jj * n + ii] = t[x][q];
  }
}

// S[d] = lower half of JJ + d0 diag(JJ) + d1 diag(1/sig^2), and J^T r as row n.
__global__ void lm_assemble(int n, int ld, const double* __restrict__ JJ,
                            const double* __restrict__ g, const double* __restrict__ sig,
                            const double* __restrict__ dm, double* __restrict__ S) {
  const int d = blockIdx.z, i = blockIdx.y * 8 + (threadIdx.x >> 5);
  const int j = blockIdx.x * 32 + (threadIdx.x & 31);
  if (i > n || j > i) return;
  double v;
  if (i == n) {
    v = j < n ? g[j] : 0.0;
  } else {
    v = JJ[(size_t)i * n + j];
    if (i == j) v = (v + dm[2 * d] * v) + dm[2 * d + 1] * (1.0 / (sig[i] * sig[i]));
  }
  S[((size_t)d * (n + 1) + i) * ld + j] = v;
}

// ---- Cholesky -----------------------------------------------------------------
constexpr int LM_NB = 64;  // columns of a panel

// Diagonal block: L L^T = A for the panel's nb columns (identity beyond), and
// 1 / L_ii.  A pivot that is not positive and finite marks the pair.
// One SM per pair, so the chain over the 64 columns is what counts: one warp forms
// 1/sqrt(pivot) (float seed, one third-order step), the block scales the
// column and updates the rest, each thread a 4 x 8 block-cyclic share in
// registers.
__global__ void __launch_bounds__(128)
    lm_potrf(int n, int k0, int nb, int ld, double* __restrict__ S, double* __restrict__ dinv,
             int* __restrict__ bad) {
  const int d = blockIdx.x;
  if (bad[d]) return;
  double* A = S + ((size_t)d * (n + 1) + k0) * ld + k0;
  __shared__ double col[2][LM_NB];  // the current column, double buffered
  __shared__ double s_inv;
  __shared__ int s_bad;
  const int tr = threadIdx.x & 15, tc = threadIdx.x >> 4;  // rows tr + 16a, columns tc + 8b
  double x[4][8];
#pragma unroll
  for (int a = 0; a < 4; a++)
#pragma unroll
    for (int b = 0; b < 8; b++) {
      const int r = tr + 16 * a, c = tc + 8 * b;
      x[a][b] = (r < nb && c <= r) ? A[(size_t)r * ld + c] : (r == c ? 1.0 : 0.0);
    }
  if (threadIdx.x == 0) s_bad = 0;
#pragma unroll
  for (int b = 0; b < 8; b++) {
    for (int cb = 0; cb < 8; cb++) {  // column c = cb + 8 b, held by tc == cb
      const int c = cb + 8 * b;
      double* cl = col[c & 1];
      if (tc == cb) {
#pragma unroll
        for (int a = 0; a < 4; a++) cl[tr + 16 * a] = x[a][b];
      }
      __syncthreads();
      if (threadIdx.x < 32) {
        const double p = cl[c];
        if (!(p > 0.0) || !(p < 1.7e308)) {
          if (threadIdx.x == 0) s_bad = 1;
        } else if (threadIdx.x == 0) {
          // 1/sqrt(p) with p = m 2^(2q), m in [1, 4)
          const int e = ((__double2hiint(p) >> 20) - 1023) >> 1;
          const double m = p * lm_pow2(-e) * lm_pow2(-e);
          const double y = (double)rsqrtf((float)m);
          const double h = fma(-m * y, y, 1.0);
          const double r = fma(y * h, fma(h, 0.375, 0.5), y);
          s_inv = r * lm_pow2(-e);
          if (c < nb) dinv[(size_t)d * n + k0 + c] = s_inv;
        }
      }
      __syncthreads();
      if (s_bad) {
        if (threadIdx.x == 0) bad[d] = 1;
        return;
      }
      const double inv = s_inv;
      double lr[4];
#pragma unroll
      for (int a = 0; a < 4; a++) lr[a] = cl[tr + 16 * a] * inv;
      if (tc == cb) {
#pragma unroll
        for (int a = 0; a < 4; a++)
          if (tr + 16 * a >= c) x[a][b] = lr[a];
      }
#pragma unroll
      for (int q = 0; q < 8; q++) {
        const int cc = tc + 8 * q;
        if (8 * q + 7 <= c) continue;  // no column of this share right of c
        const double lc = cc > c ? cl[cc] * inv : 0.0;
#pragma unroll
        for (int a = 0; a < 4; a++)
          if (16 * a + 15 > c) x[a][q] = fma(-lr[a], lc, x[a][q]);
      }
    }
  }
#pragma unroll
  for (int a = 0; a < 4; a++)
#pragma unroll
    for (int b = 0; b < 8; b++) {
      const int r = tr + 16 * a, c = tc + 8 * b;
      if (r < nb && c <= r) A[(size_t)r * ld + c] = x[a][b];
    }
}

// Rows below the diagonal block (128 per block of threads, the right-hand row
// last): X = A21 L11^-T in double, stored back, and the digits of X with a
// scale per row.  Four lanes share a row (16 columns each), so that a warp's
// FP64 instructions carry eight rows: with a thread per row a panel took one
// warp's 2,000 FP64 instructions (64 us) however few rows were left.
constexpr int TR_T = 512;
constexpr size_t TR_SMEM = (size_t)(LM_NB * LM_NB + LM_NB + OZ_M * (LM_NB + 1)) * 8 + OZ_M * 4;
__global__ void __launch_bounds__(TR_T)
    lm_trsm(int n, int k0, int nb, int ld, double* __restrict__ S, const double* __restrict__ dinv,
            unsigned char* __restrict__ dig, size_t dig_stride, int* __restrict__ ex, int ex_stride,
            const int* __restrict__ bad) {
  extern __shared__ __align__(16) double tr_smem[];
  const int d = blockIdx.y;
  if (bad[d]) return;
  double* LT = tr_smem;               // [j][k] = L11[k][j]
  double* inv = LT + LM_NB * LM_NB;   // 1 / L_jj
  double* X = inv + LM_NB;            // [128][65]
  int* se = reinterpret_cast<int*>(X + OZ_M * (LM_NB + 1));
  double* base = S + (size_t)d * (n + 1) * ld;
  const int r0 = k0 + nb + blockIdx.x * OZ_M;  // first row of this block
  for (int t = threadIdx.x; t < LM_NB * LM_NB; t += TR_T) {
    const int k = t / LM_NB, j = t % LM_NB;
    LT[j * LM_NB + k] = (k < nb && j <= k) ? base[(size_t)(k0 + k) * ld + k0 + j] : 0.0;
  }
  for (int t = threadIdx.x; t < LM_NB; t += TR_T)
    inv[t] = t < nb ? dinv[(size_t)d * n + k0 + t] : 1.0;
  for (int t = threadIdx.x; t < OZ_M * LM_NB; t += TR_T) {
    const int r = t / LM_NB, c = t % LM_NB;
    X[r * (LM_NB + 1) + c] = (r0 + r <= n && c < nb) ? base[(size_t)(r0 + r) * ld + k0 + c] : 0.0;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, g = lane & 3;
  const int row = (threadIdx.x >> 5) * 8 + (lane >> 2);
  double x[16];
#pragma unroll
  for (int m = 0; m < 16; m++) x[m] = X[row * (LM_NB + 1) + 4 * m + g];
#pragma unroll
  for (int m = 0; m < 16; m++) {
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int j = 4 * m + q;  // held by lane group q
      const double xj = __shfl_sync(0xffffffffu, x[m] * inv[j], (lane & ~3) | q);
      if (g == q) x[m] = xj;
      const double* l = LT + j * LM_NB + g;
      if (g > q) x[m] = fma(-xj, l[4 * m], x[m]);
#pragma unroll
      for (int w = m + 1; w < 16; w++) x[w] = fma(-xj, l[4 * w], x[w]);
    }
  }
  unsigned hw = 0;
#pragma unroll
  for (int m = 0; m < 16; m++) {
    X[row * (LM_NB + 1) + 4 * m + g] = x[m];
    hw = max(hw, (unsigned)__double2hiint(x[m]) & 0x7fffffffu);
  }
  hw = max(hw, __shfl_xor_sync(0xffffffffu, hw, 1));
  hw = max(hw, __shfl_xor_sync(0xffffffffu, hw, 2));
  if (g == 0) {
    // not finite: the digits are zero and the diagonal this row updates stays
    // what it is; the entries themselves keep the value for the finish
    const int e = (hw >> 20) >= 2047u ? 1 << 20 : oz_exp(hw);
    se[row] = e;
    ex[(size_t)d * ex_stride + blockIdx.x * OZ_M + row] = e == 1 << 20 ? 0 : e;
  }
  __syncthreads();
  for (int t = threadIdx.x; t < OZ_M * LM_NB; t += TR_T) {
    const int r = t / LM_NB, c = t % LM_NB;
    if (r0 + r <= n && c < nb) base[(size_t)(r0 + r) * ld + k0 + c] = X[r * (LM_NB + 1) + c];
  }
  unsigned char* out = dig + d * dig_stride + (size_t)blockIdx.x * 2 * OZ_CHUNK;
  for (int u = threadIdx.x; u < OZ_M * 8; u += TR_T) {
    const int i = u & (OZ_M - 1), k8 = u / OZ_M;
    const bool ok = se[i] != 1 << 20;
    const double sc = ok ? lm_pow2(56 - se[i]) : 0.0;
    oz_put8(out + (k8 >> 2) * OZ_CHUNK, k8 & 3, i, sc,
            [&](int k) { return ok ? X[i * (LM_NB + 1) + 8 * k8 + k] : 0.0; });
  }
}

// One block of up to 64 unknowns of L^T x = y, from the last: every block of
// threads solves the triangle (one warp), the first stores it, and each takes
// 64 of the rows above, y -= L21^T x.  y is the system's row n.
__global__ void __launch_bounds__(64)
    lm_backstep(int n, int b0, int nb, int ld, double* __restrict__ S,
                const double* __restrict__ dinv, double* __restrict__ x,
                const int* __restrict__ bad) {
  const int d = blockIdx.y;
  if (bad[d]) return;
  __shared__ double L[LM_NB][LM_NB + 1];
  __shared__ double sx[LM_NB];
  double* base = S + (size_t)d * (n + 1) * ld;
  double* y = base + (size_t)n * ld;
  for (int t = threadIdx.x; t < LM_NB * LM_NB; t += 64) {
    const int r = t / LM_NB, c = t % LM_NB;
    L[r][c] = (r < nb && c < r) ? base[(size_t)(b0 + r) * ld + b0 + c] : 0.0;
  }
  const double inv = (int)threadIdx.x < nb ? dinv[(size_t)d * n + b0 + threadIdx.x] : 0.0;
  sx[threadIdx.x] = inv;
  __syncthreads();
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    double ya = lane < nb ? y[b0 + lane] : 0.0, yb = lane + 32 < nb ? y[b0 + 32 + lane] : 0.0;
    const double ia = sx[lane], ib = sx[lane + 32];
    for (int i = LM_NB - 1; i >= 32; i--) {
      const double xi = __shfl_sync(0xffffffffu, yb * ib, i - 32);
      ya = fma(-L[i][lane], xi, ya);
      if (lane + 32 < i) yb = fma(-L[i][lane + 32], xi, yb);
    }
    for (int i = 31; i >= 0; i--) {
      const double xi = __shfl_sync(0xffffffffu, ya * ia, i);
      if (lane < i) ya = fma(-L[i][lane], xi, ya);
    }
    sx[lane] = ya * ia;
    sx[lane + 32] = yb * ib;
  }
  __syncthreads();
  if (blockIdx.x == 0 && (int)threadIdx.x < nb) x[(size_t)d * n + b0 + threadIdx.x] = sx[threadIdx.x];
  const int r = blockIdx.x * 64 + threadIdx.x;
  if (r >= b0) return;
  double s = 0.0;
#pragma unroll 8
  for (int i = 0; i < nb; i++) s = fma(base[(size_t)(b0 + i) * ld + r], sx[i], s);
  y[r] -= s;
}

// ---- the systems that are not positive definite: LU with partial pivoting --------
// Right-looking LU of the augmented matrix [A | J^T r] (row stride n + 1), LU_NB
// columns per panel, one persistent launch with a barrier of all blocks between
// the phases:
//   panel   one block per pair: per column the first row at or below the
//           diagonal with the largest |a| (the reference's pivot rule,
//           zmath.cpp:132), the swap of the two rows, the multipliers and the
//           update of the panel's remaining columns, in shared memory while its
//           rows fit; a zero pivot marks the pair singular;
//   trsm    U12 = L11^-1 A12, a thread per column (and the panel's row swaps);
//   update  A22 -= L21 U12 in 64 x 64 tiles;
//   then U x = y from the last row up, one block per pair.
constexpr int LU_NB = 8;
constexpr int LU_SMEM_ROWS = 3500;  // panels of up to this many rows in shared memory
constexpr int LU_T = 1024;
constexpr int LU_TILE = 64;

struct LuArgs {
  int n, nd;
  const double* JJ;
  const double* g;
  const double* sig;
  const double* dm;
  double* S;  // per pair (n + 1) * ld doubles: the augmented matrix goes there
  int ld;
  int* piv;
  int* singular;
  const int* bad;
  unsigned* barrier;  // zeroed before
  int* err;
  bool smem_panel;
};

// Barrier of the whole (co-resident) grid; false when the bounded wait runs out.
__device__ bool lu_barrier(const LuArgs& a, unsigned& round) {
  __shared__ int s_ok;
  __syncthreads();
  round++;
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(a.barrier, 1u);
    const unsigned want = round * gridDim.x;
    int ok = 0;
    for (unsigned it = 0; it < (1u << 26); it++) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(a.barrier) : "memory");
      if (v >= want) {
        ok = 1;
        break;
      }
      __nanosleep(100);
    }
    if (!ok) atomicOr(a.err, ZTM_DEVERR_TIMEOUT);
    s_ok = ok;
  }
  __syncthreads();
  const bool ok = s_ok != 0;
  __syncthreads();
  return ok;
}

// Row at or below c with the largest |v(r)|, the first of equals; -1 if none is
// above zero.  Whole block.
template <class F>
__device__ int lu_pivot(int c, int R, F&& v) {
  __shared__ double s_v[LU_T / 32];
  __shared__ int s_i[LU_T / 32];
  __shared__ int s_p;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double best = -1.0;
  int bi = R;
  for (int r = c + threadIdx.x; r < R; r += LU_T) {
    const double w = fabs(v(r));
    if (w > best) {
      best = w;
      bi = r;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double v2 = __shfl_down_sync(0xffffffffu, best, o);
    const int i2 = __shfl_down_sync(0xffffffffu, bi, o);
    if (v2 > best || (v2 == best && i2 < bi)) {
      best = v2;
      bi = i2;
    }
  }
  if (lane == 0) {
    s_v[warp] = best;
    s_i[warp] = bi;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double bv = s_v[0];
    int bp = s_i[0];
    for (int q = 1; q < LU_T / 32; q++)
      if (s_v[q] > bv || (s_v[q] == bv && s_i[q] < bp)) {
        bv = s_v[q];
        bp = s_i[q];
      }
    s_p = bv > 0.0 ? bp : -1;
  }
  __syncthreads();
  return s_p;
}

// The panel of columns k0 .. k0+nb-1 of matrix A (row stride w): in shared memory
// P ([rows][LU_NB]) when given, else in place with whole-row swaps.
__device__ bool lu_panel(double* A, int n, int k0, int nb, long long w, int* piv, double* P) {
  if (P) {
    const int R = n - k0;
    for (int t = threadIdx.x; t < R * LU_NB; t += LU_T) {
      const int r = t / LU_NB, m = t % LU_NB;
      P[t] = m < nb ? A[(long long)(k0 + r) * w + k0 + m] : 0.0;
    }
    __syncthreads();
    for (int c = 0; c < nb; c++) {
      const int p = lu_pivot(c, R, [&](int r) { return P[r * LU_NB + c]; });
      if (p < 0) return false;
      if (threadIdx.x == 0) piv[k0 + c] = k0 + p;
      if (p != c && threadIdx.x < LU_NB) {
        const double x = P[c * LU_NB + threadIdx.x];
        P[c * LU_NB + threadIdx.x] = P[p * LU_NB + threadIdx.x];
        P[p * LU_NB + threadIdx.x] = x;
      }
      __syncthreads();
      const double finv = 1.0 / P[c * LU_NB + c];
      for (int r = c + 1 + threadIdx.x; r < R; r += LU_T) {
        double* row = P + r * LU_NB;
        const double l = row[c] * finv;
        row[c] = l;
#pragma unroll
        for (int j = 0; j < LU_NB; j++)
          if (j > c && j < nb) row[j] = fma(-l, P[c * LU_NB + j], row[j]);
      }
      __syncthreads();
    }
    for (int t = threadIdx.x; t < R * LU_NB; t += LU_T) {
      const int r = t / LU_NB, m = t % LU_NB;
      if (m < nb) A[(long long)(k0 + r) * w + k0 + m] = P[t];
    }
    return true;
  }
  for (int c = k0; c < k0 + nb; c++) {
    const int p = lu_pivot(c, n, [&](int r) { return A[r * w + c]; });
    if (p < 0) return false;
    if (p != c)  // whole rows from the panel's first column on: its multipliers move along
      for (int j = k0 + threadIdx.x; j <= n; j += LU_T) {
        const double x = A[(long long)c * w + j];
        A[(long long)c * w + j] = A[(long long)p * w + j];
        A[(long long)p * w + j] = x;
      }
    if (threadIdx.x == 0) piv[c] = c;  // already swapped
    __syncthreads();
    const double finv = 1.0 / A[(long long)c * w + c];
    for (int r = c + 1 + threadIdx.x; r < n; r += LU_T) {
      const double l = A[r * w + c] * finv;
      A[r * w + c] = l;
      for (int j = c + 1; j < k0 + nb; j++) A[r * w + j] = fma(-l, A[(long long)c * w + j], A[r * w + j]);
    }
    __syncthreads();
  }
  return true;
}

__global__ void __launch_bounds__(LU_T, 1) lm_lu_all(LuArgs a) {
  extern __shared__ double lu_smem[];
  bool any = false;
  for (int d = 0; d < a.nd; d++) any |= a.bad[d] != 0;
  if (!any) return;  // every block alike
  const int n = a.n;
  const long long w = n + 1;
  const size_t stride = (size_t)(n + 1) * a.ld;
  unsigned round = 0;
  // the augmented matrices
  for (int d = 0; d < a.nd; d++) {
    if (!a.bad[d]) continue;
    double* A = a.S + d * stride;
    for (long long e = (long long)blockIdx.x * LU_T + threadIdx.x; e < n * w;
         e += (long long)gridDim.x * LU_T) {
      const int i = (int)(e / w), j = (int)(e % w);
      double v = j == n ? a.g[i] : a.JJ[(size_t)i * n + j];
      if (i == j) v = (v + a.dm[2 * d] * v) + a.dm[2 * d + 1] * (1.0 / (a.sig[i] * a.sig[i]));
      A[e] = v;
    }
  }
  if (!lu_barrier(a, round)) return;
  volatile int* sing = a.singular;
  for (int k0 = 0; k0 < n; k0 += LU_NB) {
    const int nb = min(LU_NB, n - k0);
    for (int d = blockIdx.x; d < a.nd; d += gridDim.x) {
      if (!a.bad[d] || sing[d]) continue;
      const bool ok = lu_panel(a.S + d * stride, n, k0, nb, w, a.piv + (size_t)d * n,
                               a.smem_panel ? lu_smem : nullptr);
      if (!ok && threadIdx.x == 0) sing[d] = 1;
      __syncthreads();
    }
    if (!lu_barrier(a, round)) return;
    const int rest = n + 1 - (k0 + nb);  // columns right of the panel, right-hand side included
    for (int d = 0; d < a.nd; d++) {
      if (!a.bad[d] || sing[d]) continue;
      double* A = a.S + d * stride;
      for (int q = blockIdx.x * LU_T + threadIdx.x; q < rest; q += gridDim.x * LU_T) {
        const int j = k0 + nb + q;
        for (int i = 0; i < nb; i++) {  // the panel's row swaps, in order, on this column
          const int p = a.piv[(size_t)d * n + k0 + i];
          if (p != k0 + i) {
            const double t = A[(long long)(k0 + i) * w + j];
            A[(long long)(k0 + i) * w + j] = A[(long long)p * w + j];
            A[(long long)p * w + j] = t;
          }
        }
        double x[LU_NB];
#pragma unroll
        for (int i = 0; i < LU_NB; i++) x[i] = i < nb ? A[(long long)(k0 + i) * w + j] : 0.0;
#pragma unroll
        for (int i = 1; i < LU_NB; i++)
#pragma unroll
          for (int m = 0; m < i; m++)
            if (i < nb) x[i] = fma(-A[(long long)(k0 + i) * w + k0 + m], x[m], x[i]);
#pragma unroll
        for (int i = 0; i < LU_NB; i++)
          if (i < nb) A[(long long)(k0 + i) * w + j] = x[i];
      }
    }
    if (!lu_barrier(a, round)) return;
    // 64 x 64 tiles of the rest, 256 threads each
    const int rows = n - (k0 + nb), tr = (rows + LU_TILE - 1) / LU_TILE, tcol = (rest + LU_TILE - 1) / LU_TILE;
    const int grp = threadIdx.x >> 8, t = threadIdx.x & 255, tx = t & 15, ty = t >> 4;
    double* Ls = lu_smem + grp * (LU_TILE * (LU_NB + 1) + LU_NB * (LU_TILE + 1));
    double* Us = Ls + LU_TILE * (LU_NB + 1);
    const long long tiles = (long long)tr * tcol * a.nd;
    for (long long b0 = (long long)blockIdx.x * 4; b0 < tiles; b0 += (long long)gridDim.x * 4) {
      const long long q = b0 + grp;
      const int d = (int)min((long long)a.nd - 1, q / ((long long)tr * tcol));
      const bool on = q < tiles && a.bad[d] && !sing[d];
      const int rem = (int)(q % ((long long)tr * tcol));
      const int r0 = k0 + nb + (rem / tcol) * LU_TILE, j0 = k0 + nb + (rem % tcol) * LU_TILE;
      double* A = a.S + d * stride;
      __syncthreads();
      if (on)
        for (int e = t; e < LU_TILE * LU_NB; e += 256) {
          const int rr = e / LU_NB, m = e % LU_NB, r = r0 + rr;
          Ls[rr * (LU_NB + 1) + m] = (r < n && m < nb) ? A[(long long)r * w + k0 + m] : 0.0;
          const int mm = e / LU_TILE, cc = e % LU_TILE, j = j0 + cc;
          Us[mm * (LU_TILE + 1) + cc] = (j <= n && mm < nb) ? A[(long long)(k0 + mm) * w + j] : 0.0;
        }
      __syncthreads();
      if (!on) continue;
#pragma unroll
      for (int p = 0; p < 4; p++)
#pragma unroll
        for (int s = 0; s < 4; s++) {
          const int r = r0 + ty + 16 * p, j = j0 + tx + 16 * s;
          if (r >= n || j > n) continue;
          double acc = 0.0;
#pragma unroll
          for (int m = 0; m < LU_NB; m++)
            acc = fma(Ls[(ty + 16 * p) * (LU_NB + 1) + m], Us[m * (LU_TILE + 1) + tx + 16 * s], acc);
          A[(long long)r * w + j] -= acc;
        }
    }
    if (!lu_barrier(a, round)) return;
  }
  // U x = y, 32 rows at a time from the bottom: a warp solves the triangle,
  // then every thread updates the right-hand sides above
  for (int d = blockIdx.x; d < a.nd; d += gridDim.x) {
    if (!a.bad[d] || sing[d]) continue;
    double* A = a.S + d * stride;
    double* s_x = lu_smem;
    const int lane = threadIdx.x & 31;
    for (int b0 = ((n - 1) / 32) * 32; b0 >= 0; b0 -= 32) {
      const int be = min(n, b0 + 32);
      if (threadIdx.x < 32) {
        const int row = b0 + lane;
        double y = row < be ? A[(long long)row * w + n] : 0.0;
        for (int i = be - 1; i >= b0; i--) {
          const double xi = __shfl_sync(0xffffffffu, y, i - b0) / A[(long long)i * w + i];
          if (lane < i - b0) y = fma(-A[(long long)row * w + i], xi, y);
          if (lane == i - b0) y = xi;
        }
        if (row < be) {
          A[(long long)row * w + n] = y;
          s_x[lane] = y;
        }
      }
      __syncthreads();
      for (int r = threadIdx.x; r < b0; r += LU_T) {
        double acc = 0.0;
        for (int i = b0; i < be; i++) acc = fma(A[(long long)r * w + i], s_x[i - b0], acc);
        A[(long long)r * w + n] -= acc;
      }
      __syncthreads();
    }
  }
}

__global__ void lm_finish(int n, int nd, int ld, const double* __restrict__ x,
                          const double* __restrict__ S, const int* __restrict__ bad,
                          const int* __restrict__ singular, const double* __restrict__ b,
                          double* __restrict__ B) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= (long long)nd * n) return;
  const int d = (int)(t / n), i = (int)(t % n);
  double step = x[t];
  if (bad[d])  // the augmented matrix's right-hand column
    step = singular[d] ? 0.0 : S[(size_t)d * (n + 1) * ld + (size_t)i * (n + 1) + n];
  B[t] = b[i] + step;
}

// ---------------------------------------------------------------------------
struct LmShape {
  int rb, tiles_j, tiles, kcs, per, slices;
};

// J in passes of kcs chunks of 32 rows (digits of at most about 1.5 GB), each
// cut into row slices so that the tiles of a narrow J fill the chip (at least
// eight chunks a slice).
LmShape lm_shape(int m, int n, int num_sms) {
  LmShape s;
  s.rb = (n + OZ_M - 1) / OZ_M;
  s.tiles_j = (n + OZ_N - 1) / OZ_N;
  s.tiles = 0;
  for (int i = 0; i < s.rb; i++) s.tiles += s.tiles_j - 2 * i;
  const int all = (m + OZ_KC - 1) / OZ_KC;
  const long long fit = std::max(16LL, 1500000000LL / ((long long)s.rb * OZ_CHUNK));
  s.kcs = (int)std::min<long long>(all, fit);
  const int want = std::max(1, (4 * std::max(num_sms, 1) + s.tiles - 1) / s.tiles);
  s.per = std::max(std::min(8, s.kcs), (s.kcs + want - 1) / want);
  s.slices = (s.kcs + s.per - 1) / s.per;
  return s;
}

}  // namespace

extern "C" int ztm_lm_steps(ztm_ctx* c, const double* J, int nrows, int ncols, const double* r,
                            const double* b, const double* sig, const double* damping, int nd,
                            double* B, double* JJ, int flags) {
  if (!c) return ZTM_ERR_ARG;
  c->err.clear();
  if (!J || !r || !b || !sig || !damping || !B) return ztm_fail(c, ZTM_ERR_ARG, "null argument");
  if (nrows < 1 || ncols < 1 || nd < 1) return ztm_fail(c, ZTM_ERR_ARG, "sizes must be >= 1");
  if (flags & ~ZTM_FLAG_DEVICE_PTRS) return ztm_fail(c, ZTM_ERR_ARG, "unknown flag");
  if (ncols > 32768 || (long long)nd * ncols * (ncols + 1) > (1LL << 31))
    return ztm_fail(c, ZTM_ERR_RANGE, "normal equations too large (ncols <= 32768, nd*ncols^2 < 2^31)");
  const bool dev = (flags & ZTM_FLAG_DEVICE_PTRS) != 0;
  const size_t n = ncols, m = nrows;
  int prev = -1;
  cudaGetDevice(&prev);
  if (prev != c->device && cudaSetDevice(c->device) != cudaSuccess)
    return ztm_fail(c, ZTM_ERR_NODEV, "cannot select device");
  struct Restore {
    int p, d;
    ~Restore() {
      if (p >= 0 && p != d) cudaSetDevice(p);
    }
  } restore{prev, c->device};
  const LmShape s = lm_shape(nrows, ncols, c->num_sms);
  const int ld = (ncols + 2) & ~1;
  const int nstat = (nrows + LM_STAT_ROWS - 1) / LM_STAT_ROWS;
  const size_t prb = (n + OZ_M) / OZ_M;  // row blocks below the first panel (the right-hand row included)
  const size_t dig_stride = prb * 2 * OZ_CHUNK;
  const size_t dig = std::max((size_t)s.rb * s.kcs * OZ_CHUNK, (size_t)nd * dig_stride);
  const size_t need = WsCarver::need(m * n * 8) + 3 * WsCarver::need(m * 8 + n * 8) +
                      WsCarver::need(n * n * 8) + WsCarver::need((size_t)nd * 16) +
                      2 * WsCarver::need((size_t)nd * n * 8) + WsCarver::need((size_t)nstat * n * 12) +
                      3 * WsCarver::need(n * 8) + WsCarver::need((size_t)s.slices * n * n * 8) +
                      WsCarver::need((size_t)nd * (n + 1) * ld * 8) + WsCarver::need(dig) +
                      WsCarver::need((size_t)nd * prb * OZ_M * 4) + 3 * WsCarver::need((size_t)nd * 8) +
                      WsCarver::need((size_t)nd * n * 4) + 16384;
  int rc = ztm_ws_reserve(c, need);
  if (rc) return rc;
  WsCarver wc(c->ws);
  double* s_J = wc.take<double>(dev ? 0 : m * n);
  double* s_r = wc.take<double>(m);
  double* s_b = wc.take<double>(n);
  double* s_sig = wc.take<double>(n);
  double* s_JJ = wc.take<double>(n * n);
  double* s_dm = wc.take<double>((size_t)nd * 2);
  double* s_B = wc.take<double>((size_t)nd * n);
  double* x = wc.take<double>((size_t)nd * n);
  double* g = wc.take<double>(n);
  double* dinv = wc.take<double>((size_t)nd * n);
  double* pdot = wc.take<double>((size_t)nstat * n);
  unsigned* pmax = wc.take<unsigned>((size_t)nstat * n);
  int* ex = wc.take<int>(n);
  int* odd = wc.take<int>(n);
  double* part = wc.take<double>((size_t)s.slices * n * n);
  double* S = wc.take<double>((size_t)nd * (n + 1) * ld);
  unsigned char* digits = wc.take<unsigned char>(dig);
  int* pex = wc.take<int>((size_t)nd * prb * OZ_M);
  int* piv = wc.take<int>((size_t)nd * n);
  int* state = wc.take<int>(2 * (size_t)nd + 1);  // bad, singular, the barrier
  if (wc.off > need) return ztm_fail(c, ZTM_ERR_ALLOC, "normal equations: workspace");
  const void *pJ, *pr, *pb, *ps, *pd;
  if ((rc = ztm_stage_in(c, J, m * n * 8, dev, s_J, &pJ))) return rc;
  if ((rc = ztm_stage_in(c, r, m * 8, dev, s_r, &pr))) return rc;
  if ((rc = ztm_stage_in(c, b, n * 8, dev, s_b, &pb))) return rc;
  if ((rc = ztm_stage_in(c, sig, n * 8, dev, s_sig, &ps))) return rc;
  if ((rc = ztm_stage_in(c, damping, (size_t)nd * 16, dev, s_dm, &pd))) return rc;
  double* oJJ = (dev && JJ) ? JJ : s_JJ;
  double* oB = dev ? B : s_B;
  int *bad = state, *singular = state + nd;
  cudaMemsetAsync(state, 0, (2 * (size_t)nd + 1) * 4, c->stream);
  cudaFuncSetAttribute(oz_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)OZ_SMEM);
  cudaFuncSetAttribute(oz_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)OZ_SMEM);
  cudaFuncSetAttribute(lm_trsm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TR_SMEM);
  long long launches = 0;
  {
    ZtmProf prof_(c, "lm");
    lm_colstat<<<dim3((unsigned)((n + 127) / 128), nstat), 128, 0, c->stream>>>(
        (const double*)pJ, nrows, ncols, (const double*)pr, pmax, pdot);
    lm_colfinish<<<(unsigned)((n + 127) / 128), 128, 0, c->stream>>>(ncols, nstat, pmax, pdot, ex,
                                                                     odd, g);
    OzArgs o = {};
    o.dig = digits;
    o.n = ncols;
    o.exps = ex;
    o.err = c->d_err;
    o.tiles_j = s.tiles_j;
    o.per = s.per;
    o.out = part;
    const int all = (nrows + OZ_KC - 1) / OZ_KC;
    for (int k = 0; k < all; k += s.kcs) {
      o.nkc = std::min(s.kcs, all - k);
      const int slices = (o.nkc + s.per - 1) / s.per;
      lm_slice<<<dim3(s.rb, o.nkc), 256, 0, c->stream>>>((const double*)pJ, k * OZ_KC, nrows, ncols,
                                                         ex, odd, digits);
      oz_kernel<0><<<dim3(s.tiles, slices), OZ_T, OZ_SMEM, c->stream>>>(o);
      const unsigned t32 = (unsigned)((n + 31) / 32);
      lm_reduce<<<dim3(t32, t32), 256, 0, c->stream>>>(ncols, slices, part, odd, k > 0, oJJ);
      launches += 3;
    }
    lm_assemble<<<dim3((unsigned)((n + 32) / 32), (unsigned)((n + 8) / 8), nd), 256, 0, c->stream>>>(
        ncols, ld, oJJ, g, (const double*)ps, (const double*)pd, S);
    launches += 3;
    OzArgs u = {};
    u.dig = digits;
    u.nkc = 2;
    u.per = 2;
    u.exps = pex;
    u.err = c->d_err;
    u.dig_stride = dig_stride;
    u.exp_stride = (int)(prb * OZ_M);
    u.S = S;
    u.s_stride = (n + 1) * (size_t)ld;
    u.ld = ld;
    u.bad = bad;
    for (int k0 = 0; k0 < ncols; k0 += LM_NB) {
      const int nb = std::min(LM_NB, ncols - k0);
      lm_potrf<<<nd, 128, 0, c->stream>>>(ncols, k0, nb, ld, S, dinv, bad);
      const int rows = ncols + 1 - (k0 + nb), rb = (rows + OZ_M - 1) / OZ_M;
      lm_trsm<<<dim3(rb, nd), TR_T, TR_SMEM, c->stream>>>(ncols, k0, nb, ld, S, dinv, digits,
                                                          dig_stride, pex, u.exp_stride, bad);
      launches += 2;
      if (rows > 1) {
        u.n = rows;
        u.r0 = k0 + nb;
        oz_kernel<1><<<dim3(rb * (rb + 1), nd), OZ_T, OZ_SMEM, c->stream>>>(u);
        launches++;
      }
    }
    for (int b0 = ((ncols - 1) / LM_NB) * LM_NB; b0 >= 0; b0 -= LM_NB) {
      lm_backstep<<<dim3(std::max(1, b0 / 64), nd), 64, 0, c->stream>>>(
          ncols, b0, std::min(LM_NB, ncols - b0), ld, S, dinv, x, bad);
      launches++;
    }
    LuArgs l = {};
    l.n = ncols;
    l.nd = nd;
    l.JJ = oJJ;
    l.g = g;
    l.sig = (const double*)ps;
    l.dm = (const double*)pd;
    l.S = S;
    l.ld = ld;
    l.piv = piv;
    l.singular = singular;
    l.bad = bad;
    l.barrier = reinterpret_cast<unsigned*>(state + 2 * (size_t)nd);
    l.err = c->d_err;
    l.smem_panel = ncols <= LU_SMEM_ROWS;
    const size_t lu_smem = std::max((size_t)(l.smem_panel ? ncols : 0) * LU_NB * 8,
                                    (size_t)4 * (LU_TILE * (LU_NB + 1) + LU_NB * (LU_TILE + 1)) * 8);
    cudaFuncSetAttribute(lm_lu_all, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lu_smem);
    void* args[] = {&l};
    cudaLaunchCooperativeKernel((const void*)lm_lu_all, dim3(std::max(c->num_sms, 1)), dim3(LU_T),
                                args, lu_smem, c->stream);
    lm_finish<<<(unsigned)(((size_t)nd * n + 255) / 256), 256, 0, c->stream>>>(
        ncols, nd, ld, x, S, bad, singular, (const double*)pb, oB);
    launches += 2;
  }
  c->launches += launches;
  if ((rc = ztm_after_launch(c, "normal equations"))) return rc;
  if (!dev) {
    if (JJ) cudaMemcpyAsync(JJ, oJJ, n * n * 8, cudaMemcpyDeviceToHost, c->stream);
    cudaMemcpyAsync(B, oB, (size_t)nd * n * 8, cudaMemcpyDeviceToHost, c->stream);
  }
  return ztm_finish(c, dev, nullptr, nullptr, 0, "normal equations");
}
