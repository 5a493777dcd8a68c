// Bordered layout of the factor and its solves (sm_103a, FP64 results).
//
// The columns of the permuted Hgamma near the roots of its elimination tree
// form the border, the subtrees below them the blocks (at most kBlkRows rows
// each with their border rows).  With A = [F B^T; B S], F block diagonal over
// the blocks:
//   per block   X = L^-1 of F = L L^T, E = B F^-1, and the update -E B^T
//   border      X = L^-1, dense, of S - sum E B^T = L L^T
//   solve       y_F = X b_F,  x_S = X^T (X (b_S - E b_F)),  x_F = X^T y_F - E^T x_S
// so that a solve is a few dense phases whatever the depth of the tree (the
// task-queue kernels pay 5-9 us per tree level and direction).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "kernels.cuh"

namespace hykkt {

// ---------------------------------------------------------------------------
// Blocks: Cholesky of a block's front [F; B] over its own columns together
// with the inverse of the factor, one CTA each, in place in the packed lower
// triangle in shared memory.  Pivot p with v = A(:,p) / sqrt(a_pp) below it
// and w = A(p,:) / sqrt(a_pp) left of it (row p of X = L^-1 so far):
//   A_ij -= v_i v_j  (i >= j > p),   A_ij -= v_i w_j  (j < p)
//   A_pj = w_j,  A_ip = -v_i / sqrt(a_pp)
// so that F ends as X, B as -E and the border part as the Schur update.  A
// block's columns are sparse (they come from a subtree), so only the nonzeros
// of v and w are visited.  Bounded by the pivots' latency.
// ---------------------------------------------------------------------------
// block columns of a back task's panel, by the rows of a border panel
__host__ __device__ constexpr int back_rows(int rb) { return rb == 8 ? 64 : 32; }
__device__ __forceinline__ int packed_lower(int i, int j) { return i * (i + 1) / 2 + j; }

__global__ void __launch_bounds__(256) k_block_sweep(DevPlan d, DevBorder bd, int blk0) {
  extern __shared__ double bsm[];
  __shared__ int wcnt[8];
  __shared__ double sroot;
  const int blk = blk0 + blockIdx.x;
  const int c0 = bd.blk_rp[blk], nt = bd.blk_rp[blk + 1] - c0;
  const int R = bd.blk_rrp[blk + 1] - bd.blk_rrp[blk];
  const int N = nt + R, tot = N * (N + 1) / 2;
  double* A = bsm;
  double* val = A + tot;                                    // nonzeros of the pivot's row and column
  short* idx = reinterpret_cast<short*>(val + blockDim.x);  // their positions, ascending
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarp = blockDim.x >> 5;
  for (int i = tid; i < tot; i += blockDim.x) A[i] = 0.0;
  __syncthreads();
  for (int e = bd.ent_rp[blk] + tid; e < bd.ent_rp[blk + 1]; e += blockDim.x) A[bd.ent_pos[e]] = d.lp_v[bd.ent_q[e]];
  __syncthreads();
  for (int p = 0; p < nt; ++p) {
    // N <= blockDim.x: one entry of the pivot's row or column per thread
    double v = 0.0;
    if (tid < N && tid != p) v = tid > p ? A[packed_lower(tid, p)] : A[packed_lower(p, tid)];
    const bool nz = v != 0.0;
    const unsigned m = __ballot_sync(0xffffffffu, nz);
    if (lane == 0) wcnt[warp] = __popc(m);
    if (tid == 0) {
      const double dp = A[packed_lower(p, p)];
      note_pivot(d, bd.blk_col[c0 + p], dp);
      sroot = rsqrt(dp);
    }
    __syncthreads();
    int base = 0, nnz = 0;
    for (int w = 0; w < nwarp; ++w) {
      if (w < warp) base += wcnt[w];
      nnz += wcnt[w];
    }
    const double rs = sroot;
    if (nz) {
      const int at = base + __popc(m & ((1u << lane) - 1));
      val[at] = v * rs;
      idx[at] = (short)tid;
    }
    __syncthreads();
    for (int a = warp; a < nnz; a += nwarp) {
      const int i = idx[a];
      const double u = val[a];
      if (i < p) {
        if (lane == 0) A[packed_lower(p, i)] = u;
        continue;
      }
      for (int b = lane; b <= a; b += 32) {
        double* g = &A[packed_lower(i, idx[b])];
        *g = fma(-u, val[b], *g);
      }
      if (lane == 0) A[packed_lower(i, p)] = -u * rs;
    }
    if (tid == 0) A[packed_lower(p, p)] = rs;
    __syncthreads();
  }
  // [X; E] in panels of 64 rows and [-E^T X^T] in panels of back_rows block columns,
  // column after column of the panel, zeros past the last row
  double* GE = bd.ge + bd.ge_off[blk];
  double* ET = bd.et + bd.et_off[blk];
  for (int e = tid; e < (N + 63) / 64 * 64 * nt; e += blockDim.x) {
    const int i = e / (64 * nt) * 64 + e % 64, t = e / 64 % nt;
    double a = 0.0;
    if (i < nt) a = i >= t ? A[packed_lower(i, t)] : 0.0;
    else if (i < N) a = -A[packed_lower(i, t)];
    GE[e] = a;
  }
  const int br = back_rows(bd.rb);
  for (int e = tid; e < (nt + br - 1) / br * br * N; e += blockDim.x) {
    const int t = e / (br * N) * br + e % br, i = e / br % N;  // entry i: border rows, then own from the last on
    double a = 0.0;
    if (t < nt) a = i < R ? A[packed_lower(nt + i, t)] : N - 1 - i >= t ? A[packed_lower(N - 1 - i, t)] : 0.0;
    ET[e] = a;
  }
  double* C = bd.cb + bd.c_off[blk];  // the border update, packed lower R x R
  for (int i = warp; i < R; i += nwarp)
    for (int j = lane; j <= i; j += 32) C[packed_lower(i, j)] = A[packed_lower(nt + i, nt + j)];
}

// The border's lower triangle: one thread per entry that has an original
// value or block updates (block order: deterministic); zeroed before.
__global__ void k_border_assemble(DevPlan d, DevBorder bd) {
  const int stride = gridDim.x * blockDim.x, tid = blockIdx.x * blockDim.x + threadIdx.x;
  for (int t = tid; t < bd.nasm; t += stride) {
    double a = bd.asm_src[t] >= 0 ? d.lp_v[bd.asm_src[t]] : 0.0;
    for (int p = bd.asm_rp[t]; p < bd.asm_rp[t + 1]; ++p) a += bd.cb[bd.asm_pos[p]];
    bd.W[(int64_t)bd.asm_col[t] * bd.ld + bd.asm_row[t]] = a;
  }
  for (int j = bd.k + tid; j < bd.npan * kBorderPanel; j += stride) bd.W[(int64_t)j * bd.ld + j] = 1.0;  // padding
}

// Schur plans (no blocks): the rows of Jc_p below the border's panels.  The
// sweep turns [Hgamma Jc^T; Jc 0] into -S = -Jc Hgamma^-1 Jc^T below them.
__global__ void k_border_constraints(DevPlan d, DevBorder bd) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= bd.mc) return;
  double* W = bd.W + bd.npan * kBorderPanel + i;
  for (int p = d.jc_rp[i]; p < d.jc_rp[i + 1]; ++p) W[(int64_t)d.jcp_ci[p] * bd.ld] = d.jc_s[p];
}

// ---------------------------------------------------------------------------
// Border: Cholesky and the inverse of the factor in one sweep, 32 columns at
// a time, in place: after panel p the rows up to it hold X = L^-1, the rows
// below the partial products of X left of the panel and the Schur complement
// right of it.  With L L^T the panel's diagonal block, per panel:
//   k_border_panel   Y = V L^-T for the rows below (V the panel's columns) and
//                    Y = L^-1 V for the columns left of it (V its rows of X),
//                    Y in digits for the update; in place X_p = Y to the left,
//                    L^-1 on the diagonal, -Y L^-1 below
//   k_border_update  A -= Y Y^T on the rows below the panel, all columns
// (An explicit W = X^T X would save a phase of every solve, but its products
// cancel: the first residual of a 1,000-bus solve rose from 2e-6 to 5e-4.)
// The update is the cost (2/3 k^3 flops in all).  FP64 runs at 1.25 TFLOP/s on
// this chip and the bf16 tensor cores at 1,900, so the products are made of
// exact bf16 pieces: every row of Y is scaled by its power of two and cut
// into seven signed 8-bit digits (55 bits), digit products are integers that
// FP32 accumulates without rounding (at most 7 * 32 * 2^14 < 2^24), and the
// digit products of equal weight share one accumulator (Ootomo, Ozaki and
// Yokota, "DGEMM on integer matrix multiplication unit", 2024, here on
// tcgen05 with bf16 operands).  What it leaves out: the digits round an entry
// at 2^-56 of its row's largest (an entry below a quarter of that keeps fewer
// bits than its double), and digit products of weight eight and more are below
// 2^-62 of the largest product; rows below 2^-958 count as zero.  The sums are
// exact and rounded twice, where a 32-term FP64 FMA chain rounds 32 times.
// Errors against FP64 FMAs in the same sweep (60 KKT systems of 60 to 160
// buses, emulated, geometric means): of the solution 0.77, of the residual 0.88
// times.  Against the task queues' FP64 factor on the GPU: Cholesky solves of
// 300 to 2,600 columns, condition 1e2 to 1e10: 0.68 to 0.95 and 0.84 to 0.93;
// unrefined KKT solves of 200 to 6,000 buses with the CG to 1e-11: 1.02 and
// 0.98, to 1e-15 (where the products with X = L^-1 show): 1.07 and 1.23.
// ---------------------------------------------------------------------------
constexpr int kDigits = 7;
constexpr int kRowBlock = 128;                                   // rows of a digit block and of an update tile
constexpr int kPlaneBytes = kRowBlock * kBorderPanel * 2;         // one digit of one row block
constexpr int kDigitBlockBytes = kDigits * kPlaneBytes;
constexpr int kTileCols = 32;                                     // columns of an update tile
constexpr int kAccs = 8;                                          // digit weights kept
constexpr int kTmemCols = kAccs * kTileCols;
constexpr int kBPlaneBytes = kTileCols * kBorderPanel * 2;
// row digits and two buffers of column digits; two CTAs per SM (their sums
// fill the 512 tensor-memory columns, their shared memory keeps a third out)
constexpr int kUpdateSmem = kDigitBlockBytes + 2 * kDigits * kBPlaneBytes;
static_assert(3 * kUpdateSmem > 227 * 1024, "a third CTA would wait for tensor memory");
constexpr int kExpZero = -100000, kExpNan = 1000000;  // row exponents of rows that are zero / not finite
constexpr unsigned kMbarLimit = 1u << 22;

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.b32 %0, 1, 0, p;\n}"
               : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}

// Bounded wait on an mbarrier phase; false (and the solve's timeout flag) when
// the limit runs out.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, DevScalars* sc) {
  for (unsigned it = 0; it < kMbarLimit; ++it)
    if (mbar_test(bar, parity)) return true;
  atomicOr(&sc->solve_flags, 1);
  return false;
}

// Test hook (dbg_unsatisfiable, 0 in use): asks for a phase that never
// completes, with the plan's poll limit, as the task-queue waits do.
__device__ __forceinline__ void mbar_wait_hook(uint32_t bar, uint32_t parity, const DevPlan& d) {
  volatile const int* flags = &d.sc->solve_flags;
  for (unsigned it = 0; !mbar_test(bar, parity); ++it) {
    if (it > d.spin_limit || (*flags & 1)) {
      atomicOr(&d.sc->solve_flags, 1);
      break;
    }
    __nanosleep(64);
  }
}

// K-major shared-memory operand without swizzle: 8-row x 16-byte core
// matrices of 128 bytes, 128 bytes apart along K, 512 along the rows.
__device__ __forceinline__ uint64_t operand_desc(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFF) >> 4) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)(512 >> 4) << 32) | (1ull << 46);
}

// power of two 2^e (0 below the normal range; NaN for the not-finite mark)
__device__ __forceinline__ double pow2_or_nan(int e) {
  if (e > 1023) return __longlong_as_double(0x7ff8000000000000ll);
  return e < -1022 ? 0.0 : __longlong_as_double((long long)(e + 1023) << 52);
}

// a - 2^(e - 32) sum_w v_w 2^(56 - 8 w) for eight exact sums |v_w| < 2^22 (e up
// to 47 below the product's exponent): the sum as a 96-bit integer, rounded to a
// double with integer instructions, then one FP64 addition.  (The SM does two
// FP64 operations a clock and 64 integer ones: three FP64 operations an element,
// which formed the sum from two biased doubles, bounded the update.  14,000
// buses, 9,472 columns: 68.5 ms of updates, 46 with these.)
__device__ __forceinline__ double minus_sums(double a, const int (&v)[8], int e) {
  const long long hi = (long long)(v[0] * 256 + v[1]) * 65536 + (v[2] * 256 + v[3]);
  const long long lo = (long long)(v[4] * 256 + v[5]) * 65536 + (v[6] * 256 + v[7]);
  const long long H = hi + (lo >> 32);  // hi 2^32 + lo = H 2^32 + L, |H| < 2^48
  const uint32_t sign = (uint32_t)(H >> 63);
  // the magnitude; of a negative sum one unit of 2^(e - 32) short, far below
  // what the digits left out
  const uint32_t w2 = (uint32_t)((unsigned long long)H >> 32) ^ sign, w1 = (uint32_t)H ^ sign, w0 = (uint32_t)lo ^ sign;
  uint32_t x = w2, y = w1, z = w0;
  int lz = 0;
  if (x == 0) {
    x = w1, y = w0, z = 0, lz = 32;
    if (x == 0) x = w0, y = 0, lz = 64;
  }
  const int n = __clz(x);
  const uint32_t m1 = __funnelshift_l(y, x, n), m0 = __funnelshift_l(z, y, n);
  // leading one at bit 63: exponent 63 + e - lz - n; a carry out of the rounded
  // fraction raises the exponent field
  const unsigned long long m = ((unsigned long long)m1 << 32 | m0);
  const bool inside = e >= -900 && e <= 900;  // else the product may leave the normal range
  const uint32_t top = (uint32_t)(1023 + 62 + (inside ? e : 0) - lz - n) << 20 | (~sign & 0x80000000u);
  const unsigned long long bits = ((unsigned long long)top << 32) + (m >> 11) + ((m0 >> 10) & 1);
  const double t = x ? __longlong_as_double((long long)bits) : 0.0;
  return inside ? dadd(a, t) : fma(pow2_or_nan(e), t, a);
}

// L D L^T of a 32 x 32 diagonal block (lower triangle in A, row stride 33) by
// 256 threads: M = L^-1 (unit lower), the reciprocals of D and of its roots.
// Gauss elimination of [A I].  FP64 instructions are what it costs (a warp's
// takes 64 clocks of its quarter of the SM), so the elements of a step are
// packed onto the threads, and warp 0 runs ahead on the next pivot's column
// (one multiply-add, reciprocal, multipliers) while the others finish the
// step.  It runs in the update kernel's first CTA (the one that completes the
// block), beside the others, so that the panel kernel starts with M ready.
__device__ void pivot_block(DevPlan& d, const DevBorder& bd, int panel, double* A, double* M) {
  constexpr int n = kBorderPanel, ld = n + 1;
  __shared__ double sinv[n], piv[n], mult[2][n];
  const int tid = threadIdx.x, lane = tid & 31;
  // threads 32 on: up to three (row, t < row) each, t the column of M, or past
  // the pivot's the column t + 1 of A
  int ei[3], et[3];
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const int f = tid - 32 + 224 * q;
    int i = 0;
    if (f >= 0 && f < n * (n - 1) / 2) {
      i = (int)((1.0f + sqrtf(1.0f + 8.0f * (float)f)) * 0.5f);
      if (i * (i - 1) / 2 > f) --i;
      if ((i + 1) * i / 2 <= f) ++i;
    }
    ei[q] = i;
    et[q] = f - i * (i - 1) / 2;
  }
  for (int e = tid; e < n * n; e += 256) M[(e / n) * ld + e % n] = e / n == e % n ? 1.0 : 0.0;
  __syncthreads();
  // warp 0, lane i: pivot k's multipliers A(i,k) / A(k,k) from the column c
  auto pivot = [&](int k, double c) {
    const double p = __shfl_sync(0xffffffffu, c, k);
    const double inv = 1.0 / p;
    mult[k & 1][lane] = c * inv;
    if (lane == 0) {
      piv[k] = p;
      sinv[k] = inv;
    }
  };
  if (tid < 32) pivot(0, A[lane * ld]);
  __syncthreads();
  for (int k = 0; k < n - 1; ++k) {
    const double* l = mult[k & 1];
    if (tid < 32) {
      // column k + 1, then its pivot
      double c = 0.0;
      if (lane > k) {
        c = fma(-l[lane], A[(k + 1) * ld + k], A[lane * ld + k + 1]);
        A[lane * ld + k + 1] = c;
      }
      pivot(k + 1, c);
    } else {
      // rows i > k: j <= k of M, j > k + 1 of A (column k + 1 is warp 0's)
#pragma unroll
      for (int q = 0; q < 3; ++q)
        if (ei[q] > k) {
          const int i = ei[q], j = et[q] <= k ? et[q] : et[q] + 1;
          double* g = j <= k ? &M[i * ld + j] : &A[i * ld + j];
          *g = fma(-l[i], j <= k ? M[k * ld + j] : A[j * ld + k], *g);
        }
    }
    __syncthreads();
  }
  double* out = bd.piv;
  for (int e = tid; e < n * n; e += 256) out[e] = M[(e / n) * ld + e % n];
  if (tid < n) {
    const int col = panel * n + tid;
    if (col < bd.k) note_pivot(d, bd.bcol[col], piv[tid]);
    out[n * n + tid] = sinv[tid];
    out[n * n + n + tid] = sqrt(sinv[tid]);
  }
}

__global__ void __launch_bounds__(256) k_border_pivot0(DevPlan d, DevBorder bd) {
  constexpr int n = kBorderPanel, ld = n + 1;
  __shared__ double A[n * ld], M[n * ld];
  for (int e = threadIdx.x; e < n * n; e += 256) A[(e % n) * ld + e / n] = bd.W[(int64_t)(e / n) * bd.ld + e % n];
  __syncthreads();
  pivot_block(d, bd, 0, A, M);
}

// One CTA per group of eight rows, a warp for two of them: with lane t the
// dot products of row a's index t and of row b's index 31 - t have 31 terms
// together, so the triangular products waste no lanes.  FP64-bound (about
// 1,000 FMA a row); eight rows a CTA spread a small border over the SMs.
__global__ void __launch_bounds__(128) k_border_panel(DevPlan d, DevBorder bd, int p) {
  constexpr int n = kBorderPanel, ld = n + 1;
  __shared__ double M[n * ld], dinv[n], rs[n];
  __shared__ double V[8][n + 1], Z[8][n + 1];
  __shared__ __align__(16) uint16_t stage[kDigits * 8 * n];
  __shared__ int ex[8];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r0 = blockIdx.x * 8, c0 = p * n;
  for (int e = tid; e < n * n; e += 128) M[(e / n) * ld + e % n] = bd.piv[e];
  if (tid < n) {
    dinv[tid] = bd.piv[n * n + tid];
    rs[tid] = bd.piv[n * n + n + tid];
  }
  const bool below = r0 >= c0 + n, own = !below && r0 >= c0;
  double* W = bd.W;
  if (below) {
    for (int e = tid; e < 8 * n; e += 128) V[e & 7][e >> 3] = W[(int64_t)(c0 + (e >> 3)) * bd.ld + r0 + (e & 7)];
  } else if (!own) {
    for (int e = tid; e < 8 * n; e += 128) V[e >> 5][e & 31] = W[(int64_t)(r0 + (e >> 5)) * bd.ld + c0 + (e & 31)];
  }
  __syncthreads();
  if (own) {
    // the panel's own rows of X: D^-1/2 M; their digits are zero
    for (int e = tid; e < 8 * n; e += 128) {
      const int i = r0 - c0 + (e & 7), j = e >> 3;
      V[e & 7][j] = rs[i] * M[i * ld + j];
    }
    for (int e = tid; e < kDigits * 8 * n / 2; e += 128) reinterpret_cast<uint32_t*>(stage)[e] = 0u;
    if (tid < 8) ex[tid] = kExpZero;
  } else {
    const int ra = 2 * warp, rb = ra + 1, t = lane, tb = n - 1 - lane;
    double ya = V[ra][t], yb = V[rb][tb];
#pragma unroll 4
    for (int s = 0; s < n - 1; ++s) {
      if (s < t) ya = fma(M[t * ld + s], V[ra][s], ya);
      else yb = fma(M[tb * ld + s - t], V[rb][s - t], yb);
    }
    Z[ra][t] = ya * dinv[t];
    Z[rb][tb] = yb * dinv[tb];
    ya *= rs[t];
    yb *= rs[tb];
    // digits of the two rows of Y
    double y2[2] = {ya, yb};
    const int row2[2] = {ra, rb}, t2[2] = {t, tb};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const double a = fabs(y2[h]);
      // exponent field of the largest entry (NaN and infinity: 2047)
      int e = (int)((unsigned long long)__double_as_longlong(a) >> 52) & 0x7ff;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
      const bool bad = e == 0x7ff, tiny = e < 64;  // |y| < 2^(e - 1022)
      long long m = 0;
      if (!bad && !tiny) m = __double2ll_rn(y2[h] * pow2_or_nan(55 - (e - 1022)));
      if (lane == 0) ex[row2[h]] = bad ? kExpNan : tiny ? kExpZero : e - 1022;
      uint16_t* st = stage + (t2[h] >> 3) * 64 + row2[h] * 8 + (t2[h] & 7);
#pragma unroll
      for (int q = kDigits - 1; q >= 0; --q) {
        int dg = q ? (int)(signed char)(m & 0xff) : (int)m;
        m = (m - dg) >> 8;
        st[q * 8 * n] = (uint16_t)(__float_as_uint((float)dg) >> 16);  // an integer of at most 8 bits: exact in bf16
      }
    }
    __syncwarp();
    if (below) {
      // Y L^-1 = M^T D^-1 M v: z_s + sum_{t > s} M[t][s] z_t
      ya = Z[ra][t];
      yb = Z[rb][tb];
#pragma unroll 4
      for (int s = 1; s < n; ++s) {
        if (s > t) ya = fma(M[s * ld + t], Z[ra][s], ya);
        else yb = fma(M[(tb + s) * ld + tb], Z[rb][tb + s], yb);
      }
      ya = -ya;
      yb = -yb;
    }
    V[ra][t] = ya;
    V[rb][tb] = yb;
  }
  __syncthreads();
  if (below || own) {
    for (int e = tid; e < 8 * n; e += 128) W[(int64_t)(c0 + (e >> 3)) * bd.ld + r0 + (e & 7)] = V[e & 7][e >> 3];
  } else {
    for (int e = tid; e < 8 * n; e += 128) W[(int64_t)(r0 + (e >> 5)) * bd.ld + c0 + (e & 31)] = V[e >> 5][e & 31];
  }
  uint8_t* dst = bd.dig + (int64_t)(r0 / kRowBlock) * kDigitBlockBytes + (r0 % kRowBlock) / 8 * 512;
  for (int e = tid; e < kDigits * 32; e += 128)
    *reinterpret_cast<uint4*>(dst + (e >> 5) * kPlaneBytes + (e & 31) * 16) =
        *reinterpret_cast<const uint4*>(reinterpret_cast<const uint8_t*>(stage) + e * 16);
  if (tid < 8) bd.ey[r0 + tid] = ex[tid];
}

// A -= Y Y^T on kRun 128 x 32 tiles of a row block below the panel.  Bounded
// by the epilogue's integer work (minus_sums) and by the read and write of A.  A
// CTA keeps the row block's digits for its run of tiles and fetches the next
// tile's 14 KB of column digits while it works on one; two CTAs an SM overlap one's products with the other's epilogue.  The column
// digits lie below one another in shared memory and the sums of a weight beside
// one another in tensor memory, so that one instruction multiplies a row digit
// with all column digits it is kept with (14 + 2 instructions instead of 68).
template <int kRun>
__global__ void __launch_bounds__(256, 2) k_border_update(DevPlan d, DevBorder bd, int p) {
  extern __shared__ __align__(1024) uint8_t usm[];
  __shared__ __align__(8) uint64_t bars[4];  // row digits, column digits (two buffers), products
  __shared__ uint32_t tmem_at;
  static_assert(kRun == 1 || kRun == 2 || kRun == 4, "runs end with the row block");
  const int pn = p + 1;  // the next panel: the run with its diagonal tile comes first, then its pivot block
  constexpr int kPer = 4 / kRun;  // runs per 128 columns
  const int rb0 = pn / 4, t_0 = kPer * (rb0 * (rb0 + 1) / 2), t_next = t_0 + pn / kRun;  // row blocks above: none
  int t = t_0 + (int)blockIdx.x;
  t = t == t_0 ? t_next : t == t_next ? t_0 : t;
  int rb = (int)((sqrtf(1.0f + 8.0f / kPer * (float)t) - 1.0f) * 0.5f);
  while (kPer * (rb * (rb + 1) / 2) > t) --rb;
  while (kPer * ((rb + 1) * (rb + 2) / 2) <= t) ++rb;
  int cb0 = (t - kPer * (rb * (rb + 1) / 2)) * kRun;
  // the run's tiles: without the panel itself; constraint rows (Schur plans)
  // have no columns of X
  const int cb1 = min(cb0 + kRun, bd.ncb);
  if (rb * kRowBlock >= bd.npan * kBorderPanel) cb0 = max(cb0, pn);
  const int skip = p >= cb0 && p < cb1 ? p : -1;
  const int ntile = cb1 - cb0 - (skip >= 0);
  if (ntile <= 0) return;
  auto tile_col = [&](int s) { return cb0 + s + (skip >= 0 && cb0 + s >= skip); };
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t sA = smem_addr(usm), sB = sA + kDigitBlockBytes;
  const uint32_t bar_a = smem_addr(&bars[0]), bar_b = smem_addr(&bars[1]), bar_mma = smem_addr(&bars[3]);
  auto load_b = [&](int s) {  // one thread
    const int cb = tile_col(s);
    const uint32_t bar = bar_b + 8 * (s & 1), dst = sB + (s & 1) * (kDigits * kBPlaneBytes);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(kDigits * kBPlaneBytes) : "memory");
    const uint8_t* gb = bd.dig + (int64_t)(cb >> 2) * kDigitBlockBytes + (cb & 3) * kBPlaneBytes;
#pragma unroll
    for (int q = 0; q < kDigits; ++q)
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                       dst + q * kBPlaneBytes),
                   "l"(gb + q * kPlaneBytes), "r"(kBPlaneBytes), "r"(bar) : "memory");
  };
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_at)),
                 "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 32) {
    for (int i = 0; i < 4; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar_a + 8 * i));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar_a), "r"(kDigitBlockBytes) : "memory");
    const uint8_t* ga = bd.dig + (int64_t)rb * kDigitBlockBytes;
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(sA),
                 "l"(ga), "r"(kDigitBlockBytes), "r"(bar_a) : "memory");
    load_b(0);
  }
  const int quad = warp & 3, half = warp >> 2;
  const int row = rb * kRowBlock + quad * 32 + lane;
  const int er = row < pn * kBorderPanel ? kExpZero : bd.ey[row] - 38;  // rows up to the panel are done
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_at;
  for (int s = 0; s < ntile; ++s) {
    const int c0 = tile_col(s) * kTileCols + half * 16;
    if (tid == 0) {
      if (s + 1 < ntile) load_b(s + 1);
      if (s == 0 && !mbar_wait(bar_a, 0, d.sc)) mbar_wait(bar_a, 0, d.sc);  // the copies in flight: once more, with a limit
      if (!mbar_wait(bar_b + 8 * (s & 1), (s >> 1) & 1, d.sc)) mbar_wait(bar_b + 8 * (s & 1), (s >> 1) & 1, d.sc);
      if (s == 0 && d.dbg_unsatisfiable) mbar_wait_hook(bar_a, 1, d);
      // D f32, A and B bf16, K-major both, M 128, N 32 per column digit
      constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kRowBlock / 16) << 24);
      auto mma = [&](int i, int j, int nj, int kk, uint32_t acc) {
        const uint64_t da = operand_desc(sA + i * kPlaneBytes + kk * 256);
        const uint64_t db = operand_desc(sB + (s & 1) * (kDigits * kBPlaneBytes) + j * kBPlaneBytes + kk * 256);
        asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(
                         tmem + (uint32_t)((i + j) * kTileCols)),
                     "l"(da), "l"(db), "r"(idesc | ((uint32_t)(nj * kTileCols / 8) << 17)), "r"(acc) : "memory");
      };
#pragma unroll 1
      for (int kk = 0; kk < 2; ++kk) {
        mma(0, 0, kDigits, kk, kk > 0);
        mma(1, kDigits - 1, 1, kk, kk > 0);  // the last weight's first product
        mma(1, 0, kDigits - 1, kk, 1);
#pragma unroll 1
        for (int i = 2; i < kDigits; ++i) mma(i, 0, kAccs - i, kk, 1);
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar_mma) : "memory");
    }
    // this thread's sixteen elements of A, on their way meanwhile
    double* g = bd.W + (int64_t)c0 * bd.ld + row;
    double a[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) a[j] = g[(int64_t)j * bd.ld];
    const int4* ecol = reinterpret_cast<const int4*>(bd.ey + c0);
    if (!mbar_wait(bar_mma, s & 1, d.sc)) mbar_wait(bar_mma, s & 1, d.sc);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t r[kAccs][8];
#pragma unroll
      for (int w = 0; w < kAccs; ++w) {
        const uint32_t ta = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(w * kTileCols + half * 16 + h * 8);
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(r[w][0]), "=r"(r[w][1]), "=r"(r[w][2]), "=r"(r[w][3]), "=r"(r[w][4]), "=r"(r[w][5]),
                       "=r"(r[w][6]), "=r"(r[w][7])
                     : "r"(ta));
      }
      const int4 e0 = ecol[2 * h], e1 = ecol[2 * h + 1];
      const int ec[8] = {e0.x, e0.y, e0.z, e0.w, e1.x, e1.y, e1.z, e1.w};
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        int v[kAccs];
#pragma unroll
        for (int w = 0; w < kAccs; ++w)  // exact: |sum| <= 7 * 2^19 < 2^22
          v[w] = __float_as_int(__uint_as_float(r[w][j]) + 12582912.0f) - 0x4B400000;
        a[h * 8 + j] = minus_sums(a[h * 8 + j], v, er + ec[j]);
      }
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) g[(int64_t)j * bd.ld] = a[j];
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();  // the sums are read: the next tile's products may replace them
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  }
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
  if (blockIdx.x == 0 && pn < bd.npan) {
    // the shared memory of the operands is free: the next panel's pivot block
    double* A = reinterpret_cast<double*>(usm);
    double* M = A + kBorderPanel * (kBorderPanel + 1);
    const double* src = bd.W + (int64_t)pn * kBorderPanel * bd.ld + pn * kBorderPanel;
    for (int e = tid; e < kBorderPanel * kBorderPanel; e += 256)
      A[(e % kBorderPanel) * (kBorderPanel + 1) + e / kBorderPanel] = src[(int64_t)(e / kBorderPanel) * bd.ld + e % kBorderPanel];
    __syncthreads();
    pivot_block(d, bd, pn, A, M);
  }
}

// Row panels of X and of X^T for the solves' products, one contiguous block
// per rb rows (column after column of the panel, zeros outside the triangle):
// in the column-major border itself a task's pieces lie a column stride apart,
// which ran the 10,000-bus products at a fifth of the streaming rate.  One CTA
// per 64 x 64 tile of the lower triangle.
__host__ __device__ inline int64_t panel_lo(int64_t b, int rb) { return (int64_t)rb * rb * (b * (b + 1) / 2); }
// X^T panels cover the columns [rb b, rb nrb): the offset from the first
__host__ __device__ inline int64_t panel_up(int64_t b, int64_t nrb, int rb) {
  return (int64_t)rb * rb * (b * nrb - b * (b - 1) / 2);
}

__global__ void __launch_bounds__(256) k_border_pack(DevBorder bd) {
  __shared__ double tile[64][65];
  int ti = (int)((sqrtf(1.0f + 8.0f * (float)blockIdx.x) - 1.0f) * 0.5f);
  while (ti * (ti + 1) / 2 > (int)blockIdx.x) --ti;
  while ((ti + 1) * (ti + 2) / 2 <= (int)blockIdx.x) ++ti;
  const int tj = blockIdx.x - ti * (ti + 1) / 2;
  const int i0 = ti * 64, j0 = tj * 64, rb = bd.rb, nrb = bd.nrb;
  for (int e = threadIdx.x; e < 64 * 64; e += 256) {
    const int i = e & 63, j = e >> 6;
    tile[j][i] = i0 + i >= j0 + j ? bd.W[(int64_t)(j0 + j) * bd.ld + i0 + i] : 0.0;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < 64 * 64; e += 256) {
    // rows of X: row block (i0 + i) / rb, column j0 + j
    const int r = e % rb, j = (e / rb) & 63, g = e / rb / 64, b = i0 / rb + g;
    if (b < nrb && j0 + j < (b + 1) * rb) bd.xlo[panel_lo(b, rb) + (int64_t)(j0 + j) * rb + r] = tile[j][g * rb + r];
  }
  for (int e = threadIdx.x; e < 64 * 64; e += 256) {
    // rows of X^T: row block (j0 + c) / rb, column i0 + i
    const int r = e % rb, i = (e / rb) & 63, g = e / rb / 64, b = j0 / rb + g;
    if (b < nrb && i0 + i >= b * rb && i0 + i < nrb * rb)
      bd.xup[panel_up(b, nrb, rb) + (int64_t)(i0 + i - b * rb) * rb + r] = tile[g * rb + r][i];
  }
}

// ---------------------------------------------------------------------------
// Solves and the CG loop: one launch each, its CTAs claiming tasks of dense
// phases from a counter in phase order.
//   0  CG: Jc^T r, Jc^T w, Jc^T s
//   1  blocks:  y_F = X b_F, u = E b_F;       CG: the vector update as well
//   2  border right-hand side  bt = b_S - sum u   (in phase 1 without blocks)
//   3  by = X bt               4  x_S = X^T by
//   5  blocks:  x_F = X^T y_F - E^T x_S
//   6  CG: w = Jc_p x and the sums of the recurrence's scalars
// A task waits (bounded) until the tasks of the phase it reads from are done;
// they were claimed before it by CTAs that are running, so the scheme cannot
// deadlock whatever the number of resident CTAs.  What a task reads that the
// launch does not change (its panel, its block, indices) it loads before it
// waits: a phase then costs little more than the round trips of its signal and
// of the vector.  Data written in the same launch is read with ld.global.cg.
// Every sum is taken in a fixed order: results do not depend on the
// scheduling.  The CG loop in one launch replaces five launches per iteration.
// ---------------------------------------------------------------------------
constexpr int kCgRows = 256;  // rows of a vector task
constexpr int kRowTask = 64;  // columns or constraints of a sparse task, four threads each

typedef unsigned long long count_t;  // tasks of all iterations of a CG run

// Part of one row of a sparse product: L threads share a row (its entries
// interleaved), each one's first eight indices and values are loaded ahead of
// the wait for the vector.  (Hub buses have rows of 60 entries and more: one
// thread per row made them the phase's length.)
struct SparseRow {
  int p, e, L;
  int c[8];
  double a[8];
};
template <class VIdx>
__device__ __forceinline__ void load_row(SparseRow& r, int p, int e, int L, int sub, const int* __restrict__ ci, const double* __restrict__ v, VIdx vidx) {
  r.p = p + sub;
  r.e = e;
  r.L = L;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const bool in = r.p + j * L < e;
    r.c[j] = in ? ci[r.p + j * L] : 0;
    r.a[j] = in ? v[vidx(r.p + j * L)] : 0.0;
  }
}
template <class VIdx, class X>
__device__ __forceinline__ double row_dot(SparseRow& r, const int* __restrict__ ci, const double* __restrict__ v, VIdx vidx, X x) {
  double acc = 0.0;
  for (;;) {
    double t[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) t[j] = r.p + j * r.L < r.e ? x(r.c[j]) : 0.0;
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (r.p + j * r.L < r.e) acc = fma(r.a[j], t[j], acc);
    const int p = r.p + 8 * r.L;
    if (p >= r.e) break;
    load_row(r, p, r.e, r.L, 0, ci, v, vidx);
  }
  return acc;
}
// the four threads' parts (neighbouring lanes)
__device__ __forceinline__ double join_row(double s) {
  s = dadd(s, __shfl_xor_sync(0xffffffffu, s, 1));
  return dadd(s, __shfl_xor_sync(0xffffffffu, s, 2));
}

// CG right-hand side Jc_p^T (r - alpha (w + beta s)): the three products come
// from a phase of their own, beside the iteration's scalars, column after
// column of the border and the blocks, so that a column's row of Jc_p^T is read
// once and the scalars are followed by two multiply-adds.  (Each task that
// needs a column formed its entry from the updated residual itself: a block of
// 232 rows did so four times, 10.5 us a task at 5,000 buses, now 4.4.  Eight
// threads a column end its phase 1 us earlier at 1,000 buses and 4 us later at
// 10,000, where its tasks fill the GPU twice.)
struct RhsParts {
  double r, w, s;
};
__device__ __forceinline__ RhsParts load_parts(const DevBorder& bd, int j) {
  return RhsParts{__ldcg(&bd.jt[j]), __ldcg(&bd.jt[bd.njt + j]), __ldcg(&bd.jt[2 * bd.njt + j])};
}
__device__ __forceinline__ double rhs_value(const RhsParts& q, const double* sc) { return fma(-sc[0], fma(sc[1], q.s, q.w), q.r); }

template <class Wait>
__device__ __forceinline__ bool rhs_parts_task(const DevPlan& d, const DevBorder& bd, int task, const double* r, const double* s, Wait wait) {
  const int j = task * kRowTask + (threadIdx.x >> 2), sub = threadIdx.x & 3;
  const int col = j >= bd.njt ? 0 : j < bd.k ? bd.bcol[j] : bd.blk_col[j - bd.k];
  const int* src = d.jctp_src;
  auto vi = [src](int p) { return src[p]; };
  SparseRow row;
  row.p = row.e = 0;
  row.L = 4;
  if (j < bd.njt) load_row(row, d.jctp_rp[col], d.jctp_rp[col + 1], 4, sub, d.jctp_ci, d.jc_s, vi);
  if (!wait()) return false;
  RhsParts q{0.0, 0.0, 0.0};
  for (;;) {
#pragma unroll
    for (int h = 0; h < 8; h += 4) {
      if (row.p + h * 4 >= row.e) break;
      double t[3][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const bool in = row.p + (h + i) * 4 < row.e;
        const int c = row.c[h + i];
        t[0][i] = in ? __ldcg(&r[c]) : 0.0;
        t[1][i] = in ? __ldcg(&d.cg_w[c]) : 0.0;
        t[2][i] = in ? __ldcg(&s[c]) : 0.0;
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (row.p + (h + i) * 4 < row.e) {
          q.r = fma(row.a[h + i], t[0][i], q.r);
          q.w = fma(row.a[h + i], t[1][i], q.w);
          q.s = fma(row.a[h + i], t[2][i], q.s);
        }
    }
    const int p = row.p + 32;
    if (p >= row.e) break;
    load_row(row, p, row.e, 4, 0, d.jctp_ci, d.jc_s, vi);
  }
  q.r = join_row(q.r);
  q.w = join_row(q.w);
  q.s = join_row(q.s);
  if (j < bd.njt && sub == 0) {
    bd.jt[j] = q.r;
    bd.jt[bd.njt + j] = q.w;
    bd.jt[2 * bd.njt + j] = q.s;
  }
  return true;
}

// every fourth of the blocks' contributions to border column j
__device__ __forceinline__ double border_updates(const DevBorder& bd, int j, int sub) {
  double s = 0.0;
  const int e = bd.ug_rp[j + 1];
  for (int p = bd.ug_rp[j] + sub; p < e; p += 16) {
    double t[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) t[i] = p + 4 * i < e ? __ldcg(&bd.u[bd.ug_pos[p + 4 * i]]) : 0.0;
#pragma unroll
    for (int i = 0; i < 4; ++i) s = dadd(s, t[i]);
  }
  return s;
}

// Products of a dense row panel, column after column of its RB rows, with a
// vector: 256 / RB threads a row over interleaved columns.  Panels stream
// through kStages shared-memory chunks by bulk copies that thread 0 issues, the
// first of them before the task waits for its vector.  A warp that has read a
// chunk says so on the chunk's second mbarrier, so that warps run apart (a CTA
// barrier per chunk was a third of their stalls).
constexpr int kChunk = 2048, kStages = 3;   // entries of a chunk
constexpr int kRed = 512, kMaxVec = 256;    // doubles: two sets of partial sums, a block's vector
constexpr int kChunkVec = 512;              // a chunk's piece of the vector (four rows a panel)
constexpr int kSolveSmem = (kRed + kMaxVec + kStages * (kChunk + kChunkVec)) * 8;
constexpr int kSchurMax = 2048;             // rows of a Schur plan, its vector in shared memory
constexpr int kSchurSmem = (kRed + kSchurMax + kStages * kChunk) * 8;
static_assert(kRed % 2 == 0 && kMaxVec % 2 == 0 && kSchurMax % 2 == 0 && kChunk % 2 == 0 && kChunkVec % 2 == 0,
              "bulk copies go to 16-byte boundaries");

// The CTA's chunk ring: barriers [chunk full, chunk read], chunks issued
// (thread 0), vector pieces issued (thread 0) and chunks consumed since the
// launch.
struct Ring {
  uint32_t bar;
  double* buf;
  int stride;  // doubles from chunk to chunk
  unsigned put, vec, got;
};
// arrivals: 1, or 2 where a chunk's piece of the vector comes with it
__device__ __forceinline__ Ring ring_init(uint64_t* bars, double* buf, int stride, int arrivals) {
  Ring g{smem_addr(bars), buf, stride, 0, 0, 0};
  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(g.bar + 8 * i), "r"(arrivals));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 8;" ::"r"(g.bar + 8 * (kStages + i)));
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  return g;
}
__device__ __forceinline__ void ring_copy(uint32_t bar, const double* dst, const double* src, int bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_addr(dst)), "l"(src),
               "r"(bytes), "r"(bar) : "memory");
}
// thread 0: n entries from M into the next buffer, once all warps have read it
__device__ __forceinline__ void ring_put(Ring& g, const double* M, int n, DevScalars* sc) {
  const int st = g.put % kStages;
  mbar_wait(g.bar + 8 * (kStages + st), ((g.put / kStages) & 1) ^ 1, sc);
  ++g.put;
  ring_copy(g.bar + 8 * st, g.buf + st * g.stride, M, n * 8);
}
// thread 0: the vector's part of the next chunk, n entries from v (0: none)
__device__ __forceinline__ void ring_vec(Ring& g, const double* v, int n) {
  const int st = g.vec % kStages;
  ++g.vec;
  if (n) ring_copy(g.bar + 8 * st, g.buf + st * g.stride + kChunk, v, (n * 8 + 15) & ~15);
  else asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(g.bar + 8 * st) : "memory");
}
// a task that gives up: thread 0 stays until the copies in flight have landed
__device__ __forceinline__ void ring_drain(Ring& g, DevScalars* sc, bool vec) {
  if (threadIdx.x == 0) {
    for (; vec && g.vec < g.put;) ring_vec(g, nullptr, 0);
    for (; g.got < g.put; ++g.got) mbar_wait(g.bar + 8 * (g.got % kStages), (g.got / kStages) & 1, sc);
  }
}

// One chunk: `left` columns from this thread's first one on, into two sums
template <int RB>
__device__ __forceinline__ void chunk_product(Ring& g, const double* v, int left, double (&a)[2], DevScalars* sc) {
  constexpr int P = 256 / RB;
  const int st = g.got % kStages;
  mbar_wait(g.bar + 8 * st, (g.got / kStages) & 1, sc);
  ++g.got;
  const double* m = g.buf + st * g.stride + threadIdx.x;
  if (!v) v = g.buf + st * g.stride + kChunk + threadIdx.x / RB;
  if (left > 7 * P) {
#pragma unroll
    for (int q = 0; q < 8; ++q) a[q & 1] = fma(m[q * 256], v[q * P], a[q & 1]);
  } else {
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (q * P < left) a[q & 1] = fma(m[q * 256], v[q * P], a[q & 1]);
  }
  __syncwarp();
  if ((threadIdx.x & 31) == 0)
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(g.bar + 8 * (kStages + st)) : "memory");
}

// The 256 / RB parts of each row: through shared memory to as many threads of
// the first warps as leave eight parts each (FP64 adds by full warps cost the
// product's time).  Row threadIdx.x in threads below RB.
template <int RB>
__device__ __forceinline__ double panel_sum(double part, double* red) {
  constexpr int P = 256 / RB, kParts = P < 8 ? P : 8, kT = 256 / kParts;  // parts per thread, threads
  red[threadIdx.x] = part;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x < kT) {
    double w[kParts];
#pragma unroll
    for (int q = 0; q < kParts; ++q) w[q] = red[q * kT + threadIdx.x];
#pragma unroll
    for (int o = 1; o < kParts; o <<= 1)
#pragma unroll
      for (int q = 0; q < kParts; q += 2 * o) w[q] = dadd(w[q], w[q + o]);
    t = w[0];
#pragma unroll
    for (int o = RB; o < kT; o <<= 1) t = dadd(t, __shfl_xor_sync(0xffffffffu, t, o));
  }
  return t;
}

// One panel with a vector that is in shared memory
struct Panel {
  const double* M;
  int n;  // entries: columns * RB
};
__device__ __forceinline__ void panel_start(Ring& g, const Panel& p, DevScalars* sc, bool vec) {
  if (threadIdx.x == 0)
    for (int c = 0; c < kStages && c * kChunk < p.n; ++c) {
      ring_put(g, p.M + c * kChunk, min(kChunk, p.n - c * kChunk), sc);
      if (vec) ring_vec(g, nullptr, 0);
    }
}
template <int RB>
__device__ __forceinline__ double panel_product(Ring& g, const Panel& p, const double* v, double* red, DevScalars* sc, bool vec) {
  constexpr int kCols = kChunk / RB;
  v += threadIdx.x / RB;
  double a[2] = {0.0, 0.0};
  int left = p.n / RB - threadIdx.x / RB;
  for (int c = 0; c * kChunk < p.n; ++c, v += kCols, left -= kCols) {
    chunk_product<RB>(g, v, left, a, sc);
    const int next = (c - 1 + kStages) * kChunk;  // into the buffer of the chunk before, which all warps have or are about to have read
    if (threadIdx.x == 0 && c > 0 && next < p.n) {
      ring_put(g, p.M + next, min(kChunk, p.n - next), sc);
      if (vec) ring_vec(g, nullptr, 0);
    }
  }
  return panel_sum<RB>(dadd(a[0], a[1]), red);
}

// by = X bt or x_S = X^T by (up): a task is every stride-th of the bins from
// `bin` on, a bin a set of whole panels; the bins hold equal work (the longest
// panel of one side with short ones), longest first.  A chunk of a panel and
// its piece of the vector come together, and the chunks of all the task's
// panels follow one another through the ring.  Bounded by the FP64 pipe (an
// entry is one multiply-add, two a clock and SM), by HBM where the panels
// exceed the L2.  Measured: 44 us a product at 10,000 buses (6,746 columns, 39
// at the FP64 peak) and 14 at 5,000 (3,342; 9).  (Tasks of one panel's piece of
// 2,048 columns, unequal and claimed one by one, left an SM without a task for
// 0.2 of the phase and with one or two for 0.25: 59 and 17 us.  Claiming the
// next task ahead, during the last chunks: the same at 5,000, 2 % slower at
// 10,000.)
struct BinCursor {
  int bin, i, next;  // bin, position in its list, the panel that follows there (read ahead; -1: none)
  int b, n, c;       // panel, its entries, chunk
  __device__ __forceinline__ void open(const DevBorder& bd, int q, bool up, int RB) {
    next = bd.bin_panel[++i];
    b = up ? bd.nrb - 1 - q : q;
    n = up ? (bd.k - b * RB) * RB : min(bd.k, (b + 1) * RB) * RB;
    c = 0;
  }
  __device__ __forceinline__ void start(const DevBorder& bd, int first, bool up, int RB) {
    bin = first;
    i = bin * bd.binw;
    open(bd, bd.bin_panel[i], up, RB);
  }
  __device__ __forceinline__ void next_panel(const DevBorder& bd, int stride, bool up, int RB) {
    if (next >= 0) {
      open(bd, next, up, RB);
      return;
    }
    bin += stride;
    if (bin < bd.nbin) start(bd, bin, up, RB);
  }
  __device__ __forceinline__ void next_chunk(const DevBorder& bd, int stride, bool up, int RB) {
    if (++c * kChunk >= n) next_panel(bd, stride, up, RB);
  }
};

template <int RB, class Wait>
__device__ __forceinline__ bool bin_task(const DevBorder& bd, Ring& g, int bin, int stride, bool up, double* x, double* sm, DevScalars* sc, Wait wait) {
  constexpr int kCols = kChunk / RB;
  BinCursor cur, put, vec;  // consumed (all threads); issued, vector pieces issued (thread 0)
  cur.start(bd, bin, up, RB);
  put = vec = cur;
  auto put_next = [&]() {
    const double* M = up ? bd.xup + panel_up(put.b, bd.nrb, RB) : bd.xlo + panel_lo(put.b, RB);
    ring_put(g, M + put.c * kChunk, min(kChunk, put.n - put.c * kChunk), sc);
    put.next_chunk(bd, stride, up, RB);
  };
  auto vec_next = [&]() {
    const int j = vec.c * kCols;
    ring_vec(g, up ? bd.by + vec.b * RB + j : bd.bt + j, min(kCols, vec.n / RB - j));
    vec.next_chunk(bd, stride, up, RB);
  };
  if (threadIdx.x == 0)
    for (int s = 0; s < kStages && put.bin < bd.nbin; ++s) put_next();
  if (!wait()) {
    ring_drain(g, sc, true);
    return false;
  }
  if (threadIdx.x == 0) {
    asm volatile("fence.proxy.async;" ::: "memory");  // the vector was written by other CTAs' stores
    while (g.vec < g.put) vec_next();
  }
  double* red = sm;
  while (cur.bin < bd.nbin) {
    const int row = cur.b * RB + threadIdx.x;
    const int at = threadIdx.x < RB && row < bd.k ? (up ? bd.bcol[row] : row) : -1;
    double a[2] = {0.0, 0.0};
    int left = cur.n / RB - threadIdx.x / RB;
    for (int e = cur.n; e > 0; e -= kChunk, left -= kCols) {
      chunk_product<RB>(g, nullptr, left, a, sc);
      if (threadIdx.x == 0)  // one chunk late, as above
        while (g.put + 1 < g.got + kStages && put.bin < bd.nbin) {
          put_next();
          vec_next();
        }
    }
    const double s = panel_sum<RB>(dadd(a[0], a[1]), red);
    if (at >= 0) (up ? x : bd.by)[at] = s;
    red = sm + (red == sm ? 256 : 0);  // warps below may still read this one
    cur.next_panel(bd, stride, up, RB);
  }
  return true;
}

// Dot product of row `lane` of a warp's block panel (kRows rows a column).
template <int kRows>
__device__ __forceinline__ double warp_rows(const double* __restrict__ M, int K, const double* v) {
  double a[2] = {0.0, 0.0};
  for (int t = 0; t < K; t += 8) {
    double m[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) m[j] = t + j < K ? M[(t + j) * kRows] : 0.0;
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (t + j < K) a[j & 1] = fma(m[j], v[t + j], a[j & 1]);
  }
  return dadd(a[0], a[1]);
}

// y_F = X b_F, u = E b_F: 64 rows of a block of more than 32 rows per CTA, or
// eight smaller blocks, one per warp.  (A block's rows on several CTAs: one
// SM's FP64 rate would make a whole large block 20-40 us.)  X is lower
// triangular: a chunk of its rows ends at its diagonal.
template <bool kCg, class Wait, class WaitScalars>
__device__ __forceinline__ bool block_fwd(const DevBorder& bd, const double* b, const double* sc, Ring& g, int task, double* sm, DevScalars* S, Wait wait,
                                          WaitScalars wait_scalars) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool big = task < bd.nfp;
  const int blk = big ? bd.fp_blk[task] : bd.nbig + (task - bd.nfp) * 8 + warp;
  const bool have = blk < bd.nblk;
  const int c0 = have ? bd.blk_rp[blk] : 0, nt = have ? bd.blk_rp[blk + 1] - c0 : 0;
  const int N = have ? nt + bd.blk_rrp[blk + 1] - bd.blk_rrp[blk] : 0;
  const int r0 = big ? 64 * (task - bd.fp_first[blk]) : 0;
  const int i = big ? (int)threadIdx.x : lane;
  const int col = i < nt ? bd.blk_col[c0 + i] : 0;
  const Panel p{bd.ge + (have ? bd.ge_off[blk] + (int64_t)r0 * nt : 0), 64 * (r0 + 64 <= nt ? r0 + 64 : nt)};
  if (big) panel_start(g, p, S, true);
  else prefetch_bytes(p.M, (int64_t)64 * nt * 8, lane, 32);
  double w = 0.0;
  if (!wait_scalars() || !wait()) {
    if (big) ring_drain(g, S, true);
    return false;
  }
  if (i < nt) w = kCg ? rhs_value(load_parts(bd, bd.k + c0 + i), sc) : b[col];
  double* v = big ? sm + kRed : sm + warp * 32;
  if (i < nt) v[i] = w;
  if (big) __syncthreads();
  else __syncwarp();
  const double t = big ? panel_product<64>(g, p, v, sm, S, true) : warp_rows<64>(p.M + lane, nt, v);
  if ((!big || i < 64) && r0 + i < N) {
    if (r0 + i < nt) bd.y[c0 + r0 + i] = t;
    else bd.u[bd.u_off[blk] + r0 + i - nt] = t;
  }
  return true;
}

// x_F = X^T y_F - E^T x_S: the same for 32 columns of a block, whose own rows
// come last and from the last one on, so that a chunk ends at its diagonal.
// (64 columns in wide systems, where tasks of 32 are more than the GPU holds:
// the phase takes 9 us with 32 and 11.5 with 64 at 5,000 buses, 17.5 and 16 at
// 10,000.)
template <int kBackRows, class Wait>
__device__ __forceinline__ bool block_bwd(const DevPlan& d, const DevBorder& bd, Ring& g, int task, double* x, double* sm, Wait wait) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool big = task < bd.nbp;
  const int blk = big ? bd.bp_blk[task] : bd.nbig + (task - bd.nbp) * 8 + warp;
  const bool have = blk < bd.nblk;
  const int c0 = have ? bd.blk_rp[blk] : 0, nt = have ? bd.blk_rp[blk + 1] - c0 : 0;
  const int b0 = have ? bd.blk_rrp[blk] : 0, R = have ? bd.blk_rrp[blk + 1] - b0 : 0, N = nt + R;
  const int t0 = big ? kBackRows * (task - bd.bp_first[blk]) : 0;
  const int i = big ? (int)threadIdx.x : lane;
  const int brow = i < R ? bd.bcol[bd.blk_row[b0 + i]] : 0;
  const Panel p{bd.et + (have ? bd.et_off[blk] + (int64_t)t0 * N : 0), kBackRows * (N - t0)};
  if (big) panel_start(g, p, d.sc, true);
  else prefetch_bytes(p.M, (int64_t)kBackRows * N * 8, lane, 32);
  const int r = t0 + (big ? (int)threadIdx.x % kBackRows : lane);
  const int col = r < nt ? bd.blk_col[c0 + r] : 0;
  if (!wait()) {
    if (big) ring_drain(g, d.sc, true);
    return false;
  }
  double* v = big ? sm + kRed : sm + warp * 32;
  if (i < N) v[i] = i < R ? __ldcg(&x[brow]) : __ldcg(&bd.y[c0 + N - 1 - i]);
  if (big) __syncthreads();
  else __syncwarp();
  const double t = big ? panel_product<kBackRows>(g, p, v, sm, d.sc, true) : warp_rows<kBackRows>(p.M + lane, N, v);
  if ((!big || threadIdx.x < kBackRows) && r < nt) x[col] = t;
  return true;
}

// Task table of one launch: phases in order (0 products Jc^T of the CG's
// vectors, 1 blocks forward and the CG's vector update, 2 border right-hand
// side, 3 and 4 its products, 5 blocks back, 6 the product Jc x and the CG's
// scalars), the phase each one waits for, counters [head, ready, done, phase
// counts].
constexpr int kPhases = 7;
struct BorderTasks {
  int n[kPhases], off[kPhases + 1], dep[kPhases];
  int n_upd;  // CG: vector update tasks of phase 1
  int n_fwd;  // block tasks of phase 1
};
// each on a 128-byte line of its own: hundreds of CTAs poll them
constexpr int kCtlReady = 16, kCtlDone = 32, kCtlCount = 48, kCtlStep = 16, kCtlWords = 48 + kPhases * 16;
__device__ __forceinline__ count_t load_acquire(const count_t* p) {
  count_t v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

// thread 0: waits until *p >= need; false when the wait gave up (wait_ge in
// kernels.cuh: the same limit, flag and test hook) or, while it was not
// satisfied, the CG has stopped.  kLast: also when it was satisfied after the
// stop, which costs a second round trip.
template <bool kLast>
__device__ __forceinline__ bool border_wait(const count_t* p, count_t need, const count_t* done, const DevPlan& d) {
  need += d.dbg_unsatisfiable;
  if (need > 0) {
    volatile const int* flags = &d.sc->solve_flags;
    for (unsigned it = 0; load_acquire(p) < need; ++it) {
      if ((it & 7) == 7 && *(volatile const count_t*)done) return false;
      if (it > d.spin_limit || ((it & 15) == 15 && (*flags & 1))) {
        atomicOr(&d.sc->solve_flags, 1);
        return false;
      }
    }
  }
  return !kLast || !*(volatile const count_t*)done;  // set before the count that a stopped CG publishes
}

// red[8] = the CTA's sum of v over every kStep-th lane (thread 0 reads it)
template <int kStep>
__device__ __forceinline__ void cta_sum(double v, double* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o >= kStep; o >>= 1) v = dadd(v, __shfl_xor_sync(0xffffffffu, v, o));
  if (lane == 0) red[warp] = v;
  __syncthreads();
  if (warp == 0) {
    double t = lane < 8 ? red[lane] : 0.0;
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) t = dadd(t, __shfl_xor_sync(0xffffffffu, t, o));
    if (lane == 0) red[8] = t;
  }
}

// red[0], red[1] = the sums of the first n0 parts of r.r and n1 parts of w.r in
// a fixed order, one warp each
__device__ __forceinline__ void sum_parts(const double* rrp, const double* dlp, int n0, int n1, double* red) {
  if (threadIdx.x < 64) {
    const double* src = threadIdx.x < 32 ? rrp : dlp;
    const int lane = threadIdx.x & 31, n = threadIdx.x < 32 ? n0 : n1;
    double v = 0.0;
    for (int i = lane; i < n; i += 128) {
      double t[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) t[j] = i + 32 * j < n ? __ldcg(&src[i + 32 * j]) : 0.0;
      v = dadd(v, dadd(dadd(t[0], t[1]), dadd(t[2], t[3])));
    }
    v = warp_sum(v);
    if (lane == 0) red[threadIdx.x >> 5] = v;
  }
  __syncthreads();
}

// The CG's recurrence after iteration `it` with the sums r.r and w.r.  Every
// iteration waits for it, and a division is 20 dependent FP64 instructions, so
// the divisions by the previous iteration's gamma and alpha are products with
// reciprocals formed beside one another then.  Where
// gamma_0 is below 2^-700 the sums are taken times the power of four near its
// reciprocal (which changes no bit of alpha and beta): the reciprocal of a sum
// below 2^-1024, or the square of a threshold below 2^-537, would leave the
// range where a quotient and the root do not.  (The two products in every run
// took 0.3 us of an iteration.)
struct CgState {
  double inv_gam, inv_alpha;  // of the scaled gamma
};
struct CgScale {
  double q, stop2;  // the power of four, the scaled r.r that stops
  int on;           // q is not 1
};
__device__ __forceinline__ CgScale cg_scale(const DevPlan& d) {
  const DevScalars* S = d.sc;
  const double gam0 = S->gam0;
  const int e = (int)((unsigned long long)__double_as_longlong(gam0) >> 52) & 0x7ff;
  const int h = gam0 == 0.0 || e > 1023 - 700 ? 0 : (e - 1023) / 2;  // -511 <= h <= 0
  const double thr = (S->rtol_cur > 0.0 ? S->rtol_cur * sqrt(gam0) : d.cg_tol) * pow2_or_nan(-h);
  return CgScale{pow2_or_nan(-2 * h), thr * thr, h != 0};
}
// 0 go on, 1 converged, 2 iteration limit; sc = alpha, beta of the next iteration
__device__ __forceinline__ int cg_step(const DevPlan& d, CgState& st, const CgScale& cs, double rr, double wr, int it, double* sc) {
  if (cs.on) {
    rr *= cs.q;
    wr *= cs.q;
  }
  if (rr < cs.stop2 || rr == 0.0) return 1;
  if (it + 1 >= d.cg_itmax) return 2;
  const double beta = rr * st.inv_gam, den = fma(-(beta * rr), st.inv_alpha, wr), inv = 1.0 / rr;
  sc[0] = rr / den;
  sc[1] = beta;
  st.inv_gam = inv;
  st.inv_alpha = den * inv;
  return 0;
}
// bd.scal: the state for the iterations of each parity, the scale
__device__ __forceinline__ CgScale cg_scale(const DevPlan& d, const DevBorder& bd, int it) {
  if (it == 0) return cg_scale(d);
  const double q = __ldcg(&bd.scal[4]);
  return CgScale{q, __ldcg(&bd.scal[5]), q != 1.0};
}
__device__ __forceinline__ CgState cg_state(const DevPlan& d, const DevBorder& bd, const CgScale& cs, int it) {
  if (it == 0) return CgState{1.0 / (d.sc->gam * cs.q), 1.0 / d.sc->alpha};
  return CgState{__ldcg(&bd.scal[2 * (it & 1)]), __ldcg(&bd.scal[2 * (it & 1) + 1])};
}
// one thread: the step for good from the state `st`, the next state, and at the
// end what the loop leaves, through `ready`
__device__ void cg_scalars(const DevPlan& d, const DevBorder& bd, const CgScale& cs, CgState st, double rr, double wr, int it, int round, count_t* ready, count_t* done) {
  DevScalars* S = d.sc;
  double sc[2];
  const int stop = cg_step(d, st, cs, rr, wr, it, sc);
  if (!stop) {
    if (it == 0) {
      bd.scal[4] = cs.q;
      bd.scal[5] = cs.stop2;
    }
    bd.scal[2 * ((it + 1) & 1)] = st.inv_gam;
    bd.scal[2 * ((it + 1) & 1) + 1] = st.inv_alpha;
  } else {
    S->gam1 = rr;
    S->delta = wr;
    S->cg_err = sqrt(rr);
    S->it = it + 1;
    S->it_total += it + 1;
    S->cond_calls = it + 1;
    if (stop == 2) S->stop_main += 1;
    S->stop = stop;
    *(volatile count_t*)done = 1;
  }
  asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(ready), "l"((count_t)round) : "memory");
}

// Whether the CG has stopped, one answer for the whole CTA (thread 0's read).
// A CTA that starts late reads the flag while another one of the same launch
// sets it: warps that read it for themselves could leave one by one, and the
// ones that stay would run on barriers and shared variables that nobody set.
__device__ __forceinline__ bool stopped_before(const DevScalars* S) {
  return __syncthreads_or(threadIdx.x == 0 && *(volatile const int*)&S->stop) != 0;
}

template <bool kCg, int RB>
__global__ void __launch_bounds__(256, 3) k_border_solve(DevPlan d, DevBorder bd, const __grid_constant__ BorderTasks tk, const double* b, double* x, int use_stop) {
  extern __shared__ __align__(128) double sm[];  // destination of bulk copies
  __shared__ double red[2 * 32];
  __shared__ int s_it, s_t, go[2], last;
  // the CG's scalars as this CTA has them: alpha and beta of iteration sc_it,
  // the recurrence's state for iteration st_it, its scale
  __shared__ double sc2[2];
  __shared__ CgScale s_scale, last_scale;
  __shared__ CgState st2, last_st;
  __shared__ int sc_it, st_it;
  if ((kCg || use_stop) && stopped_before(d.sc)) return;
  count_t* head = bd.ctl;
  count_t* ready = bd.ctl + kCtlReady;
  count_t* done = bd.ctl + kCtlDone;
  count_t* cnt = bd.ctl + kCtlCount;
  DevScalars* S = d.sc;
  const int T = tk.off[kPhases];
  __shared__ __align__(8) uint64_t bars[2 * kStages];
  Ring ring = ring_init(bars, sm + kRed + kMaxVec, kChunk + kChunkVec, 2);
  // thread 0: the first task of iteration s_it, waits known to be over (8 per
  // iteration)
  count_t base = 0, seen = 0;
  if (threadIdx.x == 0) {
    s_it = sc_it = 0;
    st_it = -1;
    sc2[0] = S->alpha;
    sc2[1] = S->beta;
  }
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) {
      const count_t next = atomicAdd(head, count_t(1));
      for (; next - base >= (count_t)T; base += T) ++s_it;
      s_t = (int)(next - base);
    }
    __syncthreads();
    const int it = s_it, t = s_t;
    if (!kCg && it > 0) return;
    trace_mark(d, t, 0);
    trace_mark(d, t, 3);
    int ph = 0;
    while (t >= tk.off[ph + 1]) ++ph;
    const int task = t - tk.off[ph];
    double* rin = it & 1 ? bd.r2 : d.cg_r;
    double* rout = it & 1 ? d.cg_r : bd.r2;
    double* sin = it & 1 ? bd.s2 : d.cg_s;
    double* sout = it & 1 ? d.cg_s : bd.s2;
    // a wait that ran out ends the CG for all CTAs
    auto gave_up = [&]() {
      if (kCg && (*(volatile int*)&S->solve_flags & 1)) {
        *(volatile int*)&S->stop = 3;
        *(volatile count_t*)done = 1;
      }
    };
    // the CTA waits for a count.  (After the CG's end only the products Jc^T of
    // the next iteration, which nobody reads, find theirs complete: what follows
    // them computes the stop itself, and what follows that waits in vain until
    // it sees the end.  So a wait costs one round trip, not two.)
    auto wait_for = [&](const count_t* p, count_t need, int mark, int* g) {
      if (threadIdx.x == 0) {
        const count_t m = (count_t)it * 8 + mark;
        *g = m < seen || border_wait<false>(p, need, done, d);
        if (m >= seen) seen = m + 1;
        if (!*g) gave_up();
      }
      __syncthreads();
      trace_mark(d, t, 1);
      return *g != 0;
    };
    // the products Jc^T follow the previous iteration's constraint tasks
    auto wait_phase = [&]() { return wait_for(&cnt[tk.dep[ph] * kCtlStep], (count_t)(ph ? it + 1 : it) * tk.n[tk.dep[ph]], ph, &go[0]); };
    // the iteration's alpha and beta in sc2, which every CTA computes itself
    // from the constraint tasks' sums (one CTA's step and a second wait for it
    // took 7.5 us an iteration, this 4.5); false at the loop's end.  Another
    // thread waits meanwhile for the scalars that the CTA of the last
    // constraint task left two iterations ago, which is nearly always over:
    // that CTA sums the parts after its task counts as done, and this
    // iteration's tasks write the buffers it read.  A CTA without a state of its
    // own takes that one.
    auto wait_scalars = [&]() {
      if (!kCg || sc_it == it) return true;
      if (threadIdx.x == 32) {
        go[0] = border_wait<false>(ready, (count_t)it - 1, done, d);
        if (!go[0]) {
          gave_up();
        } else if (st_it != it) {
          s_scale = cg_scale(d, bd, it - 1);
          st2 = cg_state(d, bd, s_scale, it - 1);
        }
      }
      if (!wait_for(&cnt[6 * kCtlStep], (count_t)it * tk.n[6], 0, &go[1]) || !go[0]) return false;
      sum_parts(bd.rrp + ((it - 1) & 1) * tk.n_upd, bd.dlp + ((it - 1) & 1) * tk.n[6], tk.n_upd, tk.n[6], red);
      if (threadIdx.x == 0) {
        CgState st = st2;
        go[1] = !cg_step(d, st, s_scale, red[0], red[1], it - 1, sc2);
        st2 = st;
        st_it = it + 1;
        sc_it = it;
      }
      __syncthreads();
      return go[1] != 0;
    };
    bool scalars = false;
    if (ph == 0) {
      if (!rhs_parts_task(d, bd, task, rin, sin, wait_phase)) return;
    } else if (ph == 1 && task < tk.n_fwd) {
      if (!block_fwd<kCg>(bd, b, sc2, ring, task, sm, S, wait_phase, wait_scalars)) return;
    } else if (ph == 1 && task < tk.n_fwd + tk.n_upd) {
      // p = r + beta p; s = w + beta s; x += alpha p; r -= alpha s; r.r
      const int c = task - tk.n_fwd, k = c * kCgRows + threadIdx.x;
      if (!wait_scalars()) return;
      double part[1] = {0.0};
      if (k < d.m_c) {
        const double r = __ldcg(&rin[k]), s0 = __ldcg(&sin[k]), w = __ldcg(&d.cg_w[k]), p0 = __ldcg(&d.cg_p[k]), x0 = __ldcg(&d.cg_x[k]);
        const double alpha = sc2[0], beta = sc2[1];
        const double sv = fma(beta, s0, w), p = fma(beta, p0, r), rn = fma(-alpha, sv, r);
        d.cg_p[k] = p;
        sout[k] = sv;
        d.cg_x[k] = fma(alpha, p, x0);
        rout[k] = rn;
        part[0] = rn * rn;
      }
      cta_sum<1>(part[0], red);
      if (threadIdx.x == 0) bd.rrp[(it & 1) * tk.n_upd + c] = red[8];
    } else if (ph <= 2) {
      // bt = b_S - sum u (in phase 1 there are no blocks)
      const int j = (ph == 2 ? task : task - tk.n_fwd - tk.n_upd) * kRowTask + (threadIdx.x >> 2), sub = threadIdx.x & 3;
      const int col = j < bd.k ? bd.bcol[j] : 0;
      if (!wait_scalars() || !wait_phase()) return;
      double v = 0.0;
      if (j < bd.k && sub == 0) v = kCg ? rhs_value(load_parts(bd, j), sc2) : b[col];
      if (ph == 2 && j < bd.k) v = dsub(v, border_updates(bd, j, sub));
      v = join_row(v);
      if (j < bd.k && sub == 0) bd.bt[j] = v;
    } else if (ph <= 4) {
      if (!bin_task<RB>(bd, ring, task, tk.n[ph], ph == 4, x, sm, S, wait_phase)) return;
    } else if (ph == 5) {
      if (!block_bwd<back_rows(RB)>(d, bd, ring, task, x, sm, wait_phase)) return;
    } else {
      // w = Jc_p x, delta = w.r
      const int k = task * kRowTask + (threadIdx.x >> 2), sub = threadIdx.x & 3;
      SparseRow row;
      row.p = row.e = 0;
      row.L = 4;
      auto vi = [](int p) { return p; };
      if (k < d.m_c) load_row(row, d.jc_rp[k], d.jc_rp[k + 1], 4, sub, d.jcp_ci, d.jc_s, vi);
      if (!wait_phase()) return;
      double part[1] = {0.0};
      const double r = k < d.m_c ? __ldcg(&rout[k]) : 0.0;
      const double acc = join_row(row_dot(row, d.jcp_ci, d.jc_s, vi, [&](int c) { return __ldcg(&x[c]); }));
      if (k < d.m_c && sub == 0) {
        d.cg_w[k] = acc;
        part[0] = acc * r;
      }
      cta_sum<4>(part[0], red);
      if (threadIdx.x == 0) bd.dlp[(it & 1) * tk.n[6] + task] = red[8];
      scalars = true;
    }
    // done: the CTA's writes, then the count
    __syncthreads();
    trace_mark(d, t, 2);
    if (!scalars) {
      if (threadIdx.x == 0)
        asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(&cnt[ph * kCtlStep]), "l"(count_t(1)) : "memory");
      continue;
    }
    if (threadIdx.x == 0) {
      count_t old;
      asm volatile("atom.acq_rel.gpu.global.add.u64 %0, [%1], 1;" : "=l"(old) : "l"(&cnt[ph * kCtlStep]) : "memory");
      last = old == (count_t)(it + 1) * tk.n[6] - 1;
    }
    __syncthreads();
    if (!last) continue;
    // the last constraint task: the step for good (k_spmv_jcp, k_cg_update).  A
    // thread beside the sums' fetches the state that it starts from, once the
    // previous iteration's step has left it.
    if (threadIdx.x == 64) {
      go[1] = border_wait<false>(ready, (count_t)it, done, d);
      if (go[1]) {
        last_scale = cg_scale(d, bd, it);
        last_st = cg_state(d, bd, last_scale, it);
      } else {
        gave_up();
      }
    }
    sum_parts(bd.rrp + (it & 1) * tk.n_upd, bd.dlp + (it & 1) * tk.n[6], tk.n_upd, tk.n[6], red);
    if (threadIdx.x == 0 && go[1]) cg_scalars(d, bd, last_scale, last_st, red[0], red[1], it, it + 1, ready, done);
  }
}

// ---------------------------------------------------------------------------
// Schur plans: a small system's S = Jc Hgamma^-1 Jc^T itself, so that a CG
// iteration is one product and one exchange of scalars instead of four
// dependent phases.  (S comes out of the border's sweep as V^T V with
// V = L^-1 Jc^T, which keeps the accuracy of the two triangular products.)
// ---------------------------------------------------------------------------
__host__ __device__ inline int64_t schur_panel(int64_t b, int rows, int mc) { return b * rows * mc; }

// S in row panels of bd.srb rows, column after column, from the lower triangle
// of -S; one CTA per 64 x 64 tile.
__global__ void __launch_bounds__(256) k_schur_pack(DevBorder bd) {
  __shared__ double tile[64][65];
  int ti = (int)((sqrtf(1.0f + 8.0f * (float)blockIdx.x) - 1.0f) * 0.5f);
  while (ti * (ti + 1) / 2 > (int)blockIdx.x) --ti;
  while ((ti + 1) * (ti + 2) / 2 <= (int)blockIdx.x) ++ti;
  const int tj = blockIdx.x - ti * (ti + 1) / 2;
  const int i0 = ti * 64, j0 = tj * 64, at = bd.npan * kBorderPanel, mc = bd.mc, rows = bd.srb;
  for (int e = threadIdx.x; e < 64 * 64; e += 256) {
    const int i = e & 63, j = e >> 6;
    if (i0 + i < mc && i0 + i >= j0 + j) {
      const double v = -bd.W[(int64_t)(at + j0 + j) * bd.ld + at + i0 + i];
      tile[j][i] = v;
      if (ti == tj) tile[i][j] = v;
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < 64 * 64; e += 256) {
    const int i = i0 + e % 64, j = j0 + e / 64;
    if (i >= mc || j >= mc) continue;
    bd.S[schur_panel(i / rows, rows, mc) + (int64_t)j * rows + i % rows] = tile[j - j0][i - i0];
  }
  if (ti == tj) return;
  for (int e = threadIdx.x; e < 64 * 64; e += 256) {
    const int j = j0 + e % 64, i = i0 + e / 64;
    if (i >= mc || j >= mc) continue;
    bd.S[schur_panel(j / rows, rows, mc) + (int64_t)i * rows + j % rows] = tile[j - j0][i - i0];
  }
}

// The whole CG run: round 0 takes r = b - S x0, round 1 w = S r, the others one
// iteration each.  A task owns RB rows: it forms the updated residual of all
// rows for its product (two multiply-adds each, cheaper than a phase of its
// own), updates its own rows of the vectors, and leaves its part of w.r and
// r.r.  Vectors that other tasks read are double-buffered.
template <int RB>
__global__ void __launch_bounds__(256, 3) k_schur_cg(DevPlan d, DevBorder bd, int tasks) {
  extern __shared__ __align__(128) double sm[];  // destination of bulk copies
  __shared__ double red[2];
  __shared__ double sc2[2];  // as in k_border_solve
  __shared__ CgScale s_scale, last_scale;
  __shared__ CgState st2, last_st;
  __shared__ int s_it, s_t, st_it, go[2], last;
  __shared__ __align__(8) uint64_t bars[2 * kStages];
  DevScalars* S = d.sc;
  if (stopped_before(S)) return;
  Ring ring = ring_init(bars, sm + kRed + kSchurMax, kChunk, 1);
  count_t *head = bd.ctl, *ready = bd.ctl + kCtlReady, *done = bd.ctl + kCtlDone, *cnt = bd.ctl + kCtlCount;
  if (threadIdx.x == 0) s_it = st_it = 0;
  const int mc = bd.mc;
  count_t base = 0;
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) {
      const count_t next = atomicAdd(head, count_t(1));
      for (; next - base >= (count_t)tasks; base += tasks) ++s_it;
      s_t = (int)(next - base);
    }
    __syncthreads();
    const int q = s_it, task = s_t, row = task * RB + threadIdx.x;
    const bool own = threadIdx.x < RB && row < mc;
    const Panel p{bd.S + schur_panel(task, RB, mc), RB * mc};
    panel_start(ring, p, S, false);
    double* const rin = q & 1 ? bd.r2 : d.cg_r;
    double* const rout = q & 1 ? d.cg_r : bd.r2;
    double* const sin = q & 1 ? bd.s2 : d.cg_s;
    double* const sout = q & 1 ? d.cg_s : bd.s2;
    double* const win = q & 1 ? bd.w2 : d.cg_w;
    double* const wout = q & 1 ? d.cg_w : bd.w2;
    // rounds 1 and 2 follow the last task's scalars, the later ones the tasks of
    // the round before: every CTA computes their scalars itself, with the last
    // task's state from two rounds before where it has none of its own.  Another
    // thread waits meanwhile for those scalars, which is nearly always over: the
    // last task's CTA sums the parts after its task counts as done, and this
    // round's tasks write the buffers it read.
    auto gave_up = [&]() {  // a wait that ran out ends the CG for all CTAs
      if (*(volatile int*)&S->solve_flags & 1) {
        *(volatile int*)&S->stop = 3;
        *(volatile count_t*)done = 1;
      }
    };
    const bool own_step = q >= 3 && st_it <= q;  // not its second task of the round
    if (threadIdx.x == 0) {
      go[0] = q < 3 ? border_wait<true>(ready, (count_t)q, done, d) : !own_step || border_wait<false>(cnt, (count_t)q * tasks, done, d);
      if (!go[0]) gave_up();
      if (q < 3) {
        sc2[0] = *(volatile double*)&S->alpha;
        sc2[1] = *(volatile double*)&S->beta;
      }
    } else if (threadIdx.x == 32) {
      go[1] = !own_step || border_wait<false>(ready, (count_t)q - 1, done, d);
      if (!go[1]) {
        gave_up();
      } else if (own_step && st_it != q) {
        s_scale = cg_scale(d, bd, q - 3);
        st2 = cg_state(d, bd, s_scale, q - 3);
      }
    }
    __syncthreads();
    bool on = go[0] && go[1];
    if (on && own_step) {
      const int old = ((q - 1) & 1) * tasks;
      sum_parts(bd.rrp + old, bd.dlp + old, tasks, tasks, red);
      if (threadIdx.x == 0) {
        CgState st = st2;
        go[0] = !cg_step(d, st, s_scale, red[0], red[1], q - 3, sc2);
        st2 = st;
        st_it = q + 1;
      }
      __syncthreads();
      on = go[0] != 0;
    }
    if (!on) {
      ring_drain(ring, S, false);
      return;
    }
    const double alpha = sc2[0], beta = sc2[1];
    double* v = sm + kRed;
    for (int h = threadIdx.x; h < mc; h += 4 * 256) {
      double r[4], w[4], s[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int k = h + j * 256;
        const bool in = k < mc;
        r[j] = in ? (q ? __ldcg(&rin[k]) : __ldcg(&d.cg_x[k])) : 0.0;
        w[j] = in && q > 1 ? __ldcg(&win[k]) : 0.0;
        s[j] = in && q > 1 ? __ldcg(&sin[k]) : 0.0;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (h + j * 256 < mc) v[h + j * 256] = q > 1 ? fma(-alpha, fma(beta, s[j], w[j]), r[j]) : r[j];
    }
    const double r0 = own ? __ldcg(&rin[row]) : 0.0, p0 = own ? __ldcg(&d.cg_p[row]) : 0.0, x0 = own ? __ldcg(&d.cg_x[row]) : 0.0;
    double sv = 0.0;
    if (own && q > 1) sv = fma(beta, __ldcg(&sin[row]), __ldcg(&win[row]));
    __syncthreads();
    const double t = panel_product<RB>(ring, p, sm + kRed, sm, S, false);
    double rr = 0.0, wr = 0.0;
    if (own) {
      double rn = r0;
      if (q == 0) {
        rn = dsub(r0, t);
      } else {
        wout[row] = t;
        if (q > 1) {
          rn = v[row];
          const double pn = fma(beta, p0, r0);
          d.cg_p[row] = pn;
          d.cg_x[row] = fma(alpha, pn, x0);
          sout[row] = sv;
        }
      }
      rout[row] = rn;
      rr = rn * rn;
      wr = t * rn;
    }
    if (threadIdx.x < 32) {
#pragma unroll
      for (int o = RB / 2; o > 0; o >>= 1) {
        rr = dadd(rr, __shfl_xor_sync(0xffffffffu, rr, o));
        wr = dadd(wr, __shfl_xor_sync(0xffffffffu, wr, o));
      }
      if (threadIdx.x == 0) {
        bd.rrp[(q & 1) * tasks + task] = rr;
        bd.dlp[(q & 1) * tasks + task] = wr;
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      count_t old;
      asm volatile("atom.acq_rel.gpu.global.add.u64 %0, [%1], 1;" : "=l"(old) : "l"(cnt) : "memory");
      last = old == (count_t)(q + 1) * tasks - 1;
    }
    __syncthreads();
    if (!last) continue;
    if (q > 1 && threadIdx.x == 64) {  // as in k_border_solve
      go[1] = border_wait<false>(ready, (count_t)q, done, d);
      if (go[1]) {
        last_scale = cg_scale(d, bd, q - 2);
        last_st = cg_state(d, bd, last_scale, q - 2);
      } else {
        gave_up();
      }
    }
    sum_parts(bd.rrp + (q & 1) * tasks, bd.dlp + (q & 1) * tasks, tasks, tasks, red);
    if (threadIdx.x == 0) {
      if (q > 1) {
        if (go[1]) cg_scalars(d, bd, last_scale, last_st, red[0], red[1], q - 2, q + 1, ready, done);
      } else {
        if (q == 0) {
          S->gam = S->gam0 = red[0];
        } else {
          S->delta = red[1];
          S->alpha = S->gam / red[1];
          S->beta = 0.0;
        }
        asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(ready), "l"((count_t)(q + 1)) : "memory");
      }
    }
  }
}

}  // namespace hykkt
