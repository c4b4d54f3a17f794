// Diffusion tensor and its Cholesky factor (FP64 parity path).
//
//   rpy_assemble   Diffusion_Tensor (func.cpp:728-804): lower triangle of
//                  the 3N x 3N RPY tensor, column-major with leading dim
//                  lda, written once (the reference writes the full matrix
//                  twice, func_cuda.cu:500-559).
//   potrf_fp64     blocked right-looking Cholesky, in place, lower: a
//                  one-CTA diagonal factor, a row-parallel triangular
//                  solve of the panel and a register-tiled FP64 SYRK/GEMM
//                  trailing update.  A negative pivot is replaced by its
//                  absolute value and counted (func.cpp:827-833).
//   trmv_lower     rd = s2dt * L p (rd_cal, func_cuda.cu:634-647), split
//                  over column chunks with a fixed-order final sum.
#include <cuda_runtime.h>

#include <algorithm>

#include "bd_internal.h"
#include "dev_physics.cuh"

using namespace bdp;

namespace {

inline int cdiv(int a, int b) { return (a + b - 1) / b; }

// tile (bi, bj <= bi) of a triangle from its row-major index t (a grid without
// the triangle's empty half: the SMs' shares of the tiles are then even)
__device__ __forceinline__ void tri_tile(int t, int& bi, int& bj) {
  bi = (int)((sqrtf(8.f * (float)t + 1.f) - 1.f) * 0.5f);
  while ((bi + 1) * (bi + 2) / 2 <= t) bi++;
  while (bi * (bi + 1) / 2 > t) bi--;
  bj = t - bi * (bi + 1) / 2;
}

// ------------------------------------------------------------ RPY
constexpr int kRpyTile = 32;

__global__ void __launch_bounds__(256) k_rpy(int nD, const double* __restrict__ r, const double* __restrict__ rad,
                                             double a1, double a2, double* __restrict__ A, int lda) {
  int bi, bj;
  tri_tile(blockIdx.x, bi, bj);
  int i = bi * kRpyTile + threadIdx.x;
  if (i >= nD) return;
  V3 ri = ld3(r + 3 * i);
  double radi = rad[i];
  for (int jj = threadIdx.y; jj < kRpyTile; jj += blockDim.y) {
    int j = bj * kRpyTile + jj;
    if (j >= nD || j > i) continue;
    if (j == i) {
      for (int l = 0; l < 3; l++)
        for (int k = l; k < 3; k++) A[(size_t)(3 * j + l) * lda + 3 * i + k] = (k == l) ? a1 / radi : 0.0;
      continue;
    }
    V3 rj = ld3(r + 3 * j);
    V3 sij{ri.x - rj.x, ri.y - rj.y, ri.z - rj.z};
    double s = sqrt(sij.x * sij.x + sij.y * sij.y + sij.z * sij.z);
    double radj = rad[j];
    double Db[3][3];
    rpy_block(sij, s, radi, radj, a1, a2, Db);
    for (int l = 0; l < 3; l++) {
      double* col = A + (size_t)(3 * j + l) * lda + 3 * i;
      for (int k = 0; k < 3; k++) col[k] = Db[k][l];
    }
  }
}

// Mixed path: the same lower triangle from the FP32 form of the RPY block
// (separations formed in FP64, then FP32), stored as the double-float pair
// (value, 0).  No FP64 arithmetic beyond the separation.
// Mixed path: FP32 blocks from the double-float positions (hi differences
// plus lo differences; radius in qh.w), no FP64 per pair; stored as (D, 0)
// pairs.  The same separations and block formula as the mixed drift.
__global__ void __launch_bounds__(256) k_rpy_mx(int nD, const float4* __restrict__ qh, const float4* __restrict__ ql,
                                                float a1f, float a2f, float2* __restrict__ A, int lda) {
  int bi = blockIdx.y, bj = blockIdx.x;
  if (bj > bi) return;
  int i = bi * kRpyTile + threadIdx.x;
  if (i >= nD) return;
  const float4 hi = qh[i], lo = ql[i];
  for (int jj = threadIdx.y; jj < kRpyTile; jj += blockDim.y) {
    int j = bj * kRpyTile + jj;
    if (j >= nD || j > i) continue;
    if (j == i) {
      for (int l = 0; l < 3; l++)
        for (int k = l; k < 3; k++)
          A[(size_t)(3 * j + l) * lda + 3 * i + k] = make_float2((k == l) ? a1f / hi.w : 0.f, 0.f);
      continue;
    }
    const float4 hj = qh[j], lj = ql[j];
    float Db[3][3];
    rpy_block_f((hi.x - hj.x) + (lo.x - lj.x), (hi.y - hj.y) + (lo.y - lj.y), (hi.z - hj.z) + (lo.z - lj.z), hi.w, hj.w,
                a1f, a2f, Db);
    for (int l = 0; l < 3; l++) {
      float2* col = A + (size_t)(3 * j + l) * lda + 3 * i;
      for (int k = 0; k < 3; k++) col[k] = make_float2(Db[k][l], 0.f);
    }
  }
}

// ------------------------------------------------------------ Cholesky
// Blocks of 64 columns, factored as two panels of kNB = 32: the FP64 pipe (two
// lanes a clock per SM) makes a diagonal block of 64 on one SM and row solves
// of 64 columns on a few SMs the serial part of a small factorisation.
constexpr int kNB = 32;

// A pivot's step: f > 0 and a column entry to a / sqrt(f), from FP32's reciprocal
// root y by one third-order step, e = 1 - f y^2: a y (1 + e / 2 + 3 e^2 / 8) (22
// bits to 2 ulp in six FP64 operations, four of them in a row, instead of a root
// and a division; the seed goes to FP32 and back as bits, off the FP64 pipe).
__device__ __forceinline__ double over_sqrt(double a, double f) {
  const int hi = __double2hiint(f);
  const unsigned e = (unsigned)hi >> 20;  // sign and exponent
  if (e < 1023 - 100 || e > 1023 + 100) return a * (1.0 / sqrt(f));
  constexpr int kBias = (1023 - 127) << 20;
  const int y32 = __float_as_int(
      rsqrtf(__int_as_float(((hi - kBias) << 3) | ((unsigned)__double2loint(f) >> 29))));
  const double y = __hiloint2double((y32 >> 3) + kBias, y32 << 29);
  const double d = fma(-f * y, y, 1.0), ay = a * y;
  return fma(ay * d, fma(0.375, d, 0.5), ay);
}

// Factor the kb x kb diagonal block at (k0, k0): right-looking, a row per lane,
// column j in the registers of warp j % 4 (one warp per FP64 pipe: a warp's
// FP64 operation holds its pipe for 64 cycles), column c to the others through
// shared memory.  The warp of column c + 1 takes column c off it alone, scales
// and publishes it, and makes up for its other columns in the next turn.  A
// negative pivot is replaced by its absolute value and counted
// (func.cpp:827-833).  Bound by the pivots' chain (six dependent FP64 operations
// and a barrier each): 64 columns by 256 threads with three barriers a column
// took 119 us, 32 by one warp 69, by four 25 without that order, 24 with it (with
// the rows' split below, 3N = 912: 5.1 -> 1.5 ms in all, 1,944: 13.3 -> 4.8).
__global__ void __launch_bounds__(128) k_potrf_diag(double* A, int lda, int k0, int kb, int* negpiv) {
  __shared__ double T[kNB][kNB];  // T[c][j] = L_jc (below the diagonal)
  __shared__ double piv[kNB];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double* col = A + (size_t)k0 * lda + k0 + lane;
  double a[kNB / 4];
#pragma unroll
  for (int i = 0; i < kNB / 4; i++) {
    const int j = 4 * i + w;
    a[i] = (lane < kb && j <= lane) ? col[(size_t)j * lda] : (j == lane ? 1.0 : 0.0);
  }
  auto pivot = [&](double& ac, int c) {  // column c, updated by all before it
    double f = __shfl_sync(0xffffffffu, ac, c);
    if (__double2hiint(f) < 0 && f < 0) {
      f = -f;
      if (lane == 0) atomicAdd(negpiv, 1);
    }
    T[c][lane] = ac = over_sqrt(ac, f);
    if (lane == c) piv[c] = f;
  };
  if (w == 0) pivot(a[0], 0);
  __syncthreads();
#pragma unroll
  for (int c = 0; c < kNB - 1; c++) {
    const double l = T[c][lane];
    if (w == ((c + 1) & 3)) {
      a[(c + 1) >> 2] = fma(-l, T[c][c + 1], a[(c + 1) >> 2]);
      pivot(a[(c + 1) >> 2], c + 1);
    } else {
      if (c > 0 && w == (c & 3)) {  // the columns left behind at c - 1
        const double lp = T[c - 1][lane];
#pragma unroll
        for (int i = (c >> 2) + 1; i < kNB / 4; i++) a[i] = fma(-lp, T[c - 1][4 * i + w], a[i]);
      }
#pragma unroll
      for (int i = c >> 2; i < kNB / 4; i++)
        if (4 * i + w > c) a[i] = fma(-l, T[c][4 * i + w], a[i]);  // (rows above the diagonal: not used)
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < kNB / 4; i++) {
    const int j = 4 * i + w;
    if (lane < kb && j < lane) col[(size_t)j * lda] = a[i];
  }
  if (w == 0 && lane < kb) col[(size_t)lane * lda] = sqrt(piv[lane]);
}

// Panel solve: rows [k0+kb, m) of columns [k0, k0+kb): X L_kk^T = A,
// right-looking in registers, the columns unscaled until the end (row c of L
// carries 1 / L_cc).  A warp takes 4 rows, lane 4 g + r the columns 8 i + g of
// row r: eight times as many warps as with a row per lane, so that the rows of
// a small matrix reach all FP64 pipes.  64 columns left-looking with a row per
// thread: 188 us at 3N = 1,944; 32 columns with a row per lane 24 us, four
// lanes a row 16; now 11.5.
constexpr int kTrsmRows = 16;  // per CTA of four warps

__global__ void __launch_bounds__(128) k_trsm_panel(double* A, int lda, int m, int k0, int kb) {
  __shared__ double L[kNB][kNB];  // L[c][j] = L_jc / L_cc, j > c; else 0
  __shared__ double rd[kNB];
  const int lane = threadIdx.x & 31, g = lane >> 2;
  const int r = k0 + kb + blockIdx.x * kTrsmRows + (threadIdx.x >> 5) * 4 + (lane & 3);
  double* col = A + (size_t)k0 * lda + r;
  double x[kNB / 8];
#pragma unroll
  for (int i = 0; i < kNB / 8; i++) x[i] = (r < m && 8 * i + g < kb) ? col[(size_t)(8 * i + g) * lda] : 0.0;
  double v[kNB / 4];
#pragma unroll
  for (int q = 0; q < kNB / 4; q++) {  // warp w: columns w, w + 4, ...; lane: row
    const int c = (threadIdx.x >> 5) + 4 * q;
    v[q] = (lane < kb && c <= lane) ? A[(size_t)(k0 + c) * lda + k0 + lane] : 0.0;
    if (lane == c) rd[c] = lane < kb ? 1.0 / v[q] : 0.0;
  }
  __syncwarp();
#pragma unroll
  for (int q = 0; q < kNB / 4; q++) {
    const int c = (threadIdx.x >> 5) + 4 * q;
    L[c][lane] = c < lane ? v[q] * rd[c] : 0.0;
  }
  __syncthreads();
#pragma unroll
  for (int c = 0; c < kNB - 1; c++) {
    const double xc = __shfl_sync(0xffffffffu, x[c >> 3], (lane & 3) + 4 * (c & 7));
#pragma unroll
    for (int i = c >> 3; i < kNB / 8; i++) x[i] = fma(-xc, L[c][8 * i + g], x[i]);
  }
  if (r < m)
#pragma unroll
    for (int i = 0; i < kNB / 8; i++)
      if (8 * i + g < kb) col[(size_t)(8 * i + g) * lda] = x[i] * rd[8 * i + g];
}

// Update of the lower triangle of A[t0:, t0:jend] by the kb columns from k0:
// A_ij -= P_i P_j^T with P = A[:, k0:k0+kb].  TM x TN output tile per CTA (a
// triangle of square ones, or one column of them), each thread an MR x NR
// register block, at least four warps: one per FP64 pipe of the SM, which
// bounds it.
constexpr int kKC = 16;  // panel columns staged per pass

template <int TM, int TN, int MR, int NR>
__global__ void __launch_bounds__(TM * TN / (MR * NR)) k_syrk_update(double* A, int lda, int m, int k0, int kb, int t0, int jend) {
  constexpr int NT = TM * TN / (MR * NR);
  int bi = blockIdx.x, bj = 0;  // TM != TN: one column of tiles
  if (TM == TN) tri_tile(blockIdx.x, bi, bj);
  const int row0 = t0 + bi * TM, col0 = t0 + bj * TN;
  __shared__ double Pr[kKC][TM + 1];  // [k][row]
  __shared__ double Pc[kKC][TN + 1];  // [k][col]
  const int tid = threadIdx.x;
  const int tr = (tid % (TM / MR)) * MR, tc = (tid / (TM / MR)) * NR;
  double acc[MR][NR];
#pragma unroll
  for (int a = 0; a < MR; a++)
#pragma unroll
    for (int b = 0; b < NR; b++) acc[a][b] = 0.0;
  for (int kc = 0; kc < kb; kc += kKC) {
    const int kn = kb - kc < kKC ? kb - kc : kKC;
    for (int e = tid; e < kKC * TM; e += NT) {
      const int k = e / TM, q = e - k * TM;
      Pr[k][q] = (k < kn && row0 + q < m) ? A[(size_t)(k0 + kc + k) * lda + row0 + q] : 0.0;
    }
    for (int e = tid; e < kKC * TN; e += NT) {
      const int k = e / TN, q = e - k * TN;
      Pc[k][q] = (k < kn && col0 + q < jend) ? A[(size_t)(k0 + kc + k) * lda + col0 + q] : 0.0;
    }
    __syncthreads();
#pragma unroll 4
    for (int k = 0; k < kKC; k++) {
      double a4[MR], b4[NR];
#pragma unroll
      for (int q = 0; q < MR; q++) a4[q] = Pr[k][tr + q];
#pragma unroll
      for (int q = 0; q < NR; q++) b4[q] = Pc[k][tc + q];
#pragma unroll
      for (int a = 0; a < MR; a++)
#pragma unroll
        for (int b = 0; b < NR; b++) acc[a][b] = fma(a4[a], b4[b], acc[a][b]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int b = 0; b < NR; b++) {
    const int cc = col0 + tc + b;
    if (cc >= jend) continue;
#pragma unroll
    for (int a = 0; a < MR; a++) {
      const int rr = row0 + tr + a;
      if (rr < m && rr >= cc) {
        double* p = A + (size_t)cc * lda + rr;
        *p = *p - acc[a][b];
      }
    }
  }
}

// ------------------------------------------------------------ L p
constexpr int kRdRows = 256;
// Columns a CTA sums: short runs at small sizes, where 512 left a few CTAs of one
// serial chain each, long ones at large ones, whose partial sums (m^2 / chunk
// values, written and read again) take memory: 34 MB at 3N = 46,200 with 512, 133 with
// 128.  32, 128, 512 columns, mixed / FP64, us: 3N = 972 16/21, 22/39, 39/123; 1,944 21/41,
// 23/39, 58/123; 3,888 31/76, 33/99, 74/127; 8,100 91/240, 64/248, 100/442; past the
// line, 8,262 93/246, 65/247, 102/363 and 10,368 127/364, 102/360, 111/477: there 128 would
// still be the faster, at 4 times the memory.
constexpr int kRdChunkMax = 512;
int rd_chunk(int m) { return m <= 2048 ? 32 : m <= 8192 ? 128 : kRdChunkMax; }

__global__ void __launch_bounds__(kRdRows) k_trmv_part(int m, const double* __restrict__ A, int lda,
                                                       const double* __restrict__ p, double s2dt, int chunk,
                                                       double* __restrict__ part) {
  int i = blockIdx.x * kRdRows + threadIdx.x;
  int kc = blockIdx.y;
  int k0 = kc * chunk, k1 = min(k0 + chunk, m);
  double s = 0.0;
  if (i < m) {
    int kend = min(k1, i + 1);
#pragma unroll 8
    for (int k = k0; k < kend; k++) s = s + (s2dt * A[(size_t)k * lda + i]) * p[k];
  }
  if (i < m) part[(size_t)kc * m + i] = s;
}

// The same over the double-float factor of the mixed path, in FP32
// arithmetic: each product L_ik p_k is formed exactly as x + ex (p split into
// FP32 hi + lo once per CTA, FMA for the rounding error of L_ik p_hi) and
// summed with a two-sum into (s, c); ~40 significant bits per partial sum.
__global__ void __launch_bounds__(kRdRows) k_trmv_part_df(int m, const float2* __restrict__ A, int lda,
                                                          const double* __restrict__ p, double s2dt, int chunk,
                                                          double* __restrict__ part) {
  __shared__ float2 ps[kRdChunkMax];
  int i = blockIdx.x * kRdRows + threadIdx.x;
  int kc = blockIdx.y;
  int k0 = kc * chunk, k1 = min(k0 + chunk, m);
  for (int k = k0 + threadIdx.x; k < k1; k += kRdRows) {
    const double pk = p[k];
    const float h = (float)pk;
    ps[k - k0] = make_float2(h, (float)(pk - (double)h));
  }
  __syncthreads();
  if (i >= m) return;
  float sh = 0.f, sc = 0.f;
  int kend = min(k1, i + 1);
  // unrolled so that eight loads of the factor are in flight per thread (the
  // sum's order is unchanged)
#pragma unroll 8
  for (int k = k0; k < kend; k++) {
    const float2 a = A[(size_t)k * lda + i];
    const float2 q = ps[k - k0];
    const float x = a.x * q.x;
    const float ex = fmaf(a.x, q.x, -x) + fmaf(a.x, q.y, a.y * q.x);
    const float t = sh + x;
    const float bp = t - sh;
    sc += ((sh - (t - bp)) + (x - bp)) + ex;
    sh = t;
  }
  part[(size_t)kc * m + i] = s2dt * ((double)sh + (double)sc);
}

__global__ void k_trmv_sum(int m, int nchunk, const double* __restrict__ part, double* __restrict__ rd) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  double s = 0.0;
#pragma unroll 8
  for (int c = 0; c < nchunk; c++) s = s + part[(size_t)c * m + i];
  rd[i] = s;
}

}  // namespace

namespace bdk {

void rpy_assemble(int nD, const double* r_all, const double* rad, double a1, double a2, double* A, int lda,
                  cudaStream_t st, const float4* qh, const float4* ql) {
  int nt = cdiv(nD, kRpyTile);
  if (qh)
    k_rpy_mx<<<dim3(nt, nt), dim3(kRpyTile, 8), 0, st>>>(nD, qh, ql, (float)a1, (float)a2,
                                                         reinterpret_cast<float2*>(A), lda);
  else
    k_rpy<<<nt * (nt + 1) / 2, dim3(kRpyTile, 8), 0, st>>>(nD, r_all, rad, a1, a2, A, lda);
}

// Blocks of 2 kNB columns: panel, the second panel's columns updated by the
// first, panel, then the trailing triangle by both (K = 64, half the passes
// over it).  The triangle's tiles are 32 wide: a tile takes 17 us on its SM's
// FP64 pipe and 64-wide ones 69, which leave SMs idle in a last wave and gain
// nothing at any size (3N = 3,888: 23.1 ms, 22.5 with 32).
int potrf_fp64(int m, double* A, int lda, double* /*rd_acc*/, const double* /*p*/, double /*s2dt*/, int* d_negpiv,
               cudaStream_t st) {
  int launches = 0;
  auto panel = [&](int k0) {  // returns its width
    const int kb = m - k0 < kNB ? m - k0 : kNB;
    k_potrf_diag<<<1, 128, 0, st>>>(A, lda, k0, kb, d_negpiv);
    launches++;
    const int rest = m - k0 - kb;
    if (rest > 0) {
      k_trsm_panel<<<cdiv(rest, kTrsmRows), 128, 0, st>>>(A, lda, m, k0, kb);
      launches++;
    }
    return kb;
  };
  for (int k0 = 0; k0 < m; k0 += 2 * kNB) {
    int kb = panel(k0);
    const int k1 = k0 + kb;
    if (k1 >= m) break;
    const int jend = k1 + kNB < m ? k1 + kNB : m;
    k_syrk_update<16, 32, 2, 2><<<cdiv(m - k1, 16), 128, 0, st>>>(A, lda, m, k0, kb, k1, jend);
    launches++;
    kb += panel(k1);
    const int t0 = k0 + kb, rest = m - t0;
    if (rest <= 0) break;
    const int nt = cdiv(rest, 32);
    k_syrk_update<32, 32, 4, 2><<<nt * (nt + 1) / 2, 128, 0, st>>>(A, lda, m, k0, kb, t0, m);
    launches++;
  }
  return launches;
}

// (for every size up to m: a smaller matrix can have more partial sums)
size_t trmv_scratch_doubles(int m) {
  auto need = [](int k) { return (size_t)cdiv(k, rd_chunk(k)) * k; };
  return std::max({need(m), need(std::min(m, 2048)), need(std::min(m, 8192))});
}

void trmv_lower_ws(int m, const double* A, int lda, const double* p, double s2dt, double* rd, double* part,
                   cudaStream_t st, bool df) {
  const int chunk = rd_chunk(m), nchunk = cdiv(m, chunk);
  if (df)
    k_trmv_part_df<<<dim3(cdiv(m, kRdRows), nchunk), kRdRows, 0, st>>>(m, reinterpret_cast<const float2*>(A), lda, p,
                                                                       s2dt, chunk, part);
  else
    k_trmv_part<<<dim3(cdiv(m, kRdRows), nchunk), kRdRows, 0, st>>>(m, A, lda, p, s2dt, chunk, part);
  k_trmv_sum<<<cdiv(m, 256), 256, 0, st>>>(m, nchunk, part, rd);
}

}  // namespace bdk
