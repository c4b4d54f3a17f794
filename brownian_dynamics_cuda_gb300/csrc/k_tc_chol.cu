// Mixed-precision Cholesky of the RPY tensor on the sm_103a tensor cores.
//
// Right-looking blocked factorisation with 128-wide panels.  The matrix is
// stored as double-float pairs (hi, lo) of FP32 (column-major, 8 bytes per
// element, ~48 significant bits), so the trailing updates accumulate without
// an FP32 rounding per panel and without FP64 arithmetic (GB300's FP64 rate
// is ~2 operations per clock per SM); the arithmetic is FP32-class.  One
// kernel, k_chol_step, runs these kinds of CTA side by side:
//   panel CTAs   solve panel k's tiles, L_ik = A_ik L_kk^-T, write them back
//                and split them into two FP16 slices (scaled by one power of
//                two: hi + lo = the FP32 value to 2^-23), stored pre-swizzled
//                in the 128-byte-swizzle K-major layout the MMA reads; one of
//                them, the chain CTA, then factors diagonal block k + 1 and
//                inverts the factor for the next launch.  A negative pivot is
//                replaced by its absolute value and counted
//                (func.cpp:827-833).
//   update CTAs  trailing update A_IJ -= L_I L_J^T of up to six earlier
//                panels, a run of tiles per CTA, warp-specialised:
//                bulk-async operand copies, three FP16 products (lo.hi,
//                hi.lo, hi.hi) per panel, up to three panels into one of
//                four FP32 tensor-memory accumulators (tcgen05.mma, M = N = 128, K = 16 per
//                instruction), tcgen05.ld epilogue subtracting into the
//                double-float tile.  The dropped product lo.lo is at most
//                2^-22 of hi.hi (both values half way between two FP16 ones).
// Two FP16 slices and three products instead of three BF16 slices and six
// (which hold the FP32 value exactly): half the tensor work, two thirds of
// the operand bytes.  3N = 11,700: 7.0 -> 6.1 ms; 3N = 46,200: 202 -> 157 ms.
// Error of L p against FP64 (2-norm, 13 fibers of 3N 912 .. 11,700):
// 2.6e-7 .. 5.4e-7 before, 2.6e-7 .. 5.1e-7 now - the sums inside the tensor
// core set it, not the split: FP32-class by that measurement.
// The launches run on one stream, one at a time (the schedule is at
// potrf_mixed).  Every mbarrier wait is bounded; on a timeout the kernel
// records an error code, frees its tensor memory and returns.
#include <algorithm>
#include <climits>
#include <cmath>
#include <type_traits>
#include <utility>
#include <vector>

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "bd_internal.h"
#include "dev_physics.cuh"
#include "sm100_ptx.cuh"

namespace {



constexpr int kT = 128;                 // tile / panel width
constexpr int kSliceBytes = kT * kT * 2;  // one FP16 slice of a 128 x 128 tile (two 64-column halves)
constexpr int kHalfBytes = kSliceBytes / 2;
constexpr int kTileSlices = 2;
constexpr int kTileBytes = kTileSlices * kSliceBytes;  // 64 KB per 128-row panel tile
constexpr uint32_t kWaitLimit = 1u << 24;
// panel p's slices are in buffer p % kBufs: a group's pass reads its panels' while the next is written
constexpr int kBufs = 7;

inline int cdiv(int a, int b) { return (a + b - 1) / b; }
__device__ __forceinline__ int cdiv_d(int a, int b) { return (a + b - 1) / b; }

// byte offset of element (row r, column k) inside one pre-swizzled slice
__device__ __forceinline__ uint32_t swz_off(int r, int k) {
  int half = k >> 6, kk = k & 63;
  return half * kHalfBytes + (r >> 3) * 1024 + (r & 7) * 128 + ((((kk >> 3) ^ (r & 7)) & 7) << 4) + (kk & 7) * 2;
}

// Two scaled FP32 values as FP16 pairs: x = hi + lo to 2^-23 |x| (two
// roundings to 11 bits each), low half first.  A value past FP16's range makes
// hi infinite and the products NaN: never a finite, wrong factor (see Range).
__device__ __forceinline__ uint32_t cvt_f16x2(float x0, float x1) {
  uint32_t r;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(x1), "f"(x0));
  return r;
}
__device__ __forceinline__ void split_f16x2(float x0, float x1, uint32_t& hi, uint32_t& lo) {
  hi = cvt_f16x2(x0, x1);
  const float2 hf = __half22float2(*reinterpret_cast<const __half2*>(&hi));
  lo = cvt_f16x2(x0 - hf.x, x1 - hf.y);
}

// Range.  The slices' common scale (mixed_scale) fits every positive definite
// tensor.  An indefinite one (its negative pivots are replaced by |f|,
// func.cpp:827-833) can grow past FP16's range at any row: such a row of a
// tile gets a power of two of its own, from its largest value (rows that fit
// keep the common one), so that slices hold whatever FP32 does.  `top`: the
// largest |hi| of the values split, NaN if one is; past(top): one of them does
// not fit.
__device__ __forceinline__ void keep_top(uint32_t& top, uint32_t hi) {
  const __half2 a = __hmax2_nan(*reinterpret_cast<const __half2*>(&top), __habs2(*reinterpret_cast<const __half2*>(&hi)));
  top = *reinterpret_cast<const uint32_t*>(&a);
}
__device__ __forceinline__ bool past(uint32_t top) { return (top & 0x7fffu) >= 0x7c00u || (top >> 16) >= 0x7c00u; }
// The power of two that puts m into [2^13, 2^14), and its inverse; false (m
// zero, infinite or NaN, or the power past 2^+-100): neither is set.
__device__ __forceinline__ bool own_scale(float m, float& up, float& down) {
  const int e = 13 + 127 - (int)(__float_as_uint(m) >> 23);
  if (!(m > 0.f) || isinf(m) || e > 100 || e < -100) return false;
  up = __uint_as_float((uint32_t)(127 + e) << 23);
  down = __uint_as_float((uint32_t)(127 - e) << 23);
  return true;
}

// (hi, lo) - v in double-float arithmetic: exact two-sums (Knuth), so the
// stored value keeps ~48 significant bits through every trailing update
// (no per-update FP32 rounding of the element) without any FP64 operation.
__device__ __forceinline__ float2 df_sub(float2 a, float v) {
  const float s = a.x - v;
  const float bb = s - a.x;
  float e = (a.x - (s - bb)) + (-v - bb);
  e += a.y;
  const float h = s + e;
  const float b2 = h - s;
  const float l = (s - (h - b2)) + (e - b2);
  return make_float2(h, l);
}

// ------------------------------------------------------------ one panel
// Launch k of the factorisation solves panel k's tiles and factors diagonal
// block k + 1:
//   tile CTAs   L_ik = A_ik W_k^T with W_k = L_kk^-1 from the launch before:
//               a product on the tensor cores in place of a substitution.
//               The tile first takes panel k - 1's update (D = L_i,k-1
//               L_k,k-1^T), also there.
//   chain CTA   the same for the tile below the diagonal, then diagonal block
//               k + 1 with the updates of panels k - 1 and k, its Cholesky
//               factor (written into A) and that factor's inverse W_k+1.
// So the serial chain of a factorisation is one CTA's work per panel, and no
// CTA repeats another's.  Bound by that chain: 26 us (copies and the panel
// k - 1 product 3, the tile and its products 5, the 128 columns 15, the last
// of W 1, the look at the range 0.6) beside 9 us of the other tiles, and ~3 us between launches.  Before,
// every panel CTA factored the diagonal block itself and solved its rows by
// substitution, 41 us.  A step of 3N = 1,944: 1.13 -> 0.94 ms, 3N = 3,888:
// 1.86 -> 1.43, 3N = 11,700: 7.6 -> 5.8 (with the FP16 slices); 24 replicas,
// where the repeated work also filled the GPU: 28.7 -> 19.0.
// The explicit inverse is as accurate as the substitution here (condition
// numbers of L_kk below 10): error of L p against FP64, 2-norm over 13 fibers
// of 3N 912 .. 11,700: 2.6e-7 .. 5.4e-7 before, 2.5e-7 .. 5.1e-7 now; 46,200: 5.3e-7, 5.1e-7.
// (A fiber pressed to a tenth of its size, condition numbers in the hundreds: up
// to a third above the substitution's 3e-6.)
constexpr int kLd = 132;  // row stride (floats) of the diagonal block in shared memory: conflict-free 16-byte rows
constexpr int kChainS = kTileBytes;                  // shared-memory offset of the FP32 diagonal block
constexpr int kChainW = 130 * 1024;                  // ... and of the inverse's slices
constexpr int kPanelMisc = kChainW + kTileBytes;     // ... and of the barriers
static_assert(kChainS + kT * kLd * 4 <= kChainW, "the diagonal block lies before the inverse's slices");

struct PanelBars {
  uint64_t fullPre, fullW, preDone, sReady, xDone, lReady, qDone, r0Free, trDone[3], trRest[2], helped[2], step[16];
  uint32_t slot;
  int again, failed;                 // some value does not fit the common scale; some wait ran out
  int lown, rown;                    // some row of L_ik, of a rank-32 product, has a scale of its own
  float rmax[2][kT];                 // a row's largest value, by column half
  float lrow[kT];                    // common scale / the row's own (L_ik)
  float rowf[2][kT];                 // undoes the scales of a row's rank-32 product (panel P in buffer P & 1)
  float colf[2][kT];                 // ... as a column of it: common scale / the row's own
  alignas(16) float xsc[kT];         // X = D * xsc, by column
  alignas(16) float dg[16][8][8];    // the 8 x 8 diagonal blocks, then L's
};
constexpr size_t kPanelSmem = kPanelMisc + sizeof(PanelBars) + 1024;

// The next 1024-byte boundary of shared memory, by an offset from smraw: a
// pointer rounded as an integer is no longer known to be shared, and every
// access through it becomes a generic one (the 128-column factorisation took
// four times as long).
__device__ __forceinline__ unsigned char* align1024(unsigned char* smraw) {
  return smraw + ((0u - sm100::smem_u32(smraw)) & 1023u);
}

// 128 consecutive K of one product: D (+)= A B^T from slice operands at sa, sb
// (two slices each), smallest products first.
__device__ __forceinline__ void mma_tile(uint32_t d, const unsigned char* sa, const unsigned char* sb, bool acc) {
  const uint32_t idesc = sm100::idesc_f16_f32(128, 128);
  const int pa[3] = {1, 0, 0};  // (A slice, B slice)
  const int pb[3] = {0, 1, 0};
#pragma unroll
  for (int h = 0; h < 2; h++)
#pragma unroll
    for (int p = 0; p < 3; p++) {
      const uint32_t aaddr = sm100::smem_u32(sa + pa[p] * kSliceBytes + h * kHalfBytes);
      const uint32_t baddr = sm100::smem_u32(sb + pb[p] * kSliceBytes + h * kHalfBytes);
#pragma unroll
      for (int kk = 0; kk < 4; kk++)
        sm100::mma_f16(d, sm100::desc_kmajor_sw128(aaddr + kk * 32), sm100::desc_kmajor_sw128(baddr + kk * 32), idesc,
                       acc || (h | p | kk) != 0);
    }
}

// 8 consecutive columns (from column c, c % 8 == 0) of row r of a slice pair at `base`
__device__ __forceinline__ void put_slices8(unsigned char* base, int r, int c, const float (&x)[8], uint32_t& top) {
  uint32_t h[4], l[4];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    split_f16x2(x[2 * j], x[2 * j + 1], h[j], l[j]);
    keep_top(top, h[j]);
  }
  const uint32_t off = swz_off(r, c);
  *reinterpret_cast<uint4*>(base + off) = make_uint4(h[0], h[1], h[2], h[3]);
  *reinterpret_cast<uint4*>(base + kSliceBytes + off) = make_uint4(l[0], l[1], l[2], l[3]);
}

// The 8 x 8 diagonal block `dg` (lower part read) factored into d; x, a row of
// the panel, solved against it.  Returns the number of negative pivots, each
// replaced by its absolute value (func.cpp:827-833).
__device__ __forceinline__ int factor8(const float (*dg)[8], float (&d)[8][8], float* x) {
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int h = 0; h <= (i >> 2); h++) {
      const float4 v = *reinterpret_cast<const float4*>(&dg[i][4 * h]);
      d[i][4 * h] = v.x, d[i][4 * h + 1] = v.y, d[i][4 * h + 2] = v.z, d[i][4 * h + 3] = v.w;
    }
  int neg = 0;
#pragma unroll
  for (int j = 0; j < 8; j++) {
    const float ad = fabsf(d[j][j]);
    if (d[j][j] < 0.f) neg++;
    const float rp = rsqrtf(ad);
    d[j][j] = ad * rp;
    x[j] *= rp;
#pragma unroll
    for (int i = j + 1; i < 8; i++) {
      d[i][j] *= rp;
      x[i] = fmaf(-x[j], d[i][j], x[i]);
    }
#pragma unroll
    for (int i = j + 1; i < 8; i++)
#pragma unroll
      for (int l = j + 1; l <= i; l++) d[i][l] = fmaf(-d[i][j], d[l][j], d[i][l]);
  }
  return neg;
}

constexpr int kTrSlice = 16 * 1024;  // one slice of a 128 x 32 operand, in 128-byte rows

// Cholesky factor and inverse of the 128 x 128 block in S (row stride kLd; its
// first 32 columns in x).  Four warps, a thread a row (r, its tensor-memory
// lane too), in four panels of 32 columns that the thread keeps in registers:
//   - 16 steps of eight columns: the 8 x 8 diagonal block goes through shared
//     memory, every thread factors it (all the same) and solves its own row
//     against it; the rows' values go to S, and every thread takes them off
//     the rest of its panel, one column after the other.
//   - the columns right of a panel take its rank-32 update on the tensor cores
//     (FP16 pairs as the tiles' slices), this thread's next panel at once, the
//     later columns by four helper warps (chol_help) beside the next panel.
// A row above a step's block has been eliminated and carries the inverse
// instead: row r of X = L^-T, started as the unit row in its own step, takes
// the same solves and updates (in the rank-32 product with a scale of its
// own: X's rows differ in size).  At the end S holds L below the 8 x 8
// diagonal blocks, X on and above them; L's 8 x 8 blocks are in dg.  step[q]
// is arrived at when step q's columns are final.
// Bound by the chain of a step (two barriers, three shared-memory round trips,
// eight reciprocal roots) and by the 16-byte loads of L's values, four cycles
// of shared memory each however few of the bytes differ: eight columns a step
// and rows in registers need the fewest of them (a register-tiled block with
// four columns a step: 1.5 times longer).  neg += negative pivots.
__device__ __forceinline__ void chol_inv128(float (*S)[kLd], PanelBars* bars, unsigned char* T, uint32_t tmem,
                                            float (&x)[32], int r, int lane, float scale, int& neg, bool& ok) {
  const float iscale = 1.f / scale;
  const uint32_t trow = tmem + ((uint32_t)(r & ~31) << 16);
  // x[j0 .. j1) of the panel P less the step s's columns; mk: 0 for a row that
  // the step eliminated (it starts as a row of X), else 1 (a product: as a
  // select it became a branch, 3 us a panel)
  auto upd = [&](int P, auto sc, auto j0c, auto j1c, float mk) {
    constexpr int s = decltype(sc)::value, j0 = decltype(j0c)::value, j1 = decltype(j1c)::value;
#pragma unroll
    for (int j = j0; j < j1; j++) {
      const float4 l0 = *reinterpret_cast<const float4*>(&S[32 * P + j][32 * P + 8 * s]);
      const float4 l1 = *reinterpret_cast<const float4*>(&S[32 * P + j][32 * P + 8 * s + 4]);
      const float l[8] = {l0.x, l0.y, l0.z, l0.w, l1.x, l1.y, l1.z, l1.w};
      x[j] *= mk;
#pragma unroll
      for (int e = 0; e < 8; e++) x[j] = fmaf(-x[8 * s + e], l[e], x[j]);
    }
  };
#pragma unroll 1
  for (int P = 0; P < 4; P++) {
    const bool mine = (r >> 5) == P;  // the panel's diagonal rows
    float rho = scale, f = iscale * iscale;
    auto step = [&](auto sc) {
      constexpr int s = decltype(sc)::value;
      const int q = 4 * P + s, c = 8 * q;  // (x[8 s ..] are columns c ..)
      const bool blk = mine && (lane >> 3) == s;
      float (*dg)[8] = bars->dg[q];
      if (blk) {
        *reinterpret_cast<float4*>(&dg[lane & 7][0]) = make_float4(x[8 * s], x[8 * s + 1], x[8 * s + 2], x[8 * s + 3]);
        *reinterpret_cast<float4*>(&dg[lane & 7][4]) = make_float4(x[8 * s + 4], x[8 * s + 5], x[8 * s + 6], x[8 * s + 7]);
      }
      asm volatile("bar.sync 2, 128;" ::: "memory");
      // the step before's update of the columns past this step's, beside this chain
      if constexpr (s > 0)
        upd(P, std::integral_constant<int, s - 1>{}, std::integral_constant<int, 8 * s + 8>{},
            std::integral_constant<int, 32>{}, mine && (lane >> 3) == s - 1 ? 0.f : 1.f);
      if (blk) {  // the block's own rows: unit rows from here on
#pragma unroll
        for (int j = 0; j < 8; j++) x[8 * s + j] = (lane & 7) == j ? 1.f : 0.f;
      }
      float d[8][8];
      neg += factor8(dg, d, &x[8 * s]);
      *reinterpret_cast<float4*>(&S[r][c]) = make_float4(x[8 * s], x[8 * s + 1], x[8 * s + 2], x[8 * s + 3]);
      *reinterpret_cast<float4*>(&S[r][c + 4]) = make_float4(x[8 * s + 4], x[8 * s + 5], x[8 * s + 6], x[8 * s + 7]);
      if constexpr (s == 3) {  // the scale of this row in the rank-32 product
        if (mine) {  // a row eliminated in this panel takes part as a row of X alone
#pragma unroll
          for (int j = 0; j < 24; j++)
            if (j < (lane & 24)) x[j] = 0.f;
        }
        float m[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int j = 0; j < 32; j++) m[j & 3] = fmaxf(m[j & 3], fabsf(x[j]));
        m[0] = fmaxf(fmaxf(m[0], m[1]), fmaxf(m[2], m[3]));
        float up = 1.f, down = 1.f, cf = 1.f;
        const bool set = own_scale(m[0], up, down);
        if ((r >> 5) <= P) {
          rho = up;
          f = down * iscale;
        } else if (m[0] * scale >= 32768.f && set) {  // a row of L past FP16's range
          rho = up;
          f = down * iscale;
          cf = scale * down;
          bars->rown = 1;
        }
        bars->rowf[P & 1][r] = f;  // (the buffer's last readers are done: helped[P - 2])
        bars->colf[P & 1][r] = cf;
      }
      asm volatile("bar.sync 2, 128;" ::: "memory");
      if (lane == 0 && (r >> 5) == 0) {
        sm100::mbar_arrive(&bars->step[q]);
        // L's block in place of the diagonal block, which every thread has
        // read before the second barrier
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
          for (int h = 0; h < 2; h++)
            *reinterpret_cast<float4*>(&dg[i][4 * h]) =
                make_float4(i >= 4 * h ? d[i][4 * h] : 0.f, i > 4 * h ? d[i][4 * h + 1] : 0.f,
                            i > 4 * h + 1 ? d[i][4 * h + 2] : 0.f, i > 4 * h + 2 ? d[i][4 * h + 3] : 0.f);
      }
      if constexpr (s < 3)  // the next step's columns
        upd(P, sc, std::integral_constant<int, 8 * s + 8>{}, std::integral_constant<int, 8 * s + 16>{}, blk ? 0.f : 1.f);
    };
    step(std::integral_constant<int, 0>{});
    step(std::integral_constant<int, 1>{});
    step(std::integral_constant<int, 2>{});
    step(std::integral_constant<int, 3>{});
    if (P == 3) break;
    // the rank-32 product: D[r][n] = row r of the panel . row 32 (P + 1) + n
    // T is free: the tile's slices have been copied, the panel before's products
    // formed and taken from tensor memory (its later columns, into S, by chol_help)
    ok = sm100::mbar_wait(P == 0 ? &bars->r0Free : &bars->helped[P - 1], 0, kWaitLimit) && ok;
#pragma unroll
    for (int j8 = 0; j8 < 4; j8++) {
      uint32_t h[4], l[4];
#pragma unroll
      for (int j = 0; j < 4; j++) split_f16x2(x[8 * j8 + 2 * j] * rho, x[8 * j8 + 2 * j + 1] * rho, h[j], l[j]);
      const uint32_t off = swz_off(r, 8 * j8);
      *reinterpret_cast<uint4*>(T + off) = make_uint4(h[0], h[1], h[2], h[3]);
      *reinterpret_cast<uint4*>(T + kTrSlice + off) = make_uint4(l[0], l[1], l[2], l[3]);
    }
    sm100::fence_proxy_async();
    sm100::tc_fence_before();
    asm volatile("bar.sync 2, 128;" ::: "memory");
    if (lane == 0 && (r >> 5) == 0) {
      sm100::tc_fence_after();
      // the next panel's columns, then the later ones
      const uint32_t ta = sm100::smem_u32(T), tb = ta + 4096u * (P + 1);
#pragma unroll
      for (int n = 0; n < 2; n++) {
        if (n == 1 && P == 2) break;
        const uint32_t idesc = sm100::idesc_f16_f32(128, n == 0 ? 32 : 64 - 32 * P);
#pragma unroll
        for (int p = 0; p < 3; p++)
#pragma unroll
          for (int kk = 0; kk < 2; kk++)
            sm100::mma_f16(tmem + 32 * n, sm100::desc_kmajor_sw128(ta + (p == 0 ? kTrSlice : 0) + kk * 32),
                           sm100::desc_kmajor_sw128(tb + 4096u * n + (p == 1 ? kTrSlice : 0) + kk * 32), idesc,
                           (p | kk) != 0);
        sm100::mma_commit(n == 0 ? &bars->trDone[P] : &bars->trRest[P]);
      }
    }
    __syncwarp();
    const bool own = bars->rown;
    ok = sm100::mbar_wait(&bars->trDone[P], 0, kWaitLimit) && ok;
    sm100::tc_fence_after();
    float v[32];
    sm100::tmem_ld32(trow, v);
    if (own) {
#pragma unroll
      for (int j = 0; j < 32; j++) v[j] *= bars->colf[P & 1][32 * (P + 1) + j];
    }
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const float4 o = *reinterpret_cast<const float4*>(&S[r][32 * (P + 1) + 4 * j]);
      x[4 * j] = fmaf(-v[4 * j], f, mine ? 0.f : o.x), x[4 * j + 1] = fmaf(-v[4 * j + 1], f, mine ? 0.f : o.y);
      x[4 * j + 2] = fmaf(-v[4 * j + 2], f, mine ? 0.f : o.z), x[4 * j + 3] = fmaf(-v[4 * j + 3], f, mine ? 0.f : o.w);
    }
    sm100::tc_fence_before();
  }
}

// The rank-32 product of panel P: the columns past the next panel, into S (beside chol_inv128).
__device__ __forceinline__ void chol_help(float (*S)[kLd], PanelBars* bars, uint32_t tmem, int P, int r, int lane,
                                          bool& ok) {
  const uint32_t trow = tmem + ((uint32_t)(r & ~31) << 16);
  ok = sm100::mbar_wait(&bars->step[4 * P + 3], 0, kWaitLimit) && ok;  // (rowf)
  ok = sm100::mbar_wait(&bars->trRest[P], 0, kWaitLimit) && ok;
  sm100::tc_fence_after();
  const float f = bars->rowf[P & 1][r];
  const bool mine = (r >> 5) == P;
#pragma unroll 1
  for (int c = 0; c < 64 - 32 * P; c += 16) {
    float v[16];
    sm100::tmem_ld16(trow + 32 + c, v);
    if (bars->rown) {
#pragma unroll
      for (int j = 0; j < 16; j++) v[j] *= bars->colf[P & 1][32 * (P + 2) + c + j];
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
      float4* o = reinterpret_cast<float4*>(&S[r][32 * (P + 2) + c + 4 * j]);
      const float4 a = mine ? make_float4(0.f, 0.f, 0.f, 0.f) : *o;
      *o = make_float4(fmaf(-v[4 * j], f, a.x), fmaf(-v[4 * j + 1], f, a.y), fmaf(-v[4 * j + 2], f, a.z),
                       fmaf(-v[4 * j + 3], f, a.w));
    }
  }
  sm100::tc_fence_before();
  __syncwarp();
  if (lane == 0) sm100::mbar_arrive(&bars->helped[P]);
}

// Beside chol_inv128, step by step:
// L's columns below the 8 x 8 diagonal blocks into A (G = A at the block), as
// (L, 0) pairs ...
__device__ __forceinline__ void chain_store_l(const float (*S)[kLd], PanelBars* bars, int lane, int kb, float2* G,
                                              int lda, bool& ok) {
#pragma unroll 1
  for (int q = 0; q < 16; q++) {
    ok = ok && sm100::mbar_wait(&bars->step[q], 0, kWaitLimit);
#pragma unroll 1
    for (int r = ((8 * q + 8) & ~31) + lane; r < kb; r += 32) {
      if (r < 8 * q + 8) continue;
      const float4 v0 = *reinterpret_cast<const float4*>(&S[r][8 * q]);
      const float4 v1 = *reinterpret_cast<const float4*>(&S[r][8 * q + 4]);
      const float v[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
#pragma unroll
      for (int j = 0; j < 8; j++) G[(size_t)(8 * q + j) * lda + r] = make_float2(v[j], 0.f);
    }
  }
}
// ... and rows 8 q .. 8 q + 7 of W = L^-1 (W[l][j] = X[j][l]) as slices in Wo
// and on to Wn, every row scaled by a power of two that puts its largest entry
// into [2^13, 2^14); wscn[l] undoes that scale and the tile's, cs.  The copies
// are in the lanes' bulk groups.
__device__ __forceinline__ void chain_store_w(const float (*S)[kLd], PanelBars* bars, int lane, int q, float cs,
                                              unsigned char* Wo, unsigned char* Wn, float* wscn, bool& ok) {
  ok = sm100::mbar_wait(&bars->step[q], 0, kWaitLimit) && ok;
  // lane (i, jc): row 8 q + i, columns 8 (jc + 4 t) .. + 7 for t = 0 .. 3
  const int i = lane & 7, jc = lane >> 3, row = 8 * q + i;
  float x[4][8];
  float m = 0.f;
#pragma unroll
  for (int t = 0; t < 4; t++) {
    const int j0 = 8 * (jc + 4 * t);
    const bool in = jc + 4 * t <= q;
#pragma unroll
    for (int j = 0; j < 8; j++) {
      x[t][j] = in ? S[j0 + j][row] : 0.f;
      m = fmaxf(m, fabsf(x[t][j]));
    }
  }
  m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 8));
  m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 16));
  float sc = 1.f, isc = 1.f;
  (void)own_scale(m, sc, isc);
  if (jc == 0) wscn[row] = 1.f / (cs * sc);
  uint32_t top = 0;  // (scaled by its own maximum: nothing to see)
#pragma unroll
  for (int t = 0; t < 4; t++) {
#pragma unroll
    for (int j = 0; j < 8; j++) x[t][j] *= sc;
    put_slices8(Wo, row, 8 * (jc + 4 * t), x[t], top);
  }
  sm100::fence_proxy_async();
  __syncwarp();
  if (lane < 2 * kTileSlices) {  // the rows' 1 KB in each half of a slice
    const int off = lane * kHalfBytes + q * 1024;
    sm100::bulk_s2g(Wn + off, Wo + off, 1024);
  }
}

// What a panel CTA works on.  tile < 0: no tile (the first launch, which only
// factors diagonal block 0).  PSpre: panel k - 1's slices, or null (k = 0).
struct PanelArgs {
  float2* A;
  int lda, m, k, tile;            // panel k, tile row
  unsigned char* PSp;             // panel k's slices
  const unsigned char* PSpre;
  const unsigned char* Wk;        // W_k's slices
  const float* wsc;               // [128] X = D * wsc, by column
  unsigned char* Wn;              // W_k+1's slices and factors (chain)
  float* wscn;
  int* negpiv;
  int* err;
  int* past;                      // [0] the first panel with rows whose scales are their own, [1 + p] panel p is such
  float* rowk;                    // [nt kT] the common scale / the row's own, of panel k ...
  const float* rowp;              // ... and of panel k - 1
  float scale, iscale2;
};

// whether p holds in either of the two warps that share 32 rows (q)
__device__ __forceinline__ bool pair_any(int q, bool p) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred a, b;\n\t"
      "setp.ne.u32 a, %1, 0;\n\t"
      "barrier.cta.red.or.pred b, %2, 64, a;\n\t"
      "selp.u32 %0, 1, 0, b;\n\t}"
      : "=r"(r)
      : "r"((uint32_t)p), "r"(4 + q)
      : "memory");
  return r != 0;
}

// The 32 rows of warps q where a row of the tile, or of L_ik, does not fit the
// slices' common scale (the product is then infinite or NaN), or panel k - 1 has
// rows with scales of their own: the tile less that panel's update, then L_ik by
// forward substitution in FP32, in A.  Such a row's values can lie further apart
// than a pair's 40 bits: no one scale holds them, and the product with the
// inverse would lose the small ones.
__device__ __forceinline__ void solve_rows(const PanelArgs& p, int q, int ch, int r, bool pre, uint32_t trow) {
  const bool in = p.tile * kT + r < p.m;
  float2* row = p.A + (size_t)(p.k * kT) * p.lda + p.tile * kT + r;
  const float2* L = p.A + (size_t)(p.k * kT) * p.lda + p.k * kT;
#pragma unroll 1
  for (int c = 0; c < 64; c += 8) {
    float v[8];
    if (pre) sm100::tmem_ld8(trow + c, v);
    if (in) {
#pragma unroll
      for (int j = 0; j < 8; j++) {
        float2* a = row + (size_t)(64 * ch + c + j) * p.lda;
        const float2 o = *a;
        const float f = pre ? p.iscale2 * p.rowp[p.tile * kT + r] * p.rowp[p.k * kT + 64 * ch + c + j] : 0.f;
        *a = make_float2((pre ? fmaf(-v[j], f, o.x) : o.x) + o.y, 0.f);
      }
    }
    __syncwarp();
  }
  (void)pair_any(q, false);
  if (ch == 0 && in) {
#pragma unroll 1
    for (int c = 0; c < kT; c++) {
      float s = row[(size_t)c * p.lda].x;
#pragma unroll 8
      for (int e = 0; e < c; e++) s = fmaf(-row[(size_t)e * p.lda].x, L[(size_t)e * p.lda + c].x, s);
      row[(size_t)c * p.lda].x = s / L[(size_t)c * p.lda + c].x;
    }
  }
  __syncwarp();
  (void)pair_any(q, false);
}

// The slices of those rows of L_ik: a row past the common scale by a power of two
// of its own, from its largest value.  Returns the common scale / the row's.
__device__ __forceinline__ float split_rows(const PanelArgs& p, PanelBars* bars, unsigned char* R0, int q, int ch, int r) {
  const float2* row = p.A + (size_t)(p.k * kT + 64 * ch) * p.lda + p.tile * kT + r;
  const bool in = p.tile * kT + r < p.m;
  float m = 0.f, s = p.scale, lrow = 1.f;
#pragma unroll 1
  for (int pass = 0; pass < 2; pass++) {
#pragma unroll 1
    for (int c = 0; c < 64; c += 8) {
      float x[8];
      uint32_t top = 0;
#pragma unroll
      for (int j = 0; j < 8; j++) {
        x[j] = in ? row[(size_t)(c + j) * p.lda].x * s : 0.f;
        m = fmaxf(m, fabsf(x[j]));
      }
      if (pass) put_slices8(R0, r, 64 * ch + c, x, top);
    }
    if (pass) break;
    bars->rmax[ch][r] = m;  // of scale * L
    (void)pair_any(q, false);
    m = fmaxf(m, bars->rmax[ch ^ 1][r]);
    float up, down;
    if (m >= 32768.f && own_scale(m, up, down)) {
      lrow = down;
      s *= up;
      bars->lown = 1;
      p.past[1 + p.k] = 1;
      atomicMin(p.past, p.k);
    }
  }
  __syncwarp();
  return lrow;
}

// The diagonal block's updates by panels k and (pre) k - 1 whose rows have scales
// of their own: row r, columns 64 ch .. + 63, in S and (the first 32) in x.
__device__ __forceinline__ void own_diag(const PanelArgs& p, PanelBars* bars, float (*S)[kLd], float (&x)[32],
                                         uint32_t trow, bool pre, int ch, int r, bool in) {
  float4* s4 = reinterpret_cast<float4*>(S[r]);
  if (ch == 0) {
#pragma unroll
    for (int j = 0; j < 8; j++) s4[j] = make_float4(x[4 * j], x[4 * j + 1], x[4 * j + 2], x[4 * j + 3]);
  }
  const int t = (p.k + 1) * kT;
  const float fk = p.iscale2 * bars->lrow[r], fp = pre ? p.iscale2 * p.rowp[t + r] : 0.f;
#pragma unroll 1
  for (int c = 64 * ch; c < 64 * ch + 64; c += 8) {
    float v[8];
    sm100::tmem_ld8(trow + c, v);
#pragma unroll
    for (int j = 0; j < 8; j++)
      if (in) S[r][c + j] = fmaf(-v[j], fk * bars->lrow[c + j], S[r][c + j]);
    __syncwarp();
    if (pre) {
      sm100::tmem_ld8(trow + 128 + c, v);
#pragma unroll
      for (int j = 0; j < 8; j++)
        if (in) S[r][c + j] = fmaf(-v[j], fp * p.rowp[t + c + j], S[r][c + j]);
      __syncwarp();
    }
  }
  if (ch == 0) {
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const float4 f = s4[j];
      x[4 * j] = f.x, x[4 * j + 1] = f.y, x[4 * j + 2] = f.z, x[4 * j + 3] = f.w;
    }
  }
}

// Shared memory: R0 L_i,k-1 then L_ik's slices; R1 L_k,k-1 then the tile's
// slices (the diagonal block from kChainS on reuses R1 and the start of R2);
// R2 W_k.  Tensor memory: P at column 0, X at 128; chain: the updates of the
// diagonal block by panel k at 256 and by panel k - 1 at 384 (apart: the tensor
// core truncates its sums, so their error grows with the length).
// Warp 0 copies, warp 1 issues the products, warps 2 .. 9 hold the tile: a
// thread one row (TMEM lane) and 64 columns.
// OWN = false returns true, with nothing written to global memory but past and
// rowk, where a value does not fit the common scale (it makes its row of the
// product infinite or NaN) or panel k - 1 has rows with scales of their own.
// OWN = true then does the work again, with solve_rows, split_rows and own_diag:
// apart, as those cost every panel 2 us in one body with the rest (registers of
// the diagonal block, loaded ahead, were waited for and spilled over them).  The
// look at every value costs one 0.6: 3N = 1,944 0.504 -> 0.514 ms, 3,888 1.03 -> 1.05,
// 11,700 4.51 -> 4.57, 24 replicas 11.4 -> 11.7; 46,200 119.2 both.
template <bool CHAIN, bool OWN>
__device__ __forceinline__ bool panel_body(unsigned char* smraw, const PanelArgs& p) {
  unsigned char* sm = align1024(smraw);
  unsigned char *R0 = sm, *R1 = sm + kTileBytes, *R2 = sm + 2 * kTileBytes;
  PanelBars* bars = reinterpret_cast<PanelBars*>(sm + kPanelMisc);
  float (*S)[kLd] = reinterpret_cast<float (*)[kLd]>(sm + kChainS);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool has_tile = p.tile >= 0, pre = has_tile && p.PSpre != nullptr;
  constexpr uint32_t kCols = CHAIN ? 512 : 256;
  if (CHAIN && !has_tile)  // the factorisation's first launch
    for (int i = tid; i <= cdiv_d(p.m, kT); i += blockDim.x) p.past[i] = i == 0 ? INT_MAX : 0;
  if (tid == 0) {
    if (OWN)
      for (uint64_t* b = &bars->fullPre; b < (CHAIN ? bars->step + 16 : &bars->r0Free); b++) sm100::mbar_inval(b);
    bars->failed = bars->again = bars->lown = bars->rown = 0;
    sm100::mbar_init(&bars->fullPre, 1);
    sm100::mbar_init(&bars->fullW, 2);
    sm100::mbar_init(&bars->preDone, 1);
    sm100::mbar_init(&bars->sReady, 8);
    sm100::mbar_init(&bars->xDone, 1);
    sm100::mbar_init(&bars->lReady, 8);
    sm100::mbar_init(&bars->qDone, 1);
    if (CHAIN) {
      sm100::mbar_init(&bars->r0Free, 1);
      for (int q = 0; q < 3; q++) sm100::mbar_init(&bars->trDone[q], 1);
      for (int q = 0; q < 2; q++) {
        sm100::mbar_init(&bars->trRest[q], 1);
        sm100::mbar_init(&bars->helped[q], 4);
      }
      for (int q = 0; q < 16; q++) sm100::mbar_init(&bars->step[q], 1);
    }
    sm100::fence_mbar_init();
  }
  if (!OWN && warp == 1) sm100::tmem_alloc(&bars->slot, kCols);
  sm100::tc_fence_before();
  __syncthreads();
  sm100::tc_fence_after();
  const uint32_t tmem = bars->slot;
  bool ok = true;

  if (warp == 0) {
    if (lane == 0 && has_tile) {
      if (pre) {
        sm100::mbar_arrive_expect_tx(&bars->fullPre, 2 * kTileBytes);
        sm100::bulk_g2s(R0, p.PSpre + (size_t)p.tile * kTileBytes, kTileBytes, &bars->fullPre);
        sm100::bulk_g2s(R1, p.PSpre + (size_t)p.k * kTileBytes, kTileBytes, &bars->fullPre);
      }
      sm100::mbar_arrive_expect_tx(&bars->fullW, kTileBytes);
      sm100::bulk_g2s(R2, p.Wk, kTileBytes, &bars->fullW);
    }
    if (has_tile) {
      *reinterpret_cast<float4*>(&bars->xsc[4 * lane]) = reinterpret_cast<const float4*>(p.wsc)[lane];
      __syncwarp();
      if (lane == 0) {
        sm100::mbar_arrive(&bars->fullW);
        ok = sm100::mbar_wait(&bars->lReady, 0, kWaitLimit);
        if (ok && !OWN && bars->again) {
        } else if (ok) {
          sm100::bulk_s2g(p.PSp + (size_t)p.tile * kTileBytes, R0, kTileBytes);
          sm100::bulk_store_wait();
        } else {  // copies in flight land before the CTA exits
          if (pre) (void)sm100::mbar_wait(&bars->fullPre, 0, kWaitLimit);
          (void)sm100::mbar_wait(&bars->fullW, 0, kWaitLimit);
        }
      }
      __syncwarp();
    }
    if (CHAIN && (OWN || !has_tile || !bars->again)) {
      const int nd = p.k + 1;
      if (lane == 0) sm100::mbar_arrive(&bars->r0Free);
      chain_store_l(S, bars, lane, min(kT, p.m - nd * kT), p.A + (size_t)(nd * kT) * p.lda + nd * kT, p.lda, ok);
    }
  } else if (warp == 1) {
    if (lane == 0 && has_tile) {
      if (pre) {
        ok = sm100::mbar_wait(&bars->fullPre, 0, kWaitLimit);
        sm100::tc_fence_after();
        if (ok) mma_tile(tmem, R0, R1, false);
        sm100::mma_commit(&bars->preDone);
        if (CHAIN && ok) mma_tile(tmem + 384, R0, R0, false);
      }
      ok = ok && sm100::mbar_wait(&bars->fullW, 0, kWaitLimit);
      ok = ok && sm100::mbar_wait(&bars->sReady, 0, kWaitLimit);
      sm100::tc_fence_after();
      if (ok) mma_tile(tmem + 128, R1, R2, false);
      sm100::mma_commit(&bars->xDone);
      if (CHAIN) {
        ok = ok && sm100::mbar_wait(&bars->lReady, 0, kWaitLimit);
        sm100::tc_fence_after();
        if (OWN || !bars->again) {
          if (ok) mma_tile(tmem + 256, R0, R0, false);
          sm100::mma_commit(&bars->qDone);
        }
      }
      if (!ok) (void)sm100::mbar_wait(&bars->xDone, 0, kWaitLimit);
    }
  } else {
    const int q = warp & 3, ch = (warp - 2) >> 2, r = 32 * q + lane;
    const uint32_t trow = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(64 * ch);
    const uint64_t pol = sm100::policy_evict_first();  // the tile's columns are read again only by the noise product
    const int nd = p.k + 1;  // the diagonal block of the chain CTA (tile row of its tile too)
    const bool pown = pre && p.past[p.k] != 0;  // rows of panel k - 1 have scales of their own
    bool subst = false;  // this row (all 32 of the warp) solved by solve_rows, in A
    // 64 columns of the thread's row of L_ik, from tensor memory into A
    auto store_l = [&](int half) {
      const int gi = p.tile * kT + r;
      float2* colp = p.A + (size_t)(p.k * kT + 64 * half) * p.lda + gi;
#pragma unroll 1
      for (int c = 0; c < 4; c++) {
        float v[16];
        sm100::tmem_ld16(tmem + ((uint32_t)(32 * q) << 16) + 128 + 64 * half + 16 * c, v);  // (the whole warp)
        if (gi < p.m) {
#pragma unroll
          for (int j4 = 0; j4 < 4; j4++) {
            const float4 f = *reinterpret_cast<const float4*>(&bars->xsc[64 * half + 16 * c + 4 * j4]);
            const float fs[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
            for (int j = 0; j < 4; j++)
              sm100::st_f2_hint(colp + (size_t)(16 * c + 4 * j4 + j) * p.lda, make_float2(v[4 * j4 + j] * fs[j], 0.f), pol);
          }
        }
        __syncwarp();
      }
    };
    float2 old[64];
    if (has_tile) {
      const int gi = p.tile * kT + r;
      float2* colp = p.A + (size_t)(p.k * kT + 64 * ch) * p.lda + gi;
      const bool in = gi < p.m;
#pragma unroll
      for (int j = 0; j < 64; j++) old[j] = sm100::ld_f2_hint_if(colp + (size_t)j * p.lda, pol, in);
      if (pre) {
        ok = sm100::mbar_wait(&bars->preDone, 0, kWaitLimit);
        sm100::tc_fence_after();
      }
      uint32_t top = 0;  // (what does not fit shows in the product)
      // the tile less panel k - 1's update, as slices of scale^2 / 16 times it
      // (positive definite: |A_ij| <= max D_ii, at most 2^14)
      const float cs = p.scale * p.scale * 0.0625f;
#pragma unroll
      for (int c = 0; c < 4; c++) {
        float v[16];
        if (pre) sm100::tmem_ld16(trow + 16 * c, v);
#pragma unroll
        for (int h = 0; h < 2; h++) {
          float x[8];
#pragma unroll
          for (int j = 0; j < 8; j++) {
            const float2 o = old[16 * c + 8 * h + j];
            x[j] = (pre ? fmaf(-v[8 * h + j], p.iscale2, o.x) + o.y : o.x + o.y) * cs;
          }
          put_slices8(R1, r, 64 * ch + 16 * c + 8 * h, x, top);
        }
      }
      sm100::fence_proxy_async();
      __syncwarp();
      if (lane == 0) sm100::mbar_arrive(&bars->sReady);
    }
    const int kb = min(kT, p.m - nd * kT);
    if (CHAIN) {  // the diagonal block's row, under the product
      const float2* colp = p.A + (size_t)(nd * kT + 64 * ch) * p.lda + nd * kT + r;
#pragma unroll
      for (int j = 0; j < 64; j++)
        old[j] = sm100::ld_f2_hint_if(colp + (size_t)j * p.lda, pol, 64 * ch + j <= r && r < kb);
    }
    bool again = false;
    if (has_tile) {
      ok = sm100::mbar_wait(&bars->fullW, 0, kWaitLimit) && ok;  // (xsc)
      ok = sm100::mbar_wait(&bars->xDone, 0, kWaitLimit) && ok;
      sm100::tc_fence_after();
      uint32_t top = 0;
#pragma unroll 1
      for (int c = 0; c < 4; c++) {
        float v[16], x[16];
        sm100::tmem_ld16(trow + 128 + 16 * c, v);
#pragma unroll
        for (int j4 = 0; j4 < 4; j4++) {
          const float4 f = *reinterpret_cast<const float4*>(&bars->xsc[64 * ch + 16 * c + 4 * j4]);
          const float fs[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
          for (int j = 0; j < 4; j++) x[4 * j4 + j] = v[4 * j4 + j] * (fs[j] * p.scale);
        }
#pragma unroll
        for (int j8 = 0; j8 < 2; j8++) {
          float y[8];
#pragma unroll
          for (int j = 0; j < 8; j++) y[j] = x[8 * j8 + j];
          put_slices8(R0, r, 64 * ch + 16 * c + 8 * j8, y, top);
        }
      }
      float lrow = 1.f;
      if (!OWN) {
        if (pown || past(top)) bars->again = 1;
      } else if (pair_any(q, pown || past(top))) {
        subst = true;
        solve_rows(p, q, ch, r, pre, trow);
        lrow = split_rows(p, bars, R0, q, ch, r);
      }
      if (ch == 0) {
        if (OWN) bars->lrow[r] = lrow;
        p.rowk[p.tile * kT + r] = lrow;
      }
      sm100::fence_proxy_async();
      __syncwarp();
      if (lane == 0) sm100::mbar_arrive(&bars->lReady);
      ok = sm100::mbar_wait(&bars->lReady, 0, kWaitLimit) && ok;  // (again; lown, lrow)
      again = !OWN && bars->again;
      if (!CHAIN && !subst && !again) store_l(ch);
    }
    if (CHAIN && !again) {
      const bool own = OWN && (pown || bars->lown);  // rows of panel k or k - 1 have scales of their own
      if (has_tile) {
        ok = sm100::mbar_wait(&bars->qDone, 0, kWaitLimit) && ok;
        sm100::tc_fence_after();
      }
      // the diagonal block less its two updates (the part above the diagonal
      // is never used); rows past the matrix: the unit block
      float x[32];
#pragma unroll
      for (int c = 0; c < 8; c++) {
        float y[8], v[8];
#pragma unroll
        for (int j = 0; j < 8; j++) y[j] = old[8 * c + j].x;
        if (has_tile && !own) {
          sm100::tmem_ld8(trow + 256 + 8 * c, v);
#pragma unroll
          for (int j = 0; j < 8; j++) y[j] = fmaf(-v[j], p.iscale2, y[j]);
        }
        if (pre && !own) {
          sm100::tmem_ld8(trow + 384 + 8 * c, v);
#pragma unroll
          for (int j = 0; j < 8; j++) y[j] = fmaf(-v[j], p.iscale2, y[j]);
        }
#pragma unroll
        for (int j = 0; j < 8; j++) {
          y[j] += old[8 * c + j].y;
          if (r >= kb) y[j] = 64 * ch + 8 * c + j == r ? 1.f : 0.f;
        }
        if (c < 4) {
#pragma unroll
          for (int j = 0; j < 8; j++) x[8 * c + j] = y[j];
        }
        if (c >= 4 || ch == 1) {  // (the first panel stays in registers)
          *reinterpret_cast<float4*>(&S[r][64 * ch + 8 * c]) = make_float4(y[0], y[1], y[2], y[3]);
          *reinterpret_cast<float4*>(&S[r][64 * ch + 8 * c + 4]) = make_float4(y[4], y[5], y[6], y[7]);
        }
      }
      if (own) own_diag(p, bars, S, x, tmem + ((uint32_t)(32 * q) << 16) + 256, pre, ch, r, r < kb);
      if (ch == 0) {
        int neg = 0;
        chol_inv128(S, bars, R0, tmem, x, r, lane, p.scale, neg, ok);
        if (neg && lane == 0 && q == 0) atomicAdd(p.negpiv, neg);
      } else {
        if (has_tile && !subst) {
          store_l(0);
          store_l(1);
        }
#pragma unroll 1
        for (int P = 0; P < 4; P++) {
          if (P < 2) chol_help(S, bars, tmem, P, r, lane, ok);
          chain_store_w(S, bars, lane, 4 * P + (warp - 6), p.scale * p.scale * 0.0625f, sm + kChainW, p.Wn, p.wscn, ok);
        }
        if (lane < 2 * kTileSlices) sm100::bulk_store_wait();
      }
      asm volatile("bar.sync 1, 256;" ::: "memory");
      // L's 8 x 8 diagonal blocks (only this CTA reads or writes the diagonal block in this launch)
      if (ch == 0 && r < kb) {
        float2* row = p.A + (size_t)(nd * kT + (r & ~7)) * p.lda + nd * kT + r;
#pragma unroll
        for (int j = 0; j < 8; j++)
          if (j <= (r & 7)) row[(size_t)j * p.lda] = make_float2(bars->dg[r >> 3][r & 7][j], 0.f);
      }
    }
  }
  if (!ok) {
    atomicExch(p.err, 6);
    bars->failed = 1;
  }
  sm100::tc_fence_before();
  __syncthreads();
  if (!OWN && bars->again && !bars->failed) return true;
  if (warp == 1) sm100::tmem_dealloc(tmem, kCols);
  return false;
}

// ------------------------------------------------------------ tensor-core trailing update
// A_IJ -= L_I L_J^T for a run of up to `group` consecutive tiles per CTA
// (row-major order over the tile triangle, so consecutive tiles share I and
// the A operand stays in shared memory).  Warp-specialised, pipelined:
//   warp 0 (one lane)  bulk-async copies: the two A slices when I changes,
//                      the two B slices per tile in two K-halves (two
//                      32 KB stages), and an L2 prefetch of the double-float
//                      tile (BD_REST_PREFETCH);
//   warp 1 (one lane)  three FP16 products per K-half into one of four TMEM
//                      accumulators (128 columns each), tcgen05.commit to
//                      release stages, the accumulator and the A operand;
//   warps 2-9          epilogue: tcgen05.ld of the accumulator (warp w reads
//                      TMEM lanes 32 (w % 4) .. + 31, half of the columns),
//                      release it, then the double-float read-modify-write.
// So the next tile's copies and MMAs run under the current tile's epilogue.
// Every wait is bounded; a timeout records an error code and raises a
// shared abort flag that ends every role's loop; copies still in flight
// are waited for (bounded) and TMEM is freed before the CTA exits.
#ifndef BD_REST_PREFETCH
#define BD_REST_PREFETCH 0  // L2 prefetch of the double-float tile ahead of the epilogue (measured slower)
#endif
#ifndef BD_EPI_EVICT_FIRST
#define BD_EPI_EVICT_FIRST 1  // L2 evict-first hint on the epilogue's tile loads and stores
#endif
#ifndef BD_EPI_AHEAD
#define BD_EPI_AHEAD 8  // chunks of 8 columns whose old values are in flight per epilogue thread (4: 8 % slower bulk)
#endif
#ifndef BD_REST_GROUP
#define BD_REST_GROUP 0  // tiles per CTA; 0: from the tile count
#endif
#ifndef BD_REST_WAVES
#define BD_REST_WAVES 3  // from the tile count: about this many CTAs per SM ...
#endif
#ifndef BD_REST_GMIN
#define BD_REST_GMIN 1  // ... with at least / at most this many tiles each
#endif
#ifndef BD_REST_GMAX
#define BD_REST_GMAX 8
#endif
constexpr int kRestThreads = 320;
constexpr int kStageBytes = kTileSlices * kHalfBytes;  // one K-half of the two B slices
constexpr size_t kRestSmem = kPanelSmem;
static_assert(kRestSmem >= (size_t)kTileBytes + 2 * kStageBytes + 1024 + 512, "the update CTAs' operands");
constexpr int kAccCols = 128;

constexpr int kAccs = 4;       // accumulators in tensor memory (all of its columns)
constexpr int kFoldPanels = 3;  // panels summed into one of them (K = 384): longer sums truncate more
struct RestBars {
  uint64_t fullA, emptyA, fullB[2], emptyB[2], accFull[kAccs], accEmpty[kAccs], done;
};
struct Slices {
  const unsigned char* base;
  size_t buf;  // bytes of one buffer
  __device__ __forceinline__ const unsigned char* at(int p) const { return base + (size_t)(p % kBufs) * buf; }
};

// Tile t of an update job's enumeration, from column jlo:
//   kRowTri  the triangle I >= J >= jlo row by row (consecutive tiles share I),
//   kBlkTri  the same by super-columns of kSuper tile columns, each row by row
//            downward: the tiles in flight read the slices of 32 columns and a
//            few dozen rows, where six panels' slices of a whole row of a large
//            matrix are more than L2 holds (3N = 46,200: 142 MB; a schedule that
//            took 145 ms row by row took 139 so, 144 with 8 columns),
//   kCol     column jlo alone (I = jlo + t).
enum { kRowTri = 0, kCol = 1, kBlkTri = 2 };
constexpr int kSuper = 32;
__device__ __forceinline__ void rest_tile(int t, int jlo, int mode, int nt, int& I, int& J) {
  if (mode == kCol) {
    I = jlo + t;
    J = jlo;
    return;
  }
  int w = nt - jlo, j0 = jlo;  // rows below (and at) the super-column's first, its width
  if (mode == kBlkTri) {
    for (; w > kSuper; w -= kSuper, j0 += kSuper) {
      const int cnt = kSuper * (kSuper + 1) / 2 + (w - kSuper) * kSuper;
      if (t < cnt) break;
      t -= cnt;
    }
    w = min(w, kSuper);
    const int u = t - w * (w + 1) / 2;
    if (u >= 0) {  // below the super-column's triangle
      I = j0 + w + u / w;
      J = j0 + u % w;
      return;
    }
  }
  int Ip = (int)((sqrtf(8.f * (float)t + 1.f) - 1.f) * 0.5f);
  while ((Ip + 1) * (Ip + 2) / 2 <= t) Ip++;
  while (Ip * (Ip + 1) / 2 > t) Ip--;
  I = j0 + Ip;
  J = j0 + (t - Ip * (Ip + 1) / 2);
}

// `cta` is the CTA's index among the update CTAs.  Panels p0 .. p0 + npan - 1.
// NF = 0: one panel, the A operand resident per row of tiles.
// NF = 1, 2, 4: up to 3 NF consecutive panels' updates in one read-modify-write of
// the tile: both operands streamed in 2 npan chunks of 64 KB per tile (panel,
// K-half) through the two stages, three panels to an accumulator, NF of them
// subtracted from the tile one after the other (as NF passes would).
// Returns true, with nothing done but the tensor memory's allocation, where one of
// the panels has rows with scales of their own (own_update's).
template <int NF>
__device__ __forceinline__ bool rest_body(unsigned char* smraw, float2* A, int lda, int m, int jlo, int mode,
                                          int tlo, int thi, int group, int cta, const Slices& sl, int p0, int npan,
                                          int fold, int* err, float iscale2, const int* past) {
  // (loaded ahead of the set-up, looked at behind it.  Looked at by the roles, in
  // their loops, the compiler places the epilogue's loads worse: 119 against 122 ms
  // at 3N = 46,200; ahead of the body, 4 us a launch of a batch)
  int first;
  asm volatile("ld.global.u32 %0, [%1];" : "=r"(first) : "l"(past));
  // (rounded as an integer, not by align1024: with the pointer known to be
  // shared the compiler places the epilogue's loads worse, 211 against 161 ms
  // for the factorisation at 3N = 46,200)
  unsigned char* sm = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smraw) + 1023) & ~uintptr_t(1023));
  unsigned char* sA = sm;                 // 2 slices x 32 KB
  unsigned char* sB = sm + kTileBytes;    // 2 stages x (2 slices x 16 KB)
  RestBars* bars = reinterpret_cast<RestBars*>(sm + kTileBytes + 2 * kStageBytes);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(bars + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tslot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t0 = tlo + cta * group, t1 = min(t0 + group, thi);
  const int nt = cdiv_d(m, kT);

  if (threadIdx.x == 0) {
    sm100::mbar_init(&bars->fullA, 1);
    sm100::mbar_init(&bars->emptyA, 1);
    for (int h = 0; h < 2; h++) {
      sm100::mbar_init(&bars->fullB[h], 1);
      sm100::mbar_init(&bars->emptyB[h], 1);
    }
    for (int h = 0; h < kAccs; h++) {
      sm100::mbar_init(&bars->accFull[h], 1);
      sm100::mbar_init(&bars->accEmpty[h], 8);
    }
    sm100::mbar_init(&bars->done, 1);
    *abort_flag = 0;
    sm100::fence_mbar_init();
  }
  if (warp == 1) sm100::tmem_alloc(tslot, kAccs * kAccCols);
  sm100::tc_fence_before();
  __syncthreads();
  sm100::tc_fence_after();
  const uint32_t tmem = *tslot;
  if (first < p0 + npan) {
    bool own = false;
    for (int i = 0; i < npan; i++) own = own || past[1 + p0 + i] != 0;
    if (own) return true;
  }

  if (warp == 0) {
    if (lane == 0) {
      // ---------------- producer
      const unsigned char* PS = sl.at(p0);  // (NF = 0)
      if constexpr (NF == 0) {
      int curI = -1;
      uint32_t nA = 0, nfill[2] = {0, 0};
      bool ok = true;
      for (int t = t0; t < t1 && ok; t++) {
        int I, J;
        rest_tile(t, jlo, mode, nt, I, J);
        if (I != curI) {
          if (nA > 0) ok = sm100::mbar_wait(&bars->emptyA, (nA - 1) & 1, kWaitLimit);
          if (!ok || *abort_flag) break;
          sm100::mbar_arrive_expect_tx(&bars->fullA, kTileBytes);
          const unsigned char* g = PS + (size_t)I * kTileBytes;
          for (int s2 = 0; s2 < kTileSlices; s2++)
            sm100::bulk_g2s(sA + s2 * kSliceBytes, g + s2 * kSliceBytes, kSliceBytes, &bars->fullA);
          curI = I;
          nA++;
        }
        if (BD_REST_PREFETCH) {  // the tile's columns into L2 ahead of the epilogue
          const int rows = min(kT, lda - I * kT);
          const int jend = min(J * kT + kT, m);
          for (int gj = J * kT; gj < jend; gj++)
            sm100::prefetch_l2(A + (size_t)gj * lda + (size_t)I * kT, (uint32_t)rows * 8u);
        }
        for (int h = 0; h < 2 && ok; h++) {
          if (nfill[h] > 0) ok = sm100::mbar_wait(&bars->emptyB[h], (nfill[h] - 1) & 1, kWaitLimit);
          if (!ok || *abort_flag) {
            ok = false;
            break;
          }
          if (I == J) {
            sm100::mbar_arrive(&bars->fullB[h]);  // diagonal tile: B is the A operand
          } else {
            sm100::mbar_arrive_expect_tx(&bars->fullB[h], kStageBytes);
            const unsigned char* g = PS + (size_t)J * kTileBytes + h * kHalfBytes;
            for (int s2 = 0; s2 < kTileSlices; s2++)
              sm100::bulk_g2s(sB + h * kStageBytes + s2 * kHalfBytes, g + s2 * kSliceBytes, kHalfBytes,
                              &bars->fullB[h]);
          }
          nfill[h]++;
        }
      }
      if (!ok) {
        atomicExch(err, 3);
        *abort_flag = 1;
      }
      // copies still in flight land before the CTA exits
      for (int h = 0; h < 2; h++)
        if (nfill[h] > 0) (void)sm100::mbar_wait(&bars->fullB[h], (nfill[h] - 1) & 1, kWaitLimit);
      if (nA > 0) (void)sm100::mbar_wait(&bars->fullA, (nA - 1) & 1, kWaitLimit);
      } else {
        // chunk q = (panel p0 + (q >> 1), K-half q & 1) of both operands
        uint32_t nfill[2] = {0, 0};
        int ctot = 0;
        bool ok = true;
        for (int t = t0; t < t1 && ok; t++) {
          int I, J;
          rest_tile(t, jlo, mode, nt, I, J);
          const bool dg = I == J;
          for (int q = 0; q < 2 * npan; q++) {
            const int st = ctot & 1;
            if (nfill[st] > 0) ok = sm100::mbar_wait(&bars->emptyB[st], (nfill[st] - 1) & 1, kWaitLimit);
            if (!ok || *abort_flag) {
              ok = false;
              break;
            }
            const unsigned char* src = sl.at(p0 + (q >> 1));
            const int h = q & 1;
            unsigned char* sa = sm + st * (2 * kStageBytes);
            sm100::mbar_arrive_expect_tx(&bars->fullB[st], dg ? kStageBytes : 2 * kStageBytes);
            for (int s2 = 0; s2 < kTileSlices; s2++)
              sm100::bulk_g2s(sa + s2 * kHalfBytes, src + (size_t)I * kTileBytes + s2 * kSliceBytes + h * kHalfBytes,
                              kHalfBytes, &bars->fullB[st]);
            if (!dg)
              for (int s2 = 0; s2 < kTileSlices; s2++)
                sm100::bulk_g2s(sa + kStageBytes + s2 * kHalfBytes,
                                src + (size_t)J * kTileBytes + s2 * kSliceBytes + h * kHalfBytes, kHalfBytes,
                                &bars->fullB[st]);
            nfill[st]++;
            ctot++;
          }
        }
        if (!ok) {
          atomicExch(err, 3);
          *abort_flag = 1;
        }
        for (int h = 0; h < 2; h++)
          if (nfill[h] > 0) (void)sm100::mbar_wait(&bars->fullB[h], (nfill[h] - 1) & 1, kWaitLimit);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // ---------------- MMA issuer
      if constexpr (NF == 0) {
      const uint32_t idesc = sm100::idesc_f16_f32(128, 128);
      const int pa[3] = {1, 0, 0};  // (A slice, B slice) products, smallest first
      const int pb[3] = {0, 1, 0};
      int curI = -1;
      uint32_t nA = 0;
      bool ok = true;
      int n = 0;
      for (int t = t0; t < t1; t++, n++) {
        int I, J;
        rest_tile(t, jlo, mode, nt, I, J);
        if (*abort_flag) break;
        if (I != curI) {
          ok = sm100::mbar_wait(&bars->fullA, nA & 1, kWaitLimit);
          if (!ok) break;
          curI = I;
          nA++;
        }
        const int acc = n & 1;
        if (n >= 2) {
          ok = sm100::mbar_wait(&bars->accEmpty[acc], ((n >> 1) - 1) & 1, kWaitLimit);
          if (!ok) break;
        }
        sm100::tc_fence_after();
        const uint32_t d = tmem + (uint32_t)(acc * kAccCols);
        for (int h = 0; h < 2 && ok; h++) {
          ok = sm100::mbar_wait(&bars->fullB[h], n & 1, kWaitLimit);
          if (!ok) break;
          sm100::tc_fence_after();
#pragma unroll
          for (int p = 0; p < 3; p++) {
            const uint32_t aaddr = sm100::smem_u32(sA + pa[p] * kSliceBytes + h * kHalfBytes);
            const uint32_t baddr = (I == J) ? sm100::smem_u32(sA + pb[p] * kSliceBytes + h * kHalfBytes)
                                            : sm100::smem_u32(sB + h * kStageBytes + pb[p] * kHalfBytes);
#pragma unroll
            for (int kk = 0; kk < 4; kk++)
              sm100::mma_f16(d, sm100::desc_kmajor_sw128(aaddr + kk * 32), sm100::desc_kmajor_sw128(baddr + kk * 32),
                              idesc, (h | p | kk) != 0);
          }
          sm100::mma_commit(&bars->emptyB[h]);
        }
        if (!ok) break;
        sm100::mma_commit(&bars->accFull[acc]);
        int In = -1, Jn;
        if (t + 1 < t1) rest_tile(t + 1, jlo, mode, nt, In, Jn);
        if (In != I) sm100::mma_commit(&bars->emptyA);
      }
      if (!ok) {
        atomicExch(err, 4);
        *abort_flag = 1;
      }
      } else {
        const uint32_t idesc = sm100::idesc_f16_f32(128, 128);
        const int pa[3] = {1, 0, 0};
        const int pb[3] = {0, 1, 0};
        uint32_t nuse[2] = {0, 0};
        int ctot = 0, nacc = 0;  // chunks, accumulators used
        bool ok = true;
        for (int t = t0; t < t1 && ok; t++) {
          int I, J;
          rest_tile(t, jlo, mode, nt, I, J);
          if (*abort_flag) break;
          const bool dg = I == J;
          for (int f = 0; f < NF && ok; f++, nacc++) {
            const int q0 = 2 * fold * f, q1 = min(q0 + 2 * fold, 2 * npan), acc = nacc % kAccs;
            if (nacc >= kAccs) ok = sm100::mbar_wait(&bars->accEmpty[acc], (nacc / kAccs - 1) & 1, kWaitLimit);
            if (!ok) break;
            sm100::tc_fence_after();
            const uint32_t d = tmem + (uint32_t)(acc * kAccCols);
            for (int q = q0; q < q1; q++) {
              const int st = ctot & 1;
              ok = sm100::mbar_wait(&bars->fullB[st], nuse[st] & 1, kWaitLimit);
              if (!ok) break;
              sm100::tc_fence_after();
              const unsigned char* sa = sm + st * (2 * kStageBytes);
              const unsigned char* sb = dg ? sa : sa + kStageBytes;
#pragma unroll
              for (int p = 0; p < 3; p++) {
                const uint32_t aaddr = sm100::smem_u32(sa + pa[p] * kHalfBytes);
                const uint32_t baddr = sm100::smem_u32(sb + pb[p] * kHalfBytes);
#pragma unroll
                for (int kk = 0; kk < 4; kk++)
                  sm100::mma_f16(d, sm100::desc_kmajor_sw128(aaddr + kk * 32),
                                  sm100::desc_kmajor_sw128(baddr + kk * 32), idesc, ((q - q0) | p | kk) != 0);
              }
              sm100::mma_commit(&bars->emptyB[st]);
              nuse[st]++;
              ctot++;
            }
            if (!ok) break;
            sm100::mma_commit(&bars->accFull[acc]);
          }
        }
        if (!ok) {
          atomicExch(err, 4);
          *abort_flag = 1;
        }
      }
      // every MMA issued has finished before TMEM is freed
      sm100::mma_commit(&bars->done);
      (void)sm100::mbar_wait(&bars->done, 0, kWaitLimit);
    }
  } else {
    // ---------------- epilogue
    // Each thread owns one row of the tile and the warp's 64-column half, in
    // chunks of kEpC columns.  The old double-float values of kEpS chunks are
    // in flight at all times: a chunk's slot is refilled as soon as it has
    // been written back, with a later chunk of this tile or the matching
    // chunk of the next one, so the loads run ahead of the accumulator and
    // across tile boundaries.
    constexpr int kEpC = 8, kEpN = 64 / kEpC, kEpS = BD_EPI_AHEAD;
    static_assert(kEpN % kEpS == 0, "slots must divide the chunks");
    const int q = warp & 3, ch = (warp - 2) >> 2;
    // the tiles stream through L2 once per launch: marked first for eviction
    // (BD_EPI_EVICT_FIRST), so the panel slices and the next launch's column
    // stay resident
    const uint64_t pol = sm100::policy_evict_first();
    auto ld_tile = [&](const float2* a) { return BD_EPI_EVICT_FIRST ? sm100::ld_f2_hint(a, pol) : *a; };
    auto st_tile = [&](float2* a, float2 v) {
      if (BD_EPI_EVICT_FIRST) sm100::st_f2_hint(a, v, pol);
      else *a = v;
    };
    // columns [0, jcnt) of this thread's row of tile t are inside the matrix
    // and the lower triangle, at colp + j lda
    auto row_of = [&](int t, float2*& colp, int& jcnt) {
      int I, J;
      rest_tile(t, jlo, mode, nt, I, J);
      const int gi = I * kT + 32 * q + lane;
      const int cbase = J * kT + 64 * ch;
      const int jlim0 = (I == J) ? max(0, gi - cbase + 1) : 64;  // diagonal tile: columns <= gi
      jcnt = gi < m ? min(min(jlim0, 64), m - cbase) : 0;
      colp = A + (size_t)cbase * lda + gi;
    };
    float2 old[kEpS][kEpC];
    auto load_chunk = [&](float2 (&o)[kEpC], const float2* colp, int jcnt, int c) {
#pragma unroll
      for (int j = 0; j < kEpC; j++)
        o[j] = (kEpC * c + j < jcnt) ? ld_tile(colp + (size_t)(kEpC * c + j) * lda) : make_float2(0.f, 0.f);
    };
    float2* colp = A;
    int jcnt = 0;
    if (t0 < t1) {
      row_of(t0, colp, jcnt);
#pragma unroll
      for (int s2 = 0; s2 < kEpS; s2++) load_chunk(old[s2], colp, jcnt, s2);
    }
    int n = 0;
    for (int t = t0; t < t1; t++, n++) {
      const bool more = t + 1 < t1;
      float2* ncolp = A;
      int njcnt = 0;
      if (more) row_of(t + 1, ncolp, njcnt);
      // the tile's accumulators (NF = 0: two in turn)
      constexpr int kNF = NF ? NF : 1, kRing = NF ? kAccs : 2;
      bool ok = true;
#pragma unroll
      for (int f = 0; f < kNF; f++)
        ok = ok && sm100::mbar_wait(&bars->accFull[(kNF * n + f) % kRing], ((kNF * n + f) / kRing) & 1, kWaitLimit);
      if (!ok || *abort_flag) {
        if (!ok && lane == 0) {
          atomicExch(err, 5);
          *abort_flag = 1;
        }
        break;
      }
      sm100::tc_fence_after();
      const int acc = kNF * n % kRing;  // (the ring holds a whole number of tiles)
      const uint32_t ta = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(acc * kAccCols + 64 * ch);
#pragma unroll
      for (int c = 0; c < kEpN; c++) {
        const int s2 = c % kEpS;
#pragma unroll
        for (int f = 0; f < kNF; f++) {
          if (f > 0 && f * fold >= npan) continue;
          float v[kEpC];
          sm100::tmem_ld8(ta + f * kAccCols + kEpC * c, v);
#pragma unroll
          for (int j = 0; j < kEpC; j++) old[s2][j] = df_sub(old[s2][j], v[j] * iscale2);
        }
        if (c == kEpN - 1) {  // read out: hand them back to the MMA issuer
          sm100::tc_fence_before();
          __syncwarp();
          if (lane == 0)
#pragma unroll
            for (int e = 0; e < kNF; e++) sm100::mbar_arrive(&bars->accEmpty[acc + e]);
        }
#pragma unroll
        for (int j = 0; j < kEpC; j++)
          if (kEpC * c + j < jcnt) st_tile(colp + (size_t)(kEpC * c + j) * lda, old[s2][j]);
        if (c + kEpS < kEpN) load_chunk(old[s2], colp, jcnt, c + kEpS);
        else if (more) load_chunk(old[s2], ncolp, njcnt, c + kEpS - kEpN);
      }
      colp = ncolp;
      jcnt = njcnt;
    }
  }
  sm100::tc_fence_before();
  __syncthreads();
  if (warp == 1) sm100::tmem_dealloc(tmem, kAccs * kAccCols);
  return false;
}

static_assert(sizeof(RestBars) + 2 * sizeof(int) <= 256, "own_update's barriers lie behind them");

// The same tiles for panels with rows whose scales are their own (rowf: the
// common scale / theirs), one panel and one tile at a time.
__device__ __forceinline__ void own_update(unsigned char* smraw, float2* A, int lda, int m, int jlo, int mode, int t0,
                                        int t1, const Slices& sl, int p0, int npan, int* err, float iscale2,
                                        const float* rowf) {
  unsigned char* sm = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smraw) + 1023) & ~uintptr_t(1023));
  unsigned char* sB = sm + kTileBytes;
  RestBars* first = reinterpret_cast<RestBars*>(sB + 2 * kStageBytes);  // rest_body's
  uint32_t* tslot = reinterpret_cast<uint32_t*>(first + 1);
  uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<unsigned char*>(first) + 256);  // copies, products
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tslot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nt = cdiv_d(m, kT);
  if (threadIdx.x == 0) {
    sm100::mbar_init(&bars[0], 1);
    sm100::mbar_init(&bars[1], 1);
    *abort_flag = 0;
    sm100::fence_mbar_init();
  }
  __syncthreads();
  const uint32_t tmem = *tslot;  // (rest_body's)
  uint32_t ph = 0;
  bool ok = true;
#pragma unroll 1
  for (int t = t0; t < t1; t++) {
    int I, J;
    rest_tile(t, jlo, mode, nt, I, J);
#pragma unroll 1
    for (int p = p0; p < p0 + npan; p++, ph ^= 1) {
      if (threadIdx.x == 0) {
        const unsigned char* src = sl.at(p);
        sm100::mbar_arrive_expect_tx(&bars[0], I == J ? kTileBytes : 2 * kTileBytes);
        sm100::bulk_g2s(sm, src + (size_t)I * kTileBytes, kTileBytes, &bars[0]);
        if (I != J) sm100::bulk_g2s(sB, src + (size_t)J * kTileBytes, kTileBytes, &bars[0]);
        if (sm100::mbar_wait(&bars[0], ph, kWaitLimit)) {
          sm100::tc_fence_after();
          mma_tile(tmem, sm, I == J ? sm : sB, false);
        } else {  // the copies in flight land before the CTA exits
          ok = false;
          (void)sm100::mbar_wait(&bars[0], ph, kWaitLimit);
        }
        sm100::mma_commit(&bars[1]);
      }
      __syncwarp();
      ok = sm100::mbar_wait(&bars[1], ph, kWaitLimit) && ok;
      sm100::tc_fence_after();
      if (warp >= 2) {
        const int q = warp & 3, ch = (warp - 2) >> 2, r = I * kT + 32 * q + lane;
        const float* f = rowf + (size_t)(p % kBufs) * (nt * kT);
        const float fr = iscale2 * f[r];
#pragma unroll 1
        for (int c = 64 * ch; c < 64 * ch + 64; c += 8) {
          float v[8];
          sm100::tmem_ld8(tmem + ((uint32_t)(32 * q) << 16) + c, v);
#pragma unroll
          for (int j = 0; j < 8; j++) {
            const int col = J * kT + c + j;
            if (r < m && col <= r) {
              float2* a = A + (size_t)col * lda + r;
              *a = df_sub(*a, v[j] * (fr * f[col]));
            }
          }
          __syncwarp();
        }
      }
      if (!ok) *abort_flag = 1;
      sm100::tc_fence_before();
      __syncthreads();  // the operands and the accumulator are free
      if (*abort_flag) t = t1, p = p0 + npan;
    }
  }
  if (!ok) atomicExch(err, 5);
  if (warp == 1) sm100::tmem_dealloc(tmem, kAccs * kAccCols);
}

// An update job: tiles [tlo, thi) of an enumeration (rest_tile) from column
// jlo, panels p0 .. p0 + npan - 1, `group` tiles per CTA.
struct UpdJob {
  int p0, npan, fold, jlo, mode, tlo, thi, group, nctas;
};
constexpr int kJobs = 2;
struct StepArgs {
  PanelArgs pan;  // panel k and the chain's tile
  int ntile;      // tile CTAs: tile rows k + 2 .. k + 1 + ntile
  Slices sl;
  const float* rowf;  // [kBufs][nt kT] the rows' factors (PanelArgs) by slice buffer
  UpdJob job[kJobs];
};

// One launch per step.  CTA 0 is the chain CTA, CTAs 1 .. ntile solve the
// other tiles of panel k; then the CTAs of the update jobs in turn.
// The parts of one launch touch disjoint tiles and slice buffers.
__device__ __forceinline__ void chol_step_body(const StepArgs& a, int b, float4* smem4) {
  unsigned char* sm = reinterpret_cast<unsigned char*>(smem4);
  if (b == 0) {
    if (panel_body<true, false>(sm, a.pan)) {
      __syncthreads();  // (its flags are set anew)
      (void)panel_body<true, true>(sm, a.pan);
    }
    return;
  }
  b -= 1;
  if (b < a.ntile) {
    PanelArgs p = a.pan;
    p.tile = a.pan.k + 2 + b;
    if (panel_body<false, false>(sm, p)) {
      __syncthreads();
      (void)panel_body<false, true>(sm, p);
    }
    return;
  }
  b -= a.ntile;
  int jn = 0;
  while (jn < kJobs - 1 && b >= a.job[jn].nctas) b -= a.job[jn++].nctas;
  const UpdJob& j = a.job[jn];
  const PanelArgs& p = a.pan;
  bool own = false;  // rows with scales of their own
  auto run = [&](auto nf) {
    own = rest_body<decltype(nf)::value>(sm, p.A, p.lda, p.m, j.jlo, j.mode, j.tlo, j.thi, j.group, b, a.sl, j.p0, j.npan,
                                   j.fold, p.err, p.iscale2, p.past);
  };
  if (j.npan > 2 * j.fold) run(std::integral_constant<int, 4>{});
  else if (j.npan > j.fold) run(std::integral_constant<int, 2>{});
  else if (j.npan > 1) run(std::integral_constant<int, 1>{});
  else run(std::integral_constant<int, 0>{});
  if (own) {
    const int t0 = j.tlo + b * j.group;
    own_update(sm, p.A, p.lda, p.m, j.jlo, j.mode, t0, min(t0 + j.group, j.thi), a.sl, j.p0, j.npan, p.err, p.iscale2,
               a.rowf);
  }
}

__global__ void __launch_bounds__(kRestThreads, 1) k_chol_step(const __grid_constant__ StepArgs a) {
  extern __shared__ float4 smem4[];
  chol_step_body(a, (int)blockIdx.x, smem4);
}

// The same step for many independent factorisations in one launch (replicas
// of a batch): each runs its own schedule's step with args[r].  The nrep
// chain CTAs come first (they take longest), then factorisation r owns CTAs
// nrep + [off[r], off[r + 1]); the factorisations share no memory.
__global__ void __launch_bounds__(kRestThreads, 1) k_chol_step_multi(const StepArgs* __restrict__ args,
                                                                      const int* __restrict__ off, int nrep) {
  extern __shared__ float4 smem4[];
  int bid = (int)blockIdx.x;
  if (bid < nrep) {
    chol_step_body(args[bid], 0, smem4);
    return;
  }
  bid -= nrep;
  int lo = 0, hi = nrep;  // off[lo] <= bid < off[lo + 1]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (off[mid] <= bid) lo = mid;
    else hi = mid;
  }
  chol_step_body(args[lo], bid - off[lo] + 1, smem4);
}

}  // namespace

namespace bdk {

// Groups of panels that share one read-modify-write of the tiles right of them:
// `fold` panels to an accumulator (K = 128 fold, summed in FP32 tensor memory: 3
// while the trailing matrix is large, 2, then 1; at most max_pass), as many
// accumulators a tile as kGroup says for that fold, each subtracted from the tile
// by itself, so that the arithmetic is that of one pass per accumulator.  The
// bulk is bound by the tiles' read-modify-write (their loads and stores share the
// SM's L1 path with the products' operands, and HBM), the products alone would
// take half; a group's column updates beside its panels cost less.  One
// accumulator a pass: 3N = 11,700 5.04 ms, 24,300 27.2, 46,200 155, 24 fibers of
// 1,992 to 7,836 together 14.9; so: 4.6, 21.7, 122, 11.6.  (Three accumulators of
// three panels: 4.8 ms at 11,700; four of two: 11.0 and 4.7; the bulk of a group
// spread over the next group's launches: 131 at 46,200.)
constexpr int kGroup[4] = {0, 4, 3, 2};  // accumulators by fold
// tile rows right of a group (fewer accumulators at the end).  2, 4, 8, 12: 3N = 1,944
// 0.532, 0.535, 0.537, 0.545 ms; at 5,184 and above within 1 %
constexpr int kGroupMin = 4;
static_assert(kBufs > kGroup[1] && kBufs > 2 * kGroup[2] && kBufs > 3 * kGroup[3], "a group's panels and the next");
// the slice buffers, then two buffers for the inverse of a diagonal factor
// (W_k in buffer k & 1: read by the launch that writes W_k+1), then its factors,
// the rows' scales by slice buffer and a flag a panel (PanelArgs)
size_t mixed_panel_bytes(int m) {
  const size_t nt = cdiv(m, kT);
  return kBufs * nt * kTileBytes + 2 * (size_t)kTileBytes + 2 * kT * sizeof(float) + kBufs * nt * kT * sizeof(float) +
         (nt + 1) * sizeof(int);
}
int mixed_max_launches(int m) { return 2 * cdiv(m, kT) + 2; }
int mixed_tiles(int m) { return cdiv(m, kT); }

// Positive definite: |L_ij| <= sqrt(max D_ii), so the slices' largest value is
// put into [2^8, 2^9): values down to 2^-34 of it stay in the pair (FP16's
// smallest subnormal is 2^-24), and the tiles' own slices (scale^2 / 16 times the
// tensor) are at most 2^14.  A factor with replaced negative pivots has 2^7 of
// room, its tiles 2^2 to 2^4; rows past that: see Range above.  Radii that give no
// finite positive diagonal: 1.
float mixed_scale(double a1, const double* rad, int nrad) {
  double dmax = 0.0;
  for (int i = 0; i < nrad; i++) dmax = std::max(dmax, std::fabs(a1 / rad[i]));
  if (!(dmax > 0.0) || !std::isfinite(dmax)) return 1.f;
  int e = 0;
  std::frexp(std::sqrt(dmax), &e);  // sqrt(dmax) in [2^(e-1), 2^e)
  e = 9 - e;
  return std::ldexp(1.f, e > 60 ? 60 : (e < -60 ? -60 : e));
}

static bool g_attr_done = false;

int set_mixed_attributes() {
  if (g_attr_done) return 0;
  cudaError_t e = cudaFuncSetAttribute(k_chol_step, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRestSmem);
  if (e != cudaSuccess) return 1;
  e = cudaFuncSetAttribute(k_chol_step_multi, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRestSmem);
  if (e != cudaSuccess) return 1;
  g_attr_done = true;
  return 0;
}

// Tiles per CTA of the bulk update: enough CTAs to fill the GPU about three
// times over, at most gmax tiles each (8; 4 with six panels a pass, 1 % faster).
static int rest_group(int tiles, int gmax) {
  if (BD_REST_GROUP > 0) return BD_REST_GROUP;
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 1;
  }
  int g = tiles / (BD_REST_WAVES * sms);
  return g < BD_REST_GMIN ? BD_REST_GMIN : (g > gmax ? gmax : g);
}

// Right-looking with a lookahead of one panel, on one stream, one launch
// after the other; every launch is one k_chol_step: panel k's tiles solved and
// diagonal block k + 1 factored (the chain and tile CTAs, which apply panel
// k - 1's update to column k themselves) beside up to two update jobs.  Panel
// p's slices live in buffer p % kBufs, W_p in buffer p & 1.  Invariant before
// the launch of panel k + 1: panels <= k are solved, column k + 1 and diagonal
// block k + 2 hold the updates of panels < k, and the launch leaves diagonal
// block k + 2 to its chain CTA (which applies panels k and k + 1).
// Groups of g panels k .. k + g - 1 (kGroup) share one read-modify-write of the
// tiles right of them (K = 128 g):
//   launch k + i, i = 1 .. g - 1: panel k + i beside panels k .. k + i - 1 on
//     column k + i + 1 and on diagonal block k + i + 2;
//   launch k + g: panel k + g beside the group on the tiles right of column k + g.
// Returns the number of kernel launches.
// Lines of the panels an accumulator sums (fold), in tile rows right of its first
// panels.  A group costs launches that hold one chain and its column updates; it
// saves read-modify-writes of the rest, so it needs rows to save.  Measured:
//   two from 48, 32, 24, 16, 8 rows: 3N = 5,184 1.57, 1.54, 1.53, 1.52, 1.52 ms, 3,888 1.10,
//   1.10, 1.09, 1.09, 1.09 - flat below 32, where one panel an accumulator is also the
//   more accurate;
//   three from 96, 64, 40, 24 rows: 3N = 8,100 2.80, 2.81, 2.68, 2.66, 12,960 6.15, 5.74,
//   5.60, 5.57, 5,184 1.53, 1.53, 1.53, 1.50 - flat from 40 down, likewise.
#ifndef BD_PAIR_MIN
#define BD_PAIR_MIN 24  // two panels an accumulator while this many tile rows remain right of column k + 2
#endif
#ifndef BD_TRIPLE_MIN
#define BD_TRIPLE_MIN 40  // three panels an accumulator while this many tile rows remain right of column k + 3
#endif
namespace {
struct Job {
  int p0 = 0, npan = 0, fold = 1, jlo = 0, mode = kCol, tlo = 0, tiles = 0, group = 1;  // tiles: the enumeration's end
};
}  // namespace

// The launches of one factorisation: issued on st, or (plan != nullptr)
// only recorded with their grid sizes.
// max_pass (1..3): most panels an accumulator sums (K = 128 max_pass; a pass has
// up to four of them).  Fewer mean fewer FP32 accumulation steps in tensor
// memory per stored update and more subtractions from the double-float tile: 3
// is the fastest, 1 the most accurate.
static int potrf_mixed_impl(int m, double* A64, int lda, unsigned char* PS, int* negpiv, int* err, cudaStream_t st,
                            cudaEvent_t* kev, int* kev_pairs, double* kflop, double* kbytes,
                            std::vector<std::pair<StepArgs, int>>* plan, int max_pass, float scale) {
  float2* A = reinterpret_cast<float2*>(A64);  // double-float storage, 8 bytes per element
  const int nt = cdiv(m, kT);
  const size_t buf = (size_t)nt * kTileBytes;
  int L = 0, timed = 0;
  auto kb_of = [&](int k) { return (m - k * kT < kT) ? m - k * kT : kT; };
  auto psb = [&](int k) { return PS + (size_t)(k % kBufs) * buf; };
  unsigned char* Wb = PS + kBufs * buf;  // the inverses' slices
  float* wsc = reinterpret_cast<float*>(Wb + 2 * (size_t)kTileBytes);
  float* rowf = wsc + 2 * kT;
  // elements of the lower triangle in tile columns [j0, j1)
  auto elems = [&](int j0, int j1) {
    double e = 0.0;
    for (int J = j0; J < j1 && J < nt; J++) {
      const double cols = kb_of(J);
      e += cols * (double)(m - J * kT) - cols * (cols - 1) / 2;
    }
    return e;
  };
  // panels p .. p + npan - 1 on column J below its diagonal block (the chain CTA's)
  auto col_job = [&](int p, int J, int npan, int fold) {
    Job j;
    j.p0 = p, j.npan = npan, j.fold = fold, j.jlo = J, j.mode = kCol, j.tlo = 1, j.tiles = nt - J;
    return j;
  };
  auto diag_job = [&](int p, int J, int npan, int fold) {  // ... on diagonal block J alone
    Job j;
    j.p0 = p, j.npan = npan, j.fold = fold, j.jlo = J, j.mode = kCol, j.tiles = J < nt ? 1 : 0;
    return j;
  };
  // ... on the triangle from column jlo but its first diagonal block
  auto tri_job = [&](int p, int npan, int fold, int jlo) {
    Job j;
    const int n = nt - jlo;
    j.p0 = p, j.npan = npan, j.fold = fold, j.jlo = jlo, j.mode = npan > kFoldPanels ? kBlkTri : kRowTri, j.tlo = 1;
    j.tiles = n > 0 ? n * (n + 1) / 2 : 0;
    j.group = rest_group(j.tiles, npan > kFoldPanels ? 4 : BD_REST_GMAX);
    return j;
  };
  // panel k's tiles (k < 0: none) and diagonal block k + 1
  auto launch = [&](int k, const Job& j0, const Job& j1 = Job()) {
    StepArgs a{};
    PanelArgs& p = a.pan;
    p.A = A, p.lda = lda, p.m = m, p.k = k, p.tile = k < 0 ? -1 : k + 1;
    p.PSp = psb(k < 0 ? 0 : k), p.PSpre = k > 0 ? psb(k - 1) : nullptr;
    p.Wk = Wb + (size_t)(k & 1) * kTileBytes, p.wsc = wsc + kT * (k & 1);
    p.Wn = Wb + (size_t)((k + 1) & 1) * kTileBytes, p.wscn = wsc + kT * ((k + 1) & 1);
    p.rowk = rowf + (size_t)((k < 0 ? 0 : k) % kBufs) * nt * kT, p.rowp = rowf + (size_t)((k > 0 ? k - 1 : 0) % kBufs) * nt * kT;
    p.past = reinterpret_cast<int*>(rowf + (size_t)kBufs * nt * kT);
    p.negpiv = negpiv, p.err = err, p.scale = scale, p.iscale2 = 1.f / (scale * scale);
    a.ntile = k < 0 ? 0 : nt - k - 2;
    a.sl = Slices{PS, buf};
    a.rowf = rowf;
    const Job* js[kJobs] = {&j0, &j1};
    int grid = 1 + a.ntile;
    for (int q = 0; q < kJobs; q++) {
      const Job& j = *js[q];
      UpdJob& u = a.job[q];
      u.p0 = j.p0, u.npan = j.npan, u.fold = j.fold, u.jlo = j.jlo, u.mode = j.mode, u.tlo = j.tlo, u.thi = j.tiles, u.group = j.group;
      u.nctas = j.tiles > j.tlo ? cdiv(j.tiles - j.tlo, j.group) : 0;
      grid += u.nctas;
    }
    if (plan) {
      plan->emplace_back(a, grid);
      return;
    }
    if (kev) cudaEventRecord(kev[2 * timed], st);
    k_chol_step<<<grid, kRestThreads, kRestSmem, st>>>(a);
    if (kev) {
      cudaEventRecord(kev[2 * timed + 1], st);
      timed++;
    }
    L++;
    if (kbytes || kflop) {
      const double tile_fl = 3.0 * 2.0 * kT * kT * kT;
      double by = 16.0 * (double)(m - (k + 1) * kT) * (k < 0 ? kb_of(0) : kT);  // panel read and written back
      double fl = k < 0 ? 0.0 : tile_fl * (2.0 * (1 + a.ntile) + 2.0);        // the panel CTAs' own products
      for (int q = 0; q < kJobs; q++) {
        const Job& j = *js[q];
        if (j.tiles <= j.tlo) continue;
        by += 16.0 * (j.tiles == 1 ? 0.5 * kT * kb_of(j.jlo) : elems(j.jlo, j.mode == kCol ? j.jlo + 1 : nt));
        fl += tile_fl * (j.tiles - j.tlo) * j.npan;  // FP16 tensor work issued
      }
      if (kbytes) *kbytes += by;
      if (kflop) *kflop += fl;
    }
  };
  launch(-1, Job());             // diagonal block 0
  if (nt > 1) launch(0, Job());  // panel 0
  int k = 0;
  while (k + 2 < nt) {
    const int fold = max_pass >= 3 && nt - (k + 4) >= BD_TRIPLE_MIN ? 3
                     : max_pass >= 2 && nt - (k + 3) >= BD_PAIR_MIN ? 2
                                                                    : 1;
    int g = fold * kGroup[fold];
    while (g > fold && nt - (k + 1 + g) < kGroupMin) g -= fold;
    for (int i = 1; i < g; i++) launch(k + i, col_job(k, k + i + 1, i, fold), diag_job(k, k + i + 2, i, fold));
    launch(k + g, tri_job(k, g, fold, k + g + 1));
    k += g;
  }
  if (plan) return L;
  if (kev_pairs) *kev_pairs = timed;
  return L;
}

int potrf_mixed(int m, double* A64, int lda, unsigned char* PS, int* negpiv, int* err, cudaStream_t st,
                cudaEvent_t* kev, int* kev_pairs, double* kflop, double* kbytes, int max_pass, float scale) {
  return potrf_mixed_impl(m, A64, lda, PS, negpiv, err, st, kev, kev_pairs, kflop, kbytes, nullptr, max_pass, scale);
}

// Factorisations of a batch advanced together: launch i of the batch runs
// step i of every factorisation whose schedule has one, each in its own CTA
// range; the step arguments and CTA offsets of every launch are uploaded
// once (the matrices and buffers do not move).
#ifndef BD_BATCH_ALIGN
#define BD_BATCH_ALIGN 0
#endif
struct MixedBatch {
  std::vector<int> nrep_at, grid_at;
  std::vector<size_t> args_at, off_at;
  StepArgs* d_args = nullptr;
  int* d_off = nullptr;
  int nrep = 0;
};

MixedBatch* mixed_batch_create(int nrep, const int* m, double* const* A, const int* lda, unsigned char* const* PS,
                               int* const* negpiv, int* const* err, const float* scale, int max_pass) {
  std::vector<std::vector<std::pair<StepArgs, int>>> plans(nrep);
  size_t steps = 0;
  MixedBatch* b = new MixedBatch();
  b->nrep = nrep;
  for (int r = 0; r < nrep; r++) {
    potrf_mixed_impl(m[r], A[r], lda[r], PS[r], negpiv[r], err[r], nullptr, nullptr, nullptr, nullptr, nullptr,
                     &plans[r], max_pass, scale[r]);
    steps = std::max(steps, plans[r].size());
  }
  std::vector<StepArgs> args;
  std::vector<int> off;
  for (size_t i = 0; i < steps; i++) {
    b->args_at.push_back(args.size());
    b->off_at.push_back(off.size());
    int n = 0, total = 0;
    for (int r = 0; r < nrep; r++) {
      // replica r's schedule starts at launch `shift` (BD_BATCH_ALIGN 1: every
      // schedule ends with the last launch; 0: every one starts with the first)
      const size_t shift = BD_BATCH_ALIGN ? steps - plans[r].size() : 0;
      if (i < shift || i - shift >= plans[r].size()) continue;
      args.push_back(plans[r][i - shift].first);
      off.push_back(total);
      total += plans[r][i - shift].second - 1;  // its chain CTA is counted apart
      n++;
    }
    off.push_back(total);
    b->nrep_at.push_back(n);
    b->grid_at.push_back(n + total);
  }
  bool ok = cudaMalloc(&b->d_args, std::max<size_t>(1, args.size()) * sizeof(StepArgs)) == cudaSuccess &&
            cudaMalloc(&b->d_off, std::max<size_t>(1, off.size()) * sizeof(int)) == cudaSuccess &&
            cudaMemcpy(b->d_args, args.data(), args.size() * sizeof(StepArgs), cudaMemcpyHostToDevice) == cudaSuccess &&
            cudaMemcpy(b->d_off, off.data(), off.size() * sizeof(int), cudaMemcpyHostToDevice) == cudaSuccess;
  if (!ok) {
    mixed_batch_free(b);
    return nullptr;
  }
  return b;
}

int mixed_batch_run(const MixedBatch* b, cudaStream_t st) {
  int L = 0;
  for (size_t i = 0; i < b->grid_at.size(); i++) {
    k_chol_step_multi<<<b->grid_at[i], kRestThreads, kRestSmem, st>>>(b->d_args + b->args_at[i],
                                                                         b->d_off + b->off_at[i], b->nrep_at[i]);
    L++;
  }
  return L;
}

void mixed_batch_free(MixedBatch* b) {
  if (!b) return;
  if (b->d_args) cudaFree(b->d_args);
  if (b->d_off) cudaFree(b->d_off);
  delete b;
}

}  // namespace bdk


