// The product of few rows (bias rows of a sentence, the pooler) as a device function: for the launch of its own
// (matmul_ffma.cu) and for the extra blocks that the tensor-core kernel takes along where its tiles leave SMs idle.
#pragma once
#include "common.cuh"

namespace fb {

// Few output tiles (the bias rows of a sentence, the pooler: M of 1 to a few hundred): the 128 x 128 tiles above would leave all
// but a handful of SMs idle, each walking K alone (32 x 128 x 128 on one block: 28 us, 32 x 512 -> 128: 99 us).  Here a
// block owns 8 rows x 32 columns and its eight warps split K, a contiguous part each: centre and radius of the rows are
// staged in shared memory and read as broadcasts, a lane owns one column and streams its part of that row of W with
// 128-bit loads (whole sectors), the eight partial sums of an output are added in warp order.  Bound by the latency of one
// pass over the operands: 4.0 us resp. 9.0 us at the sizes above.  The concretised range of the rows and the coefficients of a
// relaxation follow in the same launch where the caller wants them (two launches of 2 to 3 us each otherwise).
constexpr int kSmRows = 8, kSmCols = 32, kSmThreads = 256, kSmWarps = kSmThreads / 32, kSmChunk = 512;
constexpr uint32_t kSmSmem = sizeof(float) * (2 * kSmRows * kSmChunk + 2 * kSmWarps * kSmRows * kSmCols);

struct SmallProduct {   // (a_lo, a_up) [M, K] x W [N, K]^T + bias -> (c_lo, c_up) [M, N], split into heads where split_rows > 0
  const float *a_lo, *a_up, *W, *bias;
  float *c_lo, *c_up;
  int64_t M;
  int N, K, split_rows, split_d;
};

// Block (bx, by) of the product; threads 0 .. kSmThreads - 1.  VEC: K a multiple of four and 16-byte aligned operands.
template <bool VEC>
__device__ __forceinline__ void small_product_block(const SmallProduct& q, const RangeEpilogue& rg, int bx, int by, float* smem) {
  const float* __restrict__ a_lo = q.a_lo;
  const float* __restrict__ a_up = q.a_up;
  const float* __restrict__ W = q.W;
  const float* __restrict__ bias = q.bias;
  float* __restrict__ c_lo = q.c_lo;
  float* __restrict__ c_up = q.c_up;
  const int64_t M = q.M;
  const int N = q.N, K = q.K, split_rows = q.split_rows, split_d = q.split_d;
  float* const s_c = smem;                                  // [kSmRows][kSmChunk] centres
  float* const s_r = s_c + kSmRows * kSmChunk;              // radii
  float* const s_red = s_r + kSmRows * kSmChunk;            // [2][warps][rows][cols]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t m0 = (int64_t)bx * kSmRows;
  const int n = by * kSmCols + lane;
  const float* const wrow = W + (int64_t)(n < N ? n : N - 1) * K;   // (a column beyond N computes what is not stored)
  float sc[kSmRows], sr[kSmRows];
#pragma unroll
  for (int i = 0; i < kSmRows; ++i) { sc[i] = 0.f; sr[i] = 0.f; }
  for (int k0 = 0; k0 < K; k0 += kSmChunk) {
    const int kc = min(kSmChunk, K - k0), quads = (kc + 3) / 4;
    if (k0 > 0) __syncthreads();
    for (int f = tid; f < kSmRows * quads; f += kSmThreads) {
      const int i = f / quads, q = f % quads;
      const int64_t m = m0 + i;
      float lo[4] = {0.f, 0.f, 0.f, 0.f}, up[4] = {0.f, 0.f, 0.f, 0.f};
      if (m < M) {
        const float* pl = a_lo + m * K + k0 + 4 * q;
        const float* pu = a_up + m * K + k0 + 4 * q;
        if (VEC) {
          *reinterpret_cast<float4*>(lo) = __ldg(reinterpret_cast<const float4*>(pl));
          *reinterpret_cast<float4*>(up) = __ldg(reinterpret_cast<const float4*>(pu));
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (4 * q + e < kc) { lo[e] = __ldg(pl + e); up[e] = __ldg(pu + e); }
        }
      }
      float4 c, r;
      c.x = fmul(fadd(lo[0], up[0]), 0.5f); r.x = fmul(fsub(up[0], lo[0]), 0.5f);
      c.y = fmul(fadd(lo[1], up[1]), 0.5f); r.y = fmul(fsub(up[1], lo[1]), 0.5f);
      c.z = fmul(fadd(lo[2], up[2]), 0.5f); r.z = fmul(fsub(up[2], lo[2]), 0.5f);
      c.w = fmul(fadd(lo[3], up[3]), 0.5f); r.w = fmul(fsub(up[3], lo[3]), 0.5f);
      *reinterpret_cast<float4*>(s_c + i * kSmChunk + 4 * q) = c;
      *reinterpret_cast<float4*>(s_r + i * kSmChunk + 4 * q) = r;
    }
    __syncthreads();
    const int per = (quads + kSmWarps - 1) / kSmWarps;
    const int q_end = min(quads, (warp + 1) * per);
#pragma unroll 4
    for (int q = warp * per; q < q_end; ++q) {
      float w[4] = {0.f, 0.f, 0.f, 0.f};
      const float* pw = wrow + k0 + 4 * q;
      if (VEC) {
        *reinterpret_cast<float4*>(w) = __ldg(reinterpret_cast<const float4*>(pw));
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (4 * q + e < kc) w[e] = __ldg(pw + e);
      }
#pragma unroll
      for (int i = 0; i < kSmRows; ++i) {
        const float4 c = *reinterpret_cast<const float4*>(s_c + i * kSmChunk + 4 * q);
        const float4 r = *reinterpret_cast<const float4*>(s_r + i * kSmChunk + 4 * q);
        sc[i] = fmaf(c.x, w[0], sc[i]); sr[i] = fmaf(r.x, fabsf(w[0]), sr[i]);
        sc[i] = fmaf(c.y, w[1], sc[i]); sr[i] = fmaf(r.y, fabsf(w[1]), sr[i]);
        sc[i] = fmaf(c.z, w[2], sc[i]); sr[i] = fmaf(r.z, fabsf(w[2]), sr[i]);
        sc[i] = fmaf(c.w, w[3], sc[i]); sr[i] = fmaf(r.w, fabsf(w[3]), sr[i]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < kSmRows; ++i) {
    s_red[(warp * kSmRows + i) * kSmCols + lane] = sc[i];
    s_red[((kSmWarps + warp) * kSmRows + i) * kSmCols + lane] = sr[i];
  }
  __syncthreads();
  // thread (row i = warp, column = lane)
  const int64_t m = m0 + warp;
  if (m >= M || n >= N) return;
  float c = s_red[warp * kSmCols + lane], r = s_red[(kSmWarps * kSmRows + warp) * kSmCols + lane];
#pragma unroll
  for (int w = 1; w < kSmWarps; ++w) {
    c = fadd(c, s_red[(w * kSmRows + warp) * kSmCols + lane]);
    r = fadd(r, s_red[((kSmWarps + w) * kSmRows + warp) * kSmCols + lane]);
  }
  float lo = fsub(c, r), up = fadd(c, r);
  if (bias != nullptr) { lo = fadd(lo, bias[n]); up = fadd(up, bias[n]); }
  int64_t o = m * N + n, ot = o;
  if (split_rows > 0) {
    const int64_t g = m / split_rows, rr = m % split_rows, gh = g * (N / split_d) + n / split_d;
    o = (gh * split_rows + rr) * split_d + n % split_d;
    ot = (gh * split_d + n % split_d) * split_rows + rr;
  }
  c_lo[o] = lo;
  c_up[o] = up;
  if (rg.norm_lo == nullptr) return;
  const float lb = lo, ub = up;
  for (int w = 0; w < rg.words; ++w) {
    const int64_t at = (m * rg.words + w) * N + n;
    lo = fadd(lo, fmul(-rg.eps, __ldg(rg.norm_lo + at)));
    up = fadd(up, fmul(rg.eps, __ldg(rg.norm_up + at)));
  }
  rg.out_l[rg.transposed ? ot : o] = lo;
  rg.out_u[rg.transposed ? ot : o] = up;
  if (rg.op < 0) return;
  bool bad = false;
  const ColCoef k = relax_column(rg.op, lo, up, lb, ub, bad);
  if (rg.violation != nullptr && (bad || k.c_lu != 0.f || k.c_ul != 0.f)) atomicOr(rg.violation, bad ? 1 : 2);
  rg.k_l[m * N + n] = k.c_ll;
  rg.k_u[m * N + n] = k.c_uu;
  rg.r_lb[m * N + n] = k.nlb;
  rg.r_ub[m * N + n] = k.nub;
}

}  // namespace fb
