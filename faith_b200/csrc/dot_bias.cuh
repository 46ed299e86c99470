// Bias part of the dot product: a tile of it as a device function, for the launch of its own (dot_product.cu) and for the extra
// blocks that the kernels of the weight part take along where they leave SMs idle.
#pragma once
#include "common.cuh"

namespace fb {

constexpr int kDotBiasThreads = 256;   // threads of a block that work on a tile

// Tiled version of the bias part: one block per (b, RI i, 32 j) tile; the seven row tiles are staged in shared memory (row
// stride 33 floats: conflict-free both for the row-wise fill and for the column-wise reads), K in chunks of 32 whose global
// loads are issued before the arithmetic of the chunk before; a thread owns the outputs (warp + 8 c, lane),
// c = 0 .. RI / 8 - 1.  Same partial sums and the same final order of additions as dot_bias_kernel.  RI = 8 where 32-row
// tiles would leave SMs idle: the kernel is bound by the latency of one chunk, and four blocks of 32 rows (one sentence, four
// heads) took 7.5 us.
// y_kmajor: y_lb / y_ub are stored [b, k, j] instead of [b, j, k]; ranges_kmajor: y_l / y_u likewise.
struct DotBias {
  const float *x_lb, *x_ub, *y_lb, *y_ub, *x_l, *y_l, *y_u;
  float *z_lb, *z_ub;
  int Lx, Ly, K, n_it, n_jt, heads, y_kmajor, ranges_kmajor;
  float out_scale;
};
__host__ __device__ constexpr int dot_bias_smem_floats(int ri) { return (3 * ri + 4 * 32) * 33; }

template <int RI>
__device__ __forceinline__ void dot_bias_tile(const DotBias& q, int w, float* smem) {
  constexpr int C = RI / 8;
  float (*sx)[RI][33] = reinterpret_cast<float (*)[RI][33]>(smem);                  // x_lb, x_ub, x_l
  float (*sy)[32][33] = reinterpret_cast<float (*)[32][33]>(smem + 3 * RI * 33);    // y_lb, y_ub, y_l, y_u
  const int jt = w % q.n_jt; w /= q.n_jt;
  const int it = w % q.n_it;
  const int64_t b = w / q.n_it;
  const int i0 = it * RI, j0 = jt * 32;
  const int tid = threadIdx.x, warp = tid >> 5, j = tid & 31;
  float gl[C], gu[C], l1[C], l2[C], l3[C], l4[C], u1[C], u2[C], u3[C], u4[C];
#pragma unroll
  for (int c = 0; c < C; ++c) gl[c] = gu[c] = l1[c] = l2[c] = l3[c] = l4[c] = u1[c] = u2[c] = u3[c] = u4[c] = 0.f;
  float vx[3][C], vy[4][4];
  auto load = [&](int k0) {
    const float* const xs[3] = {q.x_lb, q.x_ub, q.x_l};
    const float* const ys[4] = {q.y_lb, q.y_ub, q.y_l, q.y_u};
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const int r = warp + 8 * c;
        vx[a][c] = (i0 + r < q.Lx && k0 + j < q.K) ? xs[a][((int64_t)b * q.Lx + i0 + r) * q.K + k0 + j] : 0.f;
      }
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const bool km = a < 2 ? q.y_kmajor != 0 : q.ranges_kmajor != 0;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int hi = warp + 8 * c, r = km ? j : hi, k = km ? hi : j;   // the fast index is the contiguous one
        const int64_t idx = km ? ((int64_t)b * q.K + k0 + k) * q.Ly + j0 + r : ((int64_t)b * q.Ly + j0 + r) * q.K + k0 + k;
        vy[a][c] = (j0 + r < q.Ly && k0 + k < q.K) ? ys[a][idx] : 0.f;
      }
    }
  };
  load(0);
  for (int k0 = 0; k0 < q.K; k0 += 32) {
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int c = 0; c < C; ++c) sx[a][warp + 8 * c][j] = vx[a][c];
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const bool km = a < 2 ? q.y_kmajor != 0 : q.ranges_kmajor != 0;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int hi = warp + 8 * c;
        sy[a][km ? j : hi][km ? hi : j] = vy[a][c];
      }
    }
    __syncthreads();
    if (k0 + 32 < q.K) load(k0 + 32);
#pragma unroll 4
    for (int k = 0; k < 32; ++k) {
      const float yl = sy[0][j][k], yu = sy[1][j][k], ly = sy[2][j][k], uy = sy[3][j][k];
      const float lyp = ly > 0.f ? ly : 0.f, lyn = ly < 0.f ? ly : 0.f;
      const float uyp = uy > 0.f ? uy : 0.f, uyn = uy < 0.f ? uy : 0.f;
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const float xl = sx[0][warp + 8 * c][k], xu = sx[1][warp + 8 * c][k], lx = sx[2][warp + 8 * c][k];
        const float lxp = lx > 0.f ? lx : 0.f, lxn = lx < 0.f ? lx : 0.f;
        gl[c] = fadd(gl[c], fmul(-ly, lx));
        gu[c] = fadd(gu[c], fmul(-uy, lx));
        l1[c] = fmaf(xl, lyp, l1[c]); l2[c] = fmaf(xu, lyn, l2[c]); l3[c] = fmaf(yl, lxp, l3[c]); l4[c] = fmaf(yu, lxn, l4[c]);
        u1[c] = fmaf(xu, uyp, u1[c]); u2[c] = fmaf(xl, uyn, u2[c]); u3[c] = fmaf(yu, lxp, u3[c]); u4[c] = fmaf(yl, lxn, u4[c]);
      }
    }
    __syncthreads();
  }
  if (j0 + j >= q.Ly) return;
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const int i = i0 + warp + 8 * c;
    if (i < q.Lx) {
      // heads > 1: head-merged output [S, Lx, heads * Ly]
      const int64_t od = (((b / q.heads) * q.Lx + i) * q.heads + b % q.heads) * q.Ly + j0 + j;
      q.z_lb[od] = fmul(fadd(fadd(fadd(fadd(gl[c], l1[c]), l2[c]), l3[c]), l4[c]), q.out_scale);
      q.z_ub[od] = fmul(fadd(fadd(fadd(fadd(gu[c], u1[c]), u2[c]), u3[c]), u4[c]), q.out_scale);
    }
  }
}

}  // namespace fb
