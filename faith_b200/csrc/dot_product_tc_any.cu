// Weight part of the bound x bound dot product on the 5th-generation tensor cores (tcgen05 / TMEM), native layout, any
// Lx, Ly, Di and K and any row pitch (dot_product_tc.cu: the attention shapes with lengths that are multiples of 32).
//
//   z_lw[b,i,m,j] = sum_k  x_c ly - x_r |ly| + y_c lx - y_r |lx|          (Bounds.py:710-823 in
//   z_uw[b,i,m,j] = sum_k  x_c uy + x_r |uy| + y_c lx + y_r |lx|           centre/radius form)
//   x_c = (x_lw + x_uw)/2, x_r = (x_uw - x_lw)/2 at [b,i,m,k];  y_c, y_r at [b,j,m,k];
//   lx = x_l[b,i,k];  ly = y_l[b,j,k], uy = y_u[b,j,k]  (concretised operand ranges)
// With y_kmajor y is given as [b,k,m,j] (contraction axis first), which is how the value projection writes it: the context
// product then needs no transposed copy of V.
//
// One tile = one b, 32 values of i, 4 of m, 32 of j; k in chunks of 32.  It is made of two sums of 128 x 64:
//   X [(i,m)][side, j] = x_c [ly; uy]^T + x_r [-|ly|; |uy|]^T
//   Y [(j,m)][side, i] = y_c [lx; lx]^T + y_r [-|lx|; |lx|]^T
// and z = X + Y^T, where the transposition (j,m),i -> (i,m),j goes through shared memory in the epilogue.  (y_c lx^T and
// y_r |lx|^T once each, 32 columns wide, and combined in the epilogue: slower, 1.0 against 0.79 ms per encoder pass of the
// size below; instructions of 32 columns take the tensor core as long as those of 64.)
//
// Numerics: these shapes ran on CUDA cores with fp32 products before, and lose nothing here.  Every fp32 operand is split
// exactly into three bf16 parts, v = h + m + l (24 bits), and a product is evaluated as hh + (hm + mh) + (mm + hl + lh), the
// same number of instructions as three TF32 products, which keep 21 bits.  What is dropped is below 2^-23 of a product, the
// error class of an fp32 multiplication.  The tensor core truncates when it adds to an accumulator, so few instructions may
// add to one of full magnitude: X and Y have two accumulators each, added with round-to-nearest in the epilogue.  One
// chunk of k: centre and radius, the small products first.  More chunks (kMulti): hh and the small products.  Error
// against fp64 over the fp32 noise of the reference: 1.3 to 1.7 at K = 32 (CUDA cores 1.4 to 1.5), below the CUDA cores' at
// K = 512; 1.5 to 2.3 for short sums, K = 7 and 16 (CUDA cores 1.2 to 1.4).  As in every centre/radius product the error of
// either side is relative to the larger of |lw| and |uw|, where the CUDA cores' is relative to the side itself: it tells for
// weights whose gap is thousands of times their value, and such a bound says nothing any more.
//
// What bounds it: about 2.8 us per tile whatever the data, i.e. the SM's shared memory (raw tiles in and out, B operands,
// transposition, result: 3000 cycles of its 128 bytes per cycle) and the hand-overs between the roles; with full tiles of 32
// positions 0.85 of that is HBM time.  CUDA-core kernel: 9.5 us per tile.  24 sentences x 21 positions, dim_in 256:
// 389 -> 131 us (scores), 719 -> 128 us (context, which needed 260 us of transposed copies besides).
//
// A operands live in tensor memory, B operands in shared memory.  x and y have converters, planes, issuers and barriers of
// their own, so that one is converted while the other is multiplied.  The B planes depend on (b, i block, j block, k chunk)
// only, and a CTA walks a contiguous range of tiles, m fastest: they are rewritten once per 32 tiles of an attention head
// instead of per tile (for every tile: 4.0 us per tile).
//
// Operands whose rows are not a multiple of 16 bytes (an attention row of 21 positions) cannot go through TMA: the
// instantiations without kTmaIn fetch them with 4-byte cp.async, each warp the part it converts.  The result leaves through
// the transposition buffer in coalesced 16-byte stores (4-byte ones without kVecOut, for rows that are not 16-byte aligned).
//
// Warp roles (28 warps, one persistent CTA per SM):
//   warps 0, 1   MMA issuers of X (two accumulators); warp 0 is also the TMA producer      warps 2, 3   issuers of Y
//   warps 4-11   epilogue, one warp per tensor-memory lane quarter and side
//   warps 12-19  converters of x and of the ranges of y (4 lane quarters x 2 halves of the chunk); warps 20-27 of y and lx
// TMEM columns: [0,128) X, [128,256) Y, [256,352) planes of x, [352,448) planes of y (centre h, m, l, radius h, m, l of 16
// columns each).
// Every mbarrier wait is bounded; on expiry the kernel raises a device-side flag, drains, frees its
// tensor memory and returns.  No cluster launch and no multicast is used.
#include <cuda.h>

#include <mutex>
#include <unordered_map>

#include "common.cuh"
#include "dot_bias.cuh"

namespace fb {
int* tc_status_sink();   // matmul_tc.cu: the status word of the pass being enqueued, if any

namespace {

#include "tc_common.cuh"

constexpr int kDaConvWarps = 16, kDaEpiWarps = 8;
constexpr int kDaFirstEpiWarp = 4, kDaFirstConvWarp = kDaFirstEpiWarp + kDaEpiWarps;
constexpr int kDaThreads = 32 * (kDaFirstConvWarp + kDaConvWarps);
constexpr uint32_t kDaTile = 128 * 32 * 4;                                   // one 128-row x 32-k fp32 tile = 16 KB
constexpr uint32_t kDaRawXl = 0, kDaRawXu = kDaTile, kDaRawYl = 2 * kDaTile, kDaRawYu = 3 * kDaTile;
constexpr uint32_t kDaRawStage = 4 * kDaTile;                                // x_lw, x_uw, y_lw, y_uw
// B planes of one accumulator: 64 rows of three 128-byte tiles, two planes of 32 bf16 per row and tile:
// planes 0-2 = h, m, l of the signed operand, 3-5 = h, m, l of the signed absolute values
constexpr uint32_t kDaBTile = 64 * 128, kDaBSet = 3 * kDaBTile;              // 24 KB
constexpr uint32_t kDaOffB = 2 * kDaRawStage, kDaOffZ = kDaOffB + 2 * kDaBSet;
constexpr uint32_t kDaOffBars = kDaOffZ + 2 * kDaTile;                       // staging of the result: two sides of 128 x 32
constexpr uint32_t kDaSmemBytes = kDaOffBars + 1024 /*align*/ + 256 /*barriers*/;
static_assert(kDaSmemBytes <= 232448, "shared memory budget");
constexpr uint32_t kDaX = 0, kDaY = 128, kDaA = 256;                         // TMEM column map
constexpr uint32_t kDaIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(64 >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);

struct DotArgs {
  const float *x_lw, *x_uw, *y_lw, *y_uw;      // read directly when !kTmaIn
  const float *x_l, *y_l, *y_u;                // ranges, rows of K (y_ranges_kmajor: [b][k][j])
  float *z_lw, *z_uw;
  int Lx, Ly, Di, K, ldx, ldy, ldz;            // ld*: floats between consecutive m of x, y, z
  int n_ib, n_jb, n_mb, n_kc, total_tiles;
  int heads, y_kmajor, y_ranges_kmajor;
  float out_scale;
};

// The MMAs of one accumulator for one chunk.  kRole 0: of the centre (kMulti: the hh products of centre and radius), 1: of the
// radius (kMulti: the small products).  a: TMEM column of the operand's planes; b: descriptor (low word) of the B set.
// ksteps: 1 or 2 steps of 16 k.  kFirst: the first MMA overwrites the accumulator.
template <bool kMulti, int kRole, bool kFirst>
__device__ __forceinline__ void issue_chunk(uint32_t d, uint32_t a, uint32_t b, uint32_t b_hi, int ksteps) {
  constexpr uint32_t T = kDaBTile >> 4;
  const uint32_t bp[6] = {b, b + 4, b + T, b + T + 4, b + 2 * T, b + 2 * T + 4};   // h, m, l of the signed operand, of the absolute values
  constexpr int pa[6] = {2, 0, 1, 1, 0, 0}, pb[6] = {0, 2, 1, 0, 1, 0};            // lh, hl, mm, mh, hm, hh
#pragma unroll
  for (int t = 0; t < 6; ++t) {
    if (kMulti && (t == 5) != (kRole == 0)) continue;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      if (j < ksteps) {
#pragma unroll
        for (int cr = 0; cr < 2; ++cr) {
          if (!kMulti && cr != kRole) continue;
          if (kFirst && j == 0 && t == (kMulti && kRole == 0 ? 5 : 0) && cr == (kMulti ? 0 : kRole)) mma_bf16_ts<false>(d, a + 48 * cr + 16 * pa[t] + 8 * j, bp[3 * cr + pb[t]] + 2 * j, b_hi, kDaIdesc);
          else mma_bf16_ts<true>(d, a + 48 * cr + 16 * pa[t] + 8 * j, bp[3 * cr + pb[t]] + 2 * j, b_hi, kDaIdesc);
        }
      }
    }
  }
}

template <bool kTmaIn, bool kVecOut, bool kMulti>
__global__ void __launch_bounds__(kDaThreads, 1)
dot_weight_tc_any(const __grid_constant__ CUtensorMap tm_xl, const __grid_constant__ CUtensorMap tm_xu,
              const __grid_constant__ CUtensorMap tm_yl, const __grid_constant__ CUtensorMap tm_yu, const DotArgs A,
              int* __restrict__ status, const DotBias bias, int n_bias) {
  extern __shared__ uint8_t smem_raw[];
  const int grid = (int)gridDim.x - n_bias;   // blocks of the weight part; the rest take a tile of the bias part each
  if ((int)blockIdx.x >= grid) {
    pdl_sync();
    if (threadIdx.x < kDotBiasThreads) dot_bias_tile<8>(bias, (int)blockIdx.x - grid, reinterpret_cast<float*>(smem_raw));
    return;
  }
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t bar0 = base + kDaOffBars;
  const uint32_t bar_full = bar0 + 0;          // [2] raw stage loaded (kTmaIn)
  const uint32_t bar_raw_empty = bar0 + 16;    // [2] raw stage read by the converters (kTmaIn)
  const uint32_t bar_ops_ready = bar0 + 32;    // [2] operands of X, Y of the item converted
  const uint32_t bar_mma_done = bar0 + 48;     // [2] MMAs of X, Y of the item complete
  const uint32_t bar_acc_ready = bar0 + 64;    // accumulators of the tile complete
  const uint32_t bar_acc_free = bar0 + 72;     // accumulators read out
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(base_ptr + kDaOffBars + 128);
  volatile int* cta_abort = reinterpret_cast<volatile int*>(base_ptr + kDaOffBars + 136);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // tiles of this CTA: a contiguous range in the order (b, i block, j block, m block), m fastest
  const int first_tile = (int)((int64_t)blockIdx.x * A.total_tiles / grid);
  const int my_tiles = (int)((int64_t)(blockIdx.x + 1) * A.total_tiles / grid) - first_tile;
  const int n_kc = kMulti ? A.n_kc : 1;
  const int n_items = my_tiles * n_kc;   // item = chunk of a tile

  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(bar_full + 8 * s, 1);
      mbar_init(bar_raw_empty + 8 * s, kDaConvWarps);
      mbar_init(bar_ops_ready + 8 * s, kDaConvWarps / 2);
      mbar_init(bar_mma_done + 8 * s, 2);
    }
    mbar_init(bar_acc_ready, 4);
    mbar_init(bar_acc_free, kDaEpiWarps);
    *cta_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {  // one warp allocates all of tensor memory for this CTA
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_sync();

  // 16 columns of X or Y: the sum of its two accumulators
  auto load_acc = [](uint32_t addr, uint32_t (&v)[16]) {
    uint32_t w[16];
    tmem_ld16(addr, v);
    tmem_ld16(addr + 64, w);
    tmem_wait_ld();
#pragma unroll
    for (int i = 0; i < 16; i += 2) {
      const uint64_t sum = add2(pack2(v[i], v[i + 1]), pack2(w[i], w[i + 1]));
      v[i] = (uint32_t)sum;
      v[i + 1] = (uint32_t)(sum >> 32);
    }
  };

  // block coordinates of tile t of this CTA
  auto tile_coords = [&](int t, int& b, int& i0, int& j0, int& m0) {
    int r = first_tile + t;
    m0 = (r % A.n_mb) * 4; r /= A.n_mb;
    j0 = (r % A.n_jb) * 32; r /= A.n_jb;
    i0 = (r % A.n_ib) * 32;
    b = r / A.n_ib;
  };

  if (warp < kDaFirstEpiWarp) {
    // ------------------------------------------------------------------ MMA issuers; warp 0 also loads
    const int op = warp >> 1, role = warp & 1;   // operand (X, Y), accumulator
    const uint64_t dsc = smem_desc_sw128(base + kDaOffB + op * kDaBSet);
    const uint32_t b_lo = (uint32_t)dsc, b_hi = (uint32_t)(dsc >> 32);
    const uint32_t d = tmem_base + (op == 0 ? kDaX : kDaY) + 64 * role, a = tmem_base + kDaA + 96 * op;
    auto load = [&](int it) {   // warp 0: raw stage of item `it`
      int b, i0, j0, m0;
      tile_coords(it / n_kc, b, i0, j0, m0);
      if (lane == 0) {
        const int k0 = 32 * (it % n_kc);
        const uint32_t full = bar_full + 8 * (it & 1), dst = base + (it & 1) * kDaRawStage;
        mbar_arrive_expect_tx(full, kDaRawStage);
        tma_load_4d(dst + kDaRawXl, &tm_xl, k0, m0, i0, b, full);
        tma_load_4d(dst + kDaRawXu, &tm_xu, k0, m0, i0, b, full);
        const int y0 = A.y_kmajor ? j0 : k0, y2 = A.y_kmajor ? k0 : j0;
        tma_load_4d(dst + kDaRawYl, &tm_yl, y0, m0, y2, b, full);
        tma_load_4d(dst + kDaRawYu, &tm_yu, y0, m0, y2, b, full);
      }
      __syncwarp();
    };
    if (kTmaIn && warp == 0) {
      if (n_items > 0) load(0);
      if (n_items > 1) load(1);
    }
    bool ok = true;
    int t = 0, kc = 0;
    for (int it = 0; it < n_items; ++it) {
      if (kTmaIn && warp == 0 && it + 2 < n_items) {
        // (the converters read the raw stage before they finish the item)
        ok = mbar_wait_warp(bar_raw_empty + 8 * (it & 1), (uint32_t)((it >> 1) & 1), cta_abort);
        if (!ok) break;
        load(it + 2);
      }
      ok = mbar_wait_warp(bar_ops_ready + 8 * op, (uint32_t)(it & 1), cta_abort);
      // the first MMA of a tile overwrites the accumulator: the previous tile must have been read out
      if (ok && kc == 0 && t > 0) ok = mbar_wait_warp(bar_acc_free, (uint32_t)((t - 1) & 1), cta_abort);
      if (!ok) break;
      tc_fence_after();
      if (lane == 0) {
        const int ksteps = A.K - 32 * kc > 16 ? 2 : 1;
        if (kc == 0) {
          if (role == 0) issue_chunk<kMulti, 0, true>(d, a, b_lo, b_hi, ksteps);
          else issue_chunk<kMulti, 1, true>(d, a, b_lo, b_hi, ksteps);
        } else {
          if (role == 0) issue_chunk<kMulti, 0, false>(d, a, b_lo, b_hi, ksteps);
          else issue_chunk<kMulti, 1, false>(d, a, b_lo, b_hi, ksteps);
        }
        tc_commit(bar_mma_done + 8 * op);
        if (kc == n_kc - 1) tc_commit(bar_acc_ready);
      }
      __syncwarp();
      if (++kc == n_kc) { kc = 0; ++t; }
    }
  } else if (warp < kDaFirstConvWarp) {
    // ------------------------------------------------------------------ epilogue (warps 4-11)
    // Warp (quarter, side): first Y of its side, transposed into the staging buffer, then X of its side into registers; the
    // accumulators go back to the issuers before anything is stored, so that the MMAs of the next tile overlap the rest.
    const int quarter = warp & 3, side = (warp - kDaFirstEpiWarp) >> 2, row = quarter * 32 + lane;   // TMEM lane = accumulator row
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const uint64_t scale2 = pack2(__float_as_uint(A.out_scale), __float_as_uint(A.out_scale));
    uint8_t* const Z = base_ptr + kDaOffZ + side * kDaTile;
    auto meet = [&](bool fine) { return side == 0 ? meet_all<1, 128>(fine) : meet_all<2, 128>(fine); };
    for (int t = 0; t < my_tiles; ++t) {
      // (the warps of a side meet here, having stored the tile before, and settle whether one has given up)
      if (!meet(mbar_wait_warp(bar_acc_ready, (uint32_t)(t & 1), cta_abort))) break;
      tc_fence_after();
      {
        const int j = row >> 2, m = row & 3;   // row of Y
        uint8_t* const T = Z + (j & 3) * 4;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t v[16];
          load_acc(tmem_base + lane_addr + kDaY + 32 * side + 16 * h, v);
#pragma unroll
          for (int i = 0; i < 16; ++i) *reinterpret_cast<uint32_t*>(T + swz(4 * (16 * h + i) + m, j >> 2)) = v[i];
        }
      }
      uint32_t x[2][16];
      load_acc(tmem_base + lane_addr + kDaX + 32 * side, x[0]);
      load_acc(tmem_base + lane_addr + kDaX + 32 * side + 16, x[1]);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_acc_free);
      meet(true);
      // this thread's row (i, m) of the transposition buffer holds Y^T: the result takes its place
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        uint8_t* const z = Z + swz(row, q);
        ulonglong2 tv = *reinterpret_cast<const ulonglong2*>(z);
        const uint32_t* v = x[q >> 2] + 4 * (q & 3);
        tv.x = mul2(add2(pack2(v[0], v[1]), tv.x), scale2);
        tv.y = mul2(add2(pack2(v[2], v[3]), tv.y), scale2);
        *reinterpret_cast<ulonglong2*>(z) = tv;
      }
      int b, i0, j0, m0;
      tile_coords(t, b, i0, j0, m0);
      float* const z0 = (side == 0 ? A.z_lw : A.z_uw) + (((int64_t)(b / A.heads) * A.Lx + i0) * A.Di + m0) * A.ldz +
                        (b % A.heads) * A.Ly + j0;
      const int ni = min(32, A.Lx - i0), nm = min(4, A.Di - m0), nj = min(32, A.Ly - j0);
      meet(true);
      // coalesced stores: eight lanes per row (i, m), so a warp writes the four (mostly adjacent) rows of one i; or, for rows
      // that are not 16-byte aligned, a lane per value
      if (kVecOut) {
        const int m = lane >> 3, j = (lane & 7) * 4;
        for (int i = quarter; i < ni; i += 4) {
          if (m < nm && j < nj) {
            const float4 v = *reinterpret_cast<const float4*>(Z + swz(4 * i + m, lane & 7));
            float* const o = z0 + ((int64_t)i * A.Di + m) * A.ldz + j;
            if (j + 4 <= nj) {
              *reinterpret_cast<float4*>(o) = v;
            } else {
              o[0] = v.x;
              if (j + 1 < nj) o[1] = v.y;
              if (j + 2 < nj) o[2] = v.z;
            }
          }
        }
      } else {
        for (int i = quarter; i < ni; i += 4) {
#pragma unroll
          for (int m = 0; m < 4; ++m)
            if (m < nm && lane < nj)
              z0[((int64_t)i * A.Di + m) * A.ldz + lane] =
                  *reinterpret_cast<const float*>(Z + swz(4 * i + m, lane >> 2) + (uint32_t)(lane & 3) * 4u);
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ converters
    const int cw = warp - kDaFirstConvWarp;   // 0..15
    const int grp = cw >> 3;                   // 0: x tile, 1: y tile
    const int gt = (threadIdx.x - 32 * kDaFirstConvWarp) & 255;   // index within the group
    const int quarter = warp & 3;
    const int half = (cw >> 2) & 1;            // which 16 of the 32 k values
    const int row = quarter * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const bool gather = grp == 1 && A.y_kmajor != 0;   // tile [k][m][j] instead of [(j, m)][k]

    // !kTmaIn: this warp's part of item `it` (the 32 rows x 16 k it converts) into raw stage it & 1, zeros outside
    auto fetch = [&](int it) {
      if (it < n_items) {
        int b, i0, j0, m0;
        tile_coords(it / n_kc, b, i0, j0, m0);
        const int k0 = (it % n_kc) * 32 + half * 16;
        const uint32_t dst = base + (it & 1) * kDaRawStage + grp * 2 * kDaTile;
        const float* const gl = grp == 0 ? A.x_lw : A.y_lw;
        const float* const gu = grp == 0 ? A.x_uw : A.y_uw;
        const int L = grp == 0 ? A.Lx : A.Ly, ld = grp == 0 ? A.ldx : A.ldy, r0 = grp == 0 ? i0 : j0;
#pragma unroll 4
        for (int q = 0; q < 16; ++q) {
          uint32_t off;
          int64_t src;
          bool ok;
          if (gather) {
            const int k = k0 + q, m = lane >> 3, j = quarter * 8 + (lane & 7);
            off = swz((half * 16 + q) * 4 + m, j >> 2) + (uint32_t)(j & 3) * 4u;
            ok = k < A.K && m0 + m < A.Di && j0 + j < A.Ly;
            src = (((int64_t)b * A.K + k) * A.Di + m0 + m) * ld + j0 + j;
          } else {
            const int r = quarter * 32 + 2 * q + (lane >> 4), kk = half * 16 + (lane & 15), l = r0 + (r >> 2), m = m0 + (r & 3);
            off = swz(r, kk >> 2) + (uint32_t)(kk & 3) * 4u;
            ok = k0 + (lane & 15) < A.K && m < A.Di && l < L;
            src = (((int64_t)b * L + l) * A.Di + m) * ld + k0 + (lane & 15);
          }
          const int bytes = ok ? 4 : 0;   // 0: zero-filled, nothing is read
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst + off), "l"(gl + (ok ? src : 0)), "r"(bytes) : "memory");
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst + kDaTile + off), "l"(gu + (ok ? src : 0)), "r"(bytes) : "memory");
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (!kTmaIn) { fetch(0); fetch(1); }
    bool ok = true;
    int last_key = -1, t = 0, kc = 0;
    for (int it = 0; it < n_items && ok; ++it) {
      const int s = it & 1;
      if (kTmaIn) {
        ok = mbar_wait_warp(bar_full + 8 * s, (uint32_t)((it >> 1) & 1), cta_abort);
        if (!ok) break;
      } else {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
      }
      const uint8_t* tl = base_ptr + s * kDaRawStage + grp * 2 * kDaTile;
      const uint8_t* tu = tl + kDaTile;
      // (arithmetic on pairs of fp32 values, fma / mul / sub .f32x2: each half rounded as the scalar instruction rounds it)
      uint64_t c2[8], r2[8];
      if (gather) {
        const int j = row >> 2, m = row & 3;
#pragma unroll
        for (int kk = 0; kk < 16; kk += 2) {
          const uint32_t off0 = swz((half * 16 + kk) * 4 + m, j >> 2) + (uint32_t)(j & 3) * 4u;
          const uint32_t off1 = swz((half * 16 + kk + 1) * 4 + m, j >> 2) + (uint32_t)(j & 3) * 4u;
          const uint64_t lo = pack2(*reinterpret_cast<const uint32_t*>(tl + off0), *reinterpret_cast<const uint32_t*>(tl + off1));
          const uint64_t up = pack2(*reinterpret_cast<const uint32_t*>(tu + off0), *reinterpret_cast<const uint32_t*>(tu + off1));
          const uint64_t hu = mul2(up, kHalf2);
          c2[kk >> 1] = fma2(lo, kHalf2, hu);
          r2[kk >> 1] = fma2(lo, kMinusHalf2, hu);
        }
      } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint32_t off = swz(row, half * 4 + q);
          const ulonglong2 vl = *reinterpret_cast<const ulonglong2*>(tl + off);
          const ulonglong2 vu = *reinterpret_cast<const ulonglong2*>(tu + off);
          const uint64_t l2[2] = {vl.x, vl.y}, u2[2] = {vu.x, vu.y};
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const uint64_t hu = mul2(u2[i], kHalf2);
            c2[q * 2 + i] = fma2(l2[i], kHalf2, hu);
            r2[q * 2 + i] = fma2(l2[i], kMinusHalf2, hu);
          }
        }
      }
      // The raw stage goes back only when every value loaded from it has been used (a shared-memory load completes
      // asynchronously); the empty asm statements keep the arithmetic above from being moved below.
#pragma unroll
      for (int i = 0; i < 8; ++i) asm volatile("" : "+l"(c2[i]), "+l"(r2[i]));
      __syncwarp();
      if (kTmaIn) {
        if (lane == 0) mbar_arrive(bar_raw_empty + 8 * s);
      } else {
        fetch(it + 2);
      }
      const int key = ((first_tile + t) / A.n_mb) * n_kc + kc;
      const bool new_b = key != last_key;
      last_key = key;
      // split while the MMAs of the previous item still run
      uint32_t pl[6][8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        split_bf16_pair(c2[i], pl[0][i], pl[1][i], pl[2][i]);
        split_bf16_pair(r2[i], pl[3][i], pl[4][i], pl[5][i]);
      }
#pragma unroll
      for (int q = 0; q < 6; ++q)
#pragma unroll
        for (int i = 0; i < 8; ++i) asm volatile("" : "+r"(pl[q][i]));
      // the planes of this operand (A and B) are free when its MMAs of the previous item are complete
      if (it >= 1) ok = mbar_wait_warp(bar_mma_done + 8 * grp, (uint32_t)((it - 1) & 1), cta_abort);
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int q = 0; q < 6; ++q) tmem_st8(tmem_base + lane_addr + kDaA + grp * 96u + 16u * q + half * 8u, pl[q]);
      if (new_b) {
        // B planes of (b, i block, j block, k chunk): four consecutive k of one row per thread
        int b, i0, j0, m0;
        tile_coords(t, b, i0, j0, m0);
        const int quad = gt & 7, k0 = 32 * kc + 4 * quad;
        auto put = [&](int r, const uint32_t (&p)[3][2], uint32_t set_sign) {
          uint8_t* const dst = base_ptr + kDaOffB + grp * kDaBSet + (quad & 1) * 8;
#pragma unroll
          for (int q = 0; q < 3; ++q) {
            const uint32_t a0 = (p[q][0] & 0x7fff7fffu) | set_sign, a1 = (p[q][1] & 0x7fff7fffu) | set_sign;
            *reinterpret_cast<uint2*>(dst + (q >> 1) * kDaBTile + swz(r, (q & 1) * 4 + (quad >> 1))) = make_uint2(p[q][0], p[q][1]);
            *reinterpret_cast<uint2*>(dst + ((q + 3) >> 1) * kDaBTile + swz(r, ((q + 3) & 1) * 4 + (quad >> 1))) = make_uint2(a0, a1);
          }
        };
        // grp 0: X set, rows 0-31 the lower range of y (absolute values negated), rows 32-63 the upper range (two rows per
        // thread); grp 1: Y set, the lower range of x in both halves, absolute values negated in the first
        for (int r = gt >> 3; r < (grp == 0 ? 64 : 32); r += 32) {
          const int l = (grp == 0 ? j0 : i0) + (r & 31), L = grp == 0 ? A.Ly : A.Lx;
          const float* const src = grp == 1 ? A.x_l : r < 32 ? A.y_l : A.y_u;
          const bool km = grp == 0 && A.y_ranges_kmajor != 0;
          float v[4];
          uint32_t p[3][2];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int64_t o = km ? ((int64_t)b * A.K + k0 + e) * L + l : ((int64_t)b * L + l) * A.K + k0 + e;
            v[e] = l < L && k0 + e < A.K ? __ldg(src + o) : 0.f;
          }
#pragma unroll
          for (int e = 0; e < 2; ++e)
            split_bf16_pair(pack2(__float_as_uint(v[2 * e]), __float_as_uint(v[2 * e + 1])), p[0][e], p[1][e], p[2][e]);
          put(r, p, r < 32 ? 0x80008000u : 0u);
          if (grp == 1) put(r + 32, p, 0u);
        }
        fence_async_smem();   // written through the generic proxy; the MMA reads them through the async proxy
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_ops_ready + 8 * grp);
      if (++kc == n_kc) { kc = 0; ++t; }
    }
    if (!kTmaIn) asm volatile("cp.async.wait_all;" ::: "memory");
  }
  // Tear-down.  On the error path, give outstanding bulk copies time to land before the shared
  // memory is released (bounded), then free the tensor memory.
  if (*cta_abort) {
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    if (threadIdx.x == 0 && status != nullptr) atomicOr(status, 4);   // bit 2 of the caller's status word
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// ------------------------------------------------------------------------ host side

// [B][R][Di][C] fp32 with rows of C values `ld` floats apart: box 32 x 4 x 32 x 1 (C, Di, R, B)
bool make_in_map(CUtensorMap* map, const float* ptr, uint64_t C, uint64_t Di, uint64_t R, uint64_t B, uint64_t ld) {
  return get_map(map, MapKey{ptr, {C, Di, R, B, 1}, {ld * 4, Di * ld * 4, R * Di * ld * 4, 0}, {32, 4, 32, 1, 1}, 4});
}
template <bool kTmaIn, bool kVecOut, bool kMulti>
int launch_variant(const CUtensorMap (&tm)[4], const DotArgs& a, cudaStream_t st, const DotBias& bias, int n_bias) {
  const int sms = device_info().sms;
  if (int rc = ensure_dynamic_smem(dot_weight_tc_any<kTmaIn, kVecOut, kMulti>, kDaSmemBytes)) return rc;
  fb::launch_tiles(a.total_tiles, dot_weight_tc_any<kTmaIn, kVecOut, kMulti>, (unsigned)((a.total_tiles < sms ? a.total_tiles : sms) + n_bias), kDaThreads, kDaSmemBytes,
               st, tm[0], tm[1], tm[2], tm[3], a, tc_status_sink(), bias, n_bias);
  FB_LAUNCH_OK();
  return FB_OK;
}

}  // namespace

// The kernel counts tiles and k chunks in 32 bits; that is its only limit.
bool dot_tc_any_supported(int B, int Lx, int Ly, int Di, int K) {
  const int64_t tiles = (int64_t)B * ceil_div(Lx, 32) * ceil_div(Ly, 32) * ceil_div(Di, 4);
  return B >= 1 && tiles < (1ll << 31) && tiles * ceil_div(K, 32) < (1ll << 31) && encode_fn() != nullptr;
}

// ldx, ldy, ldz: floats between consecutive m of the operands and of the result (0: contiguous).  y_ranges_kmajor: y_l and y_u
// are [B, K, Ly] instead of [B, Ly, K].
int launch_dot_weight_tc_any(const float* x_lw, const float* x_uw, const float* y_lw, const float* y_uw, const float* x_l,
                         const float* y_l, const float* y_u, float* z_lw, float* z_uw, int B, int Lx, int Ly, int Di, int K,
                         float out_scale, int heads, int y_kmajor, int y_ranges_kmajor, int ldx, int ldz, cudaStream_t st,
                             const DotBias& bias, bool& bias_done) {
  DotArgs a = {x_lw, x_uw, y_lw, y_uw, x_l, y_l, y_u, z_lw, z_uw, Lx, Ly, Di, K, 0, 0, 0, 0, 0, 0, 0, 0, heads, y_kmajor,
               y_ranges_kmajor, out_scale};
  a.ldx = ldx > 0 ? ldx : K;
  a.ldy = y_kmajor ? Ly : K;
  a.ldz = ldz > 0 ? ldz : heads * Ly;
  a.n_ib = (int)ceil_div(Lx, 32);
  a.n_jb = (int)ceil_div(Ly, 32);
  a.n_mb = (int)ceil_div(Di, 4);
  a.n_kc = (int)ceil_div(K, 32);
  a.total_tiles = B * a.n_ib * a.n_jb * a.n_mb;
  // TMA needs rows that are multiples of 16 bytes and 16-byte aligned bases
  const bool tma_in = a.ldx % 4 == 0 && a.ldy % 4 == 0 && aligned16(x_lw) && aligned16(x_uw) && aligned16(y_lw) && aligned16(y_uw);
  const bool vec_out = a.ldz % 4 == 0 && (heads == 1 || Ly % 4 == 0) && aligned16(z_lw) && aligned16(z_uw);
  CUtensorMap tm[4] = {};
  if (tma_in) {
    const uint64_t yc = y_kmajor ? Ly : K, yr = y_kmajor ? K : Ly;
    if (!make_in_map(&tm[0], x_lw, K, Di, Lx, B, a.ldx) || !make_in_map(&tm[1], x_uw, K, Di, Lx, B, a.ldx) ||
        !make_in_map(&tm[2], y_lw, yc, Di, yr, B, a.ldy) || !make_in_map(&tm[3], y_uw, yc, Di, yr, B, a.ldy))
      return FB_ERR_CUDA;
  }
  // the bias part goes along where that leaves a block per SM (as in the kernel for lengths of 32)
  const int64_t bias_blocks = (int64_t)B * bias.n_it * bias.n_jt;
  bias_done = a.total_tiles + bias_blocks <= device_info().sms;
  const int n_bias = bias_done ? (int)bias_blocks : 0;
#define FB_DOT_VARIANT(I, O) return a.n_kc > 1 ? launch_variant<I, O, true>(tm, a, st, bias, n_bias) : launch_variant<I, O, false>(tm, a, st, bias, n_bias)
  if (tma_in && vec_out) FB_DOT_VARIANT(true, true);
  if (tma_in) FB_DOT_VARIANT(true, false);
  if (vec_out) FB_DOT_VARIANT(false, true);
  FB_DOT_VARIANT(false, false);
#undef FB_DOT_VARIANT
}

// Reads (and clears) this file's copy of the flag raised by an expired bounded wait.
int dot_tc_any_error_flag(int* flag) {
  int v = 0;
  FB_CUDA_OK(cudaMemcpyFromSymbol(&v, g_tc_error, sizeof(int)));
  if (v != 0) {
    const int zero = 0;
    FB_CUDA_OK(cudaMemcpyToSymbol(g_tc_error, &zero, sizeof(int)));
  }
  *flag = v;
  return FB_OK;
}

}  // namespace fb
