// Split-sign product of bounds with a constant weight on the 5th-generation tensor cores, large problems: fp32 values
// as two fp16 parts under power-of-two scales, one accumulator per side, tiles of 128 x 128.
//
//   y_c = c W^T,  y_r = r |W|^T,  y_lw = y_c - y_r,  y_uw = y_c + y_r,
//   c = (x_lw + x_uw)/2,  r = (x_uw - x_lw)/2          (centre/radius form of Bounds.py:403-412)
//
// What bounds it, and why this form.  The TF32 kernel of matmul_tc.cu holds four accumulators, so a tile has 64 columns and
// the rows of x are fetched and converted again for every 64 columns of W; TMA delivers 28 bytes per cycle and SM from L2, and
// that traffic is what its products of 1 M rows wait for (K = 512 -> N = 128: 1.28 MB per 128 rows = 46 800 of the 48 700
// cycles measured).  fp16 parts take half the bytes of TF32 parts and their products half the tensor time: a tile has 128 columns,
// half the fetches and half the conversions.
//
// The product is formed transposed, y^T = W x^T: the parts of W are the A operand, in tensor memory (for good while K <= 128), the
// parts of x the B operand, in shared memory.  A lane of tensor memory is then an output feature and a column a row of x, so the
// epilogue's 32 lanes write 128 contiguous bytes of a row straight from registers and the column norms over dim_in are sums within
// a lane.  (The other way round a lane holds a row: its stores go through shared memory and bulk copies, and the read-out of the
// accumulators, which the products of the next tile wait for, took 5 000 to 8 700 cycles a tile in three forms; stores of single
// sectors from registers took 15 000.)
//
// Numerics.  A row of x is scaled by a power of two that puts its largest |x_lw|, |x_uw| just below 2^15, a row of W
// likewise; both exact, undone by one multiplication in the epilogue.  A scaled value v is hi = fp16(v) and lo = fp16(v - hi),
// both rounded to nearest: what is lost is below 2^-23 |v| or 2^-25 (2^-40 of the row's largest value), whichever is more,
// against 2^-20 |v| for the two truncated TF32 parts.  The dropped product lo * lo is below 2^-22 and of either sign.  The tensor
// core truncates when it adds into its accumulator, at K = 16 per instruction here: 24 additions for K = 128, of which the first
// eight are of the small cross terms, where the TF32 kernel has 16 of main terms.  Relative error against fp64 (2-norm, normal x,
// radii uniform to 1): 128 -> 128 8.6e-7 with the TF32 kernel, 6.1e-7 here; 512 -> 128 3.5e-6 and 2.7e-6.
//
// K > 128 (kStream).  W is converted in slices of 64 through a ring of two, by the epilogue's warps, and every further instruction
// that adds to an accumulator costs another truncation: the cross terms get accumulators of their own, for which there is room with
// 64 rows at a time (two halves of a tile one after the other).  A row's scale has to be chosen from its first 128 values: it puts
// their largest below 2^4, which leaves eleven binades for the rest of the row.  A row that needs more (or begins with zeros only)
// marks its tile; the CTA computes marked tiles again at the end, with the largest value of the whole rows read beforehand.
//
// Warps: 0 and 3 TMA producers (raw fp32 tiles of x_lw and x_uw, 32 columns of k each, into a ring), 1 and 2 MMA issuers (centre, radius: no
// accumulator is shared, so the results do not depend on how the two interleave), 4-11 epilogue, 12-27 converters (a lane a row, a
// group of warps a k-block in turn: it holds its 32 columns in registers while the largest value of every row is found, so the raw
// tiles are free again at once).
// Tensor memory: [0, 256) accumulators, [256, 512) two slices of 64 k: {W_hi, W_lo, |W|_hi, |W|_lo} x 2 k-blocks.
//
// A CTA keeps to one chunk of up to 128 columns of W and walks row tiles; the CTAs of all chunks walk the same rows at the same
// time, so x comes from HBM once.  Every wait is bounded as in matmul_tc.cu; no cluster, no multicast.

namespace hg {

constexpr int BM = 128, BK = 32, kSlice = 64;
constexpr int kEpiWarps = 8, kConvWarps = 16;
constexpr int kFirstEpi = 4, kFirstConv = 12, kThreads = 896, kWarps = kThreads / 32;
// What differs where W is streamed (K > 128): 64 rows at a time, two of them to a tile.
template <bool kStream> struct Cfg {
  static constexpr int rows = kStream ? 64 : 128;          // rows of x per accumulator
  static constexpr int subs = BM / rows;
  static constexpr int row_warps = rows / 32;              // converter warps of a group: a lane a row
  static constexpr int groups = kConvWarps / row_warps;    // converter groups: group b takes the k-blocks kb = b (mod groups)
  static constexpr uint32_t raw_bytes = rows * BK * 4;     // one line of a k-block
  static constexpr uint32_t plane_bytes = rows * kSlice * 2;   // one part of a slice of x
  static constexpr uint32_t slice_bytes = 4 * plane_bytes;     // c_hi, -c_lo, r_hi, -r_lo
  static constexpr int x_ring = kStream ? 4 : 2;           // slices of x in shared memory
  static constexpr int raw_ring = kStream ? 10 : 5;        // raw tiles in flight
};
// Shared memory.
template <bool kStream> struct Smem {
  using T = Cfg<kStream>;
  static constexpr uint32_t x = 0, raw = T::x_ring * T::slice_bytes;
  static constexpr uint32_t bars = raw + T::raw_ring * T::raw_bytes;   // 512 bytes: barriers, tensor-memory address, abort flag
  static constexpr uint32_t winv = bars + 512;               // float[128]: 1 / scale of a row of W
  static constexpr uint32_t coef = winv + 512;               // [converter groups][2 lines][32] slopes (kCoef)
  static constexpr uint32_t row_max = coef + T::groups * 256;   // uint8 [2][converter groups][rows]: exponents
  static constexpr uint32_t inv = row_max + 1024;            // float [4][128]: 1 / scale of a row of x
  static constexpr uint32_t rare = inv + 2048;               // uint8 [4][4 row warps]: a very large 1 / scale among them
  static constexpr uint32_t bits = rare + 16;                // 1024 bits, one per tile of this CTA (live, kPoint; marked, kStream)
  static constexpr uint32_t part = bits + 128;               // kNorm: float [2 tiles][2 halves of the rows][2 lines][128 columns]
  static constexpr uint32_t bytes = part + 4096;
  static_assert(bytes <= 232448, "shared memory of an SM");
};
constexpr int kBitTiles = 1024;
constexpr uint32_t kColW = 256;

// exponent field of half a row's scale: largest value below 2^15 (kTop) or, where more of the row is to come, below 2^4
constexpr int kTop = 267, kFirst = 256, kMaxField = 252;

// Bounded wait of a whole warp.  Two dozen warps wait most of the time, and every poll takes issue slots from the few that work: a
// try of the hardware lasts about 170 cycles, so the loop around it is kept to four instructions, and the clock and the abort flag
// are looked at after every 32 tries.  (With a time hint a try is itself a loop of polls and sleeps of some twenty instructions.)
__device__ __forceinline__ bool wait_warp(uint32_t bar, uint32_t parity, const WaitCtx& wc) {
  long long t0 = 0;
  for (;;) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .u32 n;\n\t"
        "mov.u32 n, 32;\n\t"
        "AGAIN:\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "@p bra OUT;\n\t"
        "sub.u32 n, n, 1;\n\t"
        "setp.ne.u32 p, n, 0;\n\t"
        "@p bra AGAIN;\n\t"
        "OUT:\n\t"
        "mov.u32 %0, n;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    if (__all_sync(0xffffffffu, ok != 0)) return true;
    const long long t = clock64();
    if (t0 == 0) t0 = t;
    if (__any_sync(0xffffffffu, *wc.cta_abort != 0 || t - t0 > (long long)wc.tries * (kTryNs * 2))) break;   // (about two cycles a nanosecond)
  }
  if (!*wc.cta_abort) {
    *wc.cta_abort = 1;
    atomicExch(&g_tc_error, 1);
  }
  __syncwarp();
  return false;
}
__device__ __forceinline__ void mbar_arrive_n(uint32_t bar, uint32_t n) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(n) : "memory");
}
__device__ __forceinline__ void mma_f16_ts(uint32_t d, uint32_t a, uint32_t b_lo, uint32_t b_hi, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 bd;\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "mov.b64 bd, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], bd, %4, {%5, %5, %5, %5}, p;\n\t}"
      ::"r"(d), "r"(a), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(0u), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const float* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ float lo_f(uint64_t v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float hi_f(uint64_t v) { return __uint_as_float((uint32_t)(v >> 32)); }
// two scaled fp32 values -> their fp16 parts, element 0 in the low half
__device__ __forceinline__ void split_f16_pair(uint64_t v, uint32_t& hi, uint32_t& lo) {
  float h0, h1;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(hi) : "f"(hi_f(v)), "f"(lo_f(v)));
  asm("{\n\t.reg .b16 a, b;\n\tmov.b32 {a, b}, %2;\n\tcvt.f32.f16 %0, a;\n\tcvt.f32.f16 %1, b;\n\t}" : "=f"(h0), "=f"(h1) : "r"(hi));
  const uint64_t r = sub2(v, pack2(__float_as_uint(h0), __float_as_uint(h1)));
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(lo) : "f"(hi_f(r)), "f"(lo_f(r)));
}
// the same with -lo in place of lo (fp16 minus fp32 in one instruction; the products with it negate their operand B)
__device__ __forceinline__ void split_f16_pair_neg(uint64_t v, uint32_t& hi, uint32_t& nlo) {
  float r0, r1;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(hi) : "f"(hi_f(v)), "f"(lo_f(v)));
  asm("{\n\t.reg .b16 a, b;\n\tmov.b32 {a, b}, %2;\n\tsub.rn.f32.f16 %0, a, %3;\n\tsub.rn.f32.f16 %1, b, %4;\n\t}"
      : "=f"(r0), "=f"(r1) : "r"(hi), "f"(lo_f(v)), "f"(hi_f(v)));
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(nlo) : "f"(r1), "f"(r0));
}
constexpr uint32_t kNegateB = 1u << 14;   // instruction descriptor
// the parts of |w| from those of w: lo takes the sign away that hi has
__device__ __forceinline__ void abs_parts(uint32_t hi, uint32_t lo, uint32_t& ahi, uint32_t& alo) {
  ahi = hi & 0x7fff7fffu;
  alo = lo ^ (hi & 0x80008000u);
}
__device__ __forceinline__ uint64_t dup2(float v) { return pack2(__float_as_uint(v), __float_as_uint(v)); }
__device__ __forceinline__ float exp_float(int field) { return __uint_as_float((uint32_t)field << 23); }
__device__ __forceinline__ int exp_field(float v) { return (int)((__float_as_uint(v) >> 23) & 255u); }
__device__ __forceinline__ int clamp_field(int f) { return f < 1 ? 1 : f > kMaxField ? kMaxField : f; }

template <int R>
__device__ __forceinline__ void reg_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R)); }
template <int R>
__device__ __forceinline__ void reg_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R)); }

struct Args {
  const float *a_lo, *a_up;    // operand (read directly for marked tiles only), and that of the bias rows
  const float *b_lo, *b_up;
  const float* W;
  float *c_lo, *c_up, *cb_lo, *cb_up;
  const float *bias, *bias_b;  // layer bias of the first segment and of the bias rows, either may be null
  int64_t M, Mb;
  int N, K, chunk, chunks;     // columns of W per CTA (a multiple of 32), number of chunks
  int main_tiles, total_tiles; // row tiles: the first segment's, all
  int split_rows, split_d;
  const float *coef_l, *coef_u;
  int coef_di;
  float *norm_lo, *norm_up;
  int norm_p;
  const float *res_lo, *res_up, *bres_lo, *bres_up;
  int* status;
  uint32_t wait_tries;
  int skip_it;                 // self-test of the give-up path only, -1 otherwise
  LiveRows live;
};

// Registers per thread after the split: what the launch was given (72 each) is dealt out and not exceeded.  With a residual the
// epilogue holds the next eight rows of it.
template <bool kResid> struct Regs {
  static constexpr int conv = 80, epi = kResid ? 80 : 72, ctrl = kResid ? 24 : 40;
  static_assert(512 * conv + 256 * epi + 128 * ctrl <= 72 * kThreads, "registers");
};

// parts of 16 values of a row of W to tensor memory
__device__ __forceinline__ void put_w16(const float* v, float scale, uint32_t col, bool radius) {
  uint32_t hi[8], lo[8];
  const uint64_t s = dup2(scale);
#pragma unroll
  for (int i = 0; i < 8; ++i) split_f16_pair(mul2(pack2(__float_as_uint(v[2 * i]), __float_as_uint(v[2 * i + 1])), s), hi[i], lo[i]);
  tmem_st8(col, hi);
  tmem_st8(col + 16, lo);
  if (radius) {
#pragma unroll
    for (int i = 0; i < 8; ++i) abs_parts(hi[i], lo[i], hi[i], lo[i]);
    tmem_st8(col + 32, hi);
    tmem_st8(col + 48, lo);
  }
}
// 32 bytes: a lane reads a row of its own, so the sector is the unit that counts
__device__ __forceinline__ void ldg_f8(const float* p, float* v) {
  asm volatile("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]) : "l"(p));
}

template <bool kStream, bool kCoef, bool kNorm, bool kResid, bool kPoint>
__global__ void __launch_bounds__(kThreads, 1)
split_sign_gemm_f16(const __grid_constant__ CUtensorMap tm_lo, const __grid_constant__ CUtensorMap tm_up,
                    const __grid_constant__ CUtensorMap tm_b_lo, const __grid_constant__ CUtensorMap tm_b_up,
                    const __grid_constant__ Args p) {
  using T = Cfg<kStream>;
  using SM = Smem<kStream>;
  constexpr int kRows = T::rows, kSubs = T::subs, kGroups = T::groups, kPasses = kStream ? 2 : 1, kLines = kPoint ? 1 : 2;
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t base = smem_u32(smem);
  if ((base & 1023u) != 0) {   // (dynamic shared memory starts at a multiple of 1024; the swizzled tiles rely on it)
    if (threadIdx.x == 0) atomicExch(&g_tc_error, 1);
    return;
  }
  const uint32_t bar0 = base + SM::bars;
  // A wait by parity is only right where the waiting warp has seen every phase before.  A k-block's arrival is therefore
  // signalled to the converter group that takes it, not per stage: a group meets a stage's phases with gaps.
  const uint32_t bar_full = bar0, bar_empty = bar0 + 64;             // [groups] converter groups; [raw_ring] raw tiles
  const uint32_t bar_ready = bar0 + 144, bar_done = bar0 + 176;      // [x_ring] slices of x in shared memory
  const uint32_t bar_acc_ready = bar0 + 208, bar_acc_free = bar0 + 216;
  const uint32_t bar_max = bar0 + 224;                               // [row_warps]: largest values of the rows
  const uint32_t bar_scale = bar0 + 256;                             // [4]: scales for the epilogue
  const uint32_t bar_w = bar0 + 296;                                 // [2] slices of W
  const uint32_t bar_all = bar0 + 312, bar_scan = bar0 + 320;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem + SM::bars + 400);
  volatile int* cta_abort = reinterpret_cast<volatile int*>(smem + SM::bars + 404);
  float* const winv_max = reinterpret_cast<float*>(smem + SM::bars + 408);
  float* const winv = reinterpret_cast<float*>(smem + SM::winv);
  uint32_t* const bits = reinterpret_cast<uint32_t*>(smem + SM::bits);

  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // (uniform, and known to be)
  const int N = p.N, K = p.K;
  const int nkb = (K + BK - 1) / BK, ns = (nkb + 1) / 2;             // k-blocks and slices of a tile
  const int chunk_i = (int)blockIdx.x % p.chunks, r0_tile = (int)blockIdx.x / p.chunks;
  const int step = ((int)gridDim.x - chunk_i + p.chunks - 1) / p.chunks;   // CTAs of this chunk
  const int my_tiles = r0_tile < p.total_tiles ? (p.total_tiles - r0_tile + step - 1) / step : 0;
  const int n0 = chunk_i * p.chunk;
  const int ncols = min(p.chunk, N - n0);                            // columns this CTA computes
  const int kbx = nkb < kGroups ? nkb : kGroups;                     // converter groups that have work
  const int kbs = nkb < 4 ? nkb : 4;                                 // k-blocks that a row's scale is chosen from

  const bool use_live = kPoint && kNorm && p.live.L > 0;
  auto live_slow = [&](int tile) -> bool {
    if (tile >= p.main_tiles) return true;   // bias rows are never known to be zero
    const unsigned bl = ((unsigned)tile * (unsigned)BM) / (unsigned)p.live.Di;
    const int l = (int)(bl % (unsigned)p.live.L), b = (int)(bl / (unsigned)p.live.L);
    bool live = false;
#pragma unroll
    for (int w = 0; w < 4; ++w)
      if (w < p.live.words)
        live |= (p.live.inst_pos != nullptr ? __ldg(p.live.inst_pos + b * p.live.words + w) : p.live.pos[w]) == l;
    return live;
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < T::x_ring; ++s) {
      mbar_init(bar_ready + 8 * s, 2 * T::row_warps);
      mbar_init(bar_done + 8 * s, 2);
    }
    for (int s = 0; s < 2; ++s) mbar_init(bar_w + 8 * s, kStream ? 8 : 4 * kbx);
    for (int s = 0; s < T::raw_ring; ++s) mbar_init(bar_empty + 8 * s, T::row_warps);
    for (int b = 0; b < kGroups; ++b) mbar_init(bar_full + 8 * b, kLines);
    for (int q = 0; q < 4; ++q) {
      mbar_init(bar_max + 8 * q, kbx);
      mbar_init(bar_scale + 8 * q, T::row_warps);
    }
    mbar_init(bar_acc_ready, 2);
    mbar_init(bar_acc_free, kEpiWarps);
    mbar_init(bar_all, kWarps);
    mbar_init(bar_scan, kConvWarps);
    *cta_abort = 0;
    *winv_max = 0.f;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x < kBitTiles / 32) bits[threadIdx.x] = 0;
  if (warp == 1) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), 512);
    tmem_relinquish();
  }
  __syncthreads();
  pdl_sync();   // (everything above needs nothing of the launches before)

  const bool live_map = use_live && !kStream && my_tiles <= kBitTiles;
  if (live_map) {
    for (int w = threadIdx.x; w < (my_tiles + 31) / 32; w += blockDim.x) {
      uint32_t b = 0;
      for (int k = 0; k < 32; ++k) {
        const int ti = w * 32 + k;
        if (ti < my_tiles && live_slow(r0_tile + ti * step)) b |= 1u << k;
      }
      bits[w] = b;
    }
  }
  // whether tile ti of this CTA is computed in this pass
  auto takes = [&](int pass, int ti) -> bool {
    if (kStream && pass == 1) return (bits[(ti & (kBitTiles - 1)) >> 5] >> (ti & 31)) & 1u;
    if (!use_live) return true;
    if (live_map) return (bits[ti >> 5] >> (ti & 31)) & 1u;
    return live_slow(r0_tile + ti * step);
  };

  // ---- scales of the rows of W (a warp per row)
  for (int n = warp; n < 128; n += kWarps) {
    float m = 0.f;
    if (n < ncols)
      for (int k = lane * 4; k < K; k += 128) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(p.W + (int64_t)(n0 + n) * K + k));
        m = fmaxf(fmaxf(m, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w)));
      }
    m = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(m)));
    if (lane == 0) {
      const float wi = exp_float(254 - min(max(268 - exp_field(m), 1), 253));
      winv[n] = wi;
      atomicMax(reinterpret_cast<int*>(winv_max), __float_as_int(wi));
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const WaitCtx wc = {cta_abort, p.wait_tries};

  // ---- parts of W: 32 k of one row per lane (the row of this warp's lane quarter of tensor memory), and their parts to slot ws
      const int wrow = (warp & 3) * 32 + lane;   // of W: the row of this warp's lane quarter of tensor memory
      const float wscale = exp_float(254 - exp_field(winv[wrow]));
      const float* const wr = p.W + (int64_t)(n0 + wrow) * K;
      const bool wide = K % 8 == 0 && (reinterpret_cast<uintptr_t>(p.W) & 31) == 0;
      auto load_w = [&](int kb, float (&v)[32]) {
        if (wide) {
  #pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int k = kb * BK + i * 8;
            if (wrow < ncols && k < K) {
              ldg_f8(wr + k, v + 8 * i);
            } else {
  #pragma unroll
              for (int e = 0; e < 8; ++e) v[8 * i + e] = 0.f;
            }
          }
        } else {
  #pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int k = kb * BK + i * 4;
            const float4 w = wrow < ncols && k < K ? __ldg(reinterpret_cast<const float4*>(wr + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
            v[4 * i] = w.x; v[4 * i + 1] = w.y; v[4 * i + 2] = w.z; v[4 * i + 3] = w.w;
          }
        }
      };
      auto put_w = [&](int kb, int ws, const float (&v)[32]) {
        const uint32_t col = tmem + ((uint32_t)((warp & 3) * 32) << 16) + kColW + ws * 128 + (kb & 1) * 64;
        put_w16(v, wscale, col, !kPoint);
        put_w16(v + 16, wscale, col + 8, !kPoint);
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
      };

  // between the passes of kStream: every warp has finished its tiles
  auto meet = [&]() -> bool {
    __syncwarp();
    if (lane == 0) mbar_arrive(bar_all);
    return wait_warp(bar_all, 0, wc);
  };
  if (warp < kFirstEpi) {
    reg_dec<Regs<kResid>::ctrl>();
    if (warp == 0 || (warp == 3 && kLines == 2)) {
      // ---------------------------------------------------------------- TMA producers, one per line
      // (a wait and an issue take 300 cycles and more: one warp for both lines was what K = 512 waited for)
      const int line = warp == 0 ? 0 : 1;
      int it = 0;
      bool ok = true;
      for (int pass = 0; pass < kPasses && ok; ++pass) {
        for (int ti = 0; ti < my_tiles && ok; ++ti) {
          if (!takes(pass, ti)) continue;
          const int tile = r0_tile + ti * step;
          const bool bseg = tile >= p.main_tiles;
          const bool coef = kCoef && !bseg && line == 0;
          const CUtensorMap* const map = line == 0 ? (bseg ? &tm_b_lo : &tm_lo) : (bseg ? &tm_b_up : &tm_up);
          for (int u = 0; u < kSubs && ok; ++u) {
            const int m0 = (bseg ? tile - p.main_tiles : tile) * BM + u * kRows;
            const int64_t rb = kCoef && !bseg ? (int64_t)m0 / p.coef_di : 0;
            for (int kb = 0; kb < nkb; ++kb, ++it) {
              const int grp = kb % kGroups;
              const uint32_t full = bar_full + 8 * grp;
              const unsigned n = (unsigned)(it * kLines + line), e = n % T::raw_ring, round = n / T::raw_ring;
              // The group's barrier (and its slopes) may be used again when the group has read its k-block before this one; the wait for
              // the ring entry covers that only where it is far enough back: with two k-blocks to a tile it is the one before the last.
              const int prev = it - kb + (kb >= kGroups ? kb - kGroups : kb + (nkb - 1 - kb) / kGroups * kGroups - nkb);
              if (prev >= 0 && prev >= it - T::raw_ring / kLines) {
                const unsigned pn = (unsigned)(prev * kLines + line);
                ok = wait_warp(bar_empty + 8 * (pn % T::raw_ring), pn / T::raw_ring & 1u, wc);
              }
              if (ok && round > 0) ok = wait_warp(bar_empty + 8 * e, (round - 1) & 1u, wc);
              if (!ok) break;
              if (lane == 0 && !(blockIdx.x == 0 && it == p.skip_it)) {
                mbar_arrive_expect_tx(full, T::raw_bytes + (coef ? 256u : 0u));
                if (coef) {
                  const uint32_t cd = base + SM::coef + grp * 256;
                  bulk_load(cd, p.coef_l + rb * K + kb * BK, 128, full);
                  bulk_load(cd + 128, p.coef_u + rb * K + kb * BK, 128, full);
                }
                tma_load_2d(base + SM::raw + e * T::raw_bytes, map, kb * BK, m0, full);
              }
              __syncwarp();
            }
          }
        }
        if (kStream && ok && pass == 0) ok = meet();
      }
    } else if (warp < 3) {
      // ------------------------------------------------------------------ MMA issuers
      const int role = warp - 1;   // 0: centre, 1: radius
      const bool idle = kPoint && role == 1;
      const uint64_t bdesc = smem_desc_sw128(base + SM::x + role * 2 * T::plane_bytes);
      const uint32_t b_hi = (uint32_t)(bdesc >> 32);
      constexpr uint32_t idesc = (1u << 4) | ((uint32_t)(kRows >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
      const uint32_t d = tmem + role * 128, dc = kStream ? d + 64 : d;   // main terms, cross terms
      bool ok = true;
      int sc = 0, lt = 0;
      // the four steps of 16 k of slice sl (ring slot ar of x, slot ws of W): the small cross terms or the main one
      auto issue = [&](int sl, int ar, int ws, bool small) {
        const int nst = min(4, (K - sl * kSlice + 15) >> 4);
        const uint32_t a0 = tmem + kColW + ws * 128 + role * 32, b0 = (uint32_t)bdesc + ((ar * T::slice_bytes) >> 4);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (j < nst) {
            const uint32_t a = a0 + (j >> 1) * 64 + (j & 1) * 8, b = b0 + j * 2;
            if (small) {
              mma_f16_ts(dc, a, b + (T::plane_bytes >> 4), b_hi, idesc | kNegateB, (sl | j) != 0);   // W_hi (-(-lo))
              mma_f16_ts(dc, a + 16, b, b_hi, idesc, 1);                                             // W_lo hi
            } else {
              mma_f16_ts(d, a, b, b_hi, idesc, !kStream || (sl | j) != 0);
            }
          }
        }
      };
      if (!kStream) ok = wait_warp(bar_w, 0, wc);
      for (int pass = 0; pass < kPasses && ok; ++pass) {
        for (int ti = 0; ti < my_tiles && ok; ++ti) {
          if (!takes(pass, ti)) continue;
          for (int u = 0; u < kSubs && ok; ++u) {
            for (int sl = 0; sl < ns; ++sl) {
              const int g = sc + sl, ar = g % T::x_ring, ws = kStream ? g & 1 : sl;
              ok = wait_warp(bar_ready + 8 * ar, (uint32_t)(g / T::x_ring) & 1u, wc);
              if (kStream && ok) ok = wait_warp(bar_w + 8 * ws, (uint32_t)(g >> 1) & 1u, wc);
              if (ok && sl == 0 && lt > 0) ok = wait_warp(bar_acc_free, (uint32_t)(lt - 1) & 1u, wc);
              if (!ok) break;
              tc_fence_after();
              if (lane == 0) {
                if (!idle) {
                  issue(sl, ar, ws, true);
                  issue(sl, ar, ws, false);
                }
                tc_commit(bar_done + 8 * ar);
                if (sl == ns - 1) tc_commit(bar_acc_ready);
              }
              __syncwarp();
            }
            sc += ns;
            ++lt;
          }
        }
        if (kStream && ok && pass == 0) ok = meet();
      }
    } else if (kStream) {
      meet();
    }
  } else if (warp < kFirstConv) {
    // ------------------------------------------------------------------ epilogue (warps 4-11)
    // Warp (q, h): output features n0 + 32 q + lane, half h of the rows, eight at a time.
    if (kResid) reg_inc<Regs<kResid>::epi>();
    const int q = warp & 3, h = (warp - kFirstEpi) >> 2, et = (int)threadIdx.x - 32 * kFirstEpi;
    const int n = q * 32 + lane, gn = n0 + n;
    const bool valid = n < ncols;
    const float wv = winv[n];
    const bool rare_w = *winv_max > 7.0e19f;
    // (with norms the epilogue's warps meet once a tile, and whether one has given up is settled there: a meeting has no limit)
    auto agree = [&](bool fine) { return kNorm ? meet_all<1, 32 * kEpiWarps>(fine) : fine; };
    bool ok = true;
    int lt = 0;
    // kStream: these warps also convert W, the two of a lane quarter a k-block in turn: they wait for the accumulators most of the time.
    // Of every part of a tile the first two slices are given before the part before it is read out, which the products wait for anyway.
    auto give_w = [&](int g0, int from, int to) -> bool {   // slices from .. to - 1 of the part whose slices begin at g0
      for (int sl = from; sl < to; ++sl) {
        const int kb = 2 * sl + h, g = g0 + sl;
        if (kb >= nkb) break;
        float v[32];
        load_w(kb, v);   // (on their way during the wait)
        if (g >= 2) {    // the products of slice g - 2 have read this slot
          if (!wait_warp(bar_done + 8 * ((g - 2) % T::x_ring), (uint32_t)((g - 2) / T::x_ring) & 1u, wc)) return false;
          tc_fence_after();
        }
        put_w(kb, g & 1, v);
        if (lane == 0) mbar_arrive_n(bar_w + 8 * (g & 1), h == 0 && kb == nkb - 1 ? 2 : 1);
      }
      return true;
    };
    if (kStream) ok = agree(give_w(0, 0, 2));
    for (int pass = 0; pass < kPasses && ok; ++pass) {
      for (int ti = 0; ti < my_tiles && ok; ++ti) {
        const bool live = takes(pass, ti);
        if (!live && (!use_live || pass == 1)) continue;
        const int tile = r0_tile + ti * step;
        const bool bseg = tile >= p.main_tiles;
        const int my = (bseg ? tile - p.main_tiles : tile) * BM;
        const int64_t left = (bseg ? p.Mb : p.M) - my;
        const int rows = left < BM ? (int)left : BM;   // rows of the tile that exist
        char* out_lo = reinterpret_cast<char*>(bseg ? p.cb_lo : p.c_lo);
        char* out_up = reinterpret_cast<char*>(bseg ? p.cb_up : p.c_up);
        const bool same = kPoint && out_lo == out_up;   // (zero radius and one buffer named twice: stored once)
        const bool split = p.split_rows > 0 && !bseg;
        const uint32_t pitch = (split ? p.split_d : N) * 4u;   // bytes
        {
          // first row of the tile, first feature of this warp (a tile lies inside one group, 32 features inside one head)
          const int wn = n0 + q * 32;
          int64_t o = (int64_t)my * N + wn;
          if (split) {
            const int grp = my / p.split_rows;
            o = ((int64_t)(grp * (N / p.split_d) + wn / p.split_d) * p.split_rows + (my - grp * p.split_rows)) * p.split_d + wn % p.split_d;
          }
          out_lo += 4 * o;
          out_up += 4 * o;
        }
        const float* tbias = bseg ? p.bias_b : p.bias;
        const float bv = tbias != nullptr && valid ? __ldg(tbias + gn) : 0.f;
        if (!live) {
          // A zero row block (kPoint): zeros and zero norms.
          if (valid)
            for (int m = h * 64; m < h * 64 + 64 && m < rows; ++m) {
              *reinterpret_cast<float*>(out_lo + (m * pitch + lane * 4)) = 0.f;
              if (!same) *reinterpret_cast<float*>(out_up + (m * pitch + lane * 4)) = 0.f;
            }
          if (valid) (h == 0 ? p.norm_lo : p.norm_up)[(int64_t)(my / BM) * N + gn] = 0.f;
          continue;
        }
        const char* rlo = nullptr;
        const char* rup = nullptr;
        if (kResid) {   // (never head-split: the pitch of the result)
          rlo = reinterpret_cast<const char*>((bseg ? p.bres_lo : p.res_lo) + (int64_t)my * N + n0 + q * 32);
          rup = reinterpret_cast<const char*>((bseg ? p.bres_up : p.res_up) + (int64_t)my * N + n0 + q * 32);
        }
        float nl[2] = {0.f, 0.f}, nu[2] = {0.f, 0.f};
#pragma unroll 1
        for (int u = 0; u < kSubs; ++u) {
          const int mu0 = u * kRows;   // first row of this part of the tile
          if (kStream) {
            ok = give_w(lt * ns, 2, ns) && give_w((lt + 1) * ns, 0, 2);
            if (!ok) break;
          }
          ok = wait_warp(bar_scale + 8 * (lt & 3), (uint32_t)(lt >> 2) & 1u, wc);
          if (!ok) break;
          const float* inv = reinterpret_cast<const float*>(smem + SM::inv) + (lt & 3) * 128 - mu0;
          const bool rare = rare_w || *reinterpret_cast<const uint32_t*>(smem + SM::rare + (lt & 3) * 4) != 0;
          const int m_lo = mu0 + h * (kRows / 2);
          const uint32_t acc = tmem + ((uint32_t)(q * 32) << 16) + h * (kRows / 2);
          float rl[8], ru[8];   // the residual of eight rows, 128 contiguous bytes of each
          auto fetch = [&](auto edge, int m0) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const bool in = !decltype(edge)::value || (valid && m0 + i < rows);
              const uint32_t o = (m0 + i) * pitch + lane * 4;
              rl[i] = in ? __ldg(reinterpret_cast<const float*>(rlo + o)) : 0.f;
              ru[i] = in ? __ldg(reinterpret_cast<const float*>(rup + o)) : 0.f;
            }
          };
          // Eight rows.  kEdge: features or rows of the tile that do not exist, or scales that overflow when multiplied;
          // everything else runs without a branch but that for the norm (with tests around single rows it took four times as long).
          auto finish = [&](auto edge, int m0) {
            constexpr bool kEdge = decltype(edge)::value;
            uint32_t Ct[8], Rt[8];
            tmem_ld8(acc + (m0 - m_lo), Ct);
            if (!kPoint) tmem_ld8(acc + 128 + (m0 - m_lo), Rt);
            if (kStream) {   // the cross terms have accumulators of their own
              uint32_t Xc[8], Xr[8];
              tmem_ld8(acc + 64 + (m0 - m_lo), Xc);
              if (!kPoint) tmem_ld8(acc + 192 + (m0 - m_lo), Xr);
              tmem_wait_ld();
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                Ct[i] = __float_as_uint(fadd(__uint_as_float(Ct[i]), __uint_as_float(Xc[i])));
                if (!kPoint) Rt[i] = __float_as_uint(fadd(__uint_as_float(Rt[i]), __uint_as_float(Xr[i])));
              }
            } else {
              tmem_wait_ld();
            }
            if (m0 == m_lo + kRows / 2 - 8) {
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive(bar_acc_free);
            }
            const uint64_t w2 = dup2(wv), b2 = dup2(bv);
            uint64_t lo[4], up[4];
#pragma unroll
            for (int i = 0; i < 4; i += 2) {
              const ulonglong2 iv = *reinterpret_cast<const ulonglong2*>(inv + m0 + 2 * i);
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                uint64_t f = mul2(w2, e ? iv.y : iv.x);
                if (kEdge) f = pack2(__float_as_uint(fminf(lo_f(f), 3.0e38f)), __float_as_uint(fminf(hi_f(f), 3.0e38f)));
                const int k = 2 * (i + e);
                const uint64_t yc = pack2(Ct[k], Ct[k + 1]);
                if (kPoint) {
                  lo[i + e] = up[i + e] = fma2(yc, f, b2);
                } else {   // (the product with the power of two is exact: one rounding, that of the bias)
                  const uint64_t yr = pack2(Rt[k], Rt[k + 1]);
                  lo[i + e] = fma2(sub2(yc, yr), f, b2);
                  up[i + e] = fma2(add2(yc, yr), f, b2);
                }
              }
            }
            if (kResid) {
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                lo[i] = add2(lo[i], pack2(__float_as_uint(rl[2 * i]), __float_as_uint(rl[2 * i + 1])));
                up[i] = add2(up[i], pack2(__float_as_uint(ru[2 * i]), __float_as_uint(ru[2 * i + 1])));
              }
              if (m0 + 8 < m_lo + kRows / 2) fetch(edge, m0 + 8);   // (on their way during the stores and the next read-out)
            }
            if (kNorm) {
              auto walk = [&](auto add) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                  nl[0] = add(nl[0], lo_f(lo[i]));
                  nl[1] = add(nl[1], hi_f(lo[i]));
                  if (!kPoint) {
                    nu[0] = add(nu[0], lo_f(up[i]));
                    nu[1] = add(nu[1], hi_f(up[i]));
                  }
                }
              };
              if (p.norm_p == FB_PINF) walk([](float s, float v) { return s + fabsf(v); });
              else if (p.norm_p == FB_P2) walk([](float s, float v) { return fmaf(v, v, s); });
              else walk([](float s, float v) { return fmaxf(s, fabsf(v)); });
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              if (!kEdge || (valid && m0 + i < rows)) {
                const uint32_t o = (m0 + i) * pitch + lane * 4;
                *reinterpret_cast<float*>(out_lo + o) = (i & 1) ? hi_f(lo[i >> 1]) : lo_f(lo[i >> 1]);
                if (!kPoint || !same) *reinterpret_cast<float*>(out_up + o) = (i & 1) ? hi_f(up[i >> 1]) : lo_f(up[i >> 1]);
              }
            }
          };
          auto walk_tile = [&](auto edge) {
            if (kResid) fetch(edge, m_lo);
            ok = wait_warp(bar_acc_ready, (uint32_t)lt & 1u, wc);
            if (!ok) return;
            tc_fence_after();
#pragma unroll 1
            for (int m0 = m_lo; m0 < m_lo + kRows / 2; m0 += 8) finish(edge, m0);
          };
          if (rows == BM && q * 32 + 32 <= ncols && !rare) walk_tile(std::false_type{});
          else walk_tile(std::true_type{});
          if (!ok) break;
          ++lt;
        }
        if (kNorm && !bseg && ok) {
          // the norms over the tile's 128 rows: the two halves' parts in order (two tiles' parts alternate: nobody overwrites what
          // another warp still reads, since it meets that warp again before)
          float* part = reinterpret_cast<float*>(smem + SM::part) + (lt / kSubs & 1) * 512;
          part[h * 256 + n] = norm_combine(p.norm_p, nl[0], nl[1]);
          part[h * 256 + 128 + n] = kPoint ? norm_combine(p.norm_p, nl[0], nl[1]) : norm_combine(p.norm_p, nu[0], nu[1]);
        }
        ok = agree(ok);
        if (!ok) break;
        if (kNorm && !bseg) {
          const float* part = reinterpret_cast<const float*>(smem + SM::part) + (lt / kSubs & 1) * 512;
          const int line = et >> 7, col = et & 127;
          if (col < ncols)
            (line == 0 ? p.norm_lo : p.norm_up)[(int64_t)(my / BM) * N + n0 + col] =
                norm_finish(p.norm_p, norm_combine(p.norm_p, part[line * 128 + col], part[256 + line * 128 + col]));
        }
      }
      if (kStream && ok && pass == 0) {
        __threadfence();   // a marked tile is stored again
        ok = agree(meet());
      }
    }
  } else {
    // ------------------------------------------------------------------ converters of x (warps 12-27)
    reg_inc<Regs<kResid>::conv>();
    const int cw = warp - kFirstConv, b = cw / T::row_warps, q = cw % T::row_warps;   // group and 32 rows of x
    const int row = q * 32 + lane;
    bool ok = true;
    if (!kStream && b < nkb) {
      float v[32];
      load_w(b, v);
      put_w(b, b >> 1, v);
      if (lane == 0) mbar_arrive(bar_w);
    }
    int lt = 0, scan_phase = 0, taken = 0;   // taken: k-blocks of this group so far
    for (int pass = 0; pass < kPasses && ok; ++pass) {
      for (int ti = 0; ti < my_tiles && ok; ++ti) {
        if (!takes(pass, ti)) continue;
        const int tile = r0_tile + ti * step;
        const bool bseg = tile >= p.main_tiles;
        for (int u = 0; u < kSubs && ok; ++u) {
          const int m0 = (bseg ? tile - p.main_tiles : tile) * BM + u * kRows;
          uint8_t* const rmax = smem + SM::row_max + (lt & 1) * 512;
          int field = 0;
          if (kStream && pass == 1) {
            // a marked tile: the largest value of its whole rows first, a warp per row (a row that needs no other scale keeps the one it
            // had: what a row gives does not depend on the others of its tile)
            const int64_t lim = bseg ? p.Mb : p.M;
            for (int r = cw * (kRows / kConvWarps); r < (cw + 1) * (kRows / kConvWarps); ++r) {
              float m = 0.f, m4 = 0.f;   // of the row, of its first four k-blocks
              if (m0 + r < lim) {
                const float* pl = (bseg ? p.b_lo : p.a_lo) + (int64_t)(m0 + r) * K;
                const float* pu = (bseg ? p.b_up : p.a_up) + (int64_t)(m0 + r) * K;
                const int64_t rb = kCoef && !bseg ? (int64_t)m0 / p.coef_di * K : 0;
                for (int k = lane; k < K; k += 32) {
                  float l = pl[k], v = pu[k];
                  if (kCoef && !bseg) {
                    l = fmul(p.coef_l[rb + k], l);
                    v = fmul(p.coef_u[rb + k], v);
                  }
                  m = fmaxf(m, fmaxf(fabsf(l), fabsf(v)));
                  if (k < 4 * BK) m4 = m;
                }
              }
              const int e = exp_field(__uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(m))));
              int f = clamp_field(kFirst - exp_field(__uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(m4)))));
              if (e + f > kTop) f = clamp_field(kTop - e);
              if (lane == 0) rmax[r] = (uint8_t)f;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_scan);
            ok = wait_warp(bar_scan, (uint32_t)scan_phase & 1u, wc);
            ++scan_phase;
            if (!ok) break;
            field = rmax[row];
          }
          // (a group that only reads the scale says that it is past the one before: a wait by parity must not miss a phase)
          if (kStream && pass == 0 && b >= 4 && b < kbx) {
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_max + 8 * q);
          }
          for (int kb = b; kb < nkb; kb += kGroups) {
            const unsigned rn = (unsigned)((lt * nkb + kb) * kLines), e0 = rn % T::raw_ring, e1 = (rn + 1) % T::raw_ring;   // raw tiles of the two lines
            ok = wait_warp(bar_full + 8 * b, (uint32_t)taken & 1u, wc);
            ++taken;
            if (!ok) break;
            const uint8_t* raw = smem + SM::raw + e0 * T::raw_bytes;
            const uint8_t* raw_up = smem + SM::raw + e1 * T::raw_bytes;
            uint64_t l2[16], u2[16];
#pragma unroll
            for (int c = 0; c < 8; ++c) {
              const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(raw + swz(row, c));
              l2[2 * c] = v.x;
              l2[2 * c + 1] = v.y;
              if (!kPoint) {
                const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(raw_up + swz(row, c));
                u2[2 * c] = w.x;
                u2[2 * c + 1] = w.y;
              }
            }
            if (kCoef && !bseg) {
              const ulonglong2* kc = reinterpret_cast<const ulonglong2*>(smem + SM::coef + b * 256);
#pragma unroll
              for (int c = 0; c < 8; ++c) {
                const ulonglong2 a = kc[c], d = kc[8 + c];
                l2[2 * c] = mul2(a.x, l2[2 * c]);
                l2[2 * c + 1] = mul2(a.y, l2[2 * c + 1]);
                u2[2 * c] = mul2(d.x, u2[2 * c]);
                u2[2 * c + 1] = mul2(d.y, u2[2 * c + 1]);
              }
            }
            float m = 0.f;
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              m = fmaxf(m, fmaxf(fabsf(lo_f(l2[i])), fabsf(hi_f(l2[i]))));
              if (!kPoint) m = fmaxf(m, fmaxf(fabsf(lo_f(u2[i])), fabsf(hi_f(u2[i]))));
            }
            const int e = exp_field(m);
            const bool first = kb == b && !(kStream && pass == 1), gives = first && b < 4;
            if (gives) rmax[b * kRows + row] = (uint8_t)e;
            // every loaded value has been used (m depends on all of them): the raw stage goes back
            asm volatile("" ::"r"(e) : "memory");
            __syncwarp();
            if (lane == 0) {
              mbar_arrive(bar_empty + 8 * e0);
              if (!kPoint) mbar_arrive(bar_empty + 8 * e1);
              if (gives) mbar_arrive(bar_max + 8 * q);
            }
            if (first) {
              ok = wait_warp(bar_max + 8 * q, (uint32_t)lt & 1u, wc);   // (only tiles of the first pass count here: lt of that pass)
              if (!ok) break;
              int em = 0;
              for (int k = 0; k < kbs; ++k) em = max(em, (int)rmax[k * kRows + row]);
              field = clamp_field((kStream ? kFirst : kTop) - em);
            }
            if (kStream && pass == 0 && e + field > kTop) {   // more than the scale leaves room for: this tile is computed again
              atomicOr(bits + ((ti & (kBitTiles - 1)) >> 5), 1u << (ti & 31));
            }
            const int g = lt * ns + (kb >> 1), ar = g % T::x_ring;
            if (g >= T::x_ring) {
              ok = wait_warp(bar_done + 8 * ar, (uint32_t)(g / T::x_ring - 1) & 1u, wc);
              if (!ok) break;
            }
            if (kb == 0) {
              // (only now: the products of at least the tile two back have ended, and they began when the epilogue had read out the
              // one before it, so the scales of the tile four back are read and their barrier has been waited for)
              const float iv = exp_float(253 - field);
              reinterpret_cast<float*>(smem + SM::inv)[(lt & 3) * 128 + row] = iv;
              const bool big = __any_sync(0xffffffffu, iv > 1.0e18f);
              if (lane == 0) smem[SM::rare + (lt & 3) * 4 + q] = big ? 1 : 0;
              __syncwarp();
              if (lane == 0) mbar_arrive(bar_scale + 8 * (lt & 3));
            }
            const uint64_t hs = dup2(exp_float(field)), nhs = dup2(-exp_float(field));
            uint8_t* const xs = smem + SM::x + ar * T::slice_bytes;
#pragma unroll
            for (int c = 0; c < 4; ++c) {   // eight k: a 16-byte piece of each part
              uint32_t ch[4], cl[4], rh[4], rl[4];
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const uint64_t l = l2[c * 4 + i], u = kPoint ? l : u2[c * 4 + i];
                // centre and radius of the scaled lines, each rounded once
                const uint64_t hu = mul2(u, hs);
                split_f16_pair_neg(fma2(l, hs, hu), ch[i], cl[i]);
                if (!kPoint) {
                  split_f16_pair_neg(fma2(l, nhs, hu), rh[i], rl[i]);
                }
              }
              uint8_t* const d = xs + swz(row, (kb & 1) * 4 + c);
              *reinterpret_cast<uint4*>(d) = make_uint4(ch[0], ch[1], ch[2], ch[3]);
              *reinterpret_cast<uint4*>(d + T::plane_bytes) = make_uint4(cl[0], cl[1], cl[2], cl[3]);
              if (!kPoint) {
                *reinterpret_cast<uint4*>(d + 2 * T::plane_bytes) = make_uint4(rh[0], rh[1], rh[2], rh[3]);
                *reinterpret_cast<uint4*>(d + 3 * T::plane_bytes) = make_uint4(rl[0], rl[1], rl[2], rl[3]);
              }
            }
            fence_async_smem();
            __syncwarp();
            // (a slice with one k-block only: its warps arrive for the missing ones)
            if (lane == 0) mbar_arrive_n(bar_ready + 8 * ar, (kb & 1) == 0 && kb == nkb - 1 ? 2 : 1);
          }
          ++lt;
        }
      }
      if (kStream && ok && pass == 0) ok = meet();
    }
  }
  // Tear-down.  On the error path, give outstanding bulk copies time to land before the shared memory is released (bounded).
  if (*cta_abort) {
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    if (threadIdx.x == 0 && p.status != nullptr) atomicOr(p.status, 4);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// ------------------------------------------------------------------------ host side
// Columns of W per CTA: as few chunks of up to 128 as there can be, all about the same width.
inline int chunks_of(int N) { return (N + 127) / 128; }
inline int chunk_of(int N) {
  const int c = chunks_of(N);
  return ((N + 32 * c - 1) / (32 * c)) * 32;
}

template <bool kStream, bool kCoef, bool kNorm, bool kResid, bool kPoint>
int launch_one(const CUtensorMap (&tm)[4], const Args& a, unsigned grid, cudaStream_t st) {
  auto kern = split_sign_gemm_f16<kStream, kCoef, kNorm, kResid, kPoint>;
  static std::once_flag once[64];
  int dev = 0;
  FB_CUDA_OK(cudaGetDevice(&dev));
  cudaError_t err = cudaSuccess;
  std::call_once(once[dev & 63], [&]() { err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Smem<kStream>::bytes); });
  FB_CUDA_OK(err);
  fb::launch_tiles((int64_t)a.total_tiles * a.chunks, kern, grid, kThreads, Smem<kStream>::bytes, st, tm[0], tm[1], tm[2], tm[3], a);
  FB_LAUNCH_OK();
  return FB_OK;
}

// q: the arguments of launch_split_sign_tc, already checked there.
template <bool kStream>
int launch(const F16Product& q, cudaStream_t st) {
  Args a = {};
  const int64_t Mb = q.br != nullptr ? q.br->M : 0;
  a.a_lo = q.a_lo, a.a_up = q.a_up, a.W = q.W, a.c_lo = q.c_lo, a.c_up = q.c_up, a.bias = q.bias;
  a.M = q.M, a.Mb = Mb, a.N = q.N, a.K = q.K;
  a.chunk = chunk_of(q.N), a.chunks = (q.N + a.chunk - 1) / a.chunk;
  a.main_tiles = (int)ceil_div(q.M, BM);
  a.total_tiles = a.main_tiles + (int)ceil_div(Mb, BM);
  a.split_rows = q.split_rows, a.split_d = q.split_d;
  a.res_lo = q.res_lo, a.res_up = q.res_up;
  a.coef_l = q.coef_l, a.coef_u = q.coef_u, a.coef_di = q.coef_di;
  a.norm_lo = q.norm_lo, a.norm_up = q.norm_up, a.norm_p = q.norm_p;
  a.status = q.status, a.wait_tries = q.wait_tries, a.skip_it = q.skip_it;
  a.live = q.live;
  CUtensorMap tm[4];
  auto in_map = [&](CUtensorMap* m, const float* ptr, int64_t rows) {
    return get_map(m, ptr, 2, (uint64_t)q.K, (uint64_t)rows, 1, (uint64_t)q.K * 4, 0, BK, Cfg<kStream>::rows);
  };
  if (!in_map(&tm[0], q.a_lo, q.M) || !in_map(&tm[1], q.a_up, q.M)) return FB_ERR_CUDA;
  tm[2] = tm[0], tm[3] = tm[1];   // (only read for tiles of the bias rows)
  if (q.br != nullptr) {
    a.b_lo = q.br->a_lo, a.b_up = q.br->a_up, a.bias_b = q.br->bias;
    a.cb_lo = q.br->c_lo, a.cb_up = q.br->c_up;
    a.bres_lo = q.br->res_lo, a.bres_up = q.br->res_up;
    if (!in_map(&tm[2], q.br->a_lo, Mb) || !in_map(&tm[3], q.br->a_up, Mb)) return FB_ERR_CUDA;
  }
  const int64_t sms = device_info().sms, tiles = (int64_t)a.total_tiles * a.chunks;
  const unsigned grid = (unsigned)(tiles < sms ? tiles : sms);
  const bool coef = q.coef_l != nullptr, resid = q.res_lo != nullptr, norm = q.norm_lo != nullptr, point = norm && q.a_lo == q.a_up;
  if (coef)
    return resid ? launch_one<kStream, true, false, true, false>(tm, a, grid, st) : launch_one<kStream, true, false, false, false>(tm, a, grid, st);
  if (point) return launch_one<kStream, false, true, false, true>(tm, a, grid, st);
  if (norm) return launch_one<kStream, false, true, false, false>(tm, a, grid, st);
  if (resid) return launch_one<kStream, false, false, true, false>(tm, a, grid, st);
  return launch_one<kStream, false, false, false, false>(tm, a, grid, st);
}

}  // namespace hg
