// Dot product, weight part, transposed layout: x [B, Lx, K, Di], y [B, Ly, K, Di] -> z [B, Lx, Ly, Di] (Di contiguous), with
// the bias part in the same launch.  Included by dot_product.cu.
//
// FP32 products on the CUDA cores (eight multiply-adds per term), so the bound is their rate.  A warp owns 4 x 4 outputs
// (i, j) of 64 symbolic coordinates, two adjacent ones per lane, and a multiply-add is a packed one (fma.rn.f32x2: half the
// instructions).  A block is WI x WJ such tiles times WK shares of k, which are summed at the end in the order of the shares;
// its operand rows travel through a ring of kStages shared-memory stages (cp.async), KS values of k each, so that loads are
// far ahead of the arithmetic and the tiles of a block share them: loaded straight into registers one k ahead, the warps
// waited half of the time for L2 (452 us against 105 us of arithmetic for [4, 64, 128, 256]).  The ranges, split by sign, are
// staged kTK values of k at a time and broadcast; the duplicates of the packed form are made in registers (in shared memory
// they double the traffic of a pipe that is as busy as the arithmetic).
// Weight part of [4, 32, 64, 128] (the middle of the reference's sweep): 49 us with one coordinate and scalar multiply-adds per
// thread and no staging, 21.7 us now, 7.5 us of it arithmetic; [4, 64, 256, 512]: 1750 us loaded straight into registers, 987 us
// now, 505 us of it arithmetic.  Twice the warps (2 x 2 x 4, 1 x 1 x 16) were slower: the sums over the shares grow.
constexpr int kDotTransposedM = 64;   // symbolic coordinates per warp
constexpr int kStages = 3;

template <int WI, int WJ, int WK>
struct DotTransposedTile {
  static constexpr int kWarps = WI * WJ * WK, kThr = kWarps * 32;
  static constexpr int kRows = 2 * (WI + WJ) * 4;                 // operand rows: x_lw, x_uw, y_lw, y_uw
  static constexpr int KS = 256 / kRows;                          // k per stage: 64 KB a stage
  static constexpr int kRangeRows = (WI + 2 * WJ) * 4;            // x_l, y_l, y_u
  static constexpr int kTK = 3072 / kRangeRows / KS * KS;         // k per staging of the ranges: 24 KB
  static constexpr int kRangeLoads = (kRangeRows * kTK + kThr - 1) / kThr;
  static constexpr int kStageFloats = kRows * KS * kDotTransposedM;
  static constexpr size_t kSmem = sizeof(float) * (kStages * kStageFloats + kRangeRows * kTK * 2);
  static_assert(KS % WK == 0 && 16 % WK == 0 && kThr / 16 >= KS, "the same number of k for every share");
};

// VEC: floats per asynchronous copy: 4 (Di % 4 == 0, 16-byte aligned operands) or 1.
template <int WI, int WJ, int WK, int VEC>
__global__ void __launch_bounds__(DotTransposedTile<WI, WJ, WK>::kThr, 1)
dot_weight_transposed(const float* __restrict__ x_lw, const float* __restrict__ x_uw, const float* __restrict__ y_lw,
                      const float* __restrict__ y_uw, float* __restrict__ z_lw, float* __restrict__ z_uw, const DotBias q, int Di,
                      int n_bias, int n_it, int n_jt, int n_mt) {
  pdl_sync();
  using T = DotTransposedTile<WI, WJ, WK>;
  constexpr int KS = T::KS, TK = T::kTK, M = kDotTransposedM;
  extern __shared__ __align__(16) float smem[];
  if ((int)blockIdx.x < n_bias) {
    if (threadIdx.x < kThreads) dot_bias_tile<8>(q, blockIdx.x, smem);   // (the other threads leave: its barriers count the rest)
    return;
  }
  float2* s_rng = reinterpret_cast<float2*>(smem + kStages * T::kStageFloats);   // [kRangeRows][TK] (positive, negative part)
  const int Lx = q.Lx, Ly = q.Ly, K = q.K;
  int64_t bid = blockIdx.x - n_bias;
  const int jt = (int)(bid % n_jt); bid /= n_jt;
  const int it = (int)(bid % n_it); bid /= n_it;
  const int mt = (int)(bid % n_mt);
  const int64_t b = bid / n_mt;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wk = warp % WK, wj = (warp / WK) % WJ, wi = warp / (WK * WJ);
  const int ib = it * WI * 4, jb = jt * WJ * 4, i0 = ib + wi * 4, j0 = jb + wj * 4, m0 = mt * M;
  const bool active = i0 < Lx && j0 < Ly;   // the same for the whole warp

  // a thread copies the same part of a row (pieces of VEC coordinates) and the same k of every stage, for several rows
  constexpr int kPieces = M / VEC;              // per row
  constexpr int kAtOnce = T::kThr / 16;         // rows of 16 pieces of 4 per pass
  const int ck = (tid / 16) % KS;
  auto copy_stage = [&](int st) {
    const int k = st * KS + ck;
    float* dst = smem + (st % kStages) * T::kStageFloats + ck * T::kRows * M;
#pragma unroll
    for (int n = 0; n < T::kRows * KS / kAtOnce; ++n) {
      const int r = tid / 16 / KS + n * (kAtOnce / KS);   // row of the stage
      const bool is_x = r < 2 * WI * 4;
      const int rr = is_x ? r : r - 2 * WI * 4, per = is_x ? WI * 4 : WJ * 4, row = rr % per, at = (is_x ? ib : jb) + row;
      const float* src = is_x ? (rr < per ? x_lw : x_uw) : (rr < per ? y_lw : y_uw);
      const bool in = at < (is_x ? Lx : Ly) && k < K;
      src += in ? ((b * (is_x ? Lx : Ly) + at) * (int64_t)K + k) * Di : 0;
#pragma unroll
      for (int e = 0; e < kPieces / 16; ++e) {
        const int m = (tid % 16 + 16 * e) * VEC;
        const bool ok = in && m0 + m < Di;
        const uint32_t to = (uint32_t)__cvta_generic_to_shared(dst + r * M + m);
        if (VEC == 4)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(src + (ok ? m0 + m : 0)), "r"(ok ? 16 : 0) : "memory");
        else
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(to), "l"(src + (ok ? m0 + m : 0)), "r"(ok ? 4 : 0) : "memory");
      }
    }
  };
  float rng[T::kRangeLoads];   // ranges of the chunk to come
  auto load_ranges = [&](int k0) {
#pragma unroll
    for (int n = 0; n < T::kRangeLoads; ++n) {
      const int f = tid + n * T::kThr, r = f / TK, k = k0 + f % TK;
      float v = 0.f;
      if (r < T::kRangeRows && k < K) {
        const bool is_x = r < WI * 4;
        const int at = is_x ? ib + r : jb + (r - WI * 4) % (WJ * 4);
        const float* src = is_x ? q.x_l : r < (WI + WJ) * 4 ? q.y_l : q.y_u;
        if (at < (is_x ? Lx : Ly)) v = __ldg(src + (b * (is_x ? Lx : Ly) + at) * (int64_t)K + k);
      }
      rng[n] = v;
    }
  };

  const int n_st = (K + KS - 1) / KS;
  load_ranges(0);
#pragma unroll
  for (int st = 0; st < kStages - 1; ++st) {
    if (st < n_st) copy_stage(st);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  uint64_t acc_l[4][4], acc_u[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc_l[a][c] = acc_u[a][c] = 0;
  for (int st = 0; st < n_st; ++st) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    __syncthreads();   // stage st has landed for every thread; the stage before it and the ranges of its chunk are read
    if (st * KS % TK == 0) {
#pragma unroll
      for (int n = 0; n < T::kRangeLoads; ++n) {
        const int f = tid + n * T::kThr;
        if (f < T::kRangeRows * TK) s_rng[f] = make_float2(fmaxf(rng[n], 0.f), fminf(rng[n], 0.f));
      }
      __syncthreads();
      load_ranges(st * KS + TK);
    }
    if (st + kStages - 1 < n_st) copy_stage(st + kStages - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (!active) continue;
    const float* tile = smem + (st % kStages) * T::kStageFloats;
    const float2* rx = s_rng + (wi * 4) * TK + st * KS % TK;
    const float2* rl = s_rng + (WI * 4 + wj * 4) * TK + st * KS % TK;
    const float2* ru = rl + WJ * 4 * TK;
#pragma unroll 2
    for (int t = 0; t < KS / WK; ++t) {   // (past K: zeros)
      const int kk = wk + WK * t;
      const float* px = tile + (kk * T::kRows + wi * 4) * M + 2 * lane;
      const float* py = tile + (kk * T::kRows + 2 * WI * 4 + wj * 4) * M + 2 * lane;
      float2 lx[4];
      uint64_t xl[4], xu[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        lx[a] = rx[a * TK + kk];
        xl[a] = *reinterpret_cast<const uint64_t*>(px + a * M);
        xu[a] = *reinterpret_cast<const uint64_t*>(px + (WI * 4 + a) * M);
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float2 ly = rl[c * TK + kk], uy = ru[c * TK + kk];
        const uint64_t lyp = pack2(ly.x, ly.x), lyn = pack2(ly.y, ly.y), uyp = pack2(uy.x, uy.x), uyn = pack2(uy.y, uy.y);
        const uint64_t yl = *reinterpret_cast<const uint64_t*>(py + c * M), yu = *reinterpret_cast<const uint64_t*>(py + (WJ * 4 + c) * M);
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          const uint64_t lxp = pack2(lx[a].x, lx[a].x), lxn = pack2(lx[a].y, lx[a].y);
          uint64_t l = acc_l[a][c], u = acc_u[a][c];
          l = fma2(xl[a], lyp, l); l = fma2(xu[a], lyn, l);
          l = fma2(yl, lxp, l);    l = fma2(yu, lxn, l);
          u = fma2(xu[a], uyp, u); u = fma2(xl[a], uyn, u);
          u = fma2(yu, lxp, u);    u = fma2(yl, lxn, u);
          acc_l[a][c] = l; acc_u[a][c] = u;
        }
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  // partial sums of the WK shares: a warp adds up 16 / WK of the tile's outputs
  uint64_t* part = reinterpret_cast<uint64_t*>(smem);   // [warp][16 outputs][2 sides][32 lanes]
  if (WK > 1) {
    __syncthreads();
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        part[((warp * 16 + a * 4 + c) * 2 + 0) * 32 + lane] = acc_l[a][c];
        part[((warp * 16 + a * 4 + c) * 2 + 1) * 32 + lane] = acc_u[a][c];
      }
    __syncthreads();
  }
  const int m = m0 + 2 * lane;
  if (!active || m >= Di) return;
#pragma unroll
  for (int e = 0; e < 16 / WK; ++e) {
    const int o = WK > 1 ? wk * (16 / WK) + e : e, i = i0 + o / 4, j = j0 + o % 4;
    if (i >= Lx || j >= Ly) continue;
    float2 l = make_float2(0.f, 0.f), u = l;
    if (WK > 1) {
#pragma unroll
      for (int w = 0; w < WK; ++w) {
        const int src = warp - wk + w;
        const float2 pl = unpack2(part[((src * 16 + o) * 2 + 0) * 32 + lane]), pu = unpack2(part[((src * 16 + o) * 2 + 1) * 32 + lane]);
        l.x = fadd(l.x, pl.x); l.y = fadd(l.y, pl.y);
        u.x = fadd(u.x, pu.x); u.y = fadd(u.y, pu.y);
      }
    } else {
      l = unpack2(acc_l[e / 4 % 4][e % 4]);
      u = unpack2(acc_u[e / 4 % 4][e % 4]);
    }
    l.x = fmul(l.x, q.out_scale); l.y = fmul(l.y, q.out_scale);
    u.x = fmul(u.x, q.out_scale); u.y = fmul(u.y, q.out_scale);
    const int64_t at = ((b * Lx + i) * (int64_t)Ly + j) * Di + m;
    if (VEC == 4) {
      *reinterpret_cast<float2*>(z_lw + at) = l;
      *reinterpret_cast<float2*>(z_uw + at) = u;
    } else {
      z_lw[at] = l.x;
      z_uw[at] = u.x;
      if (m + 1 < Di) { z_lw[at + 1] = l.y; z_uw[at + 1] = u.y; }
    }
  }
}

// Many thin products (a few rows against any number, a large batch): a thread per coordinate and 4 x 4 outputs, operands straight
// from global memory.  The kernel above has one block of 200 KB an SM and its ring to fill for each; here many small blocks hide
// each other's loads.  512 products of 64 x 1 rows, K = 8, dim_in 2: 386 us above, 156 us here; 4 x 64, K = 8, dim_in 8: 299 and
// 175 us.  With more arithmetic per loaded value the ring wins again: 512 of 4 x 16, K = 128, dim_in 16: 555 and 867 us.
constexpr int kThinM = 128, kThinK = 128;
__global__ void __launch_bounds__(kThinM)
dot_weight_transposed_thin(const float* __restrict__ x_lw, const float* __restrict__ x_uw, const float* __restrict__ y_lw,
                           const float* __restrict__ y_uw, float* __restrict__ z_lw, float* __restrict__ z_uw, const DotBias q, int Di,
                           int n_it, int n_jt) {
  pdl_sync();
  __shared__ float s_lx[4][kThinK], s_ly[4][kThinK], s_uy[4][kThinK];
  const float* __restrict__ x_l = q.x_l;
  const float* __restrict__ y_l = q.y_l;
  const float* __restrict__ y_u = q.y_u;
  const int Lx = q.Lx, Ly = q.Ly, K = q.K;
  int64_t bid = blockIdx.x;
  const int jt = (int)(bid % n_jt); bid /= n_jt;
  const int it = (int)(bid % n_it); bid /= n_it;
  const int64_t b = bid;
  const int i0 = it * 4, j0 = jt * 4;
  const int m = blockIdx.y * kThinM + threadIdx.x;
  const bool m_ok = m < Di;
  float acc_l[4][4], acc_u[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int c = 0; c < 4; ++c) { acc_l[a][c] = 0.f; acc_u[a][c] = 0.f; }
  for (int k0 = 0; k0 < K; k0 += kThinK) {
    const int nk = min(kThinK, K - k0);
    for (int f = threadIdx.x; f < 4 * kThinK; f += kThinM) {
      const int r = f / kThinK, k = f % kThinK;
      const bool kin = k < nk;
      s_lx[r][k] = (kin && i0 + r < Lx) ? x_l[(b * Lx + i0 + r) * (int64_t)K + k0 + k] : 0.f;
      s_ly[r][k] = (kin && j0 + r < Ly) ? y_l[(b * Ly + j0 + r) * (int64_t)K + k0 + k] : 0.f;
      s_uy[r][k] = (kin && j0 + r < Ly) ? y_u[(b * Ly + j0 + r) * (int64_t)K + k0 + k] : 0.f;
    }
    __syncthreads();
    if (m_ok) {
      for (int k = 0; k < nk; ++k) {
        float xl[4], xu[4], yl[4], yu[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          const bool ok = i0 + a < Lx;
          const int64_t o = ((b * Lx + i0 + a) * (int64_t)K + k0 + k) * Di + m;
          xl[a] = ok ? __ldg(x_lw + o) : 0.f;
          xu[a] = ok ? __ldg(x_uw + o) : 0.f;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const bool ok = j0 + c < Ly;
          const int64_t o = ((b * Ly + j0 + c) * (int64_t)K + k0 + k) * Di + m;
          yl[c] = ok ? __ldg(y_lw + o) : 0.f;
          yu[c] = ok ? __ldg(y_uw + o) : 0.f;
        }
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          const float lx = s_lx[a][k];
          const float lxp = fmaxf(lx, 0.f), lxn = fminf(lx, 0.f);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const float ly = s_ly[c][k], uy = s_uy[c][k];
            float l = acc_l[a][c], u = acc_u[a][c];
            l = fmaf(xl[a], fmaxf(ly, 0.f), l); l = fmaf(xu[a], fminf(ly, 0.f), l);
            l = fmaf(yl[c], lxp, l);            l = fmaf(yu[c], lxn, l);
            u = fmaf(xu[a], fmaxf(uy, 0.f), u); u = fmaf(xl[a], fminf(uy, 0.f), u);
            u = fmaf(yu[c], lxp, u);            u = fmaf(yl[c], lxn, u);
            acc_l[a][c] = l; acc_u[a][c] = u;
          }
        }
      }
    }
    __syncthreads();
  }
  if (!m_ok) return;
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (i0 + a < Lx && j0 + c < Ly) {
        const int64_t o = ((b * Lx + i0 + a) * (int64_t)Ly + j0 + c) * Di + m;
        z_lw[o] = fmul(acc_l[a][c], q.out_scale);
        z_uw[o] = fmul(acc_u[a][c], q.out_scale);
      }
}

bool dot_transposed_thin(const DotBias& q, int B, int Di) {
  const double per_sm = (double)B * ceil_div(q.Lx, 4) * ceil_div(q.Ly, 4) * ceil_div(Di, kDotTransposedM) / device_info().sms;
  return std::min(q.Lx, q.Ly) <= 4 && (int64_t)q.K * std::min(Di, kDotTransposedM) <= 800 &&
         (per_sm >= 3.0 + q.K / 16.0 || (q.Lx > 32 && per_sm >= 2.0));
}

int launch_dot_transposed_thin(const float* x_lw, const float* x_uw, const float* y_lw, const float* y_uw, float* z_lw, float* z_uw,
                               const DotBias& q, int B, int Di, cudaStream_t st) {
  if (int rc = launch_dot_bias(q, B, st)) return rc;
  const int n_it = (int)ceil_div(q.Lx, 4), n_jt = (int)ceil_div(q.Ly, 4);
  const int64_t blocks = (int64_t)B * n_it * n_jt, my = ceil_div(Di, kThinM);
  if (blocks > 0x7fffffff || my > 65535) return FB_ERR_SHAPE;
  fb::launch_k(dot_weight_transposed_thin, dim3((unsigned)blocks, (unsigned)my), kThinM, 0, st, x_lw, x_uw, y_lw, y_uw, z_lw, z_uw, q, Di, n_it,
               n_jt);
  FB_LAUNCH_OK();
  return FB_OK;
}

template <int WI, int WJ, int WK, int VEC>
int launch_dot_transposed_t(const float* x_lw, const float* x_uw, const float* y_lw, const float* y_uw, float* z_lw, float* z_uw,
                            const DotBias& q, int B, int Di, cudaStream_t st) {
  using T = DotTransposedTile<WI, WJ, WK>;
  const int n_it = (int)ceil_div(q.Lx, WI * 4), n_jt = (int)ceil_div(q.Ly, WJ * 4), n_mt = (int)ceil_div(Di, kDotTransposedM);
  const int64_t n_bias = (int64_t)B * q.n_it * q.n_jt, blocks = n_bias + (int64_t)B * n_it * n_jt * n_mt;
  if (blocks > 0x7fffffff) return FB_ERR_SHAPE;
  auto kern = dot_weight_transposed<WI, WJ, WK, VEC>;
  if (int rc = ensure_dynamic_smem(kern, T::kSmem)) return rc;
  fb::launch_k(kern, (unsigned)blocks, T::kThr, T::kSmem, st, x_lw, x_uw, y_lw, y_uw, z_lw, z_uw, q, Di, (int)n_bias, n_it, n_jt, n_mt);
  FB_LAUNCH_OK();
  return FB_OK;
}

int launch_dot_transposed(const float* x_lw, const float* x_uw, const float* y_lw, const float* y_uw, float* z_lw, float* z_uw,
                          const DotBias& q, int B, int Di, cudaStream_t st) {
  if (dot_transposed_thin(q, B, Di)) return launch_dot_transposed_thin(x_lw, x_uw, y_lw, y_uw, z_lw, z_uw, q, B, Di, st);
  const auto aligned8 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 7) == 0; };
  const bool vec = Di % 4 == 0 && aligned16(x_lw) && aligned16(x_uw) && aligned16(y_lw) && aligned16(y_uw) && aligned8(z_lw) && aligned8(z_uw);
  // Rounds of one block per SM times what a block takes: its arithmetic (in 4 x 4 tiles), the smaller tiles charged for reading
  // every operand row twice and four times as often from L2, and, in the same unit (90 ns), its start and the sums of its shares.
  // Without the latter short sums went to the smallest tiles: 353 products of 12 x 10, K = 8, dim_in 32 112 us, 57 us with it.
  const int64_t sms = device_info().sms, bm = (int64_t)B * ceil_div(Di, kDotTransposedM);
  auto rounds = [&](int t) { return ceil_div(bm * ceil_div(q.Lx, t) * ceil_div(q.Ly, t), sms); };
  const int64_t K = q.K, c16 = (16 * K + 70) * rounds(16), c8 = (5 * K + 40) * rounds(8), c4 = (2 * K + 26) * rounds(4);
#define FB_DOT_T(...) (vec ? launch_dot_transposed_t<__VA_ARGS__, 4>(x_lw, x_uw, y_lw, y_uw, z_lw, z_uw, q, B, Di, st) \
                           : launch_dot_transposed_t<__VA_ARGS__, 1>(x_lw, x_uw, y_lw, y_uw, z_lw, z_uw, q, B, Di, st))
  if (c16 <= c8 && c16 <= c4) return FB_DOT_T(4, 4, 1);
  return c8 <= c4 ? FB_DOT_T(2, 2, 2) : FB_DOT_T(1, 1, 8);
#undef FB_DOT_T
}
