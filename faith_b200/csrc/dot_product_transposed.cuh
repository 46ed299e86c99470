// Dot product, weight part, transposed layout: x [B, Lx, K, Di], y [B, Ly, K, Di] -> z [B, Lx, Ly, Di] (Di contiguous), with
// the bias part in the same launch.  Included by dot_product.cu.
//
// FP32 products on the CUDA cores (eight multiply-adds per term), so the bound is their rate.  A warp owns 4 x 4 outputs
// (i, j) of 64 symbolic coordinates, two adjacent ones per lane, and a multiply-add is a packed one (fma.rn.f32x2: half the
// instructions).  A block is WI x WJ such tiles times WK shares of k, which are summed at the end in the order of the shares.
// Its operand rows travel through a ring of kStages shared-memory stages, KS values of k each, far ahead of the arithmetic:
// four TMA boxes a stage, issued by one thread.  (Asynchronous copies of 16 bytes by all threads took 1350 of the 4400 cycles of
// a stage to issue, 6000 cycles for the first two; bulk copies of single rows, 256 bytes each, were slower than either.)  The
// ranges, split by sign, are staged kTK values of k at a time and broadcast; the duplicates of the packed form are made in
// registers (in shared memory they double the traffic of a pipe that is as busy as the arithmetic).
// LK > 1: the lanes of a warp are LK shares of k too, with 64 / LK coordinates each.  That halves or quarters the operand values
// that a block of as many multiply-adds reads, leaves fewer lanes without a coordinate where dim_in is small, and makes smaller blocks.
// Both kernels of the call (with the ranges' 7 us and the launches), us, with the threads' copies and now: [4, 32, 64, 128] (the
// middle of the reference's sweep) 38.7 and 34.5, 7.5 us of it arithmetic; [4, 64, 256, 512] 1084 and 881, 505 us arithmetic;
// [1, 128, 512, 32] 337 and 181; [4, 40, 64, 16] 34.7 and 21.7.  What is left beside the arithmetic: the start, the sums of
// the shares, and a stage's multiply-adds at 70 % of their rate.  Twice the warps (2 x 2 x 4) gained nothing.
constexpr int kDotTransposedM = 64;   // symbolic coordinates per warp (LK = 1)
constexpr int kStages = 3;

struct OperandMaps {
  CUtensorMap xl, xu, yl, yu;   // [B][rows][K][Di], boxes of a block's rows, KS values of k and kM coordinates
};

// LK: shares of k among the lanes of a warp, each with 64 / LK coordinates: for dim_in that would leave lanes without one.
template <int WI, int WJ, int WK, int LK>
struct DotTransposedTile {
  static constexpr int kWarps = WI * WJ * WK, kThr = kWarps * 32;
  static constexpr int kM = kDotTransposedM / LK, kI = WI * 4, kJ = WJ * 4;   // a block's coordinates and outputs
  static constexpr int kRows = 2 * (kI + kJ);                     // operand rows: x_lw, x_uw, y_lw, y_uw
  static constexpr int KS = 16384 / kM / kRows;                   // k per stage: 64 KB a stage
  static constexpr int kRangeRows = kI + 2 * kJ;                  // x_l, y_l, y_u
  static constexpr int kTK = 3072 / kRangeRows / KS * KS;         // k per staging of the ranges: 24 KB
  static constexpr int kRangeLoads = (kRangeRows * kTK + kThr - 1) / kThr;
  static constexpr int kStageFloats = kRows * KS * kM;
  static constexpr size_t kSmem = sizeof(float) * (kStages * kStageFloats + kRangeRows * kTK * 2 + 2 + 2 * kStages);
  static_assert(KS % (WK * LK) == 0 && kTK > 0, "the same number of k for every share");
};

// kTma: operands whose rows begin at multiples of 16 bytes arrive by TMA, four boxes a stage; other ones by 4-byte asynchronous
// copies of the threads.
template <int WI, int WJ, int WK, int LK, bool kTma>
__global__ void __launch_bounds__(DotTransposedTile<WI, WJ, WK, LK>::kThr, 1)
dot_weight_transposed(const __grid_constant__ OperandMaps maps, const float* __restrict__ x_lw, const float* __restrict__ x_uw,
                      const float* __restrict__ y_lw, const float* __restrict__ y_uw, float* __restrict__ z_lw, float* __restrict__ z_uw,
                      const DotBias q, int Di, int n_bias, int n_it, int n_jt, int n_mt) {
  using T = DotTransposedTile<WI, WJ, WK, LK>;
  constexpr int KS = T::KS, TK = T::kTK, M = T::kM, TI = T::kI, TJ = T::kJ;
  extern __shared__ __align__(128) float smem[];
  float2* s_rng = reinterpret_cast<float2*>(smem + kStages * T::kStageFloats);   // [kRangeRows][TK] (positive, negative part)
  volatile int* s_abort = reinterpret_cast<volatile int*>(s_rng + T::kRangeRows * TK);
  const uint32_t full = tma::smem_u32(s_rng + T::kRangeRows * TK + 1);              // [kStages] barriers
  if (kTma && threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) tma::mbar_init(full + 8 * s, 1);
    *s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (kTma) __syncthreads();
  pdl_sync();
  if ((int)blockIdx.x < n_bias) {
    if (threadIdx.x < kThreads) dot_bias_tile<8>(q, blockIdx.x, smem);   // (the other threads leave: its barriers count the rest)
    return;
  }
  const int Lx = q.Lx, Ly = q.Ly, K = q.K;
  int64_t bid = blockIdx.x - n_bias;
  const int jt = (int)(bid % n_jt); bid /= n_jt;
  const int it = (int)(bid % n_it); bid /= n_it;
  const int mt = (int)(bid % n_mt);
  const int64_t b = bid / n_mt;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wk = warp % WK, wj = (warp / WK) % WJ, wi = warp / (WK * WJ);
  const int lk = lane / (M / 2), lm = lane % (M / 2);   // share of k and pair of coordinates of this lane
  const int ib = it * TI, jb = jt * TJ, i0 = ib + wi * 4, j0 = jb + wj * 4, m0 = mt * M;
  const bool active = i0 < Lx && j0 < Ly;   // the same for the whole warp
  const int n_st = (K + KS - 1) / KS;

  // A stage: [row][k][coordinate].  (Rows and coordinates that do not exist only reach outputs that are not stored, and no share goes
  // past K.)
  auto copy_stage = [&](int st) {
    float* dst = smem + (st % kStages) * T::kStageFloats;
    if constexpr (kTma) {
      if (tid == 0) {
        const uint32_t bar = full + 8 * (st % kStages), to = tma::smem_u32(dst), x_bytes = TI * KS * M * 4, y_bytes = TJ * KS * M * 4;
        tma::mbar_arrive_expect_tx(bar, T::kStageFloats * 4u);
        tma::tma_load_4d(to, &maps.xl, m0, st * KS, ib, (int)b, bar);
        tma::tma_load_4d(to + x_bytes, &maps.xu, m0, st * KS, ib, (int)b, bar);
        tma::tma_load_4d(to + 2 * x_bytes, &maps.yl, m0, st * KS, jb, (int)b, bar);
        tma::tma_load_4d(to + 2 * x_bytes + y_bytes, &maps.yu, m0, st * KS, jb, (int)b, bar);
      }
    } else {
#pragma unroll 4
      for (int rk = tid / 16; rk < T::kRows * KS; rk += T::kThr / 16) {
        const int k = st * KS + rk % KS, r = rk / KS;
        const bool is_x = r < 2 * TI;
        const int rr = is_x ? r : r - 2 * TI, per = is_x ? TI : TJ, at = (is_x ? ib : jb) + rr % per, len = is_x ? Lx : Ly;
        const float* src = is_x ? (rr < per ? x_lw : x_uw) : (rr < per ? y_lw : y_uw);
        const int has = at < len && k < K ? Di : 0;
        src += has > 0 ? ((b * len + at) * (int64_t)K + k) * Di : 0;
#pragma unroll
        for (int e = 0; e < M / 16; ++e) {
          const int m = tid % 16 + 16 * e;
          if (m0 + m < has)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(tma::smem_u32(dst + rk * M + m)), "l"(src + m0 + m) : "memory");
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
  };
  float rng[T::kRangeLoads];   // ranges of the chunk to come
  auto load_ranges = [&](int k0) {
#pragma unroll
    for (int n = 0; n < T::kRangeLoads; ++n) {
      const int f = tid + n * T::kThr, r = f / TK, k = k0 + f % TK;
      float v = 0.f;
      if (r < T::kRangeRows && k < K) {
        const bool is_x = r < TI;
        const int at = is_x ? ib + r : jb + (r - TI) % TJ;
        const float* src = is_x ? q.x_l : r < TI + TJ ? q.y_l : q.y_u;
        if (at < (is_x ? Lx : Ly)) v = __ldg(src + (b * (is_x ? Lx : Ly) + at) * (int64_t)K + k);
      }
      rng[n] = v;
    }
  };

#pragma unroll
  for (int st = 0; st < kStages - 1; ++st) {
    if (st < n_st) copy_stage(st);
    else if (!kTma) asm volatile("cp.async.commit_group;" ::: "memory");
  }
  load_ranges(0);
  uint64_t acc_l[4][4], acc_u[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc_l[a][c] = acc_u[a][c] = 0;
  int ok = 1;
  for (int st = 0; st < n_st; ++st) {
    // stage st has landed for every thread; the stage before it and the ranges of its chunk are read
    if (kTma) {
      ok = __syncthreads_and(tma::mbar_wait(full + 8 * (st % kStages), (uint32_t)(st / kStages) & 1u, s_abort));
      if (!ok) break;
    } else {
      asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
      __syncthreads();
    }
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
    else if (!kTma) asm volatile("cp.async.commit_group;" ::: "memory");
    if (!active) continue;
    const float* tile = smem + (st % kStages) * T::kStageFloats;
    const float2* rx = s_rng + (wi * 4) * TK + st * KS % TK;
    const float2* rl = s_rng + (TI + wj * 4) * TK + st * KS % TK;
    const float2* ru = rl + TJ * TK;
    const int left = K - st * KS - (wk * LK + lk);   // of this share, in steps of WK * LK
    const int nt = left >= KS ? KS / (WK * LK) : left <= 0 ? 0 : min(KS / (WK * LK), (left + WK * LK - 1) / (WK * LK));
#pragma unroll 2
    for (int t = 0; t < nt; ++t) {
      const int kk = wk * LK + lk + WK * LK * t;
      const float* px = tile + (wi * 4 * KS + kk) * M + 2 * lm;
      const float* py = tile + ((2 * TI + wj * 4) * KS + kk) * M + 2 * lm;
      float2 lx[4];
      uint64_t xl[4], xu[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        lx[a] = rx[a * TK + kk];
        xl[a] = *reinterpret_cast<const uint64_t*>(px + a * KS * M);
        xu[a] = *reinterpret_cast<const uint64_t*>(px + (TI + a) * KS * M);
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float2 ly = rl[c * TK + kk], uy = ru[c * TK + kk];
        const uint64_t lyp = pack2(ly.x, ly.x), lyn = pack2(ly.y, ly.y), uyp = pack2(uy.x, uy.x), uyn = pack2(uy.y, uy.y);
        const uint64_t yl = *reinterpret_cast<const uint64_t*>(py + c * KS * M), yu = *reinterpret_cast<const uint64_t*>(py + (TJ + c) * KS * M);
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
  if (!kTma) asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (!ok) {   // (given up: the copies on their way land before the shared memory goes back, bounded)
    for (int i = 0; i < 2000; ++i) __nanosleep(1000);
    return;
  }
  // partial sums of the shares: a warp's lanes of one share add up 16 / (WK * LK) of the tile's outputs
  constexpr int kShares = WK * LK;
  uint64_t* part = reinterpret_cast<uint64_t*>(smem);   // [warp][16 outputs][2 sides][32 lanes]
  if (kShares > 1) {
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
  const int m = m0 + 2 * lm;
  if (!active || m >= Di) return;
#pragma unroll
  for (int e = 0; e < (16 + kShares - 1) / kShares; ++e) {
    const int o = kShares > 1 ? (wk * LK + lk) + e * kShares : e, i = i0 + o / 4, j = j0 + o % 4;
    if (o >= 16 || i >= Lx || j >= Ly) continue;
    float2 l = make_float2(0.f, 0.f), u = l;
    if (kShares > 1) {
#pragma unroll
      for (int w = 0; w < kShares; ++w) {
        const int src = warp - wk + w / LK, at = w % LK * (M / 2) + lm;
        const float2 pl = unpack2(part[((src * 16 + o) * 2 + 0) * 32 + at]), pu = unpack2(part[((src * 16 + o) * 2 + 1) * 32 + at]);
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
    if (kTma) {
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

template <int WI, int WJ, int WK, int LK, bool kTma>
int launch_dot_transposed_t(const float* x_lw, const float* x_uw, const float* y_lw, const float* y_uw, float* z_lw, float* z_uw,
                            const DotBias& q, int B, int Di, cudaStream_t st) {
  using T = DotTransposedTile<WI, WJ, WK, LK>;
  const int n_it = (int)ceil_div(q.Lx, T::kI), n_jt = (int)ceil_div(q.Ly, T::kJ), n_mt = (int)ceil_div(Di, T::kM);
  const int64_t n_bias = (int64_t)B * q.n_it * q.n_jt, blocks = n_bias + (int64_t)B * n_it * n_jt * n_mt;
  if (blocks > 0x7fffffff) return FB_ERR_SHAPE;
  auto kern = dot_weight_transposed<WI, WJ, WK, LK, kTma>;
  if (int rc = ensure_dynamic_smem(kern, T::kSmem)) return rc;
  OperandMaps maps = {};
  if (kTma) {
    auto map = [&](CUtensorMap* m, const float* ptr, int rows, int box) {
      const uint64_t di = (uint64_t)Di, k = (uint64_t)q.K, r = (uint64_t)rows;
      return tma::get_map(m, tma::MapKey{ptr, {di, k, r, (uint64_t)B, 1}, {di * 4, di * k * 4, di * k * r * 4, 0},
                               {(uint32_t)T::kM, (uint32_t)T::KS, (uint32_t)box, 1, 1}, 4, true});
    };
    if (!map(&maps.xl, x_lw, q.Lx, T::kI) || !map(&maps.xu, x_uw, q.Lx, T::kI) || !map(&maps.yl, y_lw, q.Ly, T::kJ) ||
        !map(&maps.yu, y_uw, q.Ly, T::kJ))
      return FB_ERR_CUDA;
  }
  fb::launch_k(kern, (unsigned)blocks, T::kThr, T::kSmem, st, maps, x_lw, x_uw, y_lw, y_uw, z_lw, z_uw, q, Di, (int)n_bias, n_it, n_jt, n_mt);
  FB_LAUNCH_OK();
  return FB_OK;
}

int launch_dot_transposed(const float* x_lw, const float* x_uw, const float* y_lw, const float* y_uw, float* z_lw, float* z_uw,
                          const DotBias& q, int B, int Di, cudaStream_t st) {
  if (dot_transposed_thin(q, B, Di)) return launch_dot_transposed_thin(x_lw, x_uw, y_lw, y_uw, z_lw, z_uw, q, B, Di, st);
  const auto aligned8 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 7) == 0; };
  // (byte strides of a tensor map stay below 2^40)
  const bool tma = tma::encode_fn() != nullptr && Di % 4 == 0 && 4.0 * Di * q.K * std::max(q.Lx, q.Ly) < 1e12 && aligned16(x_lw) &&
                   aligned16(x_uw) && aligned16(y_lw) && aligned16(y_uw) && aligned8(z_lw) && aligned8(z_uw);
#define FB_DOT_T(...) launch_dot_transposed_t<__VA_ARGS__>(x_lw, x_uw, y_lw, y_uw, z_lw, z_uw, q, B, Di, st)
  const int64_t sms = device_info().sms, K = q.K;
  auto rounds = [&](int t, int m) { return ceil_div(B * ceil_div(Di, m) * ceil_div(q.Lx, t) * ceil_div(q.Ly, t), sms); };
  if (!tma) {
    // Rounds of one block per SM times what a block takes: its arithmetic (in 4 x 4 tiles), the smaller tiles charged for reading
    // every operand row twice and four times as often from L2, and, in the same unit (90 ns), its start and the sums of its shares.
    // Without the latter short sums went to the smallest tiles: 353 products of 12 x 10, K = 8, dim_in 32 112 us, 57 us with it.
    const int64_t c16 = (16 * K + 70) * rounds(16, 64), c8 = (5 * K + 40) * rounds(8, 64), c4 = (2 * K + 26) * rounds(4, 64);
    if (c16 <= c8 && c16 <= c4) return FB_DOT_T(4, 4, 1, 1, false);
    return c8 <= c4 ? FB_DOT_T(2, 2, 2, 1, false) : FB_DOT_T(1, 1, 8, 1, false);
  }
  // The same with the times of a block in ns (start and sums, per k) as measured for each form with one to fifty rounds and K from
  // 3 to 512.  Of 25 shapes one was chosen 6 % slower than the best form, the others within 3 %.
  const struct { int tile, lanes, start, per_k; } form[] = {{16, 1, 6000, 880}, {16, 2, 5500, 460}, {16, 4, 6000, 220},
                                                            {8, 1, 4500, 250},  {8, 2, 4500, 140},  {8, 4, 3000, 66},
                                                            {4, 1, 2500, 77},   {4, 2, 3000, 35},   {4, 4, 3000, 18}};
  int best = 0;
  int64_t least = INT64_MAX;
  for (int f = 0; f < 9; ++f) {
    const int64_t c = (form[f].start + form[f].per_k * K) * rounds(form[f].tile, kDotTransposedM / form[f].lanes);
    if (c < least) least = c, best = f;
  }
  switch (best) {
    case 0: return FB_DOT_T(4, 4, 1, 1, true);
    case 1: return FB_DOT_T(4, 4, 1, 2, true);
    case 2: return FB_DOT_T(4, 4, 1, 4, true);
    case 3: return FB_DOT_T(2, 2, 2, 1, true);
    case 4: return FB_DOT_T(2, 2, 2, 2, true);
    case 5: return FB_DOT_T(2, 2, 2, 4, true);
    case 6: return FB_DOT_T(1, 1, 8, 1, true);
    case 7: return FB_DOT_T(1, 1, 8, 2, true);
    default: return FB_DOT_T(1, 1, 8, 4, true);
  }
#undef FB_DOT_T
}
