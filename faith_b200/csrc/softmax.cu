// Fused softmax bound: exp -> feature-axis sum -> reciprocal -> McCormick product, the chain of
// Bounds.softmax (Bounds.py:1005-1014 with exp :970-1003, reciprocal :1136-1161, multiply(Bounds)
// :608-651), for rows whose feature axis fits one tile of 16, 32 or 64 columns (attention scores, Do = length).
//
// One block owns one (b, l) row: the [Di, Do] tiles of lw and uw are read from HBM once, kept in
// shared memory through every stage, and the result is written once: 4 tensor passes instead of
// the 18 of the four separate kernels.  Intermediate bounds are never materialised; each stage
// recomputes the rescaled values (lw * k) with the same single-rounding product the separate
// kernels use, so the result matches the unfused chain bit for bit up to the order of the sums.
#include "common.cuh"

namespace fb {
namespace {

constexpr int kThreads = 256;

// Block-wide reduction of one value per thread (sum or max); result valid in every thread.
__device__ __forceinline__ float block_reduce(float v, int p, float* s_tmp) {
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) v = norm_combine(p, v, __shfl_xor_sync(0xffffffffu, v, s));
  __syncthreads();  // s_tmp may still be read from a previous call
  if ((threadIdx.x & 31) == 0) s_tmp[threadIdx.x >> 5] = v;
  __syncthreads();
  float r = s_tmp[0];
#pragma unroll
  for (int w = 1; w < kThreads / 32; ++w) r = norm_combine(p, r, s_tmp[w]);
  return r;
}

// kP: the norm of the perturbation (FB_P1, FB_P2, FB_PINF) as a template parameter, so that the per-element
// accumulation of the dual norms compiles to one or two instructions instead of a chain of tests.
// kCW: columns of the tile (the smallest of 16, 32, 64 that holds Do).  kVec: rows of lw, uw and of the result are ld floats
// apart with ld a multiple of four and 16-byte aligned bases (columns beyond Do are padding: read as zero, written as
// zero); otherwise (rows of an odd length, one after the other) the tile is copied between global and shared memory
// as the flat array it is, so that the accesses stay coalesced.
template <int kP, int kCW, bool kVec>
__global__ void __launch_bounds__(kThreads)
softmax_bounds_kernel(const float* __restrict__ lw, const float* __restrict__ uw, const float* __restrict__ lb,
                      const float* __restrict__ ub, float* __restrict__ o_lw, float* __restrict__ o_uw,
                      float* __restrict__ o_lb, float* __restrict__ o_ub, float* __restrict__ o_l,
                      float* __restrict__ o_u, int Di, int Do, int ld, int words, float eps,
                      int* __restrict__ violation) {
  pdl_sync();
  constexpr int p = kP;
  constexpr int CVL = kCW / 4, RG = kThreads / CVL;   // column lanes (float4) x row groups
  extern __shared__ __align__(16) float smem[];
  float* s_l = smem;                       // [Di][kCW] scores lw
  float* s_u = s_l + (size_t)Di * kCW;     // [Di][kCW] scores uw
  float* s_sl = s_u + (size_t)Di * kCW;    // [Di] row sum of exp.lw
  float* s_su = s_sl + Di;                 // [Di] row sum of exp.uw
  float* s_red = s_su + Di;                // [2][8][kCW] column partials
  float* s_col = s_red + 2 * 8 * kCW;      // [8][kCW] per-column scalars
  float* s_tmp = s_col + 8 * kCW;          // [8] block-reduce scratch, [8..16) scalars
  const int64_t row = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int cvl = tid % CVL, rg = tid / CVL;
  const int col = cvl * 4;
  const bool col_ok = col < Do;
  const int blk = Di / words;
  const float* gl = lw + (size_t)row * Di * ld;
  const float* gu = uw + (size_t)row * Di * ld;
  if (!kVec) {   // the tile as a flat array, columns beyond Do zeroed
    for (int i = tid; i < Di * kCW; i += kThreads)
      if (i % kCW >= Do) s_l[i] = s_u[i] = 0.f;
#pragma unroll 4
    for (int i = tid; i < Di * Do; i += kThreads) {
      const int r = i / Do, c = i - r * Do;
      s_l[r * kCW + c] = __ldg(gl + i);
      s_u[r * kCW + c] = __ldg(gu + i);
    }
    __syncthreads();
  }

  // column-wise dual norm of (a[r][c] * ka[c], b[r][c] * kb[c]) over the rows of every word block,
  // added word by word onto the start values in nl / nu (the bias terms), as the reference's
  // concretize does; result for threads tid < 32 (column tid)
  // With row_sums (second pass only) the same scaled values also give the sums over the features of every
  // row, s_sl / s_su: the denominator of the softmax.
  auto column_norms = [&](bool from_global, bool row_sums, const float* ka, const float* kb, float& nl, float& nu) {
    float tl = nl, tu = nu;
    for (int w = 0; w < words; ++w) {
      float al[4] = {0.f, 0.f, 0.f, 0.f}, au[4] = {0.f, 0.f, 0.f, 0.f};
      for (int r = w * blk + rg; r < (w + 1) * blk; r += RG) {
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
        if (from_global && !kVec) {
          a = *reinterpret_cast<const float4*>(s_l + r * kCW + col);
          b = *reinterpret_cast<const float4*>(s_u + r * kCW + col);
        } else if (from_global) {
          if (col_ok) {
            a = __ldg(reinterpret_cast<const float4*>(gl + (size_t)r * ld + col));
            b = __ldg(reinterpret_cast<const float4*>(gu + (size_t)r * ld + col));
            if (col + 4 > Do) {   // the last group of a row that is padded to a multiple of four
              if (col + 1 >= Do) a.y = b.y = 0.f;
              if (col + 2 >= Do) a.z = b.z = 0.f;
              a.w = b.w = 0.f;
            }
          }
          *reinterpret_cast<float4*>(s_l + r * kCW + col) = a;
          *reinterpret_cast<float4*>(s_u + r * kCW + col) = b;
        } else {
          a = *reinterpret_cast<const float4*>(s_l + r * kCW + col);
          b = *reinterpret_cast<const float4*>(s_u + r * kCW + col);
          a.x = fmul(a.x, ka[col + 0]); a.y = fmul(a.y, ka[col + 1]); a.z = fmul(a.z, ka[col + 2]); a.w = fmul(a.w, ka[col + 3]);
          b.x = fmul(b.x, kb[col + 0]); b.y = fmul(b.y, kb[col + 1]); b.z = fmul(b.z, kb[col + 2]); b.w = fmul(b.w, kb[col + 3]);
          if (row_sums) {
            // the lanes that share a row add their four columns each
            const unsigned group = CVL == 32 ? 0xffffffffu : ((1u << CVL) - 1u) << (lane & ~(CVL - 1));
            float sa = fadd(fadd(a.x, a.y), fadd(a.z, a.w));
            float sb = fadd(fadd(b.x, b.y), fadd(b.z, b.w));
#pragma unroll
            for (int s = 1; s < CVL; s <<= 1) {
              sa += __shfl_xor_sync(group, sa, s);
              sb += __shfl_xor_sync(group, sb, s);
            }
            if (cvl == 0) { s_sl[r] = sa; s_su[r] = sb; }
          }
        }
        al[0] = norm_accum(p, al[0], a.x); al[1] = norm_accum(p, al[1], a.y); al[2] = norm_accum(p, al[2], a.z); al[3] = norm_accum(p, al[3], a.w);
        au[0] = norm_accum(p, au[0], b.x); au[1] = norm_accum(p, au[1], b.y); au[2] = norm_accum(p, au[2], b.z); au[3] = norm_accum(p, au[3], b.w);
      }
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int s = CVL; s < 32; s <<= 1) {
          al[e] = norm_combine(p, al[e], __shfl_xor_sync(0xffffffffu, al[e], s));
          au[e] = norm_combine(p, au[e], __shfl_xor_sync(0xffffffffu, au[e], s));
        }
      __syncthreads();
      if (lane < CVL) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          s_red[warp * kCW + lane * 4 + e] = al[e];
          s_red[8 * kCW + warp * kCW + lane * 4 + e] = au[e];
        }
      }
      __syncthreads();
      if (tid < kCW) {
        float sl = s_red[tid], su = s_red[8 * kCW + tid];
#pragma unroll
        for (int k = 1; k < 8; ++k) {
          sl = norm_combine(p, sl, s_red[k * kCW + tid]);
          su = norm_combine(p, su, s_red[8 * kCW + k * kCW + tid]);
        }
        tl = fadd(tl, fmul(-eps, norm_finish(p, sl)));
        tu = fadd(tu, fmul(eps, norm_finish(p, su)));
      }
    }
    nl = tl;
    nu = tu;
  };

  // ---- stage 1: concretise the scores, exp relaxation per column (Bounds.py:970-1003)
  const bool mine = tid < kCW && tid < Do;
  float lbv = 0.f, ubv = 0.f;
  if (mine) { lbv = lb[row * Do + tid]; ubv = ub[row * Do + tid]; }
  float l = lbv, u = ubv;
  column_norms(true, false, nullptr, nullptr, l, u);
  float* c_kl = s_col + 0 * kCW;   // exp slope on lw
  float* c_ku = s_col + 1 * kCW;   // exp slope on uw
  float* c_elb = s_col + 2 * kCW;  // exp.lb
  float* c_eub = s_col + 3 * kCW;  // exp.ub
  float* c_la = s_col + 4 * kCW;   // concretised lower bound of exp
  if (tid < kCW) {
    ColCoef c = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    bool bad = false;
    if (mine) c = relax_column(FB_EXP, l, u, lbv, ubv, bad);
    c_kl[tid] = c.c_ll; c_ku[tid] = c.c_uu; c_elb[tid] = c.nlb; c_eub[tid] = c.nub;
  }
  __syncthreads();
  // ---- stage 2: row sums of exp.lw / exp.uw over the features, and the lower range of exp (one pass over
  // the tiles: the scaled values feed both)
  float la = mine ? c_elb[tid] : 0.f, ua_unused = mine ? c_eub[tid] : 0.f;
  column_norms(false, true, c_kl, c_ku, la, ua_unused);
  if (tid < kCW) c_la[tid] = la;
  // ---- stage 3: bounds of the sum, reciprocal relaxation (Bounds.py:1136-1161), range of 1/sum
  float s_lb = 0.f, s_ub = 0.f;
  if (warp == 0) {
    float vlb = lane < kCW ? c_elb[lane] : 0.f, vub = lane < kCW ? c_eub[lane] : 0.f;   // (zero beyond Do)
    if (kCW == 64) {
      vlb = fadd(vlb, c_elb[lane + 32]);
      vub = fadd(vub, c_eub[lane + 32]);
    }
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) { vlb += __shfl_xor_sync(0xffffffffu, vlb, s); vub += __shfl_xor_sync(0xffffffffu, vub, s); }
    if (lane == 0) { s_tmp[8] = vlb; s_tmp[9] = vub; }
  }
  __syncthreads();
  s_lb = s_tmp[8]; s_ub = s_tmp[9];
  float ls = s_lb, us = s_ub;
  for (int w = 0; w < words; ++w) {
    float al = 0.f, au = 0.f;
    for (int r = w * blk + tid; r < (w + 1) * blk; r += kThreads) { al = norm_accum(p, al, s_sl[r]); au = norm_accum(p, au, s_su[r]); }
    al = block_reduce(al, p, s_tmp);
    au = block_reduce(au, p, s_tmp);
    ls = fadd(ls, fmul(-eps, norm_finish(p, al)));
    us = fadd(us, fmul(eps, norm_finish(p, au)));
  }
  bool bad = false;
  const ColCoef rc = relax_column(FB_RECIPROCAL, ls, us, s_lb, s_ub, bad);   // same in every thread
  if (bad && tid == 0 && violation != nullptr) *violation = 1;
  const float kl_r = rc.c_lu, ku_r = rc.c_ul;    // 1/sum: lower line = kl_r * sum.uw, upper = ku_r * sum.lw
  float lr = rc.nlb, ur = rc.nub;
  for (int w = 0; w < words; ++w) {
    float al = 0.f, au = 0.f;
    for (int r = w * blk + tid; r < (w + 1) * blk; r += kThreads) {
      al = norm_accum(p, al, fmul(s_su[r], kl_r));
      au = norm_accum(p, au, fmul(s_sl[r], ku_r));
    }
    al = block_reduce(al, p, s_tmp);
    au = block_reduce(au, p, s_tmp);
    lr = fadd(lr, fmul(-eps, norm_finish(p, al)));
    ur = fadd(ur, fmul(eps, norm_finish(p, au)));
  }
  // ---- stage 4: McCormick product exp * (1/sum)  (Bounds.py:608-651, 680-688)
  // lower plane: alpha = l(1/sum) on exp, beta = l(exp) on 1/sum; upper plane: alpha = u(1/sum), beta = l(exp)
  const float al_ = lr, au_ = ur;
  __syncthreads();
  float res_lb = 0.f, res_ub = 0.f;   // bias terms of the result, column tid
  if (mine) {
    const float be = c_la[tid];
    const float gl_ = fmul(-al_, be), gu_ = fmul(-au_, be);
    const float tl = fadd(fmul(al_ > 0.f ? c_elb[tid] : c_eub[tid], al_), gl_);
    const float tu = fadd(fmul(au_ > 0.f ? c_eub[tid] : c_elb[tid], au_), gu_);
    res_lb = fadd(tl, fmul(be > 0.f ? rc.nlb : rc.nub, be));
    res_ub = fadd(tu, fmul(be > 0.f ? rc.nub : rc.nlb, be));
    o_lb[row * Do + tid] = res_lb;
    o_ub[row * Do + tid] = res_ub;
  }
  const bool want_ranges = o_l != nullptr;   // uniform
  if (kVec && !col_ok && !want_ranges) return;
  float kl[4] = {0.f, 0.f, 0.f, 0.f}, ku[4] = {0.f, 0.f, 0.f, 0.f}, be[4] = {0.f, 0.f, 0.f, 0.f};
  if (col_ok) {
#pragma unroll
    for (int e = 0; e < 4; ++e) { kl[e] = c_kl[col + e]; ku[e] = c_ku[col + e]; be[e] = c_la[col + e]; }
  }
  float* ol = o_lw + (size_t)row * Di * ld;
  float* ou = o_uw + (size_t)row * Di * ld;
  // The rows are walked word block by word block, so that the dual norms of the result (its concretised
  // range, for the product that consumes the probabilities) can be accumulated on the way out.
  for (int w = 0; w < words; ++w) {
    float nl[4] = {0.f, 0.f, 0.f, 0.f}, nu[4] = {0.f, 0.f, 0.f, 0.f};
    if (col_ok) {
      for (int r = w * blk + rg; r < (w + 1) * blk; r += RG) {
        const float4 a4 = *reinterpret_cast<const float4*>(s_l + r * kCW + col);
        const float4 b4 = *reinterpret_cast<const float4*>(s_u + r * kCW + col);
        const float a[4] = {a4.x, a4.y, a4.z, a4.w}, b[4] = {b4.x, b4.y, b4.z, b4.w};
        const float r_l = fmul(s_su[r], kl_r), r_u = fmul(s_sl[r], ku_r);
        float yl[4], yu[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float e_l = fmul(a[e], kl[e]), e_u = fmul(b[e], ku[e]);
          yl[e] = fadd(fmul(al_ > 0.f ? e_l : e_u, al_), fmul(be[e] > 0.f ? r_l : r_u, be[e]));
          yu[e] = fadd(fmul(au_ > 0.f ? e_u : e_l, au_), fmul(be[e] > 0.f ? r_u : r_l, be[e]));
          nl[e] = norm_accum(p, nl[e], yl[e]);
          nu[e] = norm_accum(p, nu[e], yu[e]);
        }
        float* const pl = kVec ? ol + (size_t)r * ld + col : s_l + r * kCW + col;   // !kVec: in place, copied out below
        float* const pu = kVec ? ou + (size_t)r * ld + col : s_u + r * kCW + col;
        *reinterpret_cast<float4*>(pl) = make_float4(yl[0], yl[1], yl[2], yl[3]);
        *reinterpret_cast<float4*>(pu) = make_float4(yu[0], yu[1], yu[2], yu[3]);
      }
    }
    if (want_ranges) {
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int s = CVL; s < 32; s <<= 1) {
          nl[e] = norm_combine(p, nl[e], __shfl_xor_sync(0xffffffffu, nl[e], s));
          nu[e] = norm_combine(p, nu[e], __shfl_xor_sync(0xffffffffu, nu[e], s));
        }
      __syncthreads();
      if (lane < CVL) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          s_red[warp * kCW + lane * 4 + e] = nl[e];
          s_red[8 * kCW + warp * kCW + lane * 4 + e] = nu[e];
        }
      }
      __syncthreads();
      if (tid < kCW) {
        float sl = s_red[tid], su = s_red[8 * kCW + tid];
#pragma unroll
        for (int k = 1; k < 8; ++k) {
          sl = norm_combine(p, sl, s_red[k * kCW + tid]);
          su = norm_combine(p, su, s_red[8 * kCW + k * kCW + tid]);
        }
        res_lb = fadd(res_lb, fmul(-eps, norm_finish(p, sl)));
        res_ub = fadd(res_ub, fmul(eps, norm_finish(p, su)));
      }
    }
  }
  if (want_ranges && mine) {
    o_l[row * Do + tid] = res_lb;
    o_u[row * Do + tid] = res_ub;
  }
  if (!kVec) {
    __syncthreads();
    for (int i = tid; i < Di * Do; i += kThreads) {
      const int r = i / Do, c = i - r * Do;
      ol[i] = s_l[r * kCW + c];
      ou[i] = s_u[r * kCW + c];
    }
  }
}

// The same operator with the tile in registers, where the rows split evenly: KR rows (of RG = T / (kCW / 4) row groups) per
// thread, a word block a multiple of RG rows.  The kernel above walks its shared-memory tile five times with eleven block-wide
// barriers between the walks; here a value is read once, scaled in place, and five barriers remain: the reductions over the rows meet in shared memory once per stage and every warp
// finishes the ones it needs itself.  Same rounding of every element; sums in another order.
// vec: rows of 16-byte aligned groups of four (columns beyond Do are padding), else 4-byte accesses.
template <int kP, int kCW, int T, int KR>
__global__ void __launch_bounds__(T, (KR > 4 ? 512 : 768) / T)
softmax_bounds_regs(const float* __restrict__ lw, const float* __restrict__ uw, const float* __restrict__ lb,
                    const float* __restrict__ ub, float* __restrict__ o_lw, float* __restrict__ o_uw,
                    float* __restrict__ o_lb, float* __restrict__ o_ub, float* __restrict__ o_l, float* __restrict__ o_u,
                    int Do, int ld, int words, float eps, int vec, int* __restrict__ violation) {
  pdl_sync();
  constexpr int p = kP, CVL = kCW / 4, RG = T / CVL, W = T / 32, Di = RG * KR;
  __shared__ float4 s_part[2][W][CVL];     // column partials of the warps, lower and upper line
  __shared__ float s_col[5][kCW];          // slopes, bias terms and lower range of exp
  __shared__ float s_row[2][Di];           // row sums of exp
  const int64_t row = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int cvl = tid % CVL, rg = tid / CVL, col = cvl * 4;
  const int kw = KR / words;               // rows per thread and word block
  const size_t base = (size_t)row * Di * ld + (size_t)rg * ld + col;
  float a[KR][4], b[KR][4];
#pragma unroll
  for (int k = 0; k < KR; ++k) {
    const float* const pl = lw + base + (size_t)k * RG * ld;
    const float* const pu = uw + base + (size_t)k * RG * ld;
    if (vec) {
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f), y = x;
      if (col < Do) { x = __ldg(reinterpret_cast<const float4*>(pl)); y = __ldg(reinterpret_cast<const float4*>(pu)); }
      a[k][0] = x.x; a[k][1] = x.y; a[k][2] = x.z; a[k][3] = x.w;
      b[k][0] = y.x; b[k][1] = y.y; b[k][2] = y.z; b[k][3] = y.w;
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        a[k][e] = col + e < Do ? __ldg(pl + e) : 0.f;
        b[k][e] = col + e < Do ? __ldg(pu + e) : 0.f;
      }
    }
  }
  if (vec && col + 4 > Do) {
#pragma unroll
    for (int k = 0; k < KR; ++k)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (col + e >= Do) a[k][e] = b[k][e] = 0.f;
  }
  // this thread's columns of one word block -> the warp's partials in s_part
  auto partials = [&](int w, const float (&x)[KR][4], const float (&y)[KR][4]) {
    float nl[4] = {0.f, 0.f, 0.f, 0.f}, nu[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 0; k < KR; ++k) {
      if (k / kw != w) continue;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        nl[e] = norm_accum(p, nl[e], x[k][e]);
        nu[e] = norm_accum(p, nu[e], y[k][e]);
      }
    }
    if constexpr (CVL == 8) {
      // every lane gives away the values it does not keep and ends with two columns of one line: 6 shuffles instead of 16
      const bool up8 = lane & 8, up16 = lane & 16;
      float h[4], g[2];
#pragma unroll
      for (int e = 0; e < 4; ++e) h[e] = norm_combine(p, up8 ? nu[e] : nl[e], __shfl_xor_sync(0xffffffffu, up8 ? nl[e] : nu[e], 8));
#pragma unroll
      for (int e = 0; e < 2; ++e)
        g[e] = norm_combine(p, up16 ? h[2 + e] : h[e], __shfl_xor_sync(0xffffffffu, up16 ? h[e] : h[2 + e], 16));
      reinterpret_cast<float2*>(&s_part[up8 ? 1 : 0][warp][cvl])[up16 ? 1 : 0] = make_float2(g[0], g[1]);
      return;
    }
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
      for (int s = CVL; s < 32; s <<= 1) {
        nl[e] = norm_combine(p, nl[e], __shfl_xor_sync(0xffffffffu, nl[e], s));
        nu[e] = norm_combine(p, nu[e], __shfl_xor_sync(0xffffffffu, nu[e], s));
      }
    if (lane < CVL) {
      s_part[0][warp][lane] = make_float4(nl[0], nl[1], nl[2], nl[3]);
      s_part[1][warp][lane] = make_float4(nu[0], nu[1], nu[2], nu[3]);
    }
  };
  auto column_norm = [&](int side, int c) -> float {   // finished norm of column c over the word block in s_part
    const float* q = reinterpret_cast<const float*>(&s_part[side][0][0]) + c;
    float v = q[0];
#pragma unroll 3
    for (int w = 1; w < W; ++w) v = norm_combine(p, v, q[w * kCW]);
    return norm_finish(p, v);
  };
  // ---- exp relaxation per column (Bounds.py:970-1003) from the range of the scores
  const bool mine = tid < Do;
  const float lbv = mine ? lb[row * Do + tid] : 0.f, ubv = mine ? ub[row * Do + tid] : 0.f;
  float l = lbv, u = ubv;
  for (int w = 0; w < words; ++w) {
    if (w > 0) __syncthreads();
    partials(w, a, b);
    __syncthreads();
    if (mine) {
      l = fadd(l, fmul(-eps, column_norm(0, tid)));
      u = fadd(u, fmul(eps, column_norm(1, tid)));
    }
  }
  if (tid < kCW) {
    ColCoef c = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    bool bad = false;
    if (mine) c = relax_column(FB_EXP, l, u, lbv, ubv, bad);
    s_col[0][tid] = c.c_ll; s_col[1][tid] = c.c_uu; s_col[2][tid] = c.nlb; s_col[3][tid] = c.nub;
  }
  __syncthreads();
  // ---- exp in place, its row sums, and the lower range of its columns
  {
    const float4 kl = *reinterpret_cast<const float4*>(&s_col[0][col]), ku = *reinterpret_cast<const float4*>(&s_col[1][col]);
#pragma unroll
    for (int k = 0; k < KR; ++k) {
      a[k][0] = fmul(a[k][0], kl.x); a[k][1] = fmul(a[k][1], kl.y); a[k][2] = fmul(a[k][2], kl.z); a[k][3] = fmul(a[k][3], kl.w);
      b[k][0] = fmul(b[k][0], ku.x); b[k][1] = fmul(b[k][1], ku.y); b[k][2] = fmul(b[k][2], ku.z); b[k][3] = fmul(b[k][3], ku.w);
    }
  }
  // row sums of exp over the CVL lanes of a row, to s_row
#pragma unroll
  for (int k0 = 0; k0 < KR; k0 += 4) {
    constexpr int NK = KR < 4 ? KR : 4;
    float v[4][2];
#pragma unroll
    for (int k = 0; k < NK; ++k) {
      v[k][0] = fadd(fadd(a[k0 + k][0], a[k0 + k][1]), fadd(a[k0 + k][2], a[k0 + k][3]));
      v[k][1] = fadd(fadd(b[k0 + k][0], b[k0 + k][1]), fadd(b[k0 + k][2], b[k0 + k][3]));
    }
    if constexpr (NK == 4 && CVL == 8) {   // eight sums over eight lanes: a lane ends with one of them, 7 shuffles instead of 24
      const bool b0 = lane & 1, b1 = lane & 2, b2 = lane & 4;
      float x[2][2], y[2];
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int e = 0; e < 2; ++e) x[k][e] = (b0 ? v[2 + k][e] : v[k][e]) + __shfl_xor_sync(0xffffffffu, b0 ? v[k][e] : v[2 + k][e], 1);
#pragma unroll
      for (int e = 0; e < 2; ++e) y[e] = (b1 ? x[1][e] : x[0][e]) + __shfl_xor_sync(0xffffffffu, b1 ? x[0][e] : x[1][e], 2);
      const float z = (b2 ? y[1] : y[0]) + __shfl_xor_sync(0xffffffffu, b2 ? y[0] : y[1], 4);
      s_row[b2 ? 1 : 0][(k0 + (b0 ? 2 : 0) + (b1 ? 1 : 0)) * RG + rg] = z;
    } else {
#pragma unroll
      for (int k = 0; k < NK; ++k) {
#pragma unroll
        for (int s = 1; s < CVL; s <<= 1) {
          v[k][0] += __shfl_xor_sync(0xffffffffu, v[k][0], s);
          v[k][1] += __shfl_xor_sync(0xffffffffu, v[k][1], s);
        }
        if (cvl == 0) { s_row[0][(k0 + k) * RG + rg] = v[k][0]; s_row[1][(k0 + k) * RG + rg] = v[k][1]; }
      }
    }
  }
  float la = mine ? s_col[2][tid] : 0.f;
  for (int w = 0; w < words; ++w) {
    if (w > 0) __syncthreads();
    partials(w, a, b);
    __syncthreads();
    if (mine) la = fadd(la, fmul(-eps, column_norm(0, tid)));
  }
  if (tid < kCW) s_col[4][tid] = la;
  // ---- bounds of the sum, reciprocal relaxation (Bounds.py:1136-1161), range of 1/sum: every warp for itself
  float s_lb = 0.f, s_ub = 0.f;
#pragma unroll
  for (int c = lane; c < kCW; c += 32) { s_lb = fadd(s_lb, s_col[2][c]); s_ub = fadd(s_ub, s_col[3][c]); }
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) { s_lb += __shfl_xor_sync(0xffffffffu, s_lb, s); s_ub += __shfl_xor_sync(0xffffffffu, s_ub, s); }
  // l - eps * sum_w ||s_row[i] * kl||, u + eps * sum_w ||s_row[j] * ku||
  auto sum_range = [&](int i, int j, float kl, float ku, float& lo, float& hi) {
    const int blk = Di / words;
    for (int w = 0; w < words; ++w) {
      float al = 0.f, au = 0.f;
      for (int r = w * blk + lane; r < (w + 1) * blk; r += 32) {
        al = norm_accum(p, al, fmul(s_row[i][r], kl));
        au = norm_accum(p, au, fmul(s_row[j][r], ku));
      }
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) {
        al = norm_combine(p, al, __shfl_xor_sync(0xffffffffu, al, s));
        au = norm_combine(p, au, __shfl_xor_sync(0xffffffffu, au, s));
      }
      lo = fadd(lo, fmul(-eps, norm_finish(p, al)));
      hi = fadd(hi, fmul(eps, norm_finish(p, au)));
    }
  };
  float ls = s_lb, us = s_ub;
  sum_range(0, 1, 1.f, 1.f, ls, us);
  bool bad = false;
  const ColCoef rc = relax_column(FB_RECIPROCAL, ls, us, s_lb, s_ub, bad);
  if (bad && tid == 0 && violation != nullptr) *violation = 1;
  const float kl_r = rc.c_lu, ku_r = rc.c_ul;    // 1/sum: lower line = kl_r * sum.uw, upper = ku_r * sum.lw
  float al_ = rc.nlb, au_ = rc.nub;
  sum_range(1, 0, kl_r, ku_r, al_, au_);
  // ---- McCormick product exp * (1/sum)  (Bounds.py:608-651, 680-688)
  __syncthreads();   // s_col[4]
  const float4 be4 = *reinterpret_cast<const float4*>(&s_col[4][col]);
  const float be[4] = {be4.x, be4.y, be4.z, be4.w};
#pragma unroll
  for (int k = 0; k < KR; ++k) {
    const float r_l = fmul(s_row[1][k * RG + rg], kl_r), r_u = fmul(s_row[0][k * RG + rg], ku_r);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float e_l = a[k][e], e_u = b[k][e];
      a[k][e] = fadd(fmul(al_ > 0.f ? e_l : e_u, al_), fmul(be[e] > 0.f ? r_l : r_u, be[e]));
      b[k][e] = fadd(fmul(au_ > 0.f ? e_u : e_l, au_), fmul(be[e] > 0.f ? r_u : r_l, be[e]));
    }
    float* const pl = o_lw + base + (size_t)k * RG * ld;
    float* const pu = o_uw + base + (size_t)k * RG * ld;
    if (vec) {
      if (col < Do) {
        *reinterpret_cast<float4*>(pl) = make_float4(a[k][0], a[k][1], a[k][2], a[k][3]);
        *reinterpret_cast<float4*>(pu) = make_float4(b[k][0], b[k][1], b[k][2], b[k][3]);
      }
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (col + e < Do) { pl[e] = a[k][e]; pu[e] = b[k][e]; }
    }
  }
  float res_l = 0.f, res_u = 0.f;   // bias terms of the result, column tid
  if (mine) {
    const float elb = s_col[2][tid], eub = s_col[3][tid];
    const float tl = fadd(fmul(al_ > 0.f ? elb : eub, al_), fmul(-al_, la));
    const float tu = fadd(fmul(au_ > 0.f ? eub : elb, au_), fmul(-au_, la));
    res_l = fadd(tl, fmul(la > 0.f ? rc.nlb : rc.nub, la));
    res_u = fadd(tu, fmul(la > 0.f ? rc.nub : rc.nlb, la));
    o_lb[row * Do + tid] = res_l;
    o_ub[row * Do + tid] = res_u;
  }
  if (o_l == nullptr) return;   // uniform
  for (int w = 0; w < words; ++w) {
    if (w > 0) __syncthreads();
    partials(w, a, b);   // (the partials of the stage before were read ahead of the last barrier)
    __syncthreads();
    if (mine) {
      res_l = fadd(res_l, fmul(-eps, column_norm(0, tid)));
      res_u = fadd(res_u, fmul(eps, column_norm(1, tid)));
    }
  }
  if (mine) {
    o_l[row * Do + tid] = res_l;
    o_u[row * Do + tid] = res_u;
  }
}

int tile_columns(int Do) { return Do <= 16 ? 16 : Do <= 32 ? 32 : 64; }
size_t smem_bytes(int Di, int cw) { return sizeof(float) * ((size_t)2 * Di * cw + 2 * Di + 2 * 8 * cw + 8 * cw + 16); }

}  // namespace
}  // namespace fb

using namespace fb;

// The whole feature axis in one tile, and the two tiles in shared memory.
bool fb::softmax_fused_shape(int Di, int Do) {
  return Do <= 64 && smem_bytes(Di, tile_columns(Do)) <= (size_t)device_info().smem_optin;
}

// out_l / out_u (both or neither): concretised range of the result, [rows, Do], as fb_concretize_f32 would return
// it for the written bounds; the kernel accumulates the dual norms while it writes the result.
// ld: floats between consecutive rows of Do values in lw, uw, out_lw, out_uw.
int fb::softmax_ex(const float* lw, const float* uw, const float* lb, const float* ub, float* out_lw, float* out_uw, float* out_lb,
                   float* out_ub, float* out_l, float* out_u, int64_t rows, int Di, int Do, int ld, int words, int p, float eps,
                   int* violation, void* stream) {
  if ((out_l == nullptr) != (out_u == nullptr)) return FB_ERR_ARG;
  if (rows == 0) return FB_OK;
  if (!lw || !uw || !lb || !ub || !out_lw || !out_uw || !out_lb || !out_ub) return FB_ERR_ARG;
  if (rows < 0 || Di <= 0 || Do <= 0 || words <= 0 || !valid_norm(p) || ld < Do) return FB_ERR_ARG;
  if (Di % words != 0) return FB_ERR_SHAPE;
  if (!softmax_fused_shape(Di, Do) || rows > 0x7fffffff) return FB_ERR_SHAPE;
  const int cw = tile_columns(Do);
  const size_t smem = smem_bytes(Di, cw);
  const bool vec = ld % 4 == 0 && aligned16(lw) && aligned16(uw) && aligned16(out_lw) && aligned16(out_uw);
  if (!vec && ld != Do) return FB_ERR_ALIGN;
  const double mw = (double)rows * Di * Do, mb = (double)rows * Do;
  ProfileScope prof(PK_RELAX, 30.0 * mw, 4.0 * (4 * mw + 4 * mb), stream);
  // The tile in registers: rows split evenly over the threads, word blocks over the row groups; blocks of up to 256 threads
  // (512, for dim_in 256 or lengths above 32, leave one block per SM and take 456 instead of 256 us for 8064 rows; 256 threads
  // with eight rows each, two blocks per SM: 2016 rows of [256, 21] 86 -> 76 us).
  // 32768 rows of [128, 32]: 483 -> 448 us, 437 -> 427 us with the exchanges that give values away; 6144 rows of [128, 12]: 88 ->
  // 46 us.
#define FB_SOFTMAX_REGS(C, T, K)                                                                                       \
  if (cw == C && Di == T / (C / 4) * K && K % words == 0) {                                                            \
    if (p == FB_PINF) FB_SOFTMAX_REGS_LAUNCH(FB_PINF, C, T, K);                                                        \
    else if (p == FB_P2) FB_SOFTMAX_REGS_LAUNCH(FB_P2, C, T, K);                                                       \
    else FB_SOFTMAX_REGS_LAUNCH(FB_P1, C, T, K);                                                                       \
    FB_LAUNCH_OK();                                                                                                    \
    return FB_OK;                                                                                                      \
  }
#define FB_SOFTMAX_REGS_LAUNCH(P, C, T, K)                                                                             \
  fb::launch_k(softmax_bounds_regs<P, C, T, K>, (unsigned)rows, T, 0, (cudaStream_t)stream, \
      lw, uw, lb, ub, out_lw, out_uw, out_lb, out_ub, out_l, out_u, Do, ld, words, eps, vec ? 1 : 0, violation)
  FB_SOFTMAX_REGS(32, 256, 4)    // Di 128
  FB_SOFTMAX_REGS(32, 256, 2)    // Di 64
  FB_SOFTMAX_REGS(32, 256, 8)    // Di 256
  FB_SOFTMAX_REGS(16, 128, 4)    // Di 128
  FB_SOFTMAX_REGS(16, 256, 4)    // Di 256
  FB_SOFTMAX_REGS(16, 128, 2)    // Di 64
#undef FB_SOFTMAX_REGS_LAUNCH
#undef FB_SOFTMAX_REGS
#define FB_SOFTMAX_LAUNCH(P, C, V)                                                                                    \
  do {                                                                                                                \
    if (int rc_ = ensure_dynamic_smem(softmax_bounds_kernel<P, C, V>, smem)) return rc_;                               \
    fb::launch_k(softmax_bounds_kernel<P, C, V>, (unsigned)rows, kThreads, smem, (cudaStream_t)stream, \
        lw, uw, lb, ub, out_lw, out_uw, out_lb, out_ub, out_l, out_u, Di, Do, ld, words, eps, violation);              \
  } while (0)
#define FB_SOFTMAX_NORM(C, V)                                  \
  do {                                                         \
    if (p == FB_PINF) FB_SOFTMAX_LAUNCH(FB_PINF, C, V);        \
    else if (p == FB_P2) FB_SOFTMAX_LAUNCH(FB_P2, C, V);       \
    else FB_SOFTMAX_LAUNCH(FB_P1, C, V);                       \
  } while (0)
  if (vec && cw == 16) FB_SOFTMAX_NORM(16, true);
  else if (vec && cw == 32) FB_SOFTMAX_NORM(32, true);
  else if (vec) FB_SOFTMAX_NORM(64, true);
  else if (cw == 16) FB_SOFTMAX_NORM(16, false);
  else if (cw == 32) FB_SOFTMAX_NORM(32, false);
  else FB_SOFTMAX_NORM(64, false);
#undef FB_SOFTMAX_NORM
#undef FB_SOFTMAX_LAUNCH
  FB_LAUNCH_OK();
  return FB_OK;
}

extern "C" int fb_softmax_ranges_f32(const float* lw, const float* uw, const float* lb, const float* ub, float* out_lw,
                                     float* out_uw, float* out_lb, float* out_ub, float* out_l, float* out_u,
                                     int64_t rows, int Di, int Do, int words, int p, float eps, int* violation,
                                     void* stream) {
  return fb::softmax_ex(lw, uw, lb, ub, out_lw, out_uw, out_lb, out_ub, out_l, out_u, rows, Di, Do, Do, words, p, eps, violation,
                        stream);
}

extern "C" int fb_softmax_f32(const float* lw, const float* uw, const float* lb, const float* ub, float* out_lw,
                              float* out_uw, float* out_lb, float* out_ub, int64_t rows, int Di, int Do, int words,
                              int p, float eps, int* violation, void* stream) {
  return fb_softmax_ranges_f32(lw, uw, lb, ub, out_lw, out_uw, out_lb, out_ub, nullptr, nullptr, rows, Di, Do, words, p,
                               eps, violation, stream);
}
