// Layer normalisation with the variance ("standard", Bounds.py:1111-1131) in one kernel.
//
// The reference's chain on a bound x is: centre by the mean (lw - mean(uw), uw - mean(lw)), variance = mean over the
// features of sqr(centred) (:860-890), + 1e-12, sqrt (:892-919), reciprocal (:1136-1161), McCormick product with the centred
// bound (:608-651), gain split by sign, shift.  Operator by operator that is twenty launches, each of which reads and writes
// the whole bound, two read-backs of a status word and a product with a constant matrix for the mean.  Here a block owns one
// (b, l) row: every step but the first and the last works on columns of [Di, Do] that the block holds, and the variance,
// its root and the reciprocal have the same value in every feature column, so they are vectors over Di.
//
// The bound is read from memory once (into shared memory, centred, where 2 * Di * Do floats fit) and written once.  Bound by
// HBM for a batch, by latency for a sentence: with one block per position 32 SMs work and each walks [128, 128] four times.
// Where rows are few a cluster of nc blocks shares a row, each with Di / nc of its lines: the partial column norms and the
// variances are exchanged through distributed shared memory, everything that is a vector over the features or over Di every
// block computes for itself.  One sentence of 32 x [128, 128]: the chain took 20 launches and 290 us of a block with two norms, a
// block per row 22 us, a cluster of four 14 us.
#include <cooperative_groups.h>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace fb {
namespace {

constexpr int kT = 512;
constexpr int kWarps = kT / 32;
constexpr float kVarianceGuard = 1e-12f;   // added to the variance before the root (Bounds.py:27, :1123)

struct NormRow {   // one (b, l) row of the operand
  const float *lw, *uw, *lb, *ub;
};

// Finishes the dual norms of a vector pair v_l, v_u [Di] in shared memory: l = lb - eps * sum_w ||v_l||, u likewise, the word
// blocks added one after the other as the reference's concretisation does.  Valid in every thread.
__device__ __forceinline__ void vector_range(const float* v_l, const float* v_u, int Di, int words, int p, float eps, float lb,
                                             float ub, float* s_tmp, float& l, float& u) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int blk = Di / words;
  l = lb;
  u = ub;
  for (int w = 0; w < words; ++w) {
    float a = 0.f, b = 0.f;
    for (int r = w * blk + threadIdx.x; r < (w + 1) * blk; r += kT) {
      a = norm_accum(p, a, v_l[r]);
      b = norm_accum(p, b, v_u[r]);
    }
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
      a = norm_combine(p, a, __shfl_xor_sync(0xffffffffu, a, s));
      b = norm_combine(p, b, __shfl_xor_sync(0xffffffffu, b, s));
    }
    __syncthreads();   // the previous word's (or call's) values have been read
    if (lane == 0) { s_tmp[warp] = a; s_tmp[kWarps + warp] = b; }
    __syncthreads();
    float sa = s_tmp[0], sb = s_tmp[kWarps];
    for (int k = 1; k < kWarps; ++k) {
      sa = norm_combine(p, sa, s_tmp[k]);
      sb = norm_combine(p, sb, s_tmp[kWarps + k]);
    }
    l = fadd(l, fmul(-eps, norm_finish(p, sa)));
    u = fadd(u, fmul(eps, norm_finish(p, sb)));
  }
}

template <bool STAGED>
__global__ void __launch_bounds__(kT)
layernorm_standard_kernel(const float* __restrict__ x_lw, const float* __restrict__ x_uw, const float* __restrict__ x_lb,
                          const float* __restrict__ x_ub, const float* __restrict__ gamma, const float* __restrict__ beta,
                          float* __restrict__ z_lw, float* __restrict__ z_uw, float* __restrict__ z_lb, float* __restrict__ z_ub,
                          int Di, int Do, int words, int p, float eps, int* __restrict__ violation, int nc) {
  pdl_sync();
  extern __shared__ __align__(16) float smem[];
  const int n = Di / nc;                           // weight rows of this block
  const int rank = nc > 1 ? (int)cg::this_cluster().block_rank() : 0, r0 = rank * n;
  const int rows = n + 1;                          // and, last, the bias row
  float* s_mu = smem;                              // [2][rows] row means of lw and uw
  float* s_v = s_mu + 2 * rows;                    // [2][Di] variance, then its root, then the reciprocal
  float* s_tmp = s_v + 2 * Di;                     // [2][kWarps]
  float* s_coef = s_tmp + 2 * kWarps;              // [4][Do] slopes of the square
  float* s_rng = s_coef + 4 * Do;                  // [2][Do] centred range l, u
  float* s_bias = s_rng + 2 * Do;                  // [4][Do] centred bias terms lb, ub; bias terms of the square
  float* s_part = s_bias + 4 * Do;                 // [words][2][Do] accumulated column norms of this block's rows
  float* s_m = s_part + 2 * words * Do;            // [2][n][Do] centred lines (STAGED)
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const size_t row = blockIdx.x / (unsigned)nc;
  const size_t first = (row * Di + r0) * Do;
  const float* gl = x_lw + first;
  const float* gu = x_uw + first;
  auto exchange = [&]() { if (nc > 1) cg::this_cluster().sync(); else __syncthreads(); };
  auto of_rank = [&](float* q, int k) -> const float* { return nc > 1 ? cg::this_cluster().map_shared_rank(q, k) : q; };
  const float* bl = x_lb + row * Do;
  const float* bu = x_ub + row * Do;
  const float inv_n = 1.0f / (float)Do;

  // 1. row means (as fb_layernorm_novar_f32: sum of t * (1/n))
  for (int r = warp; r < rows; r += kWarps) {
    const float* pl = r < n ? gl + (size_t)r * Do : bl;
    const float* pu = r < n ? gu + (size_t)r * Do : bu;
    float ml = 0.f, mu = 0.f;
    for (int j = lane; j < Do; j += 32) {
      const float a = __ldg(pl + j), b = __ldg(pu + j);
      if (STAGED && r < n) {
        s_m[(size_t)r * Do + j] = a;
        s_m[(size_t)(n + r) * Do + j] = b;
      }
      ml = fmaf(a, inv_n, ml);
      mu = fmaf(b, inv_n, mu);
    }
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
      ml += __shfl_xor_sync(0xffffffffu, ml, s);
      mu += __shfl_xor_sync(0xffffffffu, mu, s);
    }
    if (STAGED && r < n) {   // centred in place: each line minus the mean of the other (every lane its own elements)
      for (int j = lane; j < Do; j += 32) {
        s_m[(size_t)r * Do + j] = fsub(s_m[(size_t)r * Do + j], mu);
        s_m[(size_t)(n + r) * Do + j] = fsub(s_m[(size_t)(n + r) * Do + j], ml);
      }
    }
    if (lane == 0) { s_mu[r] = ml; s_mu[rows + r] = mu; }
  }
  __syncthreads();
  auto centred_l = [&](int r, int j) -> float {
    return STAGED ? s_m[(size_t)r * Do + j] : fsub(__ldg(gl + (size_t)r * Do + j), s_mu[rows + r]);
  };
  auto centred_u = [&](int r, int j) -> float {
    return STAGED ? s_m[(size_t)(n + r) * Do + j] : fsub(__ldg(gu + (size_t)r * Do + j), s_mu[r]);
  };

  // 2. range of every centred column and the slopes of its square.  A group of threads shares a column: thread t takes
  //    column c0 + t % cols of the rows t / cols, t / cols + groups, ...; the group results go through s_red, those of the
  //    blocks of a cluster are combined in the order of the blocks.
  const int cols = Do < kT ? Do : kT;
  const int groups = kT / cols;
  const int blk = Di / words;
  __shared__ float s_red[2][kT];   // (beside the dynamic part: see ensure_dynamic_smem)
  bool bad = false;
  for (int c0 = 0; c0 < Do; c0 += cols) {
    const int cc = tid % cols, g = tid / cols, j = c0 + cc;
    for (int w = 0; w < words; ++w) {
      float a = 0.f, b = 0.f;
      if (g < groups && j < Do) {
        const int lo = max(w * blk - r0, 0), hi = min((w + 1) * blk - r0, n);
#pragma unroll 4
        for (int r = lo + g; r < hi; r += groups) {
          a = norm_accum(p, a, centred_l(r, j));
          b = norm_accum(p, b, centred_u(r, j));
        }
      }
      __syncthreads();
      s_red[0][tid] = a;
      s_red[1][tid] = b;
      __syncthreads();
      if (g == 0 && j < Do) {
        for (int k = 1; k < groups; ++k) {
          a = norm_combine(p, a, s_red[0][k * cols + cc]);
          b = norm_combine(p, b, s_red[1][k * cols + cc]);
        }
        s_part[2 * w * Do + j] = a;
        s_part[(2 * w + 1) * Do + j] = b;
      }
    }
  }
  exchange();
  for (int j = tid; j < Do; j += kT) {
    const float lbv = fsub(bl[j], s_mu[rows + n]), ubv = fsub(bu[j], s_mu[n]);
    float l = lbv, u = ubv;
    for (int w = 0; w < words; ++w) {
      const float* q = of_rank(s_part, 0) + 2 * w * Do + j;
      float a = q[0], b = q[Do];
      for (int k = 1; k < nc; ++k) {
        q = of_rank(s_part, k) + 2 * w * Do + j;
        a = norm_combine(p, a, q[0]);
        b = norm_combine(p, b, q[Do]);
      }
      l = fadd(l, fmul(-eps, norm_finish(p, a)));
      u = fadd(u, fmul(eps, norm_finish(p, b)));
    }
    const ColCoef c = relax_column(FB_SQR, l, u, lbv, ubv, bad);
    s_coef[j] = c.c_ll;
    s_coef[Do + j] = c.c_lu;
    s_coef[2 * Do + j] = c.c_ul;
    s_coef[3 * Do + j] = c.c_uu;
    s_rng[j] = l;
    s_rng[Do + j] = u;
    s_bias[j] = lbv;
    s_bias[Do + j] = ubv;
    s_bias[2 * Do + j] = c.nlb;
    s_bias[3 * Do + j] = c.nub;
  }
  __syncthreads();

  // 3. variance: mean over the features of the squared lines, a warp per row (row n: the bias terms)
  float vlb = 0.f, vub = 0.f;
  for (int r = warp; r < rows; r += kWarps) {
    float a = 0.f, b = 0.f;
    for (int j = lane; j < Do; j += 32) {
      if (r < n) {
        const float ml = centred_l(r, j), mu = centred_u(r, j);
        a = fmaf(fmaf(s_coef[j], ml, fmul(s_coef[Do + j], mu)), inv_n, a);
        b = fmaf(fmaf(s_coef[3 * Do + j], mu, fmul(s_coef[2 * Do + j], ml)), inv_n, b);
      } else {
        a = fmaf(s_bias[2 * Do + j], inv_n, a);
        b = fmaf(s_bias[3 * Do + j], inv_n, b);
      }
    }
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, s);
      b += __shfl_xor_sync(0xffffffffu, b, s);
    }
    if (lane == 0) {
      if (r < n) { s_v[r0 + r] = a; s_v[Di + r0 + r] = b; }
      else { s_red[0][0] = fadd(a, kVarianceGuard); s_red[1][0] = fadd(b, kVarianceGuard); }
    }
  }
  exchange();
  if (nc > 1) {   // the variances of the other blocks' rows
    for (int r = tid; r < Di; r += kT) {
      const int k = r / n;
      if (k == rank) continue;
      const float* q = of_rank(s_v, k);
      s_v[r] = q[r];
      s_v[Di + r] = q[Di + r];
    }
    exchange();   // (nobody changes its variances, or leaves, before they have been read)
  }
  vlb = s_red[0][0];
  vub = s_red[1][0];

  // 4. root and reciprocal: the same line for every feature, so they act on the vector over Di
  for (int step = 0; step < 2; ++step) {
    float l, u;
    vector_range(s_v, s_v + Di, Di, words, p, eps, vlb, vub, s_tmp, l, u);
    const ColCoef c = relax_column(step == 0 ? FB_SQRT : FB_RECIPROCAL, l, u, vlb, vub, bad);
    for (int r = tid; r < Di; r += kT) {
      const float a = s_v[r], b = s_v[Di + r];
      s_v[r] = fmaf(c.c_ll, a, fmul(c.c_lu, b));
      s_v[Di + r] = fmaf(c.c_uu, b, fmul(c.c_ul, a));
    }
    vlb = c.nlb;
    vub = c.nub;
    __syncthreads();
  }
  if (bad && violation != nullptr) *violation = 1;
  float ly, uy;
  vector_range(s_v, s_v + Di, Di, words, p, eps, vlb, vub, s_tmp, ly, uy);

  // 5. McCormick product of the centred bound with the reciprocal (planes of col_mul_bounds_native), gain, shift
  for (int j = tid; j < Do && rank == 0; j += kT) {   // bias terms; per column the slope of the reciprocal's lines, be = l of the column
    const float be = s_rng[j];
    const bool alp = ly > 0.f, bep = be > 0.f, aup = uy > 0.f;
    const float xlb = s_bias[j], xub = s_bias[Do + j];
    const float tl = fadd(fmul(alp ? xlb : xub, ly), fmul(-ly, be));
    const float tu = fadd(fmul(aup ? xub : xlb, uy), fmul(-uy, be));
    const float zl = fadd(tl, fmul(bep ? vlb : vub, be)), zu = fadd(tu, fmul(bep ? vub : vlb, be));
    const float gv = gamma[j], gp = gv > 0.f ? gv : 0.f, gn = fsub(gv, gp);
    z_lb[row * Do + j] = fadd(fadd(fmul(zl, gp), fmul(zu, gn)), beta[j]);
    z_ub[row * Do + j] = fadd(fadd(fmul(zl, gn), fmul(zu, gp)), beta[j]);
  }
  const bool alp = ly > 0.f, aup = uy > 0.f;
  float* ol = z_lw + first;
  float* ou = z_uw + first;
  for (int c0 = 0; c0 < Do; c0 += cols) {
    const int cc = tid % cols, g = tid / cols, j = c0 + cc;
    if (g >= groups || j >= Do) continue;
    const float be = s_rng[j], gv = gamma[j], gp = gv > 0.f ? gv : 0.f, gn = fsub(gv, gp);
    const bool bep = be > 0.f;
#pragma unroll 4
    for (int r = g; r < n; r += groups) {
      const float a = centred_l(r, j), b = centred_u(r, j), c = s_v[r0 + r], d = s_v[Di + r0 + r];
      const float zl = fadd(fmul(ly, alp ? a : b), fmul(be, bep ? c : d));
      const float zu = fadd(fmul(uy, aup ? b : a), fmul(be, bep ? d : c));
      ol[(size_t)r * Do + j] = fadd(fmul(zl, gp), fmul(zu, gn));
      ou[(size_t)r * Do + j] = fadd(fmul(zl, gn), fmul(zu, gp));
    }
  }
}

}  // namespace
}  // namespace fb

using namespace fb;

extern "C" int fb_layernorm_standard_f32(const float* x_lw, const float* x_uw, const float* x_lb, const float* x_ub,
                                         const float* gamma, const float* beta, float* z_lw, float* z_uw, float* z_lb, float* z_ub,
                                         int64_t rows, int Di, int Do, int words, int p, float eps, int* violation, void* stream) {
  if (!x_lw || !x_uw || !x_lb || !x_ub || !gamma || !beta || !z_lw || !z_uw || !z_lb || !z_ub) return FB_ERR_ARG;
  if (rows < 0 || Di <= 0 || Do < 0 || words <= 0 || !valid_norm(p)) return FB_ERR_ARG;
  if (Di % words != 0 || rows > 0x7fffffff) return FB_ERR_SHAPE;
  if (z_lw == x_lw || z_lw == x_uw || z_uw == x_lw || z_uw == x_uw || z_lb == x_lb || z_lb == x_ub || z_ub == x_lb || z_ub == x_ub)
    return FB_ERR_ARG;
  if (rows == 0 || Do == 0) return FB_OK;
  // A cluster per row where the blocks would leave SMs idle: as many blocks as there are SMs for (eight at most, the portable
  // limit), with at least eight lines of Di each, since below that the exchanges cost what the walks save.
  const int64_t sms = device_info().sms;
  int nc = 1;
  while (nc < 8 && rows * nc * 2 <= sms && Di % (nc * 2) == 0 && Di / (nc * 2) >= 8) nc *= 2;
  const size_t n = (size_t)(Di / nc);
  const size_t fixed = sizeof(float) * (2 * (n + 1) + 2 * (size_t)Di + 2 * kWarps + (10 + 2 * (size_t)words) * Do);
  const size_t tile = sizeof(float) * 2 * n * Do;
  const size_t limit = (size_t)device_info().smem_optin - sizeof(float) * 2 * kT - 1024;
  if (fixed > limit) return FB_ERR_SHAPE;   // the caller runs the chain operator by operator
  const bool staged = fixed + tile <= limit;
  ProfileScope prof(PK_ELEMENTWISE, 20.0 * rows * (Di + 1) * Do, 16.0 * rows * (Di + 1) * Do, stream);
  const size_t smem = fixed + (staged ? tile : 0);
  const auto kern = staged ? layernorm_standard_kernel<true> : layernorm_standard_kernel<false>;
  if (int rc = ensure_dynamic_smem(kern, smem)) return rc;
  if (nc == 1) {
    fb::launch_k(kern, (unsigned)rows, kT, smem, (cudaStream_t)stream, x_lw, x_uw, x_lb, x_ub, gamma, beta, z_lw, z_uw, z_lb, z_ub, Di, Do, words, p, eps, violation, nc);
  } else {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)nc;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(rows * nc));
    cfg.blockDim = dim3(kT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = (cudaStream_t)stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    FB_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, x_lw, x_uw, x_lb, x_ub, gamma, beta, z_lw, z_uw, z_lb, z_ub, Di, Do, words, p, eps, violation, nc));
  }
  FB_LAUNCH_OK();
  return FB_OK;
}
