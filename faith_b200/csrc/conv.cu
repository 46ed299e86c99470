// Bound of a 2-D convolution with constant weights: the split-sign rule of the linear layer
// applied to a convolution whose batch axis is dim_in (every symbolic coordinate is an image),
// evaluated in centre/radius form like the FFMA GEMM:
//   c = (x_lw + x_uw)/2, r = (x_uw - x_lw)/2, y_c = conv(c, W), y_r = conv(r, |W|),
//   y_lw = y_c - y_r, y_uw = y_c + y_r.
// Direct convolution on CUDA cores, bound by the FP32 rate (one multiply-add per tap for the centre and one for the radius).
#include <algorithm>
#include <cstdint>
#include "common.cuh"
#include "conv_window.cuh"

namespace fb {
namespace {

// One block: the output channels [chunk * G * CPT, + G * CPT) of a tile of NI images x TH x TW output pixels.  A thread owns
// PX pixels x CPT channels, a warp of each channel group PX * 32 pixels.  The centre and the radius of a value make one packed
// multiply-add (fma.rn.f32x2: half the instructions) with a (w, |w|) pair; a tap costs a thread PX 64-bit reads of (centre,
// radius) pairs and CPT / 2 broadcast 128-bit reads of (w, |w|) pairs, two cycles each, for PX * CPT packed multiply-adds of
// two cycles on one of four pipes: with 4 x 8 the shared-memory pipe and the arithmetic are level.  CC input channels are
// staged at a time, by a table of source and destination offsets made once per block; the columns of a stride-2 layer are
// stored even ones first, so that consecutive pixels read consecutive words.  The tile is cut from the output map at run time
// (whole rows of narrow maps, several images of small ones): a fixed 16 x 16 or 8 x 32 tile spent up to two thirds of its
// threads on padding.  Every output accumulates over (input channel, tap row, tap column) in that order, whatever the tile.
// 384 images, 16 -> 32 channels, 32 x 32, 3 x 3, stride 2: 100 us with one pixel x 32 channels per thread and scalar
// multiply-adds (and 21 us more for the bias image in a launch of its own), 86 us now; 25 us are arithmetic, the staging alone
// takes 35 us and overlaps with it only across the four blocks of an SM, and the last of 1.3 rounds of blocks is thin.
struct ConvArgs {
  const float *x_lo, *x_up, *b_lo, *b_up;   // n_img images without the bias, then n_bias with it
  float *y_lo, *y_up, *yb_lo, *yb_up;
  const float *Wt, *bias;
  int64_t n_img, n_bias, blocks_bias;
  int Cin, H, W, Cout, Kh, Kw, stride, pad, Ho, Wo;
  int TH, TW, NI, tiles_h, tiles_w, chunks, G, CC;
  int in_h, in_w, pw, row, chan;   // staged tile: rows, columns, columns per phase, pairs per row and per channel
};

constexpr int kConvThreads = 256;   // at most: 8 channel groups
constexpr int kConvPos = 3, kConvLoads = 4;   // positions x input channels whose loads a thread has in flight together

__device__ __forceinline__ uint64_t lds64(uint32_t a) {
  uint64_t v;
  asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void lds128(uint32_t a, uint64_t& v, uint64_t& w) {
  asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(v), "=l"(w) : "r"(a) : "memory");
}

// KS: filter size when it is the same in both directions and known at compile time (3, 5), 0 = taken from the arguments; with
// KS the tap loops are unrolled.  ST: 2 = even columns first, 1 = stride 1, 0 = any stride, columns as they are.
template <int CPT, int PX, int KS, int ST>
__global__ void __launch_bounds__(kConvThreads)
conv_bounds_kernel(const ConvArgs q) {
  pdl_sync();
  static_assert(CPT % 2 == 0 && 32 % CPT == 0, "two channels per read; every thread stages the weights of one channel");
  extern __shared__ __align__(16) float smem[];
  const int Kh = KS ? KS : q.Kh, Kw = KS ? KS : q.Kw, taps = Kh * Kw, co_n = q.G * CPT;
  float2* s_w = reinterpret_cast<float2*>(smem);            // [CC][Kh][Kw][co_n] (w, |w|)
  float2* s_x = s_w + q.CC * taps * co_n;                   // [CC][NI][in_h][row] (centre, radius)
  int2* s_pos = reinterpret_cast<int2*>(s_x + q.CC * q.chan);   // [NI][in_h][in_w] offset in a channel of x (-1: outside), in s_x
  const int tid = threadIdx.x, nthr = blockDim.x;

  int64_t bid = blockIdx.x;
  const bool is_bias = bid < q.blocks_bias;
  if (!is_bias) bid -= q.blocks_bias;
  const int tw_i = (int)(bid % q.tiles_w); bid /= q.tiles_w;
  const int th_i = (int)(bid % q.tiles_h); bid /= q.tiles_h;
  const int cq = (int)(bid % q.chunks);
  const int64_t n0 = (bid / q.chunks) * q.NI, n_all = is_bias ? q.n_bias : q.n_img;
  const int ni = (int)min((int64_t)q.NI, n_all - n0);   // images of this block
  const int ih0 = th_i * q.TH * q.stride - q.pad, iw0 = tw_i * q.TW * q.stride - q.pad;
  const int co0 = cq * co_n, g = tid / 32;
  const int64_t hw = (int64_t)q.H * q.W;
  const float* x_lo = (is_bias ? q.b_lo : q.x_lo) + n0 * q.Cin * hw;
  const float* x_up = (is_bias ? q.b_up : q.x_up) + n0 * q.Cin * hw;

  const int n_pos = ni * q.in_h * q.in_w;
  for (int f = tid; f < n_pos; f += nthr) {
    const int rw = f % q.in_w, rh = (f / q.in_w) % q.in_h, im = f / (q.in_w * q.in_h);
    const int ih = ih0 + rh, iw = iw0 + rw;
    const bool in = ih >= 0 && ih < q.H && iw >= 0 && iw < q.W;
    s_pos[f] = make_int2(in ? (im * q.Cin * q.H + ih) * q.W + iw : -1,
                         (im * q.in_h + rh) * q.row + (ST == 2 ? (rw & 1) * q.pw + (rw >> 1) : rw));
  }
  // this thread's pixels: offset of the window in a staged channel, or the first window for a pixel it does not have
  int s0[PX];
#pragma unroll
  for (int e = 0; e < PX; ++e) {
    const int t = tid % 32 + e * 32, im = t / (q.TH * q.TW), th = (t / q.TW) % q.TH, tw = t % q.TW;
    s0[e] = im < ni ? (im * q.in_h + th * q.stride) * q.row + tw * (ST ? 1 : q.stride) : 0;
  }
  uint64_t acc[PX][CPT];
#pragma unroll
  for (int e = 0; e < PX; ++e)
#pragma unroll
    for (int o = 0; o < CPT; ++o) acc[e][o] = 0;

  // weights: 32 / CPT taps at a time, a thread always the same channel
  const int wo = tid % co_n, wt0 = tid / co_n;
  const bool w_in = co0 + wo < q.Cout;
  const float* w_src = q.Wt + (int64_t)(w_in ? co0 + wo : 0) * q.Cin * taps;
  for (int c0 = 0; c0 < q.Cin; c0 += q.CC) {
    const int cc = min(q.CC, q.Cin - c0);
    __syncthreads();
    const float* xl = x_lo + c0 * hw;
    const float* xu = x_up + c0 * hw;
    for (int t = wt0; t < cc * taps; t += 32 / CPT) {   // t = c * taps + tap
      const float w = w_in ? __ldg(w_src + (int64_t)c0 * taps + t) : 0.f;
      s_w[t * co_n + wo] = make_float2(w, fabsf(w));
    }
    for (int f0 = tid; f0 < n_pos; f0 += kConvPos * nthr) {
      int2 pos[kConvPos];
#pragma unroll
      for (int u = 0; u < kConvPos; ++u) pos[u] = f0 + u * nthr < n_pos ? s_pos[f0 + u * nthr] : make_int2(-1, -1);
      for (int c = 0; c < cc; c += kConvLoads) {
        float lo[kConvPos][kConvLoads], up[kConvPos][kConvLoads];
#pragma unroll
        for (int u = 0; u < kConvPos; ++u)
#pragma unroll
          for (int d = 0; d < kConvLoads; ++d) {
            const bool ok = pos[u].x >= 0 && c + d < cc;
            lo[u][d] = ok ? __ldg(xl + pos[u].x + (c + d) * hw) : 0.f;
            up[u][d] = ok ? __ldg(xu + pos[u].x + (c + d) * hw) : 0.f;
          }
#pragma unroll
        for (int u = 0; u < kConvPos; ++u)
#pragma unroll
          for (int d = 0; d < kConvLoads; ++d)
            if (c + d < cc && pos[u].y >= 0)
              s_x[pos[u].y + (c + d) * q.chan] = make_float2(fmul(fadd(lo[u][d], up[u][d]), 0.5f), fmul(fsub(up[u][d], lo[u][d]), 0.5f));
      }
    }
    __syncthreads();
    // addresses in shared memory by hand: one addition per row, phase and pixel, one per tap for the weights
    const uint32_t row_b = q.row * 8, chan_b = q.chan * 8, pw_b = ST == 2 ? q.pw * 8 : 0, tap_b = co_n * 8;
    uint32_t wa = (uint32_t)__cvta_generic_to_shared(s_w + g * CPT);
    uint32_t xa[PX];
#pragma unroll
    for (int e = 0; e < PX; ++e) xa[e] = (uint32_t)__cvta_generic_to_shared(s_x + s0[e]);
    for (int c = 0; c < cc; ++c) {
#pragma unroll
      for (int kh = 0; kh < (KS ? KS : Kh); ++kh) {
        uint32_t x0[PX], x1[PX];
#pragma unroll
        for (int e = 0; e < PX; ++e) {
          x0[e] = xa[e] + kh * row_b;
          x1[e] = x0[e] + pw_b;
        }
#pragma unroll
        for (int kw = 0; kw < (KS ? KS : Kw); ++kw) {
          uint64_t w[CPT];
#pragma unroll
          for (int o = 0; o < CPT; o += 2) lds128(wa + o * 8, w[o], w[o + 1]);
          wa += tap_b;
#pragma unroll
          for (int e = 0; e < PX; ++e) {
            const uint64_t v = lds64(ST == 2 ? (kw & 1 ? x1[e] : x0[e]) + (kw >> 1) * 8 : x0[e] + kw * 8);
#pragma unroll
            for (int o = 0; o < CPT; ++o) acc[e][o] = fma2(v, w[o], acc[e][o]);
          }
        }
      }
#pragma unroll
      for (int e = 0; e < PX; ++e) xa[e] += chan_b;
    }
  }
  float* y_lo = is_bias ? q.yb_lo : q.y_lo;
  float* y_up = is_bias ? q.yb_up : q.y_up;
#pragma unroll
  for (int e = 0; e < PX; ++e) {
    const int t = tid % 32 + e * 32, im = t / (q.TH * q.TW), oh = th_i * q.TH + (t / q.TW) % q.TH, ow = tw_i * q.TW + t % q.TW;
    if (im >= ni || oh >= q.Ho || ow >= q.Wo) continue;
    const int64_t off = (n0 + im) * q.Cout * (int64_t)q.Ho * q.Wo + (int64_t)oh * q.Wo + ow;
#pragma unroll
    for (int o = 0; o < CPT; ++o) {
      const int co = co0 + g * CPT + o;
      if (co >= q.Cout) break;
      const float2 v = unpack2(acc[e][o]);
      float lo = fsub(v.x, v.y), up = fadd(v.x, v.y);
      if (is_bias && q.bias != nullptr) { lo = fadd(lo, q.bias[co]); up = fadd(up, q.bias[co]); }
      y_lo[off + (int64_t)co * q.Ho * q.Wo] = lo;
      y_up[off + (int64_t)co * q.Ho * q.Wo] = up;
    }
  }
}

// Cuts the tile (`pixels` at most, up to g_max channel groups of CPT) and returns the number of blocks; 0: no tile fits.
int64_t plan_conv(ConvArgs& q, int cpt, int pixels, int g_max, int cc_max, size_t& smem) {
  const int groups = (int)ceil_div(q.Cout, cpt);
  q.chunks = (int)ceil_div(groups, g_max);
  q.G = (int)ceil_div(groups, q.chunks);
  q.TW = (int)ceil_div(q.Wo, ceil_div(q.Wo, std::min(pixels, 64)));   // even parts of at most 64 columns
  q.TH = std::max(1, std::min(q.Ho, pixels / q.TW));
  q.TH = (int)ceil_div(q.Ho, ceil_div(q.Ho, q.TH));
  q.NI = q.TW == q.Wo && q.TH == q.Ho ? std::max(1, pixels / (q.TW * q.TH)) : 1;
  q.NI = (int)std::max<int64_t>(1, std::min<int64_t>(q.NI, 0x7fffffff / ((int64_t)q.Cin * q.H * q.W)));   // 32-bit offsets
  q.CC = std::min(q.Cin, cc_max);
  for (;;) {
    const bool phases = q.stride == 2;
    q.in_h = (q.TH - 1) * q.stride + q.Kh;
    q.in_w = (q.TW - 1) * q.stride + q.Kw;
    q.pw = (q.in_w + 1) / 2;
    q.row = phases ? 2 * q.pw : q.in_w;
    q.chan = q.NI * q.in_h * q.row;
    smem = 8 * (q.CC * ((size_t)q.Kh * q.Kw * q.G * cpt + (size_t)q.chan) + (size_t)q.NI * q.in_h * q.in_w);
    // below 45 KB five blocks fit an SM; fewer channels a stage get there first, then (only if nothing fits) smaller tiles
    if (smem <= 45 * 1024 || (q.CC == 1 && smem <= (size_t)device_info().smem_optin)) break;
    if (q.CC > 1) q.CC = (q.CC + 1) / 2;
    else if (q.NI > 1) q.NI /= 2;
    else if (q.TH > 1) q.TH = (q.TH + 1) / 2;
    else if (q.TW > 1) q.TW = (q.TW + 1) / 2;
    else if (q.G > 1) { q.G = (q.G + 1) / 2; q.chunks = (int)ceil_div(groups, q.G); }
    else return 0;
  }
  q.tiles_h = (int)ceil_div(q.Ho, q.TH);
  q.tiles_w = (int)ceil_div(q.Wo, q.TW);
  const int64_t per_set = (int64_t)q.chunks * q.tiles_h * q.tiles_w;
  q.blocks_bias = ceil_div(q.n_bias, q.NI) * per_set;
  return q.blocks_bias + ceil_div(q.n_img, q.NI) * per_set;
}

template <int CPT, int PX>
int launch_conv_t(const ConvArgs& q, int64_t blocks, size_t smem, cudaStream_t st) {
  if (blocks <= 0 || blocks > 0x7fffffff) return FB_ERR_SHAPE;
  const int ks = q.Kh == q.Kw && (q.Kh == 3 || q.Kh == 5) ? q.Kh : 0;
#define FB_CONV_ST(K) (q.stride == 2 ? conv_bounds_kernel<CPT, PX, K, 2> : q.stride == 1 ? conv_bounds_kernel<CPT, PX, K, 1> \
                                     : conv_bounds_kernel<CPT, PX, K, 0>)
  auto kern = ks == 3 ? FB_CONV_ST(3) : ks == 5 ? FB_CONV_ST(5) : FB_CONV_ST(0);
#undef FB_CONV_ST
  if (int rc = ensure_dynamic_smem(kern, smem)) return rc;
  fb::launch_k(kern, (unsigned)blocks, q.G * 32, smem, st, q);
  FB_LAUNCH_OK();
  return FB_OK;
}

// n_img images without bias (the weight part) and n_bias with it (the bias part) in one launch.
int launch_conv(const float* x_lo, const float* x_up, float* y_lo, float* y_up, int64_t n_img, const float* b_lo, const float* b_up,
                float* yb_lo, float* yb_up, int64_t n_bias, const float* Wt, const float* bias, int Cin, int H, int W, int Cout,
                int Kh, int Kw, int stride, int pad, int Ho, int Wo, cudaStream_t st) {
  if (n_img + n_bias == 0) return FB_OK;
  if ((int64_t)H * W > 0x7fffffff) return FB_ERR_SHAPE;   // (offsets inside a plane are 32-bit)
  ConvArgs q = {};
  q.x_lo = x_lo, q.x_up = x_up, q.b_lo = b_lo, q.b_up = b_up;
  q.y_lo = y_lo, q.y_up = y_up, q.yb_lo = yb_lo, q.yb_up = yb_up;
  q.Wt = Wt, q.bias = bias, q.n_img = n_img, q.n_bias = n_bias;
  q.Cin = Cin, q.H = H, q.W = W, q.Cout = Cout, q.Kh = Kh, q.Kw = Kw, q.stride = stride, q.pad = pad, q.Ho = Ho, q.Wo = Wo;
  size_t smem;
  // up to 5 channel groups a block share its staged input (48 channels are 2 x 3 groups, 40 are 5)
  int64_t blocks = plan_conv(q, 8, 128, 5, 4, smem);
  if (blocks >= device_info().sms) return launch_conv_t<8, 4>(q, blocks, smem, st);
  // a few images only (the bias part alone: one image per batch element): less than a block per SM and bound by the latency
  // of the stages, so one pixel x 2 channels per thread, 32 pixels x up to 8 channels per block, all channels in one stage
  blocks = plan_conv(q, 2, 32, 4, Cin, smem);
  return launch_conv_t<2, 1>(q, blocks, smem, st);
}

// ------------------------------------------------------------------------------------------------
// Convolutions behind an identity input.  When every pixel of an image is perturbed, dim_in = Cin * H * W and the
// input bound is lw = uw = scale * I: row r of the weight tensors is the image with the single pixel
// (ci, yi, xi) = unravel(r) set.  Two consequences are used here:
//  * the first convolution needs no input at all: y_lw[r, co, y, x] is scale * W[co, ci, ky, kx] where the tap
//    (ky, kx) of output pixel (y, x) falls on (yi, xi), else zero, and the dual norm of output column (co, y, x)
//    over ALL rows is the norm of the taps of W[co] that fall inside the image -- so the concretised range, the
//    relaxation that follows and its rescale are computed from W alone and the relaxed rows are written directly;
//  * further layers keep the rows local: row r is zero outside a small window around its pixel, so a later
//    convolution only has to compute the outputs whose taps reach into that window and store zeros elsewhere.

// Per output column (co, y, x): the bias part (an ordinary convolution of the image, accumulated in the order of
// conv_bounds_kernel), the norm of the taps inside the image, and from both the slopes k_l, k_u and the relaxed bias terms of
// the relaxation `op` (op < 0: no relaxation, slopes 1).  Bound by latency (a thread per column): with KS, as above, the loads
// of an input channel's taps are in flight together, and one pass serves both sums (the image's convolution and the columns
// took 4 + 5 us as two launches for 3 -> 16 channels of 32 x 32).
template <int KS>
__global__ void __launch_bounds__(128)
identity_conv_columns_kernel(int op, const float* __restrict__ x_lb, const float* __restrict__ x_ub, const float* __restrict__ Wt,
                             const float* __restrict__ bias, float* __restrict__ y_lb, float* __restrict__ y_ub,
                             float* __restrict__ k_l, float* __restrict__ k_u, float scale, int Cin, int H, int W, int Cout,
                             int Kh_arg, int Kw_arg, int stride, int pad, int Ho, int Wo, int p, float eps,
                             int* __restrict__ violation) {
  pdl_sync();
  const int Kh = KS ? KS : Kh_arg, Kw = KS ? KS : Kw_arg;
  const int64_t n = (int64_t)Cout * Ho * Wo;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
    const int x = (int)(t % Wo), y = (int)((t / Wo) % Ho), co = (int)(t / ((int64_t)Wo * Ho));
    const int iy0 = y * stride - pad, ix0 = x * stride - pad;
    float ac = 0.f, ar = 0.f, acc = 0.f;
    for (int ci = 0; ci < Cin; ++ci) {
      const float* wp = Wt + ((int64_t)co * Cin + ci) * Kh * Kw;
      const int64_t plane = (int64_t)ci * H * W;
#pragma unroll
      for (int ky = 0; ky < (KS ? KS : Kh); ++ky)
#pragma unroll
        for (int kx = 0; kx < (KS ? KS : Kw); ++kx) {
          const int iy = iy0 + ky, ix = ix0 + kx;
          const bool in = iy >= 0 && iy < H && ix >= 0 && ix < W;
          const int64_t o = plane + (int64_t)iy * W + ix;
          const float w = __ldg(wp + ky * Kw + kx), lo = in ? __ldg(x_lb + o) : 0.f, up = in ? __ldg(x_ub + o) : 0.f;
          ac = fmaf(fmul(fadd(lo, up), 0.5f), w, ac);
          ar = fmaf(fmul(fsub(up, lo), 0.5f), fabsf(w), ar);
          acc = norm_accum(p, acc, in ? fmul(scale, w) : 0.f);
        }
    }
    float lbv = fsub(ac, ar), ubv = fadd(ac, ar);
    if (bias != nullptr) { lbv = fadd(lbv, bias[co]); ubv = fadd(ubv, bias[co]); }
    if (op < 0) {
      k_l[t] = 1.f;
      k_u[t] = 1.f;
      y_lb[t] = lbv;
      y_ub[t] = ubv;
      continue;
    }
    const float nrm = norm_finish(p, acc);
    const float l = fadd(lbv, fmul(-eps, nrm)), u = fadd(ubv, fmul(eps, nrm));
    bool bad = false;
    const ColCoef c = relax_column(op, l, u, lbv, ubv, bad);
    if (bad && violation != nullptr) *violation = 1;
    // both lines of the input coincide, so own-side and cross coefficients apply to the same numbers; for a
    // well-formed column one of each pair is zero and the sum is exact
    k_l[t] = fadd(c.c_ll, c.c_lu);
    k_u[t] = fadd(c.c_ul, c.c_uu);
    y_lb[t] = c.nlb;
    y_ub[t] = c.nub;
  }
}

__device__ __forceinline__ void store_elems(float* p, const float (&v)[4], int n) {
  if (n == 4) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  else p[0] = v[0];
}

// One block per row r = row_start + blockIdx.x: zeros everywhere, k * scale * W at the (at most Kh * Kw * Cout)
// positions whose tap falls on the row's pixel.  A thread owns output elements (V in a row of the image at a time:
// 4 when the width allows 16-byte stores, else 1), so nothing is written twice.
template <int V>
__global__ void __launch_bounds__(256)
identity_conv_rows_kernel(const float* __restrict__ Wt, const float* __restrict__ k_l, const float* __restrict__ k_u,
                          float* __restrict__ y_lw, float* __restrict__ y_uw, float scale, int64_t row_start, int Cin,
                          int H, int W, int Cout, int Kh, int Kw, int stride, int pad, int Ho, int Wo) {
  pdl_sync();
  const int64_t r = row_start + blockIdx.x;
  const int xi = (int)(r % W), yi = (int)((r / W) % H), ci = (int)(r / ((int64_t)W * H));
  const unsigned n = (unsigned)Cout * Ho * Wo, uWo = Wo, uHo = Ho;
  float* zl = y_lw + (int64_t)blockIdx.x * n;
  float* zu = y_uw + (int64_t)blockIdx.x * n;
  for (unsigned t = threadIdx.x * V; t < n; t += blockDim.x * V) {
    const unsigned q = t / uWo, x0 = t - q * uWo, co = q / uHo, y = q - co * uHo;
    const int ky = yi - ((int)y * stride - pad);
    float lo[4] = {0.f, 0.f, 0.f, 0.f}, up[4] = {0.f, 0.f, 0.f, 0.f};
    if (ky >= 0 && ky < Kh) {
#pragma unroll
      for (int e = 0; e < V; ++e) {
        const int kx = xi - ((int)(x0 + e) * stride - pad);
        if (kx >= 0 && kx < Kw) {
          const float tap = fmul(scale, __ldg(Wt + (((int64_t)co * Cin + ci) * Kh + ky) * Kw + kx));
          lo[e] = fmul(tap, k_l[t + e]);
          up[e] = fmul(tap, k_u[t + e]);
        }
      }
    }
    store_elems(zl + t, lo, V);
    store_elems(zu + t, up, V);
  }
}

// Split-sign convolution of rows that are zero outside a window (the window follows from the row's pixel and the chain
// of convolutions before this one).  One block per row: the window of the input is staged in shared memory as
// centre and radius, the outputs whose taps reach it are accumulated there in the order of the dense kernel (input
// channel, then tap row, then tap column; the skipped terms are exact zeros, so the value is the dense kernel's bit
// for bit), and the row is then streamed out, zeros outside the output window.
// Shared memory: centre and radius [Cin, win_h, win_w], then lower and upper [Cout, out_h, out_w].
template <int V>
__global__ void __launch_bounds__(256)
conv_window_kernel(const float* __restrict__ x_lo, const float* __restrict__ x_up, const float* __restrict__ Wt,
                   float* __restrict__ y_lo, float* __restrict__ y_up, int64_t row_start, int H0, int W0,
                   const ConvChain ch, int Cin, int H, int W, int Cout, int Kh, int Kw, int stride, int pad, int Ho,
                   int Wo, int win_h, int win_w, int out_h, int out_w) {
  pdl_sync();
  extern __shared__ float win_smem[];
  float* s_c = win_smem;
  float* s_r = s_c + Cin * win_h * win_w;
  float* s_ol = s_r + Cin * win_h * win_w;
  float* s_ou = s_ol + Cout * out_h * out_w;
  const int64_t r = row_start + blockIdx.x;
  const int xi = (int)(r % W0), yi = (int)((r / W0) % H0);
  Span wy, wx;
  chain_window(ch, H0, W0, yi, xi, wy, wx);
  const Span oy = span_after_conv(wy, Kh, stride, pad, Ho), ox = span_after_conv(wx, Kw, stride, pad, Wo);
  const bool empty = wy.lo > wy.hi || wx.lo > wx.hi || oy.lo > oy.hi || ox.lo > ox.hi;
  const int ah = wy.hi - wy.lo + 1, aw = wx.hi - wx.lo + 1, bh = oy.hi - oy.lo + 1, bw = ox.hi - ox.lo + 1;
  const unsigned n_out = (unsigned)Cout * Ho * Wo;
  const int64_t n_in = (int64_t)Cin * H * W;
  const float* il = x_lo + (int64_t)blockIdx.x * n_in;
  const float* iu = x_up + (int64_t)blockIdx.x * n_in;
  float* zl = y_lo + (int64_t)blockIdx.x * n_out;
  float* zu = y_up + (int64_t)blockIdx.x * n_out;
  // 1. zeros everywhere outside the output window: these stores depend on nothing and drain while the window is
  //    computed (a thread owns whole groups of V elements, so nothing is written twice).  The position (y, x0) of a
  //    thread's group is stepped without divisions: one step is blockDim.x * V elements = dq image rows and dx columns.
  {
    const unsigned uWo = Wo, uHo = Ho, step = blockDim.x * V;
    const unsigned dq = step / uWo, dx = step - dq * uWo, dy = dq % uHo;
    unsigned t = threadIdx.x * V;
    unsigned q = t / uWo, x0 = t - q * uWo, y = q % uHo;
    const float zero[4] = {0.f, 0.f, 0.f, 0.f};
    for (; t < n_out; t += step) {
      if (empty || (int)y < oy.lo || (int)y > oy.hi || (int)x0 + V - 1 < ox.lo || (int)x0 > ox.hi) {
        store_elems(zl + t, zero, V);
        store_elems(zu + t, zero, V);
      }
      x0 += dx;
      y += dy;
      if (x0 >= uWo) { x0 -= uWo; ++y; }
      if (y >= uHo) y -= uHo;
    }
  }
  if (empty) return;
  // 2. the window of the input, as centre and radius
  for (int i = threadIdx.x; i < Cin * ah * aw; i += blockDim.x) {
    const int x = i % aw, y = (i / aw) % ah, c = i / (aw * ah);
    const int64_t o = ((int64_t)c * H + wy.lo + y) * W + wx.lo + x;
    const float lo = __ldg(il + o), up = __ldg(iu + o);
    s_c[(c * win_h + y) * win_w + x] = fmul(fadd(lo, up), 0.5f);
    s_r[(c * win_h + y) * win_w + x] = fmul(fsub(up, lo), 0.5f);
  }
  __syncthreads();
  // 3. the outputs that reach it (the taps inside the window are a contiguous range per axis)
  for (int i = threadIdx.x; i < Cout * bh * bw; i += blockDim.x) {
    const int x = i % bw, y = (i / bw) % bh, co = i / (bw * bh);
    const int iy0 = (oy.lo + y) * stride - pad - wy.lo, ix0 = (ox.lo + x) * stride - pad - wx.lo;  // window coordinates
    const int ky0 = max(0, -iy0), ky1 = min(Kh, ah - iy0), kx0 = max(0, -ix0), kx1 = min(Kw, aw - ix0);
    float ac = 0.f, ar = 0.f;
    for (int c = 0; c < Cin; ++c) {
      const float* wp = Wt + ((int64_t)co * Cin + c) * Kh * Kw;
      const int sb = (c * win_h + iy0) * win_w + ix0;
      for (int ky = ky0; ky < ky1; ++ky)
        for (int kx = kx0; kx < kx1; ++kx) {
          const float w = __ldg(wp + ky * Kw + kx);
          ac = fmaf(s_c[sb + ky * win_w + kx], w, ac);
          ar = fmaf(s_r[sb + ky * win_w + kx], fabsf(w), ar);
        }
    }
    s_ol[(co * out_h + y) * out_w + x] = fsub(ac, ar);
    s_ou[(co * out_h + y) * out_w + x] = fadd(ac, ar);
  }
  __syncthreads();
  // 4. the groups of V elements that touch the output window
  const int g0 = ox.lo / V, ng = ox.hi / V - g0 + 1;
  for (int i = threadIdx.x; i < Cout * bh * ng; i += blockDim.x) {
    const int gx = i % ng, y = (i / ng) % bh, co = i / (ng * bh);
    const int x0 = (g0 + gx) * V;
    float lo[4] = {0.f, 0.f, 0.f, 0.f}, up[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int e = 0; e < V; ++e) {
      const int x = x0 + e;
      if (x >= ox.lo && x <= ox.hi) {
        const int o = (co * out_h + y) * out_w + (x - ox.lo);
        lo[e] = s_ol[o];
        up[e] = s_ou[o];
      }
    }
    const int64_t t = ((int64_t)co * Ho + oy.lo + y) * Wo + x0;
    store_elems(zl + t, lo, V);
    store_elems(zu + t, up, V);
  }
}

}  // namespace

int launch_identity_columns(int op, const float* x_lb, const float* x_ub, const float* Wt, const float* bias, float* y_lb, float* y_ub,
                            float* k_l, float* k_u, float scale, int Cin, int H, int W, int Cout, int Kh, int Kw, int stride, int pad,
                            int Ho, int Wo, int p, float eps, int* violation, cudaStream_t st) {
  const int64_t ncol = (int64_t)Cout * Ho * Wo;
  const int64_t want = ceil_div(ncol, 128), cap = (int64_t)device_info().sms * 16;
  auto kern = Kh == 3 && Kw == 3 ? identity_conv_columns_kernel<3> : identity_conv_columns_kernel<0>;
  fb::launch_k(kern, (unsigned)(want < cap ? want : cap), 128, 0, st, op, x_lb, x_ub, Wt, bias, y_lb, y_ub, k_l, k_u, scale, Cin, H, W, Cout, Kh, Kw,
                                                            stride, pad, Ho, Wo, p, eps, violation);
  FB_LAUNCH_OK();
  return FB_OK;
}

}  // namespace fb

extern "C" int fb_conv2d_identity_relax_f32(int op, const float* x_lb, const float* x_ub, const float* Wt,
                                            const float* bias, float scale, float* y_lw, float* y_uw, float* y_lb,
                                            float* y_ub, float* col_ws, int64_t rows, int64_t row_start, int Cin, int H,
                                            int W, int Cout, int Kh, int Kw, int stride, int pad, int p, float eps,
                                            int* violation, void* stream) {
  if (!x_lb || !x_ub || !Wt || !y_lw || !y_uw || !y_lb || !y_ub || !col_ws) return FB_ERR_ARG;
  if (rows < 0 || row_start < 0 || Cin <= 0 || H <= 0 || W <= 0 || Cout <= 0 || Kh <= 0 || Kw <= 0 || stride <= 0 || pad < 0 ||
      !fb::valid_norm(p) || row_start + rows > (int64_t)Cin * H * W)
    return FB_ERR_ARG;
  if (op >= 0 && !((op >= FB_RELU && op <= FB_SQRT))) return FB_ERR_ARG;
  const int Ho = (H + 2 * pad - Kh) / stride + 1, Wo = (W + 2 * pad - Kw) / stride + 1;
  if (Ho <= 0 || Wo <= 0) return FB_ERR_SHAPE;
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t ncol = (int64_t)Cout * Ho * Wo;
  fb::ProfileScope prof(fb::PK_CONV, 8.0 * (rows + 1) * ncol * Cin * Kh * Kw, 4.0 * (2.0 * (rows + 1) * ncol), stream);
  float* k_l = col_ws;
  float* k_u = col_ws + ncol;
  int rc = fb::launch_identity_columns(op, x_lb, x_ub, Wt, bias, y_lb, y_ub, k_l, k_u, scale, Cin, H, W, Cout, Kh, Kw, stride, pad, Ho, Wo,
                                       p, eps, violation, st);
  if (rc != FB_OK) return rc;
  if (rows == 0) return FB_OK;
  if (rows > 0x7fffffff) return FB_ERR_SHAPE;
  if (ncol > 0x7fffffff) return FB_ERR_SHAPE;
  if (Wo % 4 == 0 && fb::aligned16(y_lw) && fb::aligned16(y_uw))
    fb::launch_k(fb::identity_conv_rows_kernel<4>, (unsigned)rows, 256, 0, st, Wt, k_l, k_u, y_lw, y_uw, scale, row_start, Cin, H, W,
                                                                       Cout, Kh, Kw, stride, pad, Ho, Wo);
  else
    fb::launch_k(fb::identity_conv_rows_kernel<1>, (unsigned)rows, 256, 0, st, Wt, k_l, k_u, y_lw, y_uw, scale, row_start, Cin, H, W,
                                                                       Cout, Kh, Kw, stride, pad, Ho, Wo);
  FB_LAUNCH_OK();
  return FB_OK;
}

extern "C" int fb_conv2d_windowed_f32(const float* x_lw, const float* x_uw, const float* Wt, float* y_lw, float* y_uw,
                                      int64_t rows, int64_t row_start, int H0, int W0, const int* chain, int n_chain,
                                      int Cin, int H, int W, int Cout, int Kh, int Kw, int stride, int pad,
                                      void* stream) {
  if (!x_lw || !x_uw || !Wt || !y_lw || !y_uw || (n_chain > 0 && !chain)) return FB_ERR_ARG;
  if (rows < 0 || row_start < 0 || H0 <= 0 || W0 <= 0 || n_chain < 0 || Cin <= 0 || H <= 0 || W <= 0 || Cout <= 0 || Kh <= 0 ||
      Kw <= 0 || stride <= 0 || pad < 0)
    return FB_ERR_ARG;
  if (n_chain > fb::kMaxChain) return FB_ERR_SHAPE;
  fb::ConvChain ch;
  ch.n = n_chain;
  int h = H0, w = W0;
  for (int i = 0; i < n_chain; ++i) {
    ch.kh[i] = chain[4 * i], ch.kw[i] = chain[4 * i + 1], ch.stride[i] = chain[4 * i + 2], ch.pad[i] = chain[4 * i + 3];
    if (ch.kh[i] <= 0 || ch.kw[i] <= 0 || ch.stride[i] <= 0 || ch.pad[i] < 0) return FB_ERR_ARG;
    h = (h + 2 * ch.pad[i] - ch.kh[i]) / ch.stride[i] + 1;
    w = (w + 2 * ch.pad[i] - ch.kw[i]) / ch.stride[i] + 1;
  }
  if (h != H || w != W) return FB_ERR_SHAPE;   // the chain must lead from the H0 x W0 image to this layer's input
  const int Ho = (H + 2 * pad - Kh) / stride + 1, Wo = (W + 2 * pad - Kw) / stride + 1;
  if (Ho <= 0 || Wo <= 0) return FB_ERR_SHAPE;
  if (rows == 0) return FB_OK;
  const double ncol = (double)Cout * Ho * Wo;
  if (rows > 0x7fffffff || ncol > 0x7fffffff) return FB_ERR_SHAPE;
  // the largest window any pixel reaches, in and out (the kernel sizes its shared memory by it)
  int win_h = 1, win_w = 1, out_h = 1, out_w = 1;
  for (int yi = 0; yi < H0; ++yi) {
    fb::Span wy, wx;
    fb::chain_window(ch, H0, W0, yi, 0, wy, wx);
    const fb::Span oy = fb::span_after_conv(wy, Kh, stride, pad, Ho);
    win_h = std::max(win_h, wy.hi - wy.lo + 1);
    out_h = std::max(out_h, oy.hi - oy.lo + 1);
  }
  for (int xi = 0; xi < W0; ++xi) {
    fb::Span wy, wx;
    fb::chain_window(ch, H0, W0, 0, xi, wy, wx);
    const fb::Span ox = fb::span_after_conv(wx, Kw, stride, pad, Wo);
    win_w = std::max(win_w, wx.hi - wx.lo + 1);
    out_w = std::max(out_w, ox.hi - ox.lo + 1);
  }
  const size_t smem = sizeof(float) * 2 * ((size_t)Cin * win_h * win_w + (size_t)Cout * out_h * out_w);
  if (smem > (size_t)fb::device_info().smem_optin) return FB_ERR_SHAPE;   // windows too large to pay: use fb_conv2d_f32
  cudaStream_t st = (cudaStream_t)stream;
  const bool vec = Wo % 4 == 0 && fb::aligned16(y_lw) && fb::aligned16(y_uw);
  auto kern = vec ? fb::conv_window_kernel<4> : fb::conv_window_kernel<1>;
  if (int rc = fb::ensure_dynamic_smem(kern, smem)) return rc;
  fb::ProfileScope prof(fb::PK_CONV, 8.0 * rows * Cout * out_h * out_w * Cin * Kh * Kw,
                        4.0 * (2.0 * rows * Cin * win_h * win_w + 2.0 * rows * ncol), stream);
  fb::launch_k(kern, (unsigned)rows, 256, smem, st, x_lw, x_uw, Wt, y_lw, y_uw, row_start, H0, W0, ch, Cin, H, W, Cout, Kh, Kw, stride, pad,
                                          Ho, Wo, win_h, win_w, out_h, out_w);
  FB_LAUNCH_OK();
  return FB_OK;
}

extern "C" int fb_conv2d_f32(const float* x_lw, const float* x_uw, const float* x_lb, const float* x_ub,
                             const float* Wt, const float* bias, float* y_lw, float* y_uw, float* y_lb, float* y_ub,
                             int B, int Di, int Cin, int H, int W, int Cout, int Kh, int Kw, int stride, int pad,
                             void* stream) {
  if (!x_lw || !x_uw || !x_lb || !x_ub || !Wt || !y_lw || !y_uw || !y_lb || !y_ub) return FB_ERR_ARG;
  // (Di == 0: the bias part alone)
  if (B < 0 || Di < 0 || Cin <= 0 || H <= 0 || W <= 0 || Cout <= 0 || Kh <= 0 || Kw <= 0 || stride <= 0 || pad < 0)
    return FB_ERR_ARG;
  const int Ho = (H + 2 * pad - Kh) / stride + 1, Wo = (W + 2 * pad - Kw) / stride + 1;
  if (Ho <= 0 || Wo <= 0) return FB_ERR_SHAPE;
  cudaStream_t st = (cudaStream_t)stream;
  const double n1 = (double)B * (Di + 1);
  fb::ProfileScope prof(fb::PK_CONV, 8.0 * n1 * Cout * Ho * Wo * Cin * Kh * Kw,
                        4.0 * (2 * n1 * Cin * H * W + 2 * n1 * Cout * Ho * Wo + (double)Cout * Cin * Kh * Kw), stream);
  return fb::launch_conv(x_lw, x_uw, y_lw, y_uw, (int64_t)B * Di, x_lb, x_ub, y_lb, y_ub, B, Wt, bias, Cin, H, W, Cout, Kh, Kw, stride, pad,
                         Ho, Wo, st);
}
