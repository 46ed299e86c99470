// Compact rows for the convolutions behind an identity input.
//
// When every pixel of an H0 x W0 image is perturbed, row r of the weight tensors stands for pixel (ci, yi, xi) =
// unravel(r) and, after a chain of convolutions, is zero outside the window that pixel reaches (conv_window.cuh).
// The dense-row kernels of conv.cu still write and read those zeros: [rows, C, H, W] per tensor, 98 % zeros for the
// benchmark CNN.  Here a row is kept as its window only:
//
//     z[r, c, dy, dx] = row r at (c, wy.lo(r) + dy, wx.lo(r) + dx),   dy < wh, dx < ww,
//
// with (wh, ww) the largest window over all pixels (fb_cw_extent) and zeros where a pixel's own window is smaller: the form of
// the C ABI (kAbi = true below).  Between its layers the CNN driver keeps the rows as z[r, dy, dx, c] (kAbi = false): the kernels
// have their lanes on the channels, so that their loads and stores of rows are whole sectors; its windows are cut to the last map
// only (CwAxis), and where a pixel's own window is smaller nothing is written.
// The origin (wy.lo, wx.lo) is recomputed from the pixel and the chain wherever it is needed.  Every operator of the
// CNN pass has a compact form: first convolution + relaxation, later convolutions, the column norms over dim_in
// (a gather over the rows whose window holds the column, in row order: deterministic), the rescale of a relaxation,
// and the linear layer that ends the spatial part (its output is dense, [rows, N]).  fb_cw_expand_f32 writes the dense
// rows for callers that need them.  Accumulation orders follow the dense kernels, so a compact convolution expands
// to the dense kernel's values bit for bit.
//
// The reference has no counterpart (HandTunedKernels/convolution_verification.cu:228-238 is a benchmark stub); the
// operator semantics are Bounds.matmul / Bounds.relu with dim_in as batch axis (Bounds.py:397-413, :921-963).
#include <algorithm>
#include <cstdint>

#include "common.cuh"
#include "conv_window.cuh"

namespace fb {
namespace {

// Geometry of a compact tensor: its windows, its dense shape and the order of a row's elements.
template <bool kAbi>
struct CwShape;

template <>
struct CwShape<false> {
  CwAxis y, x;
  int H0, W0, C, H, W, wh, ww;
  __device__ __forceinline__ Span rows(int yi) const { return {y.lo(yi), y.hi(yi)}; }
  __device__ __forceinline__ Span cols(int xi) const { return {x.lo(xi), x.hi(xi)}; }
  // elements between neighbouring columns and between neighbouring channels
  __device__ __forceinline__ int step_x() const { return C; }
  __device__ __forceinline__ int step_c() const { return 1; }
  // element e of a row
  __device__ __forceinline__ void split(int e, int& c, int& dy, int& dx) const { c = e % C, dx = (e / C) % ww, dy = e / (C * ww); }
};

template <>
struct CwShape<true> : CwShape<false> {   // (y and x: windows that hold these, for the ranges of loops)
  ConvChain ch;
  bool same;   // y and x are these windows, as behind most chains: no walk along the chain (norms of 3072 rows: 12.3 -> 5.5 us)
  __device__ __forceinline__ Span rows(int yi) const { return same ? CwShape<false>::rows(yi) : chain_span(ch, ch.kh, ch.n, H0, yi); }
  __device__ __forceinline__ Span cols(int xi) const { return same ? CwShape<false>::cols(xi) : chain_span(ch, ch.kw, ch.n, W0, xi); }
  __device__ __forceinline__ int step_x() const { return 1; }
  __device__ __forceinline__ int step_c() const { return wh * ww; }
  __device__ __forceinline__ void split(int e, int& c, int& dy, int& dx) const { dx = e % ww, dy = (e / ww) % wh, c = e / (ww * wh); }
};

__device__ __forceinline__ void pixel_of_row(int64_t r, int H0, int W0, int& yi, int& xi) {
  xi = (int)(r % W0);
  yi = (int)((r / W0) % H0);
}

// The arguments of a launch arrive in a constant bank that no cache has seen: every 64 bytes of them cost the first reader a miss.
// The warps of a block touch one line each, so that the misses overlap.
template <typename Args>
__device__ __forceinline__ void touch_params(const Args& q) {
  const unsigned at = (threadIdx.x >> 5) * 16;
  if (at < sizeof(Args) / 4) asm volatile("" ::"r"(reinterpret_cast<const int*>(&q)[at]));
}

// First convolution (+ relaxation) of the identity input, compact: one thread per element of z.  (Behind a single convolution the
// two forms have the same windows.)
template <bool kAbi>
__global__ void __launch_bounds__(256)
cw_identity_rows_kernel(const float* __restrict__ Wt, const float* __restrict__ k_l, const float* __restrict__ k_u,
                        float* __restrict__ z_lw, float* __restrict__ z_uw, float scale, int64_t rows, int64_t row_start,
                        int Cin, int H, int W, int Cout, int Kh, int Kw, int stride, int pad, int Ho, int Wo, int wh, int ww) {
  pdl_sync();
  const int64_t per_row = (int64_t)Cout * wh * ww;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < rows * per_row; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t lr = t / per_row;
    const int e = (int)(t - lr * per_row);
    const int co = kAbi ? e / (ww * wh) : e % Cout, dx = kAbi ? e % ww : (e / Cout) % ww, dy = kAbi ? (e / ww) % wh : e / (Cout * ww);
    const int64_t r = row_start + lr;
    const int xi = (int)(r % W), yi = (int)((r / W) % H), ci = (int)(r / ((int64_t)W * H));
    Span sy = {yi, yi}, sx = {xi, xi};
    sy = span_after_conv(sy, Kh, stride, pad, Ho);
    sx = span_after_conv(sx, Kw, stride, pad, Wo);
    const int y = sy.lo + dy, x = sx.lo + dx;
    float lo = 0.f, up = 0.f;
    if (sy.lo <= sy.hi && sx.lo <= sx.hi && y <= sy.hi && x <= sx.hi) {
      const int ky = yi - (y * stride - pad), kx = xi - (x * stride - pad);
      if (ky >= 0 && ky < Kh && kx >= 0 && kx < Kw) {
        const float tap = fmul(scale, __ldg(Wt + (((int64_t)co * Cin + ci) * Kh + ky) * Kw + kx));
        const int64_t col = ((int64_t)co * Ho + y) * Wo + x;
        lo = fmul(tap, k_l[col]);
        up = fmul(tap, k_u[col]);
      }
    }
    z_lw[t] = lo;
    z_uw[t] = up;
  }
}

// A later convolution, compact -> compact.  Rows whose pixels agree modulo S, the product of all strides up to and including
// this convolution's, have the same geometry up to a shift: the same windows, the same taps for the same output.  A block takes
// G * 8 rows of one such class, so that nothing in its loops depends on the row: a thread owns one output position and channel of
// eight rows, reads a weight once for all of them, and its tap bounds are the same for the whole block.  The windows are taken
// without the borders of the maps (rows at the border are filled up with zeros, whose products leave every sum as it is), and
// what falls outside is not stored.  Every output accumulates over (input channel, tap row, tap column) in that order, as the
// dense kernel does.  Centre and radius share a packed multiply-add with a (w, |w|) pair.
// The input comes from compact rows, or (W1 != nullptr) is the first convolution and its relaxation, evaluated from the filter
// while it is staged: those rows are never written.  The first blocks compute the bias image.
// Bound by latency and shared-memory reads: 3072 rows, 16 -> 32 channels, 3 x 3 stride 2 took 35 us with a thread per output of
// one row, whose tap bounds differ from lane to lane, and 8 us before it to write its input; 20 us now for both.
constexpr int kCwR = 8;             // rows per thread
constexpr int kCwConvThreads = 512;   // at most; the items of a block in one round where that is possible
constexpr int kCwMaxRows = 32;      // rows per block at most: one per lane
constexpr size_t kCwStatic = 4096;  // static shared memory of the kernels below, at most

struct CwConvArgs {
  const float *z_lo, *z_up;                    // compact rows, or
  const float *W1, *k_l, *k_u;                 // the first convolution: filter [Cin, Cin0, kh1, kw1], slopes per column
  float scale;
  int Cin0, kh1, kw1, stride1, pad1;
  const float* Wt;
  float *y_lo, *y_up;
  const float *b_lo, *b_up, *bias;             // bias image (blocks_bias > 0)
  float *yb_lo, *yb_up;
  int blocks_bias;
  int64_t rows, row_start;
  int ci0, n_ci;                               // input channels of the image that the rows span
  int H0, W0, Cin, H, W, Cout, stride, pad, Kh, Kw, Ho, Wo, iwh, iww, owh, oww;
  int cls_x, per_class, G, CC;
  int uih, uiw;                                // largest window of the input without borders
  CwAxis iy, ix, oy, ox;                       // input and output windows
};

template <bool kAbi>
struct CwConvParams : CwConvArgs {};
template <>
struct CwConvParams<true> : CwConvArgs {
  ConvChain ch;   // up to and including this convolution
};

struct __align__(16) CwRow {
  int lr, yi, xi, ci;      // local row (-1: none), pixel
  int uy, ux;              // input window without borders: first row and column
  int iy, ix, ih, iw;      // input window: first row and column, size
  int oh, ow;              // output window: size (0 x 0: no row)
  int py, px;              // its first row and column among the positions of the class
  int64_t base;            // element (0, 0, 0) of the output row, shifted by (py, px)
};

// The bias image: an ordinary convolution, a thread per output from `first` on in steps of `step`.
template <int KS>
__device__ __forceinline__ void conv_bias_image(const CwConvArgs& q, int64_t first, int64_t step) {
  const int Kh = KS ? KS : q.Kh, Kw = KS ? KS : q.Kw, taps = Kh * Kw;
  const int64_t total = (int64_t)q.Cout * q.Ho * q.Wo;
  for (int64_t t = first; t < total; t += step) {
    const int ow = (int)(t % q.Wo), oh = (int)((t / q.Wo) % q.Ho), co = (int)(t / ((int64_t)q.Wo * q.Ho));
    const int ih0 = oh * q.stride - q.pad, iw0 = ow * q.stride - q.pad;
    float ac = 0.f, ar = 0.f;
#pragma unroll 2
    for (int c = 0; c < q.Cin; ++c) {
      const float* wp = q.Wt + ((int64_t)co * q.Cin + c) * taps;
      const int64_t plane = (int64_t)c * q.H * q.W;
#pragma unroll
      for (int kh = 0; kh < (KS ? KS : Kh); ++kh)
#pragma unroll
        for (int kw = 0; kw < (KS ? KS : Kw); ++kw) {
          const int ih = ih0 + kh, iw = iw0 + kw;
          const bool in = ih >= 0 && ih < q.H && iw >= 0 && iw < q.W;
          const int64_t o = plane + (int64_t)ih * q.W + iw;
          const float w = __ldg(wp + kh * Kw + kw), lo = in ? __ldg(q.b_lo + o) : 0.f, up = in ? __ldg(q.b_up + o) : 0.f;
          ac = fmaf(fmul(fadd(lo, up), 0.5f), w, ac);
          ar = fmaf(fmul(fsub(up, lo), 0.5f), fabsf(w), ar);
        }
    }
    float lo = fsub(ac, ar), up = fadd(ac, ar);
    if (q.bias != nullptr) { lo = fadd(lo, q.bias[co]); up = fadd(up, q.bias[co]); }
    q.yb_lo[t] = lo;
    q.yb_up[t] = up;
  }
}

// KS: filter size when it is the same in both directions and known at compile time (3), 0 = from the arguments.
// CPT: output channels per thread (2 where Cout is even: the pairs of a tap are one 128-bit read, and the inputs, which every lane
// reads, serve twice the multiply-adds).
template <int KS, int CPT, bool kAbi>
__global__ void __launch_bounds__(kCwConvThreads)
cw_conv_kernel(const __grid_constant__ CwConvParams<kAbi> q) {
  extern __shared__ __align__(16) float cw_smem[];
  __shared__ CwRow s_row[kCwMaxRows];
  touch_params(q);
  pdl_sync();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nthr = blockDim.x, nwarps = nthr >> 5;
  const int Kh = KS ? KS : q.Kh, Kw = KS ? KS : q.Kw, taps = Kh * Kw;
  if ((int)blockIdx.x < q.blocks_bias) {
    conv_bias_image<KS>(q, (int64_t)blockIdx.x * nthr + tid, (int64_t)q.blocks_bias * nthr);
    return;
  }
  const int bid = blockIdx.x - q.blocks_bias, cls = bid / q.per_class, chunk = bid - cls * q.per_class;
  const int ry = cls / q.cls_x, rx = cls - ry * q.cls_x, n_rows = q.G * kCwR;
  // geometry of the class, from its first pixel
  const int vy = q.iy.free_lo(ry), vx = q.ix.free_lo(rx), wy = q.oy.free_lo(ry), wx = q.ox.free_lo(rx);
  const int ih = max(0, q.iy.free_hi(ry) - vy + 1), iw = max(0, q.ix.free_hi(rx) - vx + 1);
  const int oh = max(0, q.oy.free_hi(ry) - wy + 1), ow = max(0, q.ox.free_hi(rx) - wx + 1);
  const int ty0 = wy * q.stride - q.pad - vy, tx0 = wx * q.stride - q.pad - vx;   // first tap of the first output
  {
    const int S = q.oy.S, ny = (q.H0 - ry + S - 1) / S, nx = (q.W0 - rx + S - 1) / S, n_cls = q.n_ci * ny * nx;
    bool live = false;
    if (tid < n_rows) {
      const int k = chunk * n_rows + tid, kl = k / nx, kx = k - kl * nx, ci = kl / ny, ky = kl - ci * ny;
      CwRow r;
      r.lr = -1;
      r.xi = rx + S * kx;
      r.yi = ry + S * ky;
      r.ci = q.ci0 + ci;
      if (k < n_cls) {
        const int64_t lr = ((int64_t)r.ci * q.H0 + r.yi) * q.W0 + r.xi - q.row_start;
        if (lr >= 0 && lr < q.rows) r.lr = (int)lr;
      }
      live = r.lr >= 0;
      r.uy = vy + q.stride * ky, r.ux = vx + q.stride * kx;
      int oy, ox;
      if constexpr (kAbi) {
        const Span sy = chain_span(q.ch, q.ch.kh, q.ch.n - 1, q.H0, r.yi), sx = chain_span(q.ch, q.ch.kw, q.ch.n - 1, q.W0, r.xi);
        const Span ty = chain_span(q.ch, q.ch.kh, q.ch.n, q.H0, r.yi), tx = chain_span(q.ch, q.ch.kw, q.ch.n, q.W0, r.xi);
        r.iy = sy.lo, r.ix = sx.lo, r.ih = sy.hi - sy.lo + 1, r.iw = sx.hi - sx.lo + 1;
        oy = ty.lo, ox = tx.lo;
        r.oh = live ? max(0, ty.hi - oy + 1) : 0, r.ow = live ? max(0, tx.hi - ox + 1) : 0;
      } else {
        r.iy = max(0, r.uy), r.ix = max(0, r.ux);
        r.ih = min(q.H, r.uy + ih) - r.iy, r.iw = min(q.W, r.ux + iw) - r.ix;
        oy = max(0, wy + ky), ox = max(0, wx + kx);
        r.oh = live ? max(0, min(q.Ho, wy + ky + oh) - oy) : 0, r.ow = live ? max(0, min(q.Wo, wx + kx + ow) - ox) : 0;
      }
      r.py = oy - wy - ky, r.px = ox - wx - kx;
      r.base = kAbi ? (int64_t)r.lr * q.Cout * q.owh * q.oww - r.py * q.oww - r.px
                    : (((int64_t)r.lr * q.owh - r.py) * q.oww - r.px) * q.Cout;
      s_row[tid] = r;
    }
    if (!__syncthreads_or(live)) return;
  }
  const int npos = oh * ow, ldw = q.Cout + CPT;                // (pairs of weights stay 8-byte aligned)
  float2* s_x = reinterpret_cast<float2*>(cw_smem);            // [CC][uih][uiw][G * 8] (centre, radius)
  float* s_w = cw_smem + 2 * (size_t)q.CC * q.uih * q.uiw * n_rows;   // [CC][Kh][Kw][ldw]
  const bool once = q.CC >= q.Cin;
  const int cgroups = q.Cout / CPT, items = npos * q.G * cgroups;
  for (int i0 = 0; i0 < items; i0 += nthr) {
    // channels fastest, then the groups of rows: the lanes of a warp that leave the channels' range keep their position
    const int item = i0 + tid, u = item / cgroups, co = (item - u * cgroups) * CPT, pos = u / q.G, g = u - pos * q.G;
    const int py = pos / ow, px = pos - py * ow;
    const int by = ty0 + py * q.stride, bx = tx0 + px * q.stride;
    const int ky0 = max(0, -by), ky1 = min(Kh, ih - by), kx0 = max(0, -bx), kx1 = min(Kw, iw - bx);
    uint64_t acc[kCwR][CPT];
#pragma unroll
    for (int j = 0; j < kCwR; ++j)
#pragma unroll
      for (int e = 0; e < CPT; ++e) acc[j][e] = 0;
    for (int c0 = 0; c0 < q.Cin; c0 += q.CC) {
      const int cc = min(q.CC, q.Cin - c0);
      if (!once || i0 == 0) {
        if (i0 > 0 || c0 > 0) __syncthreads();
        const int wn = cc * taps;
        for (int o = warp; o < q.Cout; o += nwarps) {   // asynchronous, lanes along (channel, tap)
          const float* src = q.Wt + ((int64_t)o * q.Cin + c0) * taps;
          uint32_t dst = (uint32_t)__cvta_generic_to_shared(s_w + lane * ldw + o);
          for (int t = lane; t < wn; t += 32, dst += 128 * ldw)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src + t) : "memory");
        }
        if (q.W1 != nullptr) {
          // lanes along the rows (n_rows <= 32): neighbouring columns of the slopes; two (channel, window row) pairs at a time, so
          // that eighteen loads are in flight
          const CwRow r = s_row[min(lane, n_rows - 1)];
          const int n_v = cc * ih;
          for (int v0 = warp; v0 < n_v; v0 += 2 * nwarps)
            for (int ux0 = 0; ux0 < iw; ux0 += 3) {
              float w[2][3], kl[2][3], ku[2][3];
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const int v = min(v0 + h * nwarps, n_v - 1), c = v / ih, y = r.uy + v - c * ih, ky = r.yi - (y * q.stride1 - q.pad1);
                const bool in_y = r.lr >= 0 && y >= 0 && y < q.H && ky >= 0 && ky < q.kh1;
                const float* wp = q.W1 + (((int64_t)(c0 + c) * q.Cin0 + r.ci) * q.kh1 + ky) * q.kw1;
                const int64_t col = ((int64_t)(c0 + c) * q.H + y) * q.W;
#pragma unroll
                for (int e = 0; e < 3; ++e) {
                  const int x = r.ux + ux0 + e, kx = r.xi - (x * q.stride1 - q.pad1);
                  const bool in = in_y && x >= 0 && x < q.W && kx >= 0 && kx < q.kw1;
                  w[h][e] = in ? __ldg(wp + kx) : 0.f;
                  kl[h][e] = in ? __ldg(q.k_l + col + x) : 0.f;
                  ku[h][e] = in ? __ldg(q.k_u + col + x) : 0.f;
                }
              }
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const int v = min(v0 + h * nwarps, n_v - 1), c = v / ih, uy = v - c * ih;   // (a repeated pair writes the same)
                float2* dst = s_x + ((c * q.uih + uy) * q.uiw + ux0) * n_rows + lane;
#pragma unroll
                for (int e = 0; e < 3; ++e) {
                  const float tap = fmul(q.scale, w[h][e]), lo = fmul(tap, kl[h][e]), up = fmul(tap, ku[h][e]);
                  if (ux0 + e < iw && lane < n_rows) dst[e * n_rows] = make_float2(fmul(fadd(lo, up), 0.5f), fmul(fsub(up, lo), 0.5f));
                }
              }
            }
        } else {
          // lanes along the channel: neighbouring words of a row of the driver
          for (int v = warp; v < ih * n_rows; v += nwarps) {
            const int uy = v / n_rows, t = v - uy * n_rows;
            const CwRow& r = s_row[t];
            const int dy = r.uy + uy - r.iy, dx0 = r.ux - r.ix;
            const bool in_y = r.lr >= 0 && dy >= 0 && dy < r.ih;
            const int step_x = kAbi ? 1 : q.Cin, step_c = kAbi ? q.iwh * q.iww : 1;
            const int64_t o = kAbi ? ((int64_t)r.lr * q.Cin + c0) * step_c + dy * q.iww + dx0
                                   : (((int64_t)r.lr * q.iwh + dy) * q.iww + dx0) * q.Cin + c0;
            for (int c = lane; c < cc; c += 32) {
              float2* dst = s_x + (c * q.uih + uy) * q.uiw * n_rows + t;
#pragma unroll 3
              for (int ux = 0; ux < iw; ++ux) {
                const bool in = in_y && dx0 + ux >= 0 && dx0 + ux < r.iw;
                const int64_t at = o + ux * step_x + c * step_c;
                const float lo = in ? __ldg(q.z_lo + at) : 0.f, up = in ? __ldg(q.z_up + at) : 0.f;
                dst[ux * n_rows] = make_float2(fmul(fadd(lo, up), 0.5f), fmul(fsub(up, lo), 0.5f));
              }
            }
          }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
      }
      if (item < items) {
        // all taps of all channels in one loop (the loops over a position's one to three taps would each wait for their loads),
        // the operands of the next tap loaded before the arithmetic of this one
        const int nx = kx1 - kx0, ny = ky1 - ky0, n_tap = cc * max(0, ny) * max(0, nx);
        const float2* xp = s_x + ((int64_t)(by + ky0) * q.uiw + bx + kx0) * n_rows + g * kCwR;
        const float* wp = s_w + (ky0 * Kw + kx0) * ldw + co;
        const int x_row = (q.uiw - nx) * n_rows, w_row = (Kw - nx) * ldw;
        const int x_ch = (q.uih - ny) * q.uiw * n_rows, w_ch = (taps - ny * Kw) * ldw;
        int kx = 0, ky = 0;
        auto load = [&](ulonglong2 (&x)[kCwR / 2], float (&w)[CPT]) {
#pragma unroll
          for (int j = 0; j < kCwR / 2; ++j) x[j] = reinterpret_cast<const ulonglong2*>(xp)[j];
          if (CPT == 2) {
            const float2 v = *reinterpret_cast<const float2*>(wp);
            w[0] = v.x, w[CPT - 1] = v.y;
          } else {
            w[0] = *wp;
          }
          xp += n_rows, wp += ldw;
          if (++kx == nx) {
            kx = 0, xp += x_row, wp += w_row;
            if (++ky == ny) ky = 0, xp += x_ch, wp += w_ch;
          }
        };
        auto mac = [&](const ulonglong2 (&x)[kCwR / 2], const float (&w)[CPT]) {
#pragma unroll
          for (int e = 0; e < CPT; ++e) {
            const uint64_t p = pack2(w[e], fabsf(w[e]));
#pragma unroll
            for (int j = 0; j < kCwR / 2; ++j) {
              acc[2 * j][e] = fma2(x[j].x, p, acc[2 * j][e]);
              acc[2 * j + 1][e] = fma2(x[j].y, p, acc[2 * j + 1][e]);
            }
          }
        };
        if (n_tap > 0) {
          ulonglong2 xa[kCwR / 2], xb[kCwR / 2];
          float wa[CPT], wb[CPT];
          load(xa, wa);
          int t = 1;
          for (; t + 1 < n_tap; t += 2) {
            load(xb, wb);
            mac(xa, wa);
            load(xa, wa);
            mac(xb, wb);
          }
          if (t < n_tap) load(xb, wb);
          mac(xa, wa);
          if (t < n_tap) mac(xb, wb);
        }
      }
    }
    if (item < items) {
#pragma unroll
      for (int j = 0; j < kCwR; ++j) {
        const CwRow& r = s_row[g * kCwR + j];
        if ((unsigned)(py - r.py) < (unsigned)r.oh && (unsigned)(px - r.px) < (unsigned)r.ow) {
          const int step_c = kAbi ? q.owh * q.oww : 1;
          const int64_t o = r.base + (int64_t)(py * q.oww + px) * (kAbi ? 1 : q.Cout) + (int64_t)co * step_c;
#pragma unroll
          for (int e = 0; e < CPT; ++e) {
            const float2 v = unpack2(acc[j][e]);
            q.y_lo[o + e * step_c] = fsub(v.x, v.y);
            q.y_up[o + e * step_c] = fadd(v.x, v.y);
          }
        }
      }
    }
  }
}

// The same, a thread per output that reads its taps from global memory: for windows that shared memory does not hold (they are
// taken without the borders of the maps above, so that filters larger than a small map can exceed it).
template <bool kAbi>
__global__ void __launch_bounds__(256)
cw_conv_direct_kernel(const __grid_constant__ CwConvParams<kAbi> q, const __grid_constant__ CwShape<kAbi> gi,
                      const __grid_constant__ CwShape<kAbi> go) {
  pdl_sync();
  if ((int)blockIdx.x < q.blocks_bias) {
    conv_bias_image<0>(q, (int64_t)blockIdx.x * 256 + threadIdx.x, (int64_t)q.blocks_bias * 256);
    return;
  }
  const int64_t per_in = (int64_t)gi.C * gi.wh * gi.ww, per_out = (int64_t)go.C * go.wh * go.ww;
  const int64_t step = (int64_t)(gridDim.x - q.blocks_bias) * 256;
  for (int64_t t = (int64_t)(blockIdx.x - q.blocks_bias) * 256 + threadIdx.x; t < q.rows * per_out; t += step) {
    const int64_t lr = t / per_out, r = q.row_start + lr;
    int co, dy, dx;
    go.split((int)(t - lr * per_out), co, dy, dx);
    const int xi = (int)(r % q.W0), yi = (int)((r / q.W0) % q.H0), ci = (int)(r / ((int64_t)q.W0 * q.H0));
    const Span wy = go.rows(yi), wx = go.cols(xi), vy = gi.rows(yi), vx = gi.cols(xi);
    if (wy.lo + dy > wy.hi || wx.lo + dx > wx.hi) continue;
    const int y0 = (wy.lo + dy) * q.stride - q.pad, x0 = (wx.lo + dx) * q.stride - q.pad;   // first tap
    const int ky0 = max(0, vy.lo - y0), ky1 = min(q.Kh, vy.hi + 1 - y0), kx0 = max(0, vx.lo - x0), kx1 = min(q.Kw, vx.hi + 1 - x0);
    float ac = 0.f, ar = 0.f;
    for (int c = 0; c < q.Cin; ++c)
      for (int ky = ky0; ky < ky1; ++ky)
        for (int kx = kx0; kx < kx1; ++kx) {
          const int y = y0 + ky, x = x0 + kx;
          float lo = 0.f, up = 0.f;
          if (q.W1 != nullptr) {
            const int jy = yi - (y * q.stride1 - q.pad1), jx = xi - (x * q.stride1 - q.pad1);
            if (jy >= 0 && jy < q.kh1 && jx >= 0 && jx < q.kw1) {
              const float tap = fmul(q.scale, __ldg(q.W1 + (((int64_t)c * q.Cin0 + ci) * q.kh1 + jy) * q.kw1 + jx));
              const int64_t col = ((int64_t)c * q.H + y) * q.W + x;
              lo = fmul(tap, __ldg(q.k_l + col));
              up = fmul(tap, __ldg(q.k_u + col));
            }
          } else {
            const int64_t o = lr * per_in + ((int64_t)(y - vy.lo) * gi.ww + x - vx.lo) * gi.step_x() + (int64_t)c * gi.step_c();
            lo = __ldg(q.z_lo + o);
            up = __ldg(q.z_up + o);
          }
          const float w = __ldg(q.Wt + (((int64_t)co * q.Cin + c) * q.Kh + ky) * q.Kw + kx);
          ac = fmaf(fmul(fadd(lo, up), 0.5f), w, ac);
          ar = fmaf(fmul(fsub(up, lo), 0.5f), fabsf(w), ar);
        }
    q.y_lo[t] = fsub(ac, ar);
    q.y_up[t] = fadd(ac, ar);
  }
}

// Dual-norm accumulation of every column (c, y, x) over the rows [row_start, row_start + rows): a gather over the pixels whose
// window holds (y, x).  A block takes one position and 32 channels; its warps interleave over the rows of those pixels and read 32
// consecutive words of a row of z; their sums are combined in the order of the warps, so the result depends on the geometry alone.
// op < 0: the unfinished accumulations go to part_l / part_u.  Otherwise the relaxation's coefficients follow at once (no
// exchange between ranks in between): out_lb / out_ub receive the relaxed bias terms, coef as cw_relax_columns_kernel writes it.
// 3072 rows of 3 x 3 x 32 windows, 8192 columns: 13 us with a warp per column of channel-major rows, whose 32 lanes touch 32
// sectors per load; 5 us now, coefficients included.
constexpr int kCwNormWarps = 16, kCwNormLoads = 4;

__device__ __forceinline__ void cw_relax_column(int op, float lbv, float ubv, float nl, float nu, int p, float eps, int64_t dense,
                                                int64_t at, int64_t ncol, float* out_lb, float* out_ub, float* coef, int* violation) {
  const float l = fadd(lbv, fmul(-eps, norm_finish(p, nl)));
  const float u = fadd(ubv, fmul(eps, norm_finish(p, nu)));
  bool bad = false;
  const ColCoef c = relax_column(op, l, u, lbv, ubv, bad);
  if (bad && violation != nullptr) *violation = 1;
  out_lb[dense] = c.nlb;
  out_ub[dense] = c.nub;
  coef[at] = c.c_ll;
  coef[ncol + at] = c.c_lu;
  coef[2 * ncol + at] = c.c_ul;
  coef[3 * ncol + at] = c.c_uu;
}

template <bool kAbi>
__global__ void __launch_bounds__(32 * kCwNormWarps)
cw_norm_kernel(int op, const float* __restrict__ z_lw, const float* __restrict__ z_uw, float* __restrict__ part_l,
               float* __restrict__ part_u, const float* __restrict__ lb, const float* __restrict__ ub, float* __restrict__ out_lb,
               float* __restrict__ out_ub, float* __restrict__ coef, int64_t rows, int64_t row_start, int Cin0, const __grid_constant__ CwShape<kAbi> g, int p,
               float eps, int* __restrict__ violation) {
  pdl_sync();
  __shared__ float s_part[2][kCwNormWarps][32];
  const int y = blockIdx.x / g.W, x = blockIdx.x - y * g.W, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = blockIdx.y * 32 + lane;
  // pixels whose window holds (y, x)
  const int y0 = max(0, y * g.y.S - g.y.B), ny = min(g.H0 - 1, y * g.y.S - g.y.A) - y0 + 1;
  const int x0 = max(0, x * g.x.S - g.x.B), nx = min(g.W0 - 1, x * g.x.S - g.x.A) - x0 + 1;
  float al = 0.f, au = 0.f;
  if (ny > 0) {
    for (int k = warp; k < Cin0 * ny; k += kCwNormWarps) {
      const int ci = k / ny, yi = y0 + k - ci * ny;
      const int64_t lr0 = ((int64_t)ci * g.H0 + yi) * g.W0 + x0 - row_start;
      const Span wy = g.rows(yi);
      const int dy = y - wy.lo;
      const bool in_y = !kAbi || (y >= wy.lo && y <= wy.hi);
      for (int kx = 0; kx < nx; kx += kCwNormLoads) {
        float vl[kCwNormLoads], vu[kCwNormLoads];   // zeros leave every norm as it is
#pragma unroll
        for (int e = 0; e < kCwNormLoads; ++e) {
          const int64_t lr = lr0 + kx + e;
          const Span wx = g.cols(x0 + kx + e);
          const bool in = kx + e < nx && lr >= 0 && lr < rows && c < g.C && in_y && (!kAbi || (x >= wx.lo && x <= wx.hi));
          const int64_t o = !in ? 0 : kAbi ? ((lr * g.C + c) * g.wh + dy) * g.ww + (x - wx.lo) : ((lr * g.wh + dy) * g.ww + (x - wx.lo)) * g.C + c;
          vl[e] = in ? __ldg(z_lw + o) : 0.f;
          vu[e] = in ? __ldg(z_uw + o) : 0.f;
        }
#pragma unroll
        for (int e = 0; e < kCwNormLoads; ++e) {
          al = norm_accum(p, al, vl[e]);
          au = norm_accum(p, au, vu[e]);
        }
      }
    }
  }
  s_part[0][warp][lane] = al;
  s_part[1][warp][lane] = au;
  __syncthreads();
  if (warp != 0 || c >= g.C) return;
#pragma unroll
  for (int w = 1; w < kCwNormWarps; ++w) {
    al = norm_combine(p, al, s_part[0][w][lane]);
    au = norm_combine(p, au, s_part[1][w][lane]);
  }
  const int64_t dense = ((int64_t)c * g.H + y) * g.W + x;
  if (op < 0) {
    part_l[dense] = al;
    part_u[dense] = au;
  } else {
    cw_relax_column(op, lb[dense], ub[dense], al, au, p, eps, dense, (int64_t)blockIdx.x * g.C + c, (int64_t)g.C * g.H * g.W, out_lb, out_ub,
                    coef, violation);
  }
}

// Relaxation coefficients per column from the (reduced) norms, in the order of the rows' elements: coef [4][H * W][C], or (kAbi)
// [4][C][H * W]; the relaxed bias terms go to out_lb / out_ub.
template <bool kAbi>
__global__ void __launch_bounds__(256)
cw_relax_columns_kernel(int op, const float* __restrict__ lb, const float* __restrict__ ub, const float* __restrict__ norm_l,
                        const float* __restrict__ norm_u, float* __restrict__ out_lb, float* __restrict__ out_ub,
                        float* __restrict__ coef, int C, int64_t hw, int p, float eps, int* __restrict__ violation) {
  pdl_sync();
  const int64_t ncol = C * hw;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < ncol; t += (int64_t)gridDim.x * blockDim.x)
    cw_relax_column(op, lb[t], ub[t], norm_l[t], norm_u[t], p, eps, t, kAbi ? t : (t % hw) * C + t / hw, ncol, out_lb, out_ub, coef, violation);
}

// Rescale of a relaxation on compact rows: out_lw = c_ll lw + c_lu uw, out_uw = c_uu uw + c_ul lw (the expressions of
// the dense kernel).  A warp per row: the window is worked out once, the lanes interleave over its elements.
template <bool kAbi>
__global__ void __launch_bounds__(256)
cw_rescale_kernel(const float* __restrict__ z_lw, const float* __restrict__ z_uw, const float* __restrict__ coef,
                  float* __restrict__ o_lw, float* __restrict__ o_uw, int64_t rows, int64_t row_start, const __grid_constant__ CwShape<kAbi> g) {
  pdl_sync();
  const int lane = threadIdx.x & 31;
  const int64_t lr = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (lr >= rows) return;
  const int per_row = g.C * g.wh * g.ww;
  const int64_t ncol = (int64_t)g.C * g.H * g.W;
  int yi, xi;
  pixel_of_row(row_start + lr, g.H0, g.W0, yi, xi);
  const Span wy = g.rows(yi), wx = g.cols(xi);
  for (int e = lane; e < per_row; e += 32) {
    int c, dy, dx;
    g.split(e, c, dy, dx);
    float lo = 0.f, up = 0.f;
    if (wy.lo + dy <= wy.hi && wx.lo + dx <= wx.hi) {
      const int64_t pos = (int64_t)(wy.lo + dy) * g.W + wx.lo + dx, col = kAbi ? (int64_t)c * g.H * g.W + pos : pos * g.C + c;
      const float a = z_lw[lr * per_row + e], b = z_uw[lr * per_row + e];
      lo = fmaf(coef[col], a, fmul(coef[ncol + col], b));
      up = fmaf(coef[3 * ncol + col], b, fmul(coef[2 * ncol + col], a));
    }
    o_lw[lr * per_row + e] = lo;
    o_uw[lr * per_row + e] = up;
  }
}

// Linear layer on compact rows: y[r, n] = sum_e c_e W[n, col(e)] -/+ r_e |W[n, col(e)]|, where (coef != nullptr) the rows go
// through the rescale of a relaxation on the way.  A block takes the pixels of one image row, kCwPx of its columns and every
// channel of the image: their windows overlap, so the weights they need (the union of the windows) are staged in shared memory
// once, [position][32 channels][NB outputs], 32 channels and as many rows of positions at a time as fit.  A warp owns a row
// of the result, its lanes the channels; the sums over the lanes go through a transposing butterfly (31 shuffles for 32 values).
// Where this is the last layer (part != nullptr), the rows are not written: what is left of them is their dual norm, one partial
// accumulation per block, tile and output.  The first bias_blocks blocks compute the bias part, an output each.
// Bound by L2 reads: with W^T in global memory every row read its own copy of the weights (20 us and 2 us for the transpose at
// 3072 rows, 288 elements, 10 outputs, and 9 us to write the rescaled rows first; 12 us now).
constexpr int kCwPx = 8, kCwLinWarps = 24, kCwLinThreads = 32 * kCwLinWarps;   // 24: the rows of 8 pixels of 3 channels

template <bool kAbi>
struct CwLinearArgs {
  const float *z_lw, *z_uw, *coef, *W;
  float *y_lw, *y_uw, *part;
  const float *lb, *ub, *bias;
  float *y_lb, *y_ub;
  int bias_blocks;
  int64_t rows, row_start;
  int ci0, n_ci, N, nb, ny_max, nx_max, p;
  CwShape<kAbi> g;
};

template <int NB, bool kAbi>
__global__ void __launch_bounds__(kCwLinThreads)
cw_linear_kernel(const __grid_constant__ CwLinearArgs<kAbi> q) {
  touch_params(q);
  pdl_sync();
  constexpr int LDN = NB + 2, LDP = 32 * LDN + 2;   // the lanes' 64-bit reads, along the channels, and the stores, along the
                                                    // positions, fall on different banks
  extern __shared__ __align__(16) float cw_smem[];
  __shared__ float s_red[2][kCwLinWarps][16];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const CwShape<kAbi>& g = q.g;
  const int64_t ncol = (int64_t)g.C * g.H * g.W;
  if ((int)blockIdx.x < q.bias_blocks) {
    if (blockIdx.y > 0) return;
    const float* w = q.W + (int64_t)blockIdx.x * ncol;
    float c = 0.f, r = 0.f;
#pragma unroll 4
    for (int64_t f = tid; f < ncol; f += kCwLinThreads) {
      const float lo = __ldg(q.lb + f), up = __ldg(q.ub + f), v = __ldg(w + f);
      c = fmaf(fmul(fadd(lo, up), 0.5f), v, c);
      r = fmaf(fmul(fsub(up, lo), 0.5f), fabsf(v), r);
    }
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
      c += __shfl_xor_sync(0xffffffffu, c, s);
      r += __shfl_xor_sync(0xffffffffu, r, s);
    }
    if (lane == 0) s_red[0][warp][0] = c, s_red[1][warp][0] = r;
    __syncthreads();
    if (tid == 0) {
      for (int i = 1; i < kCwLinWarps; ++i) c += s_red[0][i][0], r += s_red[1][i][0];
      const float b = q.bias != nullptr ? q.bias[blockIdx.x] : 0.f;
      q.y_lb[blockIdx.x] = fadd(fsub(c, r), b);
      q.y_ub[blockIdx.x] = fadd(fadd(c, r), b);
    }
    return;
  }
  const int tiles_x = (g.W0 + kCwPx - 1) / kCwPx, tile = blockIdx.x - q.bias_blocks;
  const int yi = tile / tiles_x, x0 = (tile - yi * tiles_x) * kCwPx, npx = min(kCwPx, g.W0 - x0);
  const int n0 = blockIdx.y * q.nb, nb = min(q.nb, q.N - n0);
  // the union of the windows (their ends do not decrease along the pixels)
  const int ylo = g.y.lo(yi), yhi = g.y.hi(yi), xl = g.x.lo(x0), nxr = max(0, g.x.hi(x0 + npx - 1) - xl + 1), rows_here = npx * q.n_ci;
  const int64_t per_pos = g.step_x(), per_row = (int64_t)g.wh * g.ww * g.C;
  const int wy0 = kAbi ? g.rows(yi).lo : ylo;   // first row of the windows of the tile's pixels
  float pl = 0.f, pu = 0.f;   // accumulated norms of this lane's output
  for (int r0 = 0; r0 < rows_here; r0 += kCwLinWarps) {
    float sc[NB], sr[NB];
#pragma unroll
    for (int n = 0; n < NB; ++n) sc[n] = sr[n] = 0.f;
    const int t = r0 + warp, px = t % npx, ci = q.ci0 + t / npx;
    int64_t lr = -1;
    const int wlo = g.cols(x0 + px).lo, aw = g.cols(x0 + px).hi - wlo + 1;
    if (t < rows_here) {
      const int64_t l = ((int64_t)ci * g.H0 + yi) * g.W0 + x0 + px - q.row_start;
      if (l >= 0 && l < q.rows) lr = l;
    }
    for (int c0 = 0; c0 < g.C; c0 += 32) {
      const int c = c0 + lane;
      for (int ya = ylo; ya <= yhi; ya += q.ny_max) {
        const int yb = min(yhi, ya + q.ny_max - 1), npos = (yb - ya + 1) * nxr;
        __syncthreads();
        for (int pos = lane; pos < npos; pos += 32) {   // asynchronous; a warp per (output, channel), lanes along the positions
          const int yy = pos / nxr;
          const float* src = q.W + (int64_t)n0 * ncol + ((int64_t)c0 * g.H + ya + yy) * g.W + xl + pos - yy * nxr;
          const uint32_t dst = (uint32_t)__cvta_generic_to_shared(cw_smem + pos * LDP);
          for (int u = warp; u < 32 * NB; u += kCwLinWarps) {
            const int cl = u % 32, n = u / 32;
            const bool in = n < nb && c0 + cl < g.C;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst + 4 * (cl * LDN + n)),
                         "l"(src + (in ? n * ncol + (int64_t)cl * g.H * g.W : 0)), "r"(in ? 4 : 0) : "memory");
          }
        }
        // the row's elements, three at a time: those of the next step are loaded before the arithmetic of this one
        const bool mine = lr >= 0 && c < g.C && aw > 0;
        const int y_first = kAbi ? max(ya, wy0) : ya, n_y = kAbi ? max(0, min(yb, g.rows(yi).hi) - y_first + 1) : yb - ya + 1;
        const int steps_x = (aw + 2) / 3, steps = mine ? n_y * steps_x : 0;
        float zl[3], zu[3], kf[4][3];
        int sy = y_first, sx = 0;   // the next step: row, first column of the window
        auto load = [&] {
          const int64_t zb = lr * per_row + ((int64_t)(sy - wy0) * g.ww + sx) * per_pos + (kAbi ? (int64_t)c * g.step_c() : c), cb = ((int64_t)sy * g.W + wlo + sx) * g.C + c;
#pragma unroll
          for (int e = 0; e < 3; ++e) {
            const bool in = sx + e < aw;
            zl[e] = in ? __ldg(q.z_lw + zb + e * per_pos) : 0.f;
            zu[e] = in ? __ldg(q.z_uw + zb + e * per_pos) : 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) kf[i][e] = in && q.coef != nullptr ? __ldg(q.coef + i * ncol + cb + e * g.C) : 0.f;
          }
        };
        if (steps > 0) load();
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        for (int st = 0; st < steps; ++st) {
          const float* wb = cw_smem + ((sy - ya) * nxr + wlo + sx - xl) * LDP + lane * LDN;
          const int left = aw - sx;
          float vc[3], vr[3];
#pragma unroll
          for (int e = 0; e < 3; ++e) {
            const float lo = q.coef != nullptr ? fmaf(kf[0][e], zl[e], fmul(kf[1][e], zu[e])) : zl[e];
            const float up = q.coef != nullptr ? fmaf(kf[3][e], zu[e], fmul(kf[2][e], zl[e])) : zu[e];
            vc[e] = fmul(fadd(lo, up), 0.5f), vr[e] = fmul(fsub(up, lo), 0.5f);
          }
          sx += 3;
          if (sx >= aw) sx = 0, ++sy;
          if (st + 1 < steps) load();
#pragma unroll
          for (int e = 0; e < 3; ++e) {
            const float2* w = reinterpret_cast<const float2*>(wb + (e < left ? e : 0) * LDP);
#pragma unroll
            for (int n = 0; n < NB; n += 2) {
              const float2 v = w[n / 2];
              sc[n] = fmaf(vc[e], v.x, sc[n]);
              sr[n] = fmaf(vr[e], fabsf(v.x), sr[n]);
              sc[n + 1] = fmaf(vc[e], v.y, sc[n + 1]);
              sr[n + 1] = fmaf(vr[e], fabsf(v.y), sr[n + 1]);
            }
          }
        }
      }
    }
    // lane i ends with the sum of value i of (sc[0 .. 15], sr[0 .. 15])
    float v[32];
#pragma unroll
    for (int n = 0; n < 16; ++n) {
      v[n] = n < NB ? sc[n < NB ? n : 0] : 0.f;
      v[16 + n] = n < NB ? sr[n < NB ? n : 0] : 0.f;
    }
#pragma unroll
    for (int s = 16; s > 0; s >>= 1)
#pragma unroll
      for (int i = 0; i < s; ++i) {
        const bool upper = (lane & s) != 0;
        const float keep = upper ? v[i + s] : v[i], give = upper ? v[i] : v[i + s];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, give, s);
      }
    const float other = __shfl_xor_sync(0xffffffffu, v[0], 16);
    if (lr >= 0 && lane < nb) {   // (the lanes below 16 hold the centres)
      const float lo = fsub(v[0], other), up = fadd(v[0], other);
      if (q.part != nullptr) {
        pl = norm_accum(q.p, pl, lo);
        pu = norm_accum(q.p, pu, up);
      } else {
        q.y_lw[lr * q.N + n0 + lane] = lo;
        q.y_uw[lr * q.N + n0 + lane] = up;
      }
    }
  }
  if (q.part == nullptr) return;
  if (lane < 16) s_red[0][warp][lane] = pl, s_red[1][warp][lane] = pu;
  __syncthreads();
  if (tid < nb) {
    pl = s_red[0][0][tid], pu = s_red[1][0][tid];
    for (int i = 1; i < kCwLinWarps; ++i) pl = norm_combine(q.p, pl, s_red[0][i][tid]), pu = norm_combine(q.p, pu, s_red[1][i][tid]);
    q.part[((int64_t)tile * 2 + 0) * q.N + n0 + tid] = pl;
    q.part[((int64_t)tile * 2 + 1) * q.N + n0 + tid] = pu;
  }
}

// Concretised range of output blockIdx.x from the partial norms of cw_linear_kernel: warp 0 the lower, warp 1 the upper side.
__global__ void __launch_bounds__(64)
cw_linear_range_kernel(const float* __restrict__ part, const float* __restrict__ lb, const float* __restrict__ ub, float* __restrict__ l,
                       float* __restrict__ u, int tiles, int N, int p, float eps) {
  pdl_sync();
  const int lane = threadIdx.x & 31, side = threadIdx.x >> 5, n = blockIdx.x;
  float a = 0.f;
#pragma unroll 4
  for (int t = lane; t < tiles; t += 32) a = norm_combine(p, a, __ldg(part + ((int64_t)t * 2 + side) * N + n));
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) a = norm_combine(p, a, __shfl_xor_sync(0xffffffffu, a, s));
  if (lane == 0) {
    if (side == 0) l[n] = fadd(lb[n], fmul(-eps, norm_finish(p, a)));
    else u[n] = fadd(ub[n], fmul(eps, norm_finish(p, a)));
  }
}

// Dense rows from compact ones: one block per row, zeros outside the window.
template <bool kAbi>
__global__ void __launch_bounds__(256)
cw_expand_kernel(const float* __restrict__ z_lw, const float* __restrict__ z_uw, float* __restrict__ y_lw,
                 float* __restrict__ y_uw, int64_t row_start, const __grid_constant__ CwShape<kAbi> g) {
  pdl_sync();
  const int64_t r = row_start + blockIdx.x;
  int yi, xi;
  pixel_of_row(r, g.H0, g.W0, yi, xi);
  const Span wy = g.rows(yi), wx = g.cols(xi);
  const int per_row = g.C * g.wh * g.ww;
  const unsigned n = (unsigned)g.C * g.H * g.W, uW = g.W, uH = g.H;
  const float* zl = z_lw + (int64_t)blockIdx.x * per_row;
  const float* zu = z_uw + (int64_t)blockIdx.x * per_row;
  float* ol = y_lw + (int64_t)blockIdx.x * n;
  float* ou = y_uw + (int64_t)blockIdx.x * n;
  for (unsigned t = threadIdx.x; t < n; t += blockDim.x) {
    const unsigned q = t / uW, x = t - q * uW, c = q / uH, y = q - c * uH;
    float lo = 0.f, up = 0.f;
    if ((int)y >= wy.lo && (int)y <= wy.hi && (int)x >= wx.lo && (int)x <= wx.hi) {
      const int e = (((int)y - wy.lo) * g.ww + ((int)x - wx.lo)) * g.step_x() + (int)c * g.step_c();
      lo = zl[e];
      up = zu[e];
    }
    ol[t] = lo;
    ou[t] = up;
  }
}

template <bool kAbi>
int make_shape(const int* chain, int n_chain, int H0, int W0, int C, int H, int W, CwShape<kAbi>& g) {
  int h, w;
  ConvChain ch;
  int rc = chain_from_host(chain, n_chain, H0, W0, ch, h, w);
  if (rc != FB_OK) return rc;
  if (n_chain == 0 || C <= 0 || h != H || w != W) return FB_ERR_SHAPE;
  g.H0 = H0, g.W0 = W0, g.C = C, g.H = H, g.W = W;
  rc = axis_from_chain(ch, ch.kh, H, g.y);
  if (rc == FB_OK) rc = axis_from_chain(ch, ch.kw, W, g.x);
  if (rc != FB_OK) return rc;
  if constexpr (kAbi) {
    g.ch = ch;
    g.wh = chain_extent(ch, ch.kh, H0), g.ww = chain_extent(ch, ch.kw, W0);
    g.same = axis_is_chain(g.y, ch, ch.kh, H0) && axis_is_chain(g.x, ch, ch.kw, W0);
  } else {
    g.wh = axis_extent(g.y, H0), g.ww = axis_extent(g.x, W0);
  }
  if ((int64_t)C * H * W > 0x7fffffff || (int64_t)C * g.wh * g.ww > 0x7fffffff) return FB_ERR_SHAPE;
  return FB_OK;
}

inline unsigned grid_for(int64_t items, int per_block) {
  const int64_t want = ceil_div(items, per_block), cap = (int64_t)device_info().sms * 16;
  return (unsigned)std::max<int64_t>(1, std::min(want, cap));
}

// Channels of the image that the rows [row_start, row_start + rows) span.
inline void row_channels(int64_t row_start, int64_t rows, int H0, int W0, int& ci0, int& n_ci) {
  const int64_t hw = (int64_t)H0 * W0;
  ci0 = (int)(row_start / hw);
  n_ci = (int)((row_start + rows - 1) / hw) - ci0 + 1;
}

// z_lo == nullptr: the rows of the first convolution, from its filter W1 and the slopes k_l, k_u (chain has one entry).
// b_lo != nullptr: the bias image goes along (b_lo, b_up [Cin, H, W] -> yb_lo, yb_up).
template <bool kAbi>
int conv_rows(const float* z_lo, const float* z_up, const float* W1, const float* k_l, const float* k_u, float scale, int Cin0,
               const float* Wt, float* y_lo, float* y_up, const float* b_lo, const float* b_up, const float* bias, float* yb_lo,
               float* yb_up, int64_t rows, int64_t row_start, int H0, int W0, const int* chain, int n_chain, int Cin, int H, int W,
               int Cout, int Kh, int Kw, int stride, int pad, cudaStream_t st) {
  if (rows < 0 || row_start < 0 || Cin <= 0 || Cout <= 0 || Kh <= 0 || Kw <= 0 || stride <= 0 || pad < 0 || n_chain < 1)
    return FB_ERR_ARG;
  if (n_chain >= kMaxChain) return FB_ERR_SHAPE;
  CwShape<kAbi> gi, go;
  int rc = make_shape(chain, n_chain, H0, W0, Cin, H, W, gi);
  if (rc != FB_OK) return rc;
  const int Ho = (H + 2 * pad - Kh) / stride + 1, Wo = (W + 2 * pad - Kw) / stride + 1;
  if (Ho <= 0 || Wo <= 0) return FB_ERR_SHAPE;
  int out_chain[4 * kMaxChain];
  std::copy(chain, chain + 4 * n_chain, out_chain);
  out_chain[4 * n_chain] = Kh, out_chain[4 * n_chain + 1] = Kw, out_chain[4 * n_chain + 2] = stride, out_chain[4 * n_chain + 3] = pad;
  rc = make_shape(out_chain, n_chain + 1, H0, W0, Cout, Ho, Wo, go);
  if (rc != FB_OK) return rc;
  if (rows == 0) return FB_OK;
  if (rows > 0x7fffffff) return FB_ERR_SHAPE;

  CwConvParams<kAbi> q = {};
  if constexpr (kAbi) q.ch = go.ch;
  q.z_lo = z_lo, q.z_up = z_up, q.W1 = W1, q.k_l = k_l, q.k_u = k_u, q.scale = scale, q.Cin0 = Cin0;
  q.Wt = Wt, q.y_lo = y_lo, q.y_up = y_up;
  q.b_lo = b_lo, q.b_up = b_up, q.bias = bias, q.yb_lo = yb_lo, q.yb_up = yb_up;
  q.rows = rows, q.row_start = row_start;
  row_channels(row_start, rows, H0, W0, q.ci0, q.n_ci);
  q.H0 = H0, q.W0 = W0, q.Cin = Cin, q.H = H, q.W = W, q.Cout = Cout, q.Kh = Kh, q.Kw = Kw, q.stride = stride, q.pad = pad;
  q.Ho = Ho, q.Wo = Wo, q.iwh = gi.wh, q.iww = gi.ww, q.owh = go.wh, q.oww = go.ww;
  q.iy = gi.y, q.ix = gi.x, q.oy = go.y, q.ox = go.x;
  q.kh1 = chain[0], q.kw1 = chain[1], q.stride1 = chain[2], q.pad1 = chain[3];
  const int S = go.y.S, cls_y = std::min(S, H0);
  q.cls_x = std::min(S, W0);
  q.uih = q.uiw = 1;
  for (int yi = 0; yi < cls_y; ++yi) q.uih = std::max(q.uih, gi.y.free_hi(yi) - gi.y.free_lo(yi) + 1);
  for (int xi = 0; xi < q.cls_x; ++xi) q.uiw = std::max(q.uiw, gi.x.free_hi(xi) - gi.x.free_lo(xi) + 1);
  const int64_t n_cls = (int64_t)q.n_ci * ceil_div(H0, S) * ceil_div(W0, S);   // rows of the largest class
  if (n_cls > 0x7fffffff / 64) return FB_ERR_SHAPE;
  // about a block per SM, the weights being staged once per block
  q.G = (int)std::max<int64_t>(1, std::min<int64_t>(kCwMaxRows / kCwR, ceil_div((int64_t)cls_y * q.cls_x * n_cls, (int64_t)kCwR * device_info().sms)));
  const int cpt = Cout % 2 == 0 ? 2 : 1;
  static_assert(sizeof(CwRow) * kCwMaxRows <= kCwStatic, "static shared memory");
  const size_t limit = device_info().smem_optin - 2 * kCwStatic;
  auto bytes = [&] {
    return sizeof(float) * q.CC * ((size_t)Kh * Kw * (Cout + cpt) + 2 * (size_t)q.uih * q.uiw * q.G * kCwR);
  };
  q.CC = Cin;
  while (bytes() > limit && (q.CC > 1 || q.G > 1)) {
    if (q.CC > 1) q.CC = (q.CC + 1) / 2;
    else q.G = (q.G + 1) / 2;
  }
  const bool direct = bytes() > limit;
  q.per_class = (int)ceil_div(n_cls, (int64_t)q.G * kCwR);
  const int64_t items = (int64_t)q.G * go.wh * go.ww * (Cout / cpt);
  const int threads = direct ? 256 : (int)(ceil_div(ceil_div(items, ceil_div(items, kCwConvThreads)), 32) * 32);
  const int64_t out = (int64_t)Cout * Ho * Wo;
  q.blocks_bias = b_lo != nullptr ? (int)std::min<int64_t>(ceil_div(out, threads), device_info().sms) : 0;
  const int64_t blocks = q.blocks_bias + (direct ? grid_for(rows * Cout * go.wh * go.ww, 256) : (int64_t)cls_y * q.cls_x * q.per_class);
  if (blocks > 0x7fffffff) return FB_ERR_SHAPE;
  auto kern = Kh == 3 && Kw == 3 ? (cpt == 2 ? cw_conv_kernel<3, 2, kAbi> : cw_conv_kernel<3, 1, kAbi>)
                                 : (cpt == 2 ? cw_conv_kernel<0, 2, kAbi> : cw_conv_kernel<0, 1, kAbi>);
  if (!direct)
    if (int rc = ensure_dynamic_smem(kern, bytes())) return rc;
  ProfileScope prof(PK_CONV, 8.0 * rows * Cout * go.wh * go.ww * Cin * Kh * Kw,
                    4.0 * 2.0 * rows * ((double)Cin * gi.wh * gi.ww + (double)Cout * go.wh * go.ww), (void*)st);
  if (kAbi) {   // (the kernel stores the pixels' own windows)
    const size_t n = sizeof(float) * (size_t)rows * Cout * go.wh * go.ww;
    FB_CUDA_OK(cudaMemsetAsync(y_lo, 0, n, st));
    FB_CUDA_OK(cudaMemsetAsync(y_up, 0, n, st));
  }
  if (direct) fb::launch_k(cw_conv_direct_kernel<kAbi>, (unsigned)blocks, threads, 0, st, q, gi, go);
  else fb::launch_k(kern, (unsigned)blocks, threads, bytes(), st, q);
  FB_LAUNCH_OK();
  return FB_OK;
}

inline int64_t linear_tiles(int H0, int W0) { return (int64_t)H0 * ceil_div(W0, kCwPx); }

// coef != nullptr: the rows go through that rescale first.  part != nullptr: no rows are written, but the partial norms
// [linear_tiles][2][N].  lb != nullptr: the bias part goes along.
template <bool kAbi>
int linear_rows(const float* z_lw, const float* z_uw, const float* coef, const float* Wl, float* y_lw, float* y_uw, float* part,
                 const float* lb, const float* ub, const float* bias, float* y_lb, float* y_ub, int64_t rows, int64_t row_start, int H0,
                 int W0, const int* chain, int n_chain, int C, int H, int W, int N, int p, cudaStream_t st) {
  if (rows < 0 || row_start < 0 || N <= 0) return FB_ERR_ARG;
  CwLinearArgs<kAbi> q = {};
  int rc = make_shape(chain, n_chain, H0, W0, C, H, W, q.g);
  if (rc != FB_OK) return rc;
  if (rows == 0) return FB_OK;
  q.z_lw = z_lw, q.z_uw = z_uw, q.coef = coef, q.W = Wl, q.y_lw = y_lw, q.y_uw = y_uw, q.part = part;
  q.lb = lb, q.ub = ub, q.bias = bias, q.y_lb = y_lb, q.y_ub = y_ub;
  q.bias_blocks = lb != nullptr ? N : 0;
  q.rows = rows, q.row_start = row_start, q.N = N, q.p = p;
  row_channels(row_start, rows, H0, W0, q.ci0, q.n_ci);
  // widest union of the windows of a tile
  q.nx_max = 1;
  for (int x0 = 0; x0 < W0; x0 += kCwPx) q.nx_max = std::max(q.nx_max, q.g.x.hi(std::min(W0, x0 + kCwPx) - 1) - q.g.x.lo(x0) + 1);
  // outputs a block: at most 16, fewer where a row of positions would not fit otherwise
  const size_t limit = device_info().smem_optin - 2 * kCwStatic;
  int NB = 16;
  auto row_bytes = [&] { return sizeof(float) * (32 * (NB + 2) + 2) * (size_t)q.nx_max; };
  while (NB > 4 && row_bytes() > limit) NB -= 4;
  if (row_bytes() > limit) return FB_ERR_SHAPE;
  const int groups = (int)ceil_div(N, NB);
  q.nb = (int)ceil_div(N, groups);
  NB = (int)ceil_div(q.nb, 4) * 4;
  q.ny_max = (int)std::max<int64_t>(1, std::min<int64_t>(q.g.wh, (int64_t)(limit / 2 / row_bytes())));   // two blocks per SM where that is possible
  const int64_t blocks = q.bias_blocks + linear_tiles(H0, W0);
  if (blocks > 0x7fffffff || groups > 65535) return FB_ERR_SHAPE;
  const size_t smem = row_bytes() * q.ny_max;
  auto kern = NB == 4    ? cw_linear_kernel<4, kAbi>
              : NB == 8  ? cw_linear_kernel<8, kAbi>
              : NB == 12 ? cw_linear_kernel<12, kAbi>
                         : cw_linear_kernel<16, kAbi>;
  if (int rc = ensure_dynamic_smem(kern, smem)) return rc;
  ProfileScope prof(PK_MATMUL, 8.0 * rows * C * q.g.wh * q.g.ww * N,
                    4.0 * (2.0 * rows * C * q.g.wh * q.g.ww + 2.0 * rows * N + (double)C * H * W * N), (void*)st);
  fb::launch_k(kern, dim3((unsigned)blocks, (unsigned)groups), kCwLinThreads, smem, st, q);
  FB_LAUNCH_OK();
  return FB_OK;
}

// op < 0: partial accumulations to part_l / part_u; else the coefficients of the relaxation and the relaxed bias terms.
template <bool kAbi>
int norm_columns(int op, const float* z_lw, const float* z_uw, float* part_l, float* part_u, const float* lb, const float* ub, float* out_lb,
               float* out_ub, float* coef, int64_t rows, int64_t row_start, int Cin0, int H0, int W0, const int* chain, int n_chain, int C,
               int H, int W, int p, float eps, int* violation, cudaStream_t st) {
  if (rows < 0 || row_start < 0 || Cin0 <= 0 || !valid_norm(p) || row_start + rows > (int64_t)Cin0 * H0 * W0) return FB_ERR_ARG;
  CwShape<kAbi> g;
  int rc = make_shape(chain, n_chain, H0, W0, C, H, W, g);
  if (rc != FB_OK) return rc;
  if (ceil_div(C, 32) > 65535 || (int64_t)Cin0 * H0 * W0 > 0x7fffffff) return FB_ERR_SHAPE;
  ProfileScope prof(PK_RELAX, 4.0 * rows * C * g.wh * g.ww, 4.0 * (2.0 * rows * C * g.wh * g.ww + 2.0 * C * H * W), (void*)st);
  fb::launch_k(cw_norm_kernel<kAbi>, dim3((unsigned)(H * W), (unsigned)ceil_div(C, 32)), 32 * kCwNormWarps, 0, st, op, z_lw, z_uw, part_l, part_u, lb, ub, out_lb, out_ub, coef, rows, row_start, Cin0, g, p, eps, violation);
  FB_LAUNCH_OK();
  return FB_OK;
}

template <bool kAbi>
int relax_columns(int op, const float* lb, const float* ub, const float* norm_l, const float* norm_u, float* out_lb, float* out_ub,
                  float* coef, int C, int64_t hw, int p, float eps, int* violation, cudaStream_t st) {
  fb::launch_k(cw_relax_columns_kernel<kAbi>, grid_for(C * hw, 256), 256, 0, st, op, lb, ub, norm_l, norm_u, out_lb, out_ub, coef, C, hw, p, eps, violation);
  FB_LAUNCH_OK();
  return FB_OK;
}

template <bool kAbi>
int rescale_rows(const float* z_lw, const float* z_uw, const float* coef, float* out_lw, float* out_uw, int64_t rows, int64_t row_start,
                    int H0, int W0, const int* chain, int n_chain, int C, int H, int W, cudaStream_t st) {
  CwShape<kAbi> g;
  int rc = make_shape(chain, n_chain, H0, W0, C, H, W, g);
  if (rc != FB_OK || rows == 0) return rc;
  fb::launch_k(cw_rescale_kernel<kAbi>, (unsigned)ceil_div(rows, 8), 256, 0, st, z_lw, z_uw, coef, out_lw, out_uw, rows, row_start, g);
  FB_LAUNCH_OK();
  return FB_OK;
}

// First convolution and relaxation (op < 0: none): the columns' slopes, then the rows.
template <bool kAbi>
int identity_rows(int op, const float* x_lb, const float* x_ub, const float* Wt, const float* bias, float scale, float* z_lw, float* z_uw,
                  float* y_lb, float* y_ub, float* col_ws, int64_t rows, int64_t row_start, int Cin, int H, int W, int Cout, int Kh, int Kw,
                  int stride, int pad, int p, float eps, int* violation, cudaStream_t st) {
  if (rows < 0 || row_start < 0 || Cin <= 0 || H <= 0 || W <= 0 || Cout <= 0 || Kh <= 0 || Kw <= 0 || stride <= 0 || pad < 0 ||
      !valid_norm(p) || row_start + rows > (int64_t)Cin * H * W)
    return FB_ERR_ARG;
  if (op >= 0 && !(op >= FB_RELU && op <= FB_SQRT)) return FB_ERR_ARG;
  const int chain[4] = {Kh, Kw, stride, pad};
  CwShape<kAbi> g;
  const int Ho = (H + 2 * pad - Kh) / stride + 1, Wo = (W + 2 * pad - Kw) / stride + 1;
  if (Ho <= 0 || Wo <= 0) return FB_ERR_SHAPE;
  int rc = make_shape(chain, 1, H, W, Cout, Ho, Wo, g);
  if (rc != FB_OK) return rc;
  const int64_t ncol = (int64_t)Cout * Ho * Wo;
  ProfileScope prof(PK_CONV, 2.0 * rows * Cout * g.wh * g.ww, 4.0 * 2.0 * rows * Cout * g.wh * g.ww, (void*)st);
  float* k_l = col_ws;
  float* k_u = col_ws + ncol;
  rc = launch_identity_columns(op, x_lb, x_ub, Wt, bias, y_lb, y_ub, k_l, k_u, scale, Cin, H, W, Cout, Kh, Kw, stride, pad, Ho, Wo, p, eps,
                               violation, st);
  if (rc != FB_OK || rows == 0) return rc;
  fb::launch_k(cw_identity_rows_kernel<kAbi>, grid_for(rows * Cout * g.wh * g.ww, 256), 256, 0, st, Wt, k_l, k_u, z_lw, z_uw, scale, rows, row_start,
                                                                                   Cin, H, W, Cout, Kh, Kw, stride, pad, Ho, Wo,
                                                                                   g.wh, g.ww);
  FB_LAUNCH_OK();
  return FB_OK;
}

// Dense rows [rows, C, H, W].
template <bool kAbi>
int expand_rows(const float* z_lw, const float* z_uw, float* y_lw, float* y_uw, int64_t rows, int64_t row_start, int H0, int W0,
                const int* chain, int n_chain, int C, int H, int W, cudaStream_t st) {
  if (rows < 0 || row_start < 0) return FB_ERR_ARG;
  CwShape<kAbi> g;
  int rc = make_shape(chain, n_chain, H0, W0, C, H, W, g);
  if (rc != FB_OK) return rc;
  if (rows == 0) return FB_OK;
  if (rows > 0x7fffffff) return FB_ERR_SHAPE;
  ProfileScope prof(PK_ELEMENTWISE, 0.0, 4.0 * 2.0 * rows * C * H * W, (void*)st);
  fb::launch_k(cw_expand_kernel<kAbi>, (unsigned)rows, 256, 0, st, z_lw, z_uw, y_lw, y_uw, row_start, g);
  FB_LAUNCH_OK();
  return FB_OK;
}

}  // namespace

int cw_identity_rows(int op, const float* x, const float* Wt, const float* bias, float* z_lw, float* z_uw, float* y_lb, float* y_ub,
                     float* col_ws, int64_t rows, int64_t row_start, int Cin, int H, int W, int Cout, int Kh, int Kw, int stride, int pad,
                     int p, float eps, int* violation, cudaStream_t st) {
  return identity_rows<false>(op, x, x, Wt, bias, 1.0f, z_lw, z_uw, y_lb, y_ub, col_ws, rows, row_start, Cin, H, W, Cout, Kh, Kw, stride, pad,
                              p, eps, violation, st);
}

int cw_conv_ex(const float* z_lo, const float* z_up, const float* W1, const float* k_l, const float* k_u, float scale, int Cin0,
               const float* Wt, float* y_lo, float* y_up, const float* b_lo, const float* b_up, const float* bias, float* yb_lo,
               float* yb_up, int64_t rows, int64_t row_start, int H0, int W0, const int* chain, int n_chain, int Cin, int H, int W,
               int Cout, int Kh, int Kw, int stride, int pad, cudaStream_t st) {
  return conv_rows<false>(z_lo, z_up, W1, k_l, k_u, scale, Cin0, Wt, y_lo, y_up, b_lo, b_up, bias, yb_lo, yb_up, rows, row_start, H0, W0,
                          chain, n_chain, Cin, H, W, Cout, Kh, Kw, stride, pad, st);
}

int64_t cw_linear_tiles(int H0, int W0) { return linear_tiles(H0, W0); }

int cw_linear_ex(const float* z_lw, const float* z_uw, const float* coef, const float* Wl, float* y_lw, float* y_uw, float* part,
                 const float* lb, const float* ub, const float* bias, float* y_lb, float* y_ub, int64_t rows, int64_t row_start, int H0,
                 int W0, const int* chain, int n_chain, int C, int H, int W, int N, int p, cudaStream_t st) {
  return linear_rows<false>(z_lw, z_uw, coef, Wl, y_lw, y_uw, part, lb, ub, bias, y_lb, y_ub, rows, row_start, H0, W0, chain, n_chain, C, H,
                            W, N, p, st);
}

int cw_linear_range(const float* part, const float* lb, const float* ub, float* l, float* u, int H0, int W0, int N, int p, float eps,
                    cudaStream_t st) {
  fb::launch_k(cw_linear_range_kernel, (unsigned)N, 64, 0, st, part, lb, ub, l, u, (int)cw_linear_tiles(H0, W0), N, p, eps);
  FB_LAUNCH_OK();
  return FB_OK;
}

int cw_norm_ex(int op, const float* z_lw, const float* z_uw, float* part_l, float* part_u, const float* lb, const float* ub, float* out_lb,
               float* out_ub, float* coef, int64_t rows, int64_t row_start, int Cin0, int H0, int W0, const int* chain, int n_chain, int C,
               int H, int W, int p, float eps, int* violation, cudaStream_t st) {
  return norm_columns<false>(op, z_lw, z_uw, part_l, part_u, lb, ub, out_lb, out_ub, coef, rows, row_start, Cin0, H0, W0, chain, n_chain, C,
                             H, W, p, eps, violation, st);
}

int cw_relax_columns(int op, const float* lb, const float* ub, const float* norm_l, const float* norm_u, float* out_lb, float* out_ub,
                     float* coef, int C, int64_t hw, int p, float eps, int* violation, cudaStream_t st) {
  return relax_columns<false>(op, lb, ub, norm_l, norm_u, out_lb, out_ub, coef, C, hw, p, eps, violation, st);
}

int cw_rescale_rows(const float* z_lw, const float* z_uw, const float* coef, float* out_lw, float* out_uw, int64_t rows, int64_t row_start,
                    int H0, int W0, const int* chain, int n_chain, int C, int H, int W, cudaStream_t st) {
  return rescale_rows<false>(z_lw, z_uw, coef, out_lw, out_uw, rows, row_start, H0, W0, chain, n_chain, C, H, W, st);
}

int cw_expand_rows(const float* z_lw, const float* z_uw, float* y_lw, float* y_uw, int64_t rows, int64_t row_start, int H0, int W0,
                   const int* chain, int n_chain, int C, int H, int W, cudaStream_t st) {
  return expand_rows<false>(z_lw, z_uw, y_lw, y_uw, rows, row_start, H0, W0, chain, n_chain, C, H, W, st);
}

}  // namespace fb

using namespace fb;

extern "C" int fb_cw_extent(int H0, int W0, const int* chain, int n_chain, int* wh, int* ww) {
  if (!wh || !ww) return FB_ERR_ARG;
  ConvChain ch;
  int h, w;
  int rc = chain_from_host(chain, n_chain, H0, W0, ch, h, w);
  if (rc != FB_OK) return rc;
  *wh = chain_extent(ch, ch.kh, H0), *ww = chain_extent(ch, ch.kw, W0);
  return FB_OK;
}

extern "C" int fb_cw_identity_relax_f32(int op, const float* x_lb, const float* x_ub, const float* Wt, const float* bias,
                                        float scale, float* z_lw, float* z_uw, float* y_lb, float* y_ub, float* col_ws,
                                        int64_t rows, int64_t row_start, int Cin, int H, int W, int Cout, int Kh, int Kw,
                                        int stride, int pad, int p, float eps, int* violation, void* stream) {
  if (!x_lb || !x_ub || !Wt || !z_lw || !z_uw || !y_lb || !y_ub || !col_ws) return FB_ERR_ARG;
  return identity_rows<true>(op, x_lb, x_ub, Wt, bias, scale, z_lw, z_uw, y_lb, y_ub, col_ws, rows, row_start, Cin, H, W, Cout, Kh, Kw,
                             stride, pad, p, eps, violation, (cudaStream_t)stream);
}

extern "C" int fb_cw_conv2d_f32(const float* x_lw, const float* x_uw, const float* Wt, float* y_lw, float* y_uw, int64_t rows,
                                int64_t row_start, int H0, int W0, const int* chain, int n_chain, int Cin, int H, int W,
                                int Cout, int Kh, int Kw, int stride, int pad, void* stream) {
  if (!x_lw || !x_uw || !Wt || !y_lw || !y_uw) return FB_ERR_ARG;
  return conv_rows<true>(x_lw, x_uw, nullptr, nullptr, nullptr, 1.f, 0, Wt, y_lw, y_uw, nullptr, nullptr, nullptr, nullptr, nullptr, rows,
                         row_start, H0, W0, chain, n_chain, Cin, H, W, Cout, Kh, Kw, stride, pad, (cudaStream_t)stream);
}

extern "C" int fb_cw_norm_partials_f32(const float* z_lw, const float* z_uw, float* part_l, float* part_u, int64_t rows,
                                       int64_t row_start, int Cin0, int H0, int W0, const int* chain, int n_chain, int C, int H,
                                       int W, int p, void* stream) {
  if (!z_lw || !z_uw || !part_l || !part_u) return FB_ERR_ARG;
  return norm_columns<true>(-1, z_lw, z_uw, part_l, part_u, nullptr, nullptr, nullptr, nullptr, nullptr, rows, row_start, Cin0, H0, W0, chain,
                            n_chain, C, H, W, p, 0.f, nullptr, (cudaStream_t)stream);
}

extern "C" int fb_cw_relax_apply_f32(int op, const float* z_lw, const float* z_uw, const float* lb, const float* ub,
                                     const float* norm_l, const float* norm_u, float* out_lw, float* out_uw, float* out_lb,
                                     float* out_ub, float* coef_ws, int64_t rows, int64_t row_start, int H0, int W0,
                                     const int* chain, int n_chain, int C, int H, int W, int p, float eps, int* violation,
                                     void* stream) {
  if (op < FB_RELU || op > FB_SQRT) return FB_ERR_ARG;
  if (!z_lw || !z_uw || !lb || !ub || !norm_l || !norm_u || !out_lw || !out_uw || !out_lb || !out_ub || !coef_ws) return FB_ERR_ARG;
  if (rows < 0 || row_start < 0 || !valid_norm(p)) return FB_ERR_ARG;
  CwShape<true> g;
  int rc = make_shape(chain, n_chain, H0, W0, C, H, W, g);
  if (rc != FB_OK) return rc;
  const int64_t ncol = (int64_t)C * H * W, per_row = (int64_t)C * g.wh * g.ww;
  ProfileScope prof(PK_RELAX, 4.0 * rows * per_row, 4.0 * (4.0 * rows * per_row + 10.0 * ncol), stream);
  rc = relax_columns<true>(op, lb, ub, norm_l, norm_u, out_lb, out_ub, coef_ws, C, (int64_t)H * W, p, eps, violation, (cudaStream_t)stream);
  if (rc != FB_OK) return rc;
  return rescale_rows<true>(z_lw, z_uw, coef_ws, out_lw, out_uw, rows, row_start, H0, W0, chain, n_chain, C, H, W, (cudaStream_t)stream);
}

extern "C" int fb_cw_linear_f32(const float* z_lw, const float* z_uw, const float* Wl, float* y_lw, float* y_uw, float* wt_ws,
                                int64_t rows, int64_t row_start, int H0, int W0, const int* chain, int n_chain, int C, int H,
                                int W, int N, void* stream) {
  if (!z_lw || !z_uw || !Wl || !y_lw || !y_uw || !wt_ws) return FB_ERR_ARG;
  return linear_rows<true>(z_lw, z_uw, nullptr, Wl, y_lw, y_uw, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, rows, row_start, H0, W0,
                           chain, n_chain, C, H, W, N, FB_PINF, (cudaStream_t)stream);
}

extern "C" int fb_cw_expand_f32(const float* z_lw, const float* z_uw, float* y_lw, float* y_uw, int64_t rows, int64_t row_start,
                                int H0, int W0, const int* chain, int n_chain, int C, int H, int W, void* stream) {
  if (!z_lw || !z_uw || !y_lw || !y_uw) return FB_ERR_ARG;
  return expand_rows<true>(z_lw, z_uw, y_lw, y_uw, rows, row_start, H0, W0, chain, n_chain, C, H, W, (cudaStream_t)stream);
}
