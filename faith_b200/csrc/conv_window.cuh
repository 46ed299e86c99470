// Window arithmetic of the convolutions behind an identity input (all pixels of an H0 x W0 image perturbed): row r of
// the weight tensors stands for one pixel, and after a chain of convolutions it is zero outside the window that pixel
// reaches.  Shared by the dense-row kernels (conv.cu) and the compact-row kernels (conv_compact.cu).
#pragma once
#include <algorithm>

#include "common.cuh"

namespace fb {

// The convolutions a row has been through before the one being computed: enough to know, from the row's pixel alone,
// the window outside of which the row is zero.
constexpr int kMaxChain = 8;
struct ConvChain {
  int n;
  int kh[kMaxChain], kw[kMaxChain], stride[kMaxChain], pad[kMaxChain];
};

struct Span { int lo, hi; };   // inclusive; lo > hi: empty

// Outputs (along one axis) of a convolution (k, stride, pad, n_out outputs) that have a tap inside the input span.
__host__ __device__ inline Span span_after_conv(Span s, int k, int stride, int pad, int n_out) {
  if (s.lo > s.hi) return s;
  const int a = s.lo + pad - (k - 1);
  Span o;
  o.lo = a > 0 ? (a + stride - 1) / stride : 0;
  o.hi = (s.hi + pad) / stride;
  if (o.hi > n_out - 1) o.hi = n_out - 1;
  return o;
}

// Window, along one axis (k: the filter sizes of the chain along it) and in the coordinates of the output of the first n
// convolutions, reached by pixel i of n0.
__host__ __device__ inline Span chain_span(const ConvChain& ch, const int* k, int n, int n0, int i) {
  Span s = {i, i};
  for (int j = 0; j < n; ++j) {
    n0 = (n0 + 2 * ch.pad[j] - k[j]) / ch.stride[j] + 1;
    s = span_after_conv(s, k[j], ch.stride[j], ch.pad[j], n0);
  }
  return s;
}

// Window (in the coordinates of the chain's last output) reached by pixel (yi, xi) of the H0 x W0 image.
__host__ __device__ inline void chain_window(const ConvChain& ch, int H0, int W0, int yi, int xi, Span& wy, Span& wx) {
  wy = chain_span(ch, ch.kh, ch.n, H0, yi);
  wx = chain_span(ch, ch.kw, ch.n, W0, xi);
}

// Largest window along one axis that any pixel of n0 reaches through the chain (at least 1).
inline int chain_extent(const ConvChain& ch, const int* k, int n0) {
  int win = 1;
  for (int i = 0; i < n0; ++i) {
    const Span s = chain_span(ch, k, ch.n, n0, i);
    win = std::max(win, s.hi - s.lo + 1);
  }
  return win;
}

// Host side: the chain as the C ABI passes it (n x 4 ints: kernel height, kernel width, stride, padding).  Fills `ch`
// and the size (h, w) of the chain's last output; FB_ERR_ARG / FB_ERR_SHAPE on malformed input.
inline int chain_from_host(const int* chain, int n_chain, int H0, int W0, ConvChain& ch, int& h, int& w) {
  if (n_chain < 0 || (n_chain > 0 && !chain) || H0 <= 0 || W0 <= 0) return FB_ERR_ARG;
  if (n_chain > kMaxChain) return FB_ERR_SHAPE;
  ch.n = n_chain;
  h = H0, w = W0;
  for (int i = 0; i < n_chain; ++i) {
    ch.kh[i] = chain[4 * i], ch.kw[i] = chain[4 * i + 1], ch.stride[i] = chain[4 * i + 2], ch.pad[i] = chain[4 * i + 3];
    if (ch.kh[i] <= 0 || ch.kw[i] <= 0 || ch.stride[i] <= 0 || ch.pad[i] < 0) return FB_ERR_ARG;
    h = (h + 2 * ch.pad[i] - ch.kh[i]) / ch.stride[i] + 1;
    w = (w + 2 * ch.pad[i] - ch.kw[i]) / ch.stride[i] + 1;
    if (h <= 0 || w <= 0) return FB_ERR_SHAPE;
  }
  return FB_OK;
}

// The same for the compact rows of the CNN driver (conv_compact.cu), along one axis.  Without the borders of the maps the nested
// divisions of a chain collapse into one: pixel i reaches [ceil((i + A) / S), floor((i + B) / S)], S the product of the strides, so that a shift
// of the pixel by S shifts the window by one; the compact window is that interval cut to the map.  (It holds the window above,
// and is larger only where a padding exceeds its filter or a stride its filter; what is more is zero.)  Turned round, output y is
// reached by the pixels [y S - B, y S - A].
struct CwAxis {
  int S, sh, A, B, n;   // sh: log2(S), or -1; n: outputs of the chain
  __host__ __device__ int floor_s(int a) const { return sh >= 0 ? a >> sh : a >= 0 ? a / S : -((-a + S - 1) / S); }
  __host__ __device__ int free_lo(int i) const { return floor_s(i + A + S - 1); }
  __host__ __device__ int free_hi(int i) const { return floor_s(i + B); }
  __host__ __device__ int lo(int i) const { const int v = free_lo(i); return v > 0 ? v : 0; }
  __host__ __device__ int hi(int i) const { const int v = free_hi(i); return v < n - 1 ? v : n - 1; }
};

inline int axis_from_chain(const ConvChain& ch, const int* k, int n, CwAxis& ax) {
  int64_t S = 1, A = 0, B = 0;
  for (int i = 0; i < ch.n; ++i) {
    A += (ch.pad[i] - (k[i] - 1)) * S;
    B += ch.pad[i] * S;
    S *= ch.stride[i];
    if (S > (1 << 24) || A < -(1 << 28) || B > (1 << 28)) return FB_ERR_SHAPE;
  }
  ax.S = (int)S, ax.A = (int)A, ax.B = (int)B, ax.n = n;
  ax.sh = -1;
  for (int i = 0; i < 25; ++i)
    if (S == (int64_t)1 << i) ax.sh = i;
  return FB_OK;
}

// Largest window any pixel of n0 reaches (at least 1).
inline int axis_extent(const CwAxis& ax, int n0) {
  int win = 1;
  for (int i = 0; i < n0; ++i) win = std::max(win, ax.hi(i) - ax.lo(i) + 1);
  return win;
}

// Whether these are the windows of chain_span for every pixel of n0.
inline bool axis_is_chain(const CwAxis& ax, const ConvChain& ch, const int* k, int n0) {
  for (int i = 0; i < n0; ++i) {
    const Span s = chain_span(ch, k, ch.n, n0, i);
    if (ax.lo(i) != s.lo || ax.hi(i) != s.hi) return false;
  }
  return true;
}

// Bias part, slopes and relaxed bias terms of the first convolution and the relaxation behind it, per output column (conv.cu).
int launch_identity_columns(int op, const float* x_lb, const float* x_ub, const float* Wt, const float* bias, float* y_lb, float* y_ub,
                            float* k_l, float* k_u, float scale, int Cin, int H, int W, int Cout, int Kh, int Kw, int stride, int pad,
                            int Ho, int Wo, int p, float eps, int* violation, cudaStream_t st);

}  // namespace fb
