// Shared host/device helpers of libfaith_b200 (sm_100a only).
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "faith_b200.h"

namespace fb {

// ---------------------------------------------------------------- host side
void set_last_cuda_error(int e);

struct DeviceInfo {
  int sms;
  int smem_optin;  // max dynamic shared memory per block (opt-in), bytes
};
// Properties of the current device, queried once per device and cached.
const DeviceInfo& device_info();

#define FB_CUDA_OK(expr)                                   \
  do {                                                     \
    cudaError_t fb_e_ = (expr);                            \
    if (fb_e_ != cudaSuccess) {                            \
      fb::set_last_cuda_error((int)fb_e_);                 \
      return FB_ERR_CUDA;                                  \
    }                                                      \
  } while (0)

// Checks the launches just enqueued (n of them, for the launch counter of fb_profile_*).
#define FB_LAUNCH_OK_N(n)                \
  do {                                   \
    fb::count_launches(n);               \
    FB_CUDA_OK(cudaGetLastError());      \
  } while (0)
#define FB_LAUNCH_OK() FB_LAUNCH_OK_N(1)

void count_launches(int n);

// A launch whose blocks may become resident while the launch before on the stream still drains (programmatic dependent launch):
// the passes over one sentence are chains of kernels of 3 to 10 us with 2 us between them, most of it launch latency and
// prologues (barriers, tensor memory, tensor maps).  The kernel must call pdl_sync() first thing.  Work of many waves keeps the
// plain launch: the gap before it is nothing beside it, and the hand-over cost the 4096 blocks of a relaxation 2 % of 135 us.
// tiles: what a persistent kernel walks, the number of blocks for any other; kManyTiles where the blocks run long and there are more
// of them than two an SM: those that come early fill the gaps as these appear, two more on one SM than on another, and that costs
// more than the launch.  us plain and programmatic: product of two bounds, 420 blocks of 320 rows 22.8 and 32.4; relu, 440 blocks of
// 384 rows re-read from L2 3.3 more, tanh 4.2 more; 16 columns of K = 400, 580 blocks 9.7 more.
constexpr int64_t kManyTiles = INT64_MAX;
template <typename... P, typename... A>
inline void launch_tiles(int64_t tiles, void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = tiles <= 4 * (int64_t)device_info().sms ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);   // (errors are picked up by FB_LAUNCH_OK)
}
template <typename... P, typename... A>
inline void launch_k(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  launch_tiles((int64_t)grid.x * grid.y * grid.z, kern, grid, block, smem, st, args...);
}

// Hint for the tensor-core GEMM (thread-local, set by the encoder driver around the projections of the first layer):
// the operand has M rows in blocks of Di per (sentence, position) pair, L positions per sentence, and only the
// blocks of the perturbed positions are non-zero (the input bound is an identity at those positions and zero
// elsewhere, VerifierForward.py:127-156).  Positions: `pos` (one set for all sentences) or `inst_pos` (device,
// [sentences, words]).  The zero-radius GEMM then writes zeros for the other blocks without reading or multiplying.
struct LiveRows {
  int L, Di, words;
  int pos[4];
  const int* inst_pos;
  int64_t M;
};
void tc_set_live_rows(const LiveRows* lr);   // nullptr clears

// The bias terms of a bound riding in the GEMM launch of its weight rows (extra tiles at the end of the grid):
// operand a_lo / a_up [M, K], the layer bias (may be null), results c_lo / c_up [M, N] stored plain, and the
// residual res_lo / res_up [M, N] when the weight rows add one.
struct TcBiasRows {
  const float* a_lo;
  const float* a_up;
  const float* bias;
  float* c_lo;
  float* c_up;
  int64_t M;
  const float* res_lo;
  const float* res_up;
};

// Layer norm (mode no_var) applied by the epilogue of a product with residual: gain and shift [N], the weight itself
// (its column means give the row means of the product), the row sums of the residual as its producer left them and
// those of the result for the next consumer: [2 lines][4 partial sums][rs_stride rows], weight rows first, then bias rows.
struct TcLnArgs {
  const float* gamma;
  const float* beta;
  const float* w_raw;
  const float* rs_in;
  float* rs_out;
  int64_t rs_stride;
};

// A large product for the fp16-split kernels (matmul_tc_f16.cuh), as launch_split_sign_tc has checked it: operands [M, K], W [N, K],
// results [M, N] (head-split where split_rows > 0), slopes, norms, residual and bias rows as there, null where absent.
struct F16Product {
  const float *a_lo, *a_up, *W, *bias;
  float *c_lo, *c_up;
  int64_t M;
  int N, K, split_rows, split_d;
  const float *coef_l, *coef_u;
  int coef_di;
  float *norm_lo, *norm_up;
  int norm_p;
  const float *res_lo, *res_up;
  const TcBiasRows* br;
  int* status;
  uint32_t wait_tries;
  int skip_it;
  LiveRows live;
};
int launch_split_sign_f16(const F16Product& q, cudaStream_t st);          // K <= 128
int launch_split_sign_f16_stream(const F16Product& q, cudaStream_t st);   // K > 128
int f16_error_flag(int* flag);
int f16_stream_error_flag(int* flag);

// fb_layernorm_novar_f32 that can also leave the row sums of its result behind (rowsum, may be null; 128 features
// only): [2 lines][4 partial sums][rows * (Di + 1)], of which it writes the first partial sum of each line.
int layernorm_novar_rowsum(const float* x_lw, const float* x_uw, const float* x_lb, const float* x_ub, const float* r_lw,
                           const float* r_uw, const float* r_lb, const float* r_ub, const float* gamma, const float* beta,
                           float* z_lw, float* z_uw, float* z_lb, float* z_ub, int64_t rows, int Di, int Do, float* rowsum,
                           void* stream);

// column_ops.cu: the concretised ranges of two bounds over the same dim_in in one launch.
int concretize_pair(const float* x_lw, const float* x_uw, const float* x_lb, const float* x_ub, float* x_l, float* x_u, int64_t x_rows,
                    int x_do, const float* y_lw, const float* y_uw, const float* y_lb, const float* y_ub, float* y_l, float* y_u,
                    int64_t y_rows, int y_do, int Di, int words, int p, float eps, int layout, cudaStream_t st);

// conv_compact.cu: the operators on compact rows in the CNN driver's form and with its options (see the definitions).
int cw_identity_rows(int op, const float* x, const float* Wt, const float* bias, float* z_lw, float* z_uw, float* y_lb, float* y_ub,
                     float* col_ws, int64_t rows, int64_t row_start, int Cin, int H, int W, int Cout, int Kh, int Kw, int stride, int pad,
                     int p, float eps, int* violation, cudaStream_t st);
int cw_expand_rows(const float* z_lw, const float* z_uw, float* y_lw, float* y_uw, int64_t rows, int64_t row_start, int H0, int W0,
                   const int* chain, int n_chain, int C, int H, int W, cudaStream_t st);
int cw_conv_ex(const float* z_lo, const float* z_up, const float* W1, const float* k_l, const float* k_u, float scale, int Cin0,
               const float* Wt, float* y_lo, float* y_up, const float* b_lo, const float* b_up, const float* bias, float* yb_lo,
               float* yb_up, int64_t rows, int64_t row_start, int H0, int W0, const int* chain, int n_chain, int Cin, int H, int W,
               int Cout, int Kh, int Kw, int stride, int pad, cudaStream_t st);
int cw_norm_ex(int op, const float* z_lw, const float* z_uw, float* part_l, float* part_u, const float* lb, const float* ub, float* out_lb,
               float* out_ub, float* coef, int64_t rows, int64_t row_start, int Cin0, int H0, int W0, const int* chain, int n_chain, int C,
               int H, int W, int p, float eps, int* violation, cudaStream_t st);
int cw_relax_columns(int op, const float* lb, const float* ub, const float* norm_l, const float* norm_u, float* out_lb, float* out_ub,
                     float* coef, int C, int64_t hw, int p, float eps, int* violation, cudaStream_t st);
int cw_rescale_rows(const float* z_lw, const float* z_uw, const float* coef, float* out_lw, float* out_uw, int64_t rows, int64_t row_start,
                    int H0, int W0, const int* chain, int n_chain, int C, int H, int W, cudaStream_t st);
int64_t cw_linear_tiles(int H0, int W0);
int cw_linear_ex(const float* z_lw, const float* z_uw, const float* coef, const float* Wl, float* y_lw, float* y_uw, float* part,
                 const float* lb, const float* ub, const float* bias, float* y_lb, float* y_ub, int64_t rows, int64_t row_start, int H0,
                 int W0, const int* chain, int n_chain, int C, int H, int W, int N, int p, cudaStream_t st);
int cw_linear_range(const float* part, const float* lb, const float* ub, float* l, float* u, int H0, int W0, int N, int p, float eps,
                    cudaStream_t st);

// What the product of a few bias rows does with its result besides storing it (matmul_ffma.cu): the concretised range, from the
// column norms [row * words + w][N] of the weight rows, to out_l / out_u in the layout of the result or (transposed) as
// [group * head][feature][row in group]; with op >= 0 the slopes k_l, k_u and the relaxed bias terms r_lb, r_ub of that
// relaxation, [M, N], as fb_relax_coef_given_f32 returns them.
struct RangeEpilogue {
  const float *norm_lo, *norm_up;
  float *out_l, *out_u;
  int words;
  float eps;
  int transposed, op;
  float *k_l, *k_u, *r_lb, *r_ub;
  int* violation;
};
bool small_product(int64_t M, int N, int K);   // whether the kernel for few rows takes a product of that size
int launch_split_sign_small(const float* a_lo, const float* a_up, const float* W, const float* bias, float* c_lo, float* c_up, int64_t M,
                            int N, int K, cudaStream_t st, int split_rows, int split_d, const RangeEpilogue* range);
// matmul.cu: fb_matmul_heads_ranges_f32 with the wishes of the driver: ranges transposed, relaxation coefficients of the result.
// Both are extras of the kernel for few bias rows; `granted` tells whether they were done.
struct RangeWishes {
  int transposed, op;
  float *k_l, *k_u, *r_lb, *r_ub;
  int* violation;
  bool granted;
};
int matmul_ranges_ex(const float* x_lw, const float* x_uw, const float* x_lb, const float* x_ub, const float* W, const float* bias,
                     float* y_lw, float* y_uw, float* y_lb, float* y_ub, float* y_l, float* y_u, float* norm_ws, int64_t rows, int Di,
                     int Do, int Dy, int L, int heads, int words, int p, float eps, RangeWishes* wishes, void* stream);

// softmax.cu: fb_softmax_ranges_f32 with rows `ld` floats apart.
int softmax_ex(const float* lw, const float* uw, const float* lb, const float* ub, float* out_lw, float* out_uw, float* out_lb,
               float* out_ub, float* out_l, float* out_u, int64_t rows, int Di, int Do, int ld, int words, int p, float eps,
               int* violation, void* stream);

bool softmax_fused_shape(int Di, int Do);   // whether the fused kernel takes the shape

// dot_product.cu: whether the tensor-core kernel takes the shape (rows of any pitch; more than a few query rows).
bool dot_pitched_supported(int B, int Lx, int Ly, int Di, int K);
// The dot product and the context product with the options of the encoder driver (see the definitions).
int dot_product_ex(const float* x_lw, const float* x_uw, const float* x_lb, const float* x_ub, const float* y_lw, const float* y_uw,
                   const float* y_lb, const float* y_ub, float* z_lw, float* z_uw, float* z_lb, float* z_ub, float* x_l, float* x_u,
                   float* y_l, float* y_u, int B, int Lx, int Ly, int Di, int K, int words, int p, float eps, float out_scale,
                   int layout, int merge_heads, int given, int ldz, void* stream);
int context_ex(const float* x_lw, const float* x_uw, const float* x_lb, const float* x_ub, const float* v_lw, const float* v_uw,
               const float* v_lb, const float* v_ub, float* z_lw, float* z_uw, float* z_lb, float* z_ub, float* x_l, float* x_u,
               float* y_l, float* y_u, int B, int Lx, int Ly, int Di, int K, int words, int p, float eps, float out_scale,
               int merge_heads, int given, int ldx, bool transposed_ranges, void* stream);

// Opts `kernel` in to `bytes` of dynamic shared memory on the current device (nothing to do up to 40 KB, or when it
// already has that much): FB_OK or FB_ERR_CUDA.
int ensure_dynamic_smem_impl(const void* func, size_t bytes);
template <typename K>
inline int ensure_dynamic_smem(K kernel, size_t bytes) {
  return ensure_dynamic_smem_impl(reinterpret_cast<const void*>(kernel), bytes);
}

// Optional per-operator timing (fb_profile_enable): the outermost C-ABI operator call on a thread
// brackets its launches with a pair of CUDA events on the caller's stream and records the
// algorithmic work of the call.  Disabled (the default), a scope costs one branch.
enum ProfileKind { PK_MATMUL = 0, PK_RELAX = 1, PK_DOT = 2, PK_MUL = 3, PK_ELEMENTWISE = 4, PK_CONV = 5, PK_COUNT = 6 };
class ProfileScope {
 public:
  ProfileScope(int kind, double flops, double bytes, void* stream);
  ~ProfileScope();
 private:
  int slot_;
  void* stream_;
};

__host__ __device__ inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
inline bool valid_norm(int p) { return p == FB_P1 || p == FB_P2 || p == FB_PINF; }
inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

// -------------------------------------------------------------- device side
// Scalar arithmetic with the rounding of the reference's PyTorch expressions: one rounding
// per operation, no contraction into fused multiply-adds.
__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fdiv(float a, float b) { return __fdiv_rn(a, b); }

// Every kernel launched through launch_k calls this before it reads or writes anything another launch may touch: it waits for
// the launches before to complete, and lets the next one start its prologue.  Unconditional: with a test of the grid's size
// around it, kernels overlapped the launch before them and read what it had not written yet.
__device__ __forceinline__ void pdl_sync() {
  asm volatile("griddepcontrol.wait;\n\tgriddepcontrol.launch_dependents;" ::: "memory");
}

// Two FP32 multiply-adds per instruction (fma.rn.f32x2), lanes in a 64-bit register pair.
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
  float2 d;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(v));
  return d;
}

constexpr float kGuard = 1e-12f;  // additive guard of every chord slope (Bounds.py:27)

// Accumulation of the dual norm over dim_in: sum |x| (p = inf), sum x^2 (p = 2), max |x| (p = 1).
__device__ __forceinline__ float norm_accum(int p, float acc, float x) {
  if (p == FB_PINF) return acc + fabsf(x);
  if (p == FB_P2) return fmaf(x, x, acc);
  return fmaxf(acc, fabsf(x));
}
__device__ __forceinline__ float norm_combine(int p, float a, float b) {
  return (p == FB_P1) ? fmaxf(a, b) : a + b;
}
__device__ __forceinline__ float norm_finish(int p, float acc) {
  return (p == FB_P2) ? sqrtf(acc) : acc;
}

// Coefficients of one column after a relaxation:
//   out_lw = c_ll * lw + c_lu * uw      out_lb = nlb
//   out_uw = c_ul * lw + c_uu * uw      out_ub = nub
// For every well-formed column (l <= u) exactly one coefficient per line is non-zero, so the
// rescale is a single rounded product as in the reference.
struct ColCoef {
  float c_ll, c_lu, c_ul, c_uu, nlb, nub;
};

// One call of the reference's add_linear (Bounds.py:362-381) at the level of a column:
// adds mask * (line with slope k through (x0, y0) applied to the input bound) to the lower
// (lower = true) or upper output line.  A positive slope keeps the side, any other swaps it.
__device__ __forceinline__ void add_line(ColCoef& c, float mask, bool lower, float k, float x0, float y0,
                                         float lb, float ub) {
  const float kp = (k > 0.f) ? 1.f : 0.f;
  const float kn = 1.f - kp;
  const float own_b = lower ? lb : ub;
  const float oth_b = lower ? ub : lb;
  const float t_own = fmul(fmul(mask, kp), fadd(fmul(fsub(own_b, x0), k), y0));
  const float t_oth = fmul(fmul(mask, kn), fadd(fmul(fsub(oth_b, x0), k), y0));
  const float w_own = fmul(fmul(mask, kp), k);
  const float w_oth = fmul(fmul(mask, kn), k);
  if (lower) {
    c.c_ll = fadd(c.c_ll, w_own);
    c.c_lu = fadd(c.c_lu, w_oth);
    c.nlb = fadd(fadd(c.nlb, t_own), t_oth);
  } else {
    c.c_uu = fadd(c.c_uu, w_own);
    c.c_ul = fadd(c.c_ul, w_oth);
    c.nub = fadd(fadd(c.nub, t_own), t_oth);
  }
}

__device__ __forceinline__ float dtanh_ref(float x) {
  const float ch = coshf(x);
  return fdiv(1.f, fmul(ch, ch));
}

// exp continued linearly above 12 (Bounds.py:984-989)
__device__ __forceinline__ float exp_capped(float x) {
  const float thres = 12.f;
  if (x < thres) return expf(fminf(x, thres));
  return fmul(expf(thres), fadd(fsub(x, thres), 1.f));
}

// Tangent points of tanh on a range that crosses zero (Bounds.py:1027-1103): upper = false: the point in [l, 0] whose tangent
// passes through (u, tanh u), else the point in [0, u] whose tangent passes through (l, tanh l); ten bisection steps.  One step
// is an evaluation of tanh_right_of and a move of (d, lo, hi).
struct TanhSearch {
  float d, lo, hi;
};
__device__ __forceinline__ TanhSearch tanh_search(bool upper, float l, float u) {
  return upper ? TanhSearch{fmul(u, 0.5f), 0.f, u} : TanhSearch{fmul(l, 0.5f), l, 0.f};
}
// does the search go on to the right of d?  x, tx: the point the tangent has to meet (u for the lower line, l for the upper)
__device__ __forceinline__ bool tanh_right_of(bool upper, float d, float x, float tx) {
  const float td = tanhf(d);
  const float v = upper ? fsub(fdiv(fsub(td, tx), fadd(fsub(d, x), kGuard)), dtanh_ref(d))
                        : fsub(fdiv(fsub(tx, td), fadd(fsub(x, d), kGuard)), dtanh_ref(d));
  return upper ? !(v > 0.f) : v > 0.f;
}
__device__ __forceinline__ TanhSearch tanh_move(TanhSearch q, bool right) {
  if (right) return TanhSearch{fmul(fadd(q.d, q.hi), 0.5f), q.d, q.hi};
  return TanhSearch{fmul(fadd(q.d, q.lo), 0.5f), q.lo, q.d};
}
constexpr int kTanhSteps = 10;
__device__ __forceinline__ float tanh_point(bool upper, float l, float u) {
  const float x = upper ? l : u, tx = tanhf(x);
  TanhSearch q = tanh_search(upper, l, u);
#pragma unroll 1
  for (int t = 0; t < kTanhSteps; ++t) q = tanh_move(q, tanh_right_of(upper, q.d, x, tx));
  return q.d;
}

// Per-column relaxation: from the concretised range (l, u) and the bias terms (lb, ub) to
// the column coefficients.  `bad` is set when FB_RECIPROCAL sees l < 1e-12.  tangent: the two tangent points of tanh where
// the caller has them already (lower line, upper line), else they are searched here.
__device__ inline ColCoef relax_column(int op, float l, float u, float lb, float ub, bool& bad, const float* tangent = nullptr) {
  ColCoef c = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (op >= FB_INTERVAL) {
    // interval form (the reference's `ibp` branches): constant bounds, no dependence on the weights
    switch (op - FB_INTERVAL) {
      case FB_RELU: c.nlb = fmaxf(l, 0.f); c.nub = fmaxf(u, 0.f); break;       // Bounds.py:924-926
      case FB_TANH: c.nlb = tanhf(l); c.nub = tanhf(u); break;                  // :1030-1032
      case FB_EXP: c.nlb = expf(l); c.nub = expf(u); break;                     // :973-975
      case FB_RECIPROCAL: c.nlb = fdiv(1.f, u); c.nub = fdiv(1.f, l); break;    // :1139-1143
      case FB_SQR: {                                                            // :863-866
        const float a = fmul(l, l), b = fmul(u, u);
        const float both = 1.f - ((l > 0.f) ? 1.f : 0.f) - ((u < 0.f) ? 1.f : 0.f);
        const float lo = fminf(a, b);
        c.nlb = fsub(lo, fmul(both, lo));   // zero when the range crosses zero
        c.nub = fmaxf(a, b);
        break;
      }
      default:                                                                  // FB_SQRT, :894-898
        if (!(l > 0.f)) bad = true;
        c.nlb = sqrtf(l);
        c.nub = sqrtf(u);
        break;
    }
    return c;
  }
  if (op == FB_SQR) {  // Bounds.py:867-885: chord above; tangent below, placed so that it never goes negative
    add_line(c, 1.f, false, fadd(u, l), l, fmul(l, l), lb, ub);
    if (u < 0.f) {
      const float m = fmaxf(fmul(fadd(l, u), 0.5f), fmul(2.f, u));
      add_line(c, 1.f, true, fmul(2.f, m), m, fmul(m, m), lb, ub);
    }
    if (l > 0.f) {
      const float m = fminf(fmul(fadd(l, u), 0.5f), fmul(2.f, l));
      add_line(c, 1.f, true, fmul(2.f, m), m, fmul(m, m), lb, ub);
    }
    return c;
  }
  if (op == FB_SQRT) {  // Bounds.py:892-913: chord below, tangent at the midpoint above
    if (!(l > 0.f)) bad = true;
    const float sl = sqrtf(l);
    add_line(c, 1.f, true, fdiv(fsub(sqrtf(u), sl), fadd(fsub(u, l), kGuard)), l, sl, lb, ub);
    const float m = fmul(fadd(l, u), 0.5f);
    const float sm = sqrtf(m);
    add_line(c, 1.f, false, fdiv(0.5f, sm), m, sm, lb, ub);
    return c;
  }
  if (op == FB_EXP) {  // Bounds.py:982-997; both slopes are applied to the own side
    const float m = fminf(fmul(fadd(l, u), 0.5f), fadd(l, 0.99f));
    const float kl = expf(fminf(m, 12.f));
    const float el = exp_capped(l);
    const float ku = fdiv(fsub(exp_capped(u), el), fadd(fsub(u, l), kGuard));
    c.c_ll = kl;
    c.nlb = fmul(kl, fadd(fsub(lb, m), 1.f));
    c.c_uu = ku;
    c.nub = fadd(fsub(fmul(ub, ku), fmul(ku, l)), el);
    return c;
  }
  if (op == FB_RECIPROCAL) {  // Bounds.py:1145-1155; both slopes negative: sides swap
    if (!(l >= kGuard)) bad = true;
    const float m = fmul(fadd(l, u), 0.5f);
    const float kl = fdiv(-1.f, fmul(m, m));
    const float ku = fdiv(-1.f, fmul(l, u));
    c.c_lu = kl;
    c.nlb = fadd(fmul(ub, kl), fdiv(2.f, m));
    c.c_ul = ku;
    c.nub = fadd(fsub(fmul(lb, ku), fmul(ku, l)), fdiv(1.f, l));
    return c;
  }
  const float pos = (l > 0.f) ? 1.f : 0.f;
  const float neg = (u < 0.f) ? 1.f : 0.f;
  const float both = 1.f - pos - neg;
  if (op == FB_RELU) {  // Bounds.py:921-963
    if (pos != 0.f) {
      add_line(c, pos, true, 1.f, 0.f, 0.f, lb, ub);
      add_line(c, pos, false, 1.f, 0.f, 0.f, lb, ub);
    }
    if (both != 0.f) {
      const float k_up = fdiv(u, fadd(fsub(u, l), kGuard));
      add_line(c, both, false, k_up, l, 0.f, lb, ub);
      const float k_lo = (fabsf(u) > fabsf(l)) ? 1.f : 0.f;
      add_line(c, both, true, k_lo, 0.f, 0.f, lb, ub);
    }
    return c;
  }
  // FB_TANH, Bounds.py:1027-1103
  if (pos != 0.f || neg != 0.f) {
    const float m = fmul(fadd(l, u), 0.5f);
    const float k_tan = dtanh_ref(m);
    const float y_tan = tanhf(m);
    const float tl = tanhf(l);
    const float k_chd = fdiv(fsub(tanhf(u), tl), fadd(fsub(u, l), kGuard));
    if (neg != 0.f) {
      add_line(c, neg, true, k_tan, m, y_tan, lb, ub);
      add_line(c, neg, false, k_chd, l, tl, lb, ub);
    }
    if (pos != 0.f) {
      add_line(c, pos, false, k_tan, m, y_tan, lb, ub);
      add_line(c, pos, true, k_chd, l, tl, lb, ub);
    }
  }
  if (both != 0.f) {
    const float tu = tanhf(u), tl = tanhf(l);
    float d = tangent != nullptr ? tangent[0] : tanh_point(false, l, u);
    float td = tanhf(d);
    float k = fdiv(fsub(td, tu), fadd(fsub(d, u), kGuard));
    add_line(c, both, true, k, d, td, lb, ub);
    d = tangent != nullptr ? tangent[1] : tanh_point(true, l, u);
    td = tanhf(d);
    k = fdiv(fsub(td, tl), fadd(fsub(d, l), kGuard));
    add_line(c, both, false, k, d, td, lb, ub);
  }
  return c;
}

}  // namespace fb
