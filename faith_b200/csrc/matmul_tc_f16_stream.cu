// Instantiations of the fp16-split product of matmul_tc_f16.cuh, K > 128: W is converted in slices.
#include <cuda.h>

#include <mutex>
#include <type_traits>
#include <unordered_map>

#include "common.cuh"

namespace fb {
namespace {
#include "tc_common.cuh"
#include "matmul_tc_f16.cuh"
}  // namespace

int launch_split_sign_f16_stream(const F16Product& q, cudaStream_t st) { return hg::launch<true>(q, st); }

int f16_stream_error_flag(int* flag) {
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
