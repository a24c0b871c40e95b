// FP8-path int4 GEMM, output mode 1 (bf16 output through a bulk store): its token tiles, in a translation unit of their
// own to build in parallel.
#include "gemm_w4a4_int4_f8.cuh"

namespace dq {
namespace f8 {

cudaError_t run_out1(int tn, const Launch& l) {
  switch (tn) {
    case 32: return run<32, 1>(l);
    case 64: return run<64, 1>(l);
    case 96: return run<96, 1>(l);
    case 128: return run<128, 1>(l);
    case 160: return run<160, 1>(l);
    case 192: return run<192, 1>(l);
    case 224: return run<224, 1>(l);
    case 256: return run<256, 1>(l);
    default: return cudaErrorInvalidValue;
  }
}
cudaError_t init_out1() {
  cudaError_t e = cudaSuccess;
  if (e == cudaSuccess) e = allow_smem<32, 1>();
  if (e == cudaSuccess) e = allow_smem<64, 1>();
  if (e == cudaSuccess) e = allow_smem<96, 1>();
  if (e == cudaSuccess) e = allow_smem<128, 1>();
  if (e == cudaSuccess) e = allow_smem<160, 1>();
  if (e == cudaSuccess) e = allow_smem<192, 1>();
  if (e == cudaSuccess) e = allow_smem<224, 1>();
  if (e == cudaSuccess) e = allow_smem<256, 1>();
  return e;
}

}  // namespace f8
}  // namespace dq
