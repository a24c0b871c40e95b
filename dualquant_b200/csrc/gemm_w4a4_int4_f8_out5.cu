// FP8-path int4 GEMM, output mode 5 (bf16 output with a bias): its token tiles, in a translation unit of their
// own to build in parallel.
#include "gemm_w4a4_int4_f8.cuh"

namespace dq {
namespace f8 {

cudaError_t run_out5(int tn, const Launch& l) {
  switch (tn) {
    case 32: return run<32, 5>(l);
    case 64: return run<64, 5>(l);
    case 96: return run<96, 5>(l);
    case 128: return run<128, 5>(l);
    case 160: return run<160, 5>(l);
    case 192: return run<192, 5>(l);
    case 224: return run<224, 5>(l);
    case 256: return run<256, 5>(l);
    default: return cudaErrorInvalidValue;
  }
}
cudaError_t init_out5() {
  cudaError_t e = cudaSuccess;
  if (e == cudaSuccess) e = allow_smem<32, 5>();
  if (e == cudaSuccess) e = allow_smem<64, 5>();
  if (e == cudaSuccess) e = allow_smem<96, 5>();
  if (e == cudaSuccess) e = allow_smem<128, 5>();
  if (e == cudaSuccess) e = allow_smem<160, 5>();
  if (e == cudaSuccess) e = allow_smem<192, 5>();
  if (e == cudaSuccess) e = allow_smem<224, 5>();
  if (e == cudaSuccess) e = allow_smem<256, 5>();
  return e;
}

}  // namespace f8
}  // namespace dq
