// FP8-path int4 GEMM, output mode 0 (direct stores, and the scatter mode of the tensor-parallel prompt pass): its token tiles, in a translation unit of their
// own to build in parallel.
#include "gemm_w4a4_int4_f8.cuh"

namespace dq {
namespace f8 {

cudaError_t run_out0(int tn, const Launch& l) {
  switch (tn) {
    case 32: return run<32, 0>(l);
    case 128: return run<128, 0>(l);
    case 256: return run<256, 0>(l);
    default: return cudaErrorInvalidValue;
  }
}
cudaError_t run_scatter(const Launch& l) { return run<256, 4>(l); }
cudaError_t init_out0() {
  cudaError_t e = cudaSuccess;
  if (e == cudaSuccess) e = allow_smem<32, 0>();
  if (e == cudaSuccess) e = allow_smem<128, 0>();
  if (e == cudaSuccess) e = allow_smem<256, 0>();
  if (e == cudaSuccess) e = allow_smem<256, 4>();
  return e;
}

}  // namespace f8
}  // namespace dq
