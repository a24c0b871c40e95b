// Walsh-Hadamard stages over values in registers.
#pragma once

namespace dq {

// Butterflies over V values in registers, stages h = 1, 2, ... V / 2 of their index; pairs of neighbours share an
// instruction from the second stage on.
template <int V>
__device__ __forceinline__ void wht_registers(float2 (&p)[V / 2]) {
#pragma unroll
  for (int k = 0; k < V / 2; ++k) p[k] = make_float2(__fadd_rn(p[k].x, p[k].y), __fsub_rn(p[k].x, p[k].y));
#pragma unroll
  for (int h = 1; h < V / 2; h <<= 1) {
#pragma unroll
    for (int k = 0; k < V / 2; ++k) {
      if ((k & h) == 0) {
        const float2 u = p[k], w = p[k + h];
        p[k] = __fadd2_rn(u, w);
        p[k + h] = __ffma2_rn(w, make_float2(-1.0f, -1.0f), u);
      }
    }
  }
}

}  // namespace dq
