// The online Hadamard with a factor of more than 32 rows (orders 36 ... 172 of the reference's table, e.g. 11008 = 172 * 64 and
// 13824 = 108 * 128) for segments of 32, 64 or 128 values, in front of the int4 quantiser.  Included by act_quant_int4.cu.
#pragma once
#include "act_quant_common.cuh"
#include "wht_registers.cuh"

#include <type_traits>

namespace dq {

constexpr int kBigWarps = 12, kBigThreads = kBigWarps * 32, kBigCols = 128;

// RPW: output rows of the factor per warp.
__host__ __device__ constexpr int big_pitch(int rpw) { return kBigWarps * ((rpw + 3) / 4 * 4); }  // of a row of coefficients, floats
__host__ __device__ constexpr int big_smem(int had_k, int rpw) { return had_k * (kBigCols + big_pitch(rpw)) * 4; }

// A CTA holds 128 columns of the matrix stage - one, two or four token rows - as [segment][column] in shared memory, and the
// coefficients of its output rows as [segment][row]; it walks over groups of token rows.  Per segment j a lane reads its four
// columns (one 16-byte load, conflict-free) and the warp's RPW coefficients (broadcasts) for 2 RPW packed FMAs, j ascending as
// in act_quant_had_big_kernel, which read two values from shared memory for every addition.  With few token rows a cluster of
// `split` CTAs shares a group: each transforms all segments and sums its own output rows; the rows' maxima are exchanged.
// Bound at many rows by the FP32 pipe (172 additions a value: 120 us for 2048 rows of 11008) and the phases around it, which
// one CTA per SM does not overlap.  Against that kernel, us: 11008 gated, 1 row 77 -> 16, 66 rows 79 -> 20, 300 237 -> 75, 2048
// 1108 -> 248; 13824, 8 rows 68 -> 12.5, 2048 954 -> 226; 5120 = 40 * 128, 2048 rows 195 -> 74.
template <int RPW, typename XT>
__global__ void __launch_bounds__(kBigThreads, 1)
act_quant_had_wide_kernel(const XT* x, const XT* up, int64_t ldx, const float* a, int M,
                          int K, int had_k, float had_scale, const float* had_mat, int split,
                          int8_t* __restrict__ codes, float* __restrict__ sx, float* __restrict__ out, int mode,
                          int scale_fp16) {
  constexpr int RP = (RPW + 3) / 4 * 4, kPitch = big_pitch(RPW);
  extern __shared__ float sm[];
  __shared__ float red[4][kBigWarps], pmax[8][4];
  float* vals = sm;                       // [had_k][128]
  float* coef = sm + had_k * kBigCols;    // [had_k][12][RP]
  if (split > 1) cluster_arrive();
  grid_dep_launch_dependents();
  grid_dep_wait();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = split > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  const int P = K / had_k, T = kBigCols / P;  // segment length, token rows per group
  const int first_row = rank * kBigWarps * RPW;
  // (rows fastest: neighbouring threads write neighbouring coefficients)
  for (int u = tid; u < had_k * kBigWarps * RP; u += kBigThreads) {
    const int j = u / (kBigWarps * RP), at = u - j * (kBigWarps * RP), w = at / RP, r = at - w * RP;
    const int i = first_row + w * RPW + r;
    coef[u] = (r < RPW && i < had_k) ? had_mat[i * had_k + j] : 0.f;
  }
  if (split > 1) cluster_wait();  // the peers have started: their shared memory may be written (the rows' maxima)
  const int groups = (M + T - 1) / T;
  for (int grp = blockIdx.x / split; grp < groups; grp += gridDim.x / split) {
    const int row0 = grp * T;
    constexpr int kAhead = 4;  // vectors of eight in flight per thread
    const int vectors = had_k * kBigCols / 8;
    for (int u0 = tid; u0 < vectors; u0 += kAhead * kBigThreads) {
      Raw8<XT> xw[kAhead], uw[kAhead];
#pragma unroll
      for (int n = 0; n < kAhead; ++n) {
        const int idx = (u0 + n * kBigThreads) * 8, t = idx / K, k = idx - t * K;
        if (idx < vectors * 8 && row0 + t < M) {
          const int64_t at = static_cast<int64_t>(row0 + t) * ldx + k;
          xw[n].load(x + at);
          if (up != nullptr) uw[n].load(up + at);
        }
      }
#pragma unroll
      for (int n = 0; n < kAhead; ++n) {
        const int idx = (u0 + n * kBigThreads) * 8, t = idx / K, k = idx - t * K;
        if (idx >= vectors * 8) break;
        float2 p[4] = {};
        if (row0 + t < M) {
          float v[8];
          if (up != nullptr) gated8(xw[n], uw[n], v);
          else xw[n].expand(v);
#pragma unroll
          for (int e = 0; e < 4; ++e) p[e] = make_float2(v[2 * e], v[2 * e + 1]);
          if (a != nullptr) {
            float av[8];
            load8(a + k, av);
#pragma unroll
            for (int e = 0; e < 4; ++e) p[e] = __fmul2_rn(p[e], make_float2(av[2 * e], av[2 * e + 1]));
          }
          wht_registers<8>(p);
        }
        float* dst = vals + (k / P) * kBigCols + t * P + k % P;
        *reinterpret_cast<float4*>(dst) = make_float4(p[0].x, p[0].y, p[1].x, p[1].y);
        *reinterpret_cast<float4*>(dst + 4) = make_float4(p[2].x, p[2].y, p[3].x, p[3].y);
      }
    }
    __syncthreads();
    auto segments = [&](auto values) {  // the stages from 8 on of every segment, then the transform's scale
      constexpr int V = decltype(values)::value;
      for (int t = tid; t < had_k * kBigCols / V; t += kBigThreads) {
        float* q = vals + (t >> 3) * (8 * V) + (t & 7);
        float2 p[V / 2];
#pragma unroll
        for (int k = 0; k < V; k += 2) p[k / 2] = make_float2(q[8 * k], q[8 * k + 8]);
        wht_registers<V>(p);
#pragma unroll
        for (int k = 0; k < V; k += 2) {
          const float2 w = __fmul2_rn(p[k / 2], make_float2(had_scale, had_scale));
          q[8 * k] = w.x;
          q[8 * k + 8] = w.y;
        }
      }
    };
    if (P == 32) segments(std::integral_constant<int, 4>());
    else if (P == 64) segments(std::integral_constant<int, 8>());
    else segments(std::integral_constant<int, 16>());
    __syncthreads();

    float2 acc[RPW][2];
#pragma unroll
    for (int r = 0; r < RPW; ++r) acc[r][0] = acc[r][1] = make_float2(0.f, 0.f);
    const float* vp = vals + 4 * lane;
    const float* cp = coef + warp * RP;
#pragma unroll 2
    for (int j = 0; j < had_k; ++j) {
      const float4 v = *reinterpret_cast<const float4*>(vp + j * kBigCols);
#pragma unroll
      for (int r4 = 0; r4 < RP; r4 += 4) {
        const float4 h4 = *reinterpret_cast<const float4*>(cp + j * kPitch + r4);
        const float h[4] = {h4.x, h4.y, h4.z, h4.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (r4 + e < RPW) {
            acc[r4 + e][0] = __ffma2_rn(make_float2(h[e], h[e]), make_float2(v.x, v.y), acc[r4 + e][0]);
            acc[r4 + e][1] = __ffma2_rn(make_float2(h[e], h[e]), make_float2(v.z, v.w), acc[r4 + e][1]);
          }
        }
      }
    }
    float amax = 0.f;  // of this lane's token row; rows past the factor's are zero
#pragma unroll
    for (int r = 0; r < RPW; ++r)
      amax = fmaxf(amax, fmaxf(fmaxf(fabsf(acc[r][0].x), fabsf(acc[r][0].y)), fmaxf(fabsf(acc[r][1].x), fabsf(acc[r][1].y))));
    for (int o = P / 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if (lane % (P / 4) == 0) red[4 * lane / P][warp] = amax;
    __syncthreads();  // every warp has read its inputs
#pragma unroll
    for (int r = 0; r < RPW; ++r) {
      const int i = first_row + warp * RPW + r;
      if (i < had_k)
        *reinterpret_cast<float4*>(vals + i * kBigCols + 4 * lane) =
            make_float4(acc[r][0].x, acc[r][0].y, acc[r][1].x, acc[r][1].y);
    }
    if (tid < T) {
      float m = red[tid][0];
#pragma unroll
      for (int w = 1; w < kBigWarps; ++w) m = fmaxf(m, red[tid][w]);
      if (split == 1) pmax[0][tid] = m;
      else
        for (int p = 0; p < split; ++p) dsmem_store_f32(dsmem_map(smem_u32(&pmax[rank][tid]), static_cast<uint32_t>(p)), m);
    }
    if (split == 1) __syncthreads();
    else cluster_sync_all();
    // (kBigThreads is a multiple of the 16 vectors of a row of values: a thread stays in its columns)
    const int own = min(had_k - first_row, kBigWarps * RPW);  // output rows of this CTA (none for the last CTAs of a small factor)
    const int c = tid % (kBigCols / 8) * 8, t = c / P;
    if (row0 + t < M) {
      TokenQuant tq = {1.f, 1.f, false};
      if (mode != MODE_RAW) {
        float m = pmax[0][t];
        for (int p = 1; p < split; ++p) m = fmaxf(m, pmax[p][t]);
        tq = token_quant(m, token_scale(m, scale_fp16));
        if (rank == 0 && tid < kBigCols / 8 && c % P == 0 && sx != nullptr) sx[row0 + t] = tq.s;
      }
      int8_t* crow = codes != nullptr ? codes + static_cast<int64_t>(row0 + t) * K : nullptr;
      float* orow = out_row_ptr(out, row0 + t, K, mode);
#pragma unroll 2
      for (int i = tid / (kBigCols / 8); i < own; i += kBigThreads / (kBigCols / 8)) {
        const float* src = vals + (first_row + i) * kBigCols + c;
        const float4 f = *reinterpret_cast<const float4*>(src), g = *reinterpret_cast<const float4*>(src + 4);
        const float v[8] = {f.x, f.y, f.z, f.w, g.x, g.y, g.z, g.w};
        emit8(v, tq, mode, crow, orow, (first_row + i) * P + c % P, scale_fp16);
      }
    }
    // the next group overwrites the values, and its maxima the peers'
    if (split == 1) __syncthreads();
    else cluster_sync_all();
  }
}

template <typename XT, typename F>
static cudaError_t for_each_wide(F&& f) {
  cudaError_t e = f(act_quant_had_wide_kernel<2, XT>);
  if (e == cudaSuccess) e = f(act_quant_had_wide_kernel<4, XT>);
  if (e == cudaSuccess) e = f(act_quant_had_wide_kernel<5, XT>);
  if (e == cudaSuccess) e = f(act_quant_had_wide_kernel<8, XT>);
  if (e == cudaSuccess) e = f(act_quant_had_wide_kernel<9, XT>);
  if (e == cudaSuccess) e = f(act_quant_had_wide_kernel<13, XT>);
  if (e == cudaSuccess) e = f(act_quant_had_wide_kernel<15, XT>);
  return e;
}

static bool had_wide_covers(int had_k, int K) {
  const int P = K / had_k;
  return had_k > 32 && had_k <= 15 * kBigWarps && (P == 32 || P == 64 || P == 128);
}

// A group's output rows on one CTA where the groups fill the chip, else on clusters of two, four or eight.
template <typename XT>
static int launch_had_wide(const XT* x, const XT* up, int64_t ldx, const float* a, int M, int K, int had_k, float had_scale,
                           const float* had_mat, int8_t* codes, float* sx, float* out, int mode, int scale_fp16,
                           cudaStream_t stream) {
  const DeviceState* st = current_state();
  if (st == nullptr) return DQ_ERR_NOT_INIT;
  const int T = kBigCols / (K / had_k), groups = (M + T - 1) / T;
  // places for clusters of 8 and 4 CTAs of one CTA per SM: 15 and 33 on 148 SMs (a cluster stays inside one GPC)
  int split = 1;
  if (groups <= 15 * st->sm_count / 148) split = 8;
  else if (groups <= 33 * st->sm_count / 148) split = 4;
  else if (groups <= st->sm_count / 2) split = 2;
  const int need = (had_k + kBigWarps * split - 1) / (kBigWarps * split);  // rows per warp
  const int rpw = need <= 2 ? 2 : need <= 4 ? 4 : need <= 5 ? 5 : need <= 8 ? 8 : need <= 9 ? 9 : need <= 13 ? 13 : 15;
  int clusters = st->sm_count / split;
  if (clusters > groups) clusters = groups;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(clusters * split));
  cfg.blockDim = dim3(kBigThreads);
  cfg.dynamicSmemBytes = static_cast<size_t>(big_smem(had_k, rpw));
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = split;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  auto kernel = rpw == 2   ? act_quant_had_wide_kernel<2, XT>
                : rpw == 4 ? act_quant_had_wide_kernel<4, XT>
                : rpw == 5 ? act_quant_had_wide_kernel<5, XT>
                : rpw == 8 ? act_quant_had_wide_kernel<8, XT>
                : rpw == 9 ? act_quant_had_wide_kernel<9, XT>
                : rpw == 13 ? act_quant_had_wide_kernel<13, XT>
                            : act_quant_had_wide_kernel<15, XT>;
  DQ_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kernel, x, up, ldx, a, M, K, had_k, had_scale, had_mat, split, codes, sx, out, mode,
                                   scale_fp16));
  return DQ_OK;
}

}  // namespace dq
