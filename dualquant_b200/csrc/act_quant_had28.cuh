// Many rows of 28 * P values (P = 64, 128, 256, 512): the online Hadamard with the 28 x 28 factor of the reference's table,
// in front of the int4 quantiser.  Included by act_quant_had.cuh.
#pragma once
#include "act_quant_common.cuh"
#include "wht_registers.cuh"

#include <type_traits>

namespace dq {
namespace {

// ---------------------------------------------------------------------------------------------
// the factor at compile time
// ---------------------------------------------------------------------------------------------
// Paley's second construction over GF(13), what the reference stores as a literal
// (quarot/vendor/hadamard_utils.py:277-391): [[S + I, S - I], [S - I, -S - I]], S = [[0, 1], [1, Q]] with
// Q[i][j] = (j - i | 13).
__host__ __device__ constexpr int legendre13(int a) {
  a = ((a % 13) + 13) % 13;
  for (int r = 1; r <= 6; ++r)
    if (r * r % 13 == a) return 1;
  return a == 0 ? 0 : -1;
}
__host__ __device__ constexpr int had28_entry(int i, int j) {
  const int r = i % 14, c = j % 14;
  const int s = r == c ? 0 : (r == 0 || c == 0) ? 1 : legendre13(c - r), d = r == c ? 1 : 0;
  return i < 14 ? (j < 14 ? s + d : s - d) : (j < 14 ? s - d : -s - d);
}
__host__ __device__ constexpr uint32_t had28_minus(int j) {  // rows with -1 in column j
  uint32_t m = 0;
  for (int i = 0; i < 28; ++i) m |= had28_entry(i, j) < 0 ? 1u << i : 0u;
  return m;
}
struct Had28Columns {
  uint32_t minus[28];
};
constexpr Had28Columns had28_columns() {
  Had28Columns c = {};
  for (int j = 0; j < 28; ++j) c.minus[j] = had28_minus(j);
  return c;
}
__constant__ Had28Columns c_had28 = had28_columns();

// The sums of the rows in ROWS from column J on; `acc` is their common sum of the columns before.  Rows that begin with
// the same signs share those additions: 637 packed additions per column pair instead of 784, each rounded where the
// j-ascending chain of its row rounds.
template <uint32_t ROWS, int J, typename F>
__device__ __forceinline__ void had28_sums(const float2 (&v)[28], float2 acc, F&& emit) {
  if constexpr (J == 28) {
    static_assert((ROWS & (ROWS - 1)) == 0, "the rows of the factor differ");
    constexpr int row = [] {
      int i = 0;
      while ((ROWS >> i) != 1u) ++i;
      return i;
    }();
    emit(row, acc);
  } else {
    constexpr uint32_t minus = ROWS & had28_minus(J), plus = ROWS & ~had28_minus(J);
    if constexpr (plus != 0) had28_sums<plus, J + 1>(v, __fadd2_rn(acc, v[J]), emit);
    if constexpr (minus != 0) had28_sums<minus, J + 1>(v, __ffma2_rn(v[J], make_float2(-1.0f, -1.0f), acc), emit);
  }
}

__device__ __forceinline__ float max3_abs(float m, float a, float b) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(m), "f"(fabsf(a)), "f"(fabsf(b)));
  return r;
}

constexpr int kHad28Threads = 256;

template <int P>
struct Had28 {
  static constexpr int kRows = 512 / P;          // rows per CTA: always 14336 values, 56 a thread
  static constexpr int kSegments = 28 * kRows;
  static constexpr int kPitch = P + 8;           // of a segment: the four segments of a warp sit eight banks apart
  static constexpr int kSmem = kSegments * kPitch * 4;
};

// Three CTAs of 256 threads per SM, 14336 values each in shared memory; three passes over them:
//   load     eight neighbours a thread: SiLU * up, column scale, stages 1, 2, 4, two 16-byte stores
//   segment  P / 8 values a thread, eight apart, in registers: the stages from 8 on, then the transform's scale
//   matrix   a column pair a thread, 28 pairs in registers: the sums of the factor's rows, the row's absmax
// and the codes, four neighbours a thread at a time.  Element o of a segment sits at o ^ ((o & 32) >> 3), so that the 16-byte
// accesses of eight lanes, two vectors apart in the load pass, touch every bank once.
// The factor is compiled in; a CTA compares the caller's matrix with it and takes coefficients from memory if they differ.
// EXPAND: some of the CTAs expand a weight instead (expand_w_e4m3.cuh).
template <int P, typename XT, bool EXPAND = false>
__global__ void __launch_bounds__(kHad28Threads, 3)
act_quant_had28_kernel(const XT* x, const XT* up, int64_t ldx, const float* a, int M,
                       float had_scale, const float* had_mat, int8_t* __restrict__ codes,
                       float* __restrict__ sx, float* __restrict__ out, int mode, int scale_fp16, const ExpansionShare ex) {
  using H = Had28<P>;
  constexpr int T = kHad28Threads, K = 28 * P, V = P / 8;
  extern __shared__ float sm_row[];
  __shared__ float red[T / 32];
  grid_dep_launch_dependents();
  grid_dep_wait();
  const int tid = threadIdx.x;
  const int cta = EXPAND ? quantiser_cta<T>(ex) : static_cast<int>(blockIdx.x);
  if (EXPAND && cta < 0) return;
  const int row0 = cta * H::kRows;

  bool known = true;
#pragma unroll
  for (int t = 0; t < (28 * 28 + T - 1) / T; ++t) {
    const int u = t * T + tid;
    if (u < 28 * 28) known &= had_mat[u] == (((c_had28.minus[u % 28] >> (u / 28)) & 1u) != 0 ? -1.0f : 1.0f);
  }

  // vector u = eight values; 1792 of them, seven a thread, four and three in flight
  auto swizzle = [](int o) { return o ^ ((o & 32) >> 3); };
  auto load_pass = [&](auto count, int first) {
    constexpr int N = decltype(count)::value;
    Raw8<XT> xw[N], uw[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int idx = ((first + i) * T + tid) * 8, n = H::kRows > 1 ? idx / K : 0, k = idx - n * K;
      if (H::kRows == 1 || row0 + n < M) {
        const int64_t at = static_cast<int64_t>(row0 + n) * ldx + k;
        xw[i].load(x + at);
        if (up != nullptr) uw[i].load(up + at);
      }
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int idx = ((first + i) * T + tid) * 8, n = H::kRows > 1 ? idx / K : 0, k = idx - n * K;
      if (H::kRows == 1 || row0 + n < M) {
        float v[8];
        if (up != nullptr) gated8(xw[i], uw[i], v);
        else xw[i].expand(v);
        float2 p[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) p[e] = make_float2(v[2 * e], v[2 * e + 1]);
        if (a != nullptr) {
          float av[8];
          load8(a + k, av);
#pragma unroll
          for (int e = 0; e < 4; ++e) p[e] = __fmul2_rn(p[e], make_float2(av[2 * e], av[2 * e + 1]));
        }
        wht_registers<8>(p);
        const int o = idx % P;
        float* seg = sm_row + (idx / P) * H::kPitch;
        *reinterpret_cast<float4*>(seg + swizzle(o)) = make_float4(p[0].x, p[0].y, p[1].x, p[1].y);
        *reinterpret_cast<float4*>(seg + swizzle(o + 4)) = make_float4(p[2].x, p[2].y, p[3].x, p[3].y);
      }
    }
  };
  load_pass(std::integral_constant<int, 4>(), 0);
  load_pass(std::integral_constant<int, 3>(), 4);
  known = __syncthreads_and(known) != 0;

  for (int t = tid; t < H::kSegments * 8; t += T) {
    float* p0 = sm_row + (t >> 3) * H::kPitch + (t & 7);  // values with bit 2 of their index clear, and set
    float* p1 = sm_row + (t >> 3) * H::kPitch + ((t & 7) ^ 4);
    float2 p[V / 2];
#pragma unroll
    for (int k = 0; k < V; k += 2) {
      const float* q = (k & 4) != 0 ? p1 : p0;
      p[k / 2] = make_float2(q[8 * k], q[8 * k + 8]);
    }
    wht_registers<V>(p);
#pragma unroll
    for (int k = 0; k < V; k += 2) {
      float* q = (k & 4) != 0 ? p1 : p0;
      const float2 w = __fmul2_rn(p[k / 2], make_float2(had_scale, had_scale));
      q[8 * k] = w.x;
      q[8 * k + 8] = w.y;
    }
  }
  __syncthreads();

  const int n = tid / (P / 2), lt = tid % (P / 2);  // row of the CTA, and thread of that row
  float* rowp = sm_row + n * 28 * H::kPitch;
  float amax = 0.f;
  {
    float* col = rowp + swizzle(2 * lt);
    float2 v[28];
#pragma unroll
    for (int j = 0; j < 28; ++j) v[j] = *reinterpret_cast<const float2*>(col + j * H::kPitch);
    if (known) {
      had28_sums<0xFFFFFFFu, 0>(v, make_float2(0.f, 0.f), [&](int i, float2 acc) {
        *reinterpret_cast<float2*>(col + i * H::kPitch) = acc;
        amax = max3_abs(amax, acc.x, acc.y);
      });
    } else {
      for (int i = 0; i < 28; ++i) {
        float2 acc = make_float2(0.f, 0.f);
#pragma unroll
        for (int j = 0; j < 28; ++j) {
          const float h = had_mat[i * 28 + j];
          acc = __ffma2_rn(make_float2(h, h), v[j], acc);
        }
        *reinterpret_cast<float2*>(col + i * H::kPitch) = acc;
        amax = max3_abs(amax, acc.x, acc.y);
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  if ((tid & 31) == 0) red[tid >> 5] = amax;
  __syncthreads();
  const int row = row0 + n;
  if (H::kRows > 1 && row >= M) return;
  constexpr int kWarps = P / 64;  // of a row
#pragma unroll
  for (int w = 0; w < kWarps; ++w) amax = fmaxf(amax, red[n * kWarps + w]);
  TokenQuant tq = {1.f, 1.f, false};
  if (mode != MODE_RAW) {
    tq = token_quant(amax, token_scale(amax, scale_fp16));
    if (lt == 0 && sx != nullptr) sx[row] = tq.s;
  }
  auto quad = [&](int o) {
    return *reinterpret_cast<const float4*>(rowp + (o / P) * H::kPitch + swizzle(o % P));
  };
  if (mode == MODE_CODES && (scale_fp16 & 0xFF) != 2) {
    const bool e4m3 = (scale_fp16 & kCodesE4M3) != 0;
    int8_t* crow = codes + static_cast<int64_t>(row) * K + 4 * lt;
#pragma unroll
    for (int i = 0; i < 14; i += 2) {
      const float4 f = quad(i * 2 * P + 4 * lt), g = quad((i + 1) * 2 * P + 4 * lt);
      const float v[8] = {f.x, f.y, f.z, f.w, g.x, g.y, g.z, g.w};
      const uint2 w = quant_pack8(v, tq, e4m3);
      *reinterpret_cast<uint32_t*>(crow + i * 2 * P) = w.x;
      *reinterpret_cast<uint32_t*>(crow + (i + 1) * 2 * P) = w.y;
    }
  } else {
    int8_t* crow = (codes != nullptr) ? codes + static_cast<int64_t>(row) * K : nullptr;
    float* orow = out_row_ptr(out, row, K, mode);
    for (int i = 0; i < 7; ++i) {
      const int o = i * 4 * P + 8 * lt;
      const float4 f = quad(o), g = quad(o + 4);
      const float v[8] = {f.x, f.y, f.z, f.w, g.x, g.y, g.z, g.w};
      emit8(v, tq, mode, crow, orow, o, scale_fp16);
    }
  }
}

}  // namespace
}  // namespace dq
