// DualQuant's offline scale search and block quantisation of a whole weight (see bcd.py for the method and
// its reference lines): all column blocks at once, one pass over the matrix per iteration.
//
// A block is bs columns of all rows; alpha[row, block] scales rows, beta[column] scales columns.  An iteration
// is a least-squares row step followed by a least-squares column step.  The row step of a row needs only that
// row's bs values, and the column step of the same row needs only its new alpha, so both happen while the row
// sits in registers: a warp owns a row of a block (bs / 32 columns per lane), forms the two row sums with
// shuffles, computes alpha, and adds the row to its column sums.  What crosses rows - numerator and
// denominator of every beta - goes through a small buffer of partial sums, one slot per row chunk, that the next
// pass adds up in chunk order.  Written as tensor expressions the same search was ~200 element-wise and
// reduction launches, each reading and writing the matrix: 3.8 ms for 4096 x 4096 with five iterations; bound
// here by instruction issue and latency (60 % of issue slots): 0.19 ms including the packing, of which about 25 us
// are one iteration.  Half as many row chunks ran alike.
//
// Passes: column statistic (beta's first value), num_iter iterations (the first also sets alpha's first value),
// and the block quantisation.  The chunking depends on the number of rows alone, so a block searched on its own
// gives the same bits as the same block inside a wider matrix.
#include "dq_common.h"
#include "dq_ptx.cuh"

namespace dq {
namespace bcd {

constexpr int kThreads = 256, kWarps = kThreads / 32;
constexpr int kRowsAtOnce = 4;  // rows a warp works on together: their reductions share shuffles and divisions
constexpr int kMaxChunks = 32;
constexpr float kEps = 1e-12f;

enum { COL_L1 = 0, COL_L2 = 1, COL_ONE = 2, COL_MAX = 3 };
enum { ROW_MAX = 0, ROW_ONE = 1 };
enum { FMT_NONE = 0, FMT_E8M0 = 1, FMT_E4M3 = 2 };
enum { OPT_BOTH = 0, OPT_COLUMN = 1, OPT_ROW = 2 };

struct Params {
  const float* w;  // [R, C]
  int R, C, blocks, chunks, rows_per_chunk;
  int option, row_init, col_init, scale_format;
  float qmin, qmax;
  float* alpha;     // [R, blocks]
  float* beta;      // [C]
  float* partials;  // two buffers of [chunks][2][C]: (numerator, denominator) or (statistic, -)
};

// minimum / maximum that pass a NaN on, as torch's clamp and amax do
__device__ __forceinline__ float max_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float min_nan(float a, float b) {
  float r;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
// clamp(rint(v), qmin, qmax): the bounds are integers, so clamping first gives the same value, and adding and
// subtracting 1.5 * 2^23 then rounds half to even
__device__ __forceinline__ float code_of(float v, float qmin, float qmax) {
  const float c = min_nan(max_nan(v, qmin), qmax);
  return __fsub_rn(__fadd_rn(c, 12582912.0f), 12582912.0f);
}

// The same for a lane's VPL columns of a row, two at a time where they come in pairs: m = code(a * w * beta) * f, with
// num += w * m and den += m * m.  Packed fp32 instructions round each half like the scalar ones.
template <int VPL>
__device__ __forceinline__ void row_sums(const float* w, const float* beta, float a, const float* f, float f_all,
                                         float qmin, float qmax, float* num, float* den) {
  if constexpr (VPL % 2 == 0) {
    const float2 a2 = make_float2(a, a), magic = make_float2(12582912.0f, 12582912.0f),
                 back = make_float2(-12582912.0f, -12582912.0f);
#pragma unroll
    for (int i = 0; i < VPL; i += 2) {
      const float2 w2 = make_float2(w[i], w[i + 1]);
      float2 v = __fmul2_rn(__fmul2_rn(a2, w2), make_float2(beta[i], beta[i + 1]));
      v.x = min_nan(max_nan(v.x, qmin), qmax);
      v.y = min_nan(max_nan(v.y, qmin), qmax);
      v = __fadd2_rn(__fadd2_rn(v, magic), back);
      v = __fmul2_rn(v, f != nullptr ? make_float2(f[i], f[i + 1]) : make_float2(f_all, f_all));
      const float2 n2 = __ffma2_rn(w2, v, make_float2(num[i], num[i + 1]));
      const float2 d2 = __ffma2_rn(v, v, make_float2(den[i], den[i + 1]));
      num[i] = n2.x; num[i + 1] = n2.y;
      den[i] = d2.x; den[i + 1] = d2.y;
    }
  } else {
    const float m = __fmul_rn(code_of(__fmul_rn(__fmul_rn(a, w[0]), beta[0]), qmin, qmax), f != nullptr ? f[0] : f_all);
    num[0] = fmaf(w[0], m, num[0]);
    den[0] = fmaf(m, m, den[0]);
  }
}

// row scale 1 / alpha in its storage format
__device__ __forceinline__ float store_format(float s, int fmt) {
  if (fmt == FMT_E4M3) {
    const float c = min_nan(max_nan(s, 0.015625f), 448.0f);
    unsigned short q;
    uint32_t h2;
    asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(q) : "f"(0.f), "f"(c));
    asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h2) : "h"(q));
    float f;
    asm("{\n.reg .b16 lo, hi;\nmov.b32 {lo, hi}, %1;\ncvt.f32.f16 %0, lo;\n}" : "=f"(f) : "r"(h2));
    return f;
  }
  if (fmt == FMT_E8M0) {  // nearest power of two by the leading mantissa bit; NaN becomes the biased exponent 255
    const uint32_t bits = __float_as_uint(s);
    const uint32_t e = ((bits >> 23) & 0xFFu) + ((bits >> 22) & 1u);
    const float p = (s != s) ? __uint_as_float(255u << 23) : __uint_as_float((e < 255u ? e : 255u) << 23);
    return fmaxf(p, 5.877471754111438e-39f);  // 2^-127
  }
  return s;
}

template <int VPL>
__device__ __forceinline__ void load_cols(const float* p, float* v) {
  if constexpr (VPL % 4 == 0) {
#pragma unroll
    for (int i = 0; i < VPL; i += 4) {
      const float4 t = *reinterpret_cast<const float4*>(p + i);
      v[i] = t.x; v[i + 1] = t.y; v[i + 2] = t.z; v[i + 3] = t.w;
    }
  } else if constexpr (VPL == 2) {
    const float2 t = *reinterpret_cast<const float2*>(p);
    v[0] = t.x; v[1] = t.y;
  } else {
    v[0] = *p;
  }
}

// The sum (or maximum) of N values in pairs: its rounding error grows with log N.  Added in order, the partial sums of a
// column left its scale further from the 64-bit one than a tensor reduction does (median of 4096 rows, one iteration: in
// order 9.2e-8, in pairs 4.6e-8, tensor expressions 5.2e-8); the time is the same.
template <int N>
__device__ __forceinline__ float pairwise(float* v, bool is_max) {
#pragma unroll
  for (int step = N / 2; step > 0; step /= 2)
#pragma unroll
    for (int k = 0; k < step; ++k) v[k] = is_max ? max_nan(v[k], v[k + step]) : v[k] + v[k + step];
  return v[0];
}

// Adds the warps' column sums (num, den; VPL columns per lane) and writes them to this chunk's slot.
template <int VPL>
__device__ __forceinline__ void write_partials(float* sm, const float* num, const float* den, bool is_max, float* slot,
                                               int C, int c0) {
  constexpr int BS = 32 * VPL;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    sm[(warp * 2) * BS + lane * VPL + i] = num[i];
    sm[(warp * 2 + 1) * BS + lane * VPL + i] = den[i];
  }
  __syncthreads();
  for (int t = threadIdx.x; t < 2 * BS; t += kThreads) {
    float s[kWarps];
#pragma unroll
    for (int w = 0; w < kWarps; ++w) s[w] = sm[w * 2 * BS + t];
    slot[static_cast<size_t>(t / BS) * C + c0 + t % BS] = pairwise<kWarps>(s, is_max);
  }
}

// The block's column scales from the previous pass's partial sums: beta and beta_inv into shared memory.
// `first`: the partial sums are the column statistic, beta = 1 / max(stat, 1e-8); otherwise
// beta_inv = numerator / (denominator + eps).  One thread per sum, all its loads in flight.
template <int VPL>
__device__ __forceinline__ void read_beta(const Params& p, const float* partials, int c0, bool first, float* s_beta,
                                          float* s_inv) {
  constexpr int BS = 32 * VPL;
  const bool none = p.option == OPT_ROW || (first && p.col_init == COL_ONE);
  const bool is_max = first && p.col_init == COL_MAX;
  if (!none) {
    for (int t = threadIdx.x; t < 2 * BS; t += kThreads) {
      const float* src = partials + static_cast<size_t>(t / BS) * p.C + c0 + t % BS;
      float v[kMaxChunks];
#pragma unroll
      for (int k = 0; k < kMaxChunks; ++k) v[k] = k < p.chunks ? src[static_cast<size_t>(2 * k) * p.C] : 0.f;
      (t < BS ? s_beta : s_inv)[t % BS] = pairwise<kMaxChunks>(v, is_max);
    }
    __syncthreads();
  }
  for (int c = threadIdx.x; c < BS; c += kThreads) {
    float b = 1.f, inv = 1.f;
    if (!none && first) {
      b = 1.0f / max_nan(p.col_init == COL_L2 ? sqrtf(s_beta[c]) : s_beta[c], 1e-8f);
      inv = 1.0f / b;
    } else if (!none) {
      inv = s_beta[c] / (s_inv[c] + kEps);
      b = 1.0f / inv;
    }
    s_beta[c] = b;
    s_inv[c] = inv;
  }
  __syncthreads();
}

// The statistic behind beta's first value: sum |w|, sum w^2 or max |w| over the rows of a column.
template <int VPL>
__global__ void __launch_bounds__(kThreads) column_stat_kernel(const Params p) {
  constexpr int BS = 32 * VPL;
  extern __shared__ float sm[];
  // (every kernel here waits before it lets the next one start, so the next one may read w before its own wait)
  grid_dep_wait();
  grid_dep_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c0 = blockIdx.x * BS;
  const int r_end = min(p.R, (static_cast<int>(blockIdx.y) + 1) * p.rows_per_chunk);
  float acc[VPL], none[VPL];
#pragma unroll
  for (int i = 0; i < VPL; ++i) acc[i] = none[i] = 0.f;
#pragma unroll 8
  for (int r = blockIdx.y * p.rows_per_chunk + warp; r < r_end; r += kWarps) {
    float v[VPL];
    load_cols<VPL>(p.w + static_cast<size_t>(r) * p.C + c0 + lane * VPL, v);
#pragma unroll
    for (int i = 0; i < VPL; ++i) {
      if (p.col_init == COL_L1) acc[i] += fabsf(v[i]);
      else if (p.col_init == COL_L2) acc[i] = fmaf(v[i], v[i], acc[i]);
      else acc[i] = max_nan(acc[i], fabsf(v[i]));
    }
  }
  write_partials<VPL>(sm, acc, none, p.col_init == COL_MAX, p.partials + static_cast<size_t>(blockIdx.y) * 2 * p.C, p.C,
                      c0);
}

// The sums of n[j] and d[j] (j < 4 rows) over the warp: lane L ends up with both sums of row
// 2 * (L >> 4) + ((L >> 3) & 1).  Ten shuffles in place of forty.
__device__ __forceinline__ void reduce_rows(const float* n, const float* d, int lane, float& nr, float& dr) {
  const bool h16 = (lane & 16) != 0, h8 = (lane & 8) != 0, h4 = (lane & 4) != 0;
  float n0 = h16 ? n[2] : n[0], n1 = h16 ? n[3] : n[1], d0 = h16 ? d[2] : d[0], d1 = h16 ? d[3] : d[1];
  n0 += __shfl_xor_sync(0xffffffffu, h16 ? n[0] : n[2], 16);
  n1 += __shfl_xor_sync(0xffffffffu, h16 ? n[1] : n[3], 16);
  d0 += __shfl_xor_sync(0xffffffffu, h16 ? d[0] : d[2], 16);
  d1 += __shfl_xor_sync(0xffffffffu, h16 ? d[1] : d[3], 16);
  float nn = h8 ? n1 : n0, dd = h8 ? d1 : d0;
  nn += __shfl_xor_sync(0xffffffffu, h8 ? n0 : n1, 8);
  dd += __shfl_xor_sync(0xffffffffu, h8 ? d0 : d1, 8);
  float v = h4 ? dd : nn;
  v += __shfl_xor_sync(0xffffffffu, h4 ? nn : dd, 4);
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  const float other = __shfl_xor_sync(0xffffffffu, v, 4);
  nr = h4 ? other : v;
  dr = h4 ? v : other;
}
// max of m[j] (j < 4 rows) over the warp, for the same row-to-lane assignment
__device__ __forceinline__ float reduce_rows_max(const float* m, int lane) {
  const bool h16 = (lane & 16) != 0, h8 = (lane & 8) != 0;
  float m0 = h16 ? m[2] : m[0], m1 = h16 ? m[3] : m[1];
  m0 = max_nan(m0, __shfl_xor_sync(0xffffffffu, h16 ? m[0] : m[2], 16));
  m1 = max_nan(m1, __shfl_xor_sync(0xffffffffu, h16 ? m[1] : m[3], 16));
  float v = h8 ? m1 : m0;
  v = max_nan(v, __shfl_xor_sync(0xffffffffu, h8 ? m0 : m1, 8));
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) v = max_nan(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float from_row(float v, int j) {  // the value that row j's lanes hold
  return __shfl_sync(0xffffffffu, v, (j >> 1) * 16 + (j & 1) * 8);
}

// One iteration: row step (unless only columns are scaled), then the column step's sums (unless only rows are).
// FIRST also forms alpha's first value.
template <int VPL, bool FIRST>
__global__ void __launch_bounds__(kThreads, VPL <= 4 ? 4 : 2) iteration_kernel(const Params p, const float* partials_in,
                                                             float* partials_out) {
  constexpr int BS = 32 * VPL;
  extern __shared__ float sm[];
  __shared__ float s_beta[BS], s_inv[BS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c0 = blockIdx.x * BS;
  const int r_end = min(p.R, (static_cast<int>(blockIdx.y) + 1) * p.rows_per_chunk);
  const int r_first = blockIdx.y * p.rows_per_chunk + warp * kRowsAtOnce;
  auto load_rows = [&](int r0, float (*w)[VPL]) {  // past the end: the last row again, left out of the sums below
    const float* src = p.w + static_cast<size_t>(r0) * p.C + c0 + lane * VPL;
    if (r0 + kRowsAtOnce <= r_end) {
#pragma unroll
      for (int j = 0; j < kRowsAtOnce; ++j, src += p.C) load_cols<VPL>(src, w[j]);
    } else {
#pragma unroll
      for (int j = 0; j < kRowsAtOnce; ++j)
        load_cols<VPL>(p.w + static_cast<size_t>(min(r0 + j, r_end - 1)) * p.C + c0 + lane * VPL, w[j]);
    }
  };
  float w[kRowsAtOnce][VPL], ahead[kRowsAtOnce][VPL];
  if (FIRST) grid_dep_wait();  // no kernel of this file may have run before this one
  load_rows(r_first, ahead);
  if (!FIRST) grid_dep_wait();
  grid_dep_launch_dependents();
  read_beta<VPL>(p, partials_in, c0, FIRST, s_beta, s_inv);
  float beta[VPL], beta_inv[VPL], num[VPL], den[VPL];
#pragma unroll
  for (int i = 0; i < VPL; ++i) {
    beta[i] = s_beta[lane * VPL + i];
    beta_inv[i] = s_inv[lane * VPL + i];
    num[i] = den[i] = 0.f;
  }
  const int my_row = 2 * (lane >> 4) + ((lane >> 3) & 1);  // of four: the one whose scale this lane computes
  const float qmin = p.qmin, qmax = p.qmax;
  for (int r0 = r_first; r0 < r_end; r0 += kWarps * kRowsAtOnce) {
#pragma unroll
    for (int j = 0; j < kRowsAtOnce; ++j)
#pragma unroll
      for (int i = 0; i < VPL; ++i) w[j][i] = ahead[j][i];
    if (r0 + kWarps * kRowsAtOnce < r_end) load_rows(r0 + kWarps * kRowsAtOnce, ahead);
    const int row_l = min(r0 + my_row, r_end - 1);
    float a_l = 1.f, a_inv_l = 1.f;
    if (p.option != OPT_COLUMN) {
      float* alpha = p.alpha + static_cast<size_t>(row_l) * p.blocks + blockIdx.x;
      if (FIRST) {
        if (p.row_init == ROW_MAX) {
          float m[kRowsAtOnce];
#pragma unroll
          for (int j = 0; j < kRowsAtOnce; ++j) {
            m[j] = 0.f;
#pragma unroll
            for (int i = 0; i < VPL; ++i) m[j] = max_nan(m[j], fabsf(__fmul_rn(w[j][i], beta[i])));
          }
          a_l = 1.0f / (reduce_rows_max(m, lane) / qmax);
        }
      } else {
        a_l = *alpha;
      }
      float n[kRowsAtOnce], d[kRowsAtOnce];
#pragma unroll
      for (int j = 0; j < kRowsAtOnce; ++j) {
        const float a = from_row(a_l, j);
        float nv[VPL], dv[VPL];
#pragma unroll
        for (int i = 0; i < VPL; ++i) nv[i] = dv[i] = 0.f;
        row_sums<VPL>(w[j], beta, a, beta_inv, 0.f, qmin, qmax, nv, dv);
        n[j] = d[j] = 0.f;
#pragma unroll
        for (int i = 0; i < VPL; ++i) {
          n[j] += nv[i];
          d[j] += dv[i];
        }
      }
      float nr, dr;
      reduce_rows(n, d, lane, nr, dr);
      a_inv_l = store_format(nr / (dr + kEps), p.scale_format);
      a_l = 1.0f / a_inv_l;
      if ((lane & 7) == 0 && r0 + my_row < r_end) *alpha = a_l;
    }
    if (p.option != OPT_ROW) {
#pragma unroll
      for (int j = 0; j < kRowsAtOnce; ++j) {
        const float a = from_row(a_l, j), a_inv = from_row(a_inv_l, j);
        if (r0 + j < r_end) row_sums<VPL>(w[j], beta, a, nullptr, a_inv, qmin, qmax, num, den);
      }
    }
  }
  if (p.option != OPT_ROW)
    write_partials<VPL>(sm, num, den, false, partials_out + static_cast<size_t>(blockIdx.y) * 2 * p.C, p.C, c0);
}

// beta from the last iteration's sums and, with mat_q, the stored weight: (1 / alpha) * RTN(alpha * w * beta), one
// RTN scale per row of a block; column_scales = 1 / beta.
template <int VPL>
__global__ void __launch_bounds__(kThreads) finish_kernel(const Params p, const float* partials_in, float* mat_q,
                                                          float* column_scales) {
  constexpr int BS = 32 * VPL;
  __shared__ float s_beta[BS], s_inv[BS];
  grid_dep_wait();
  grid_dep_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c0 = blockIdx.x * BS;
  read_beta<VPL>(p, partials_in, c0, false, s_beta, s_inv);
  if (blockIdx.y == 0) {
    for (int c = threadIdx.x; c < BS; c += kThreads) {
      p.beta[c0 + c] = s_beta[c];
      if (column_scales != nullptr) column_scales[c0 + c] = 1.0f / s_beta[c];
    }
  }
  if (p.option == OPT_COLUMN) {  // alpha is part of the result: ones
    for (int r = blockIdx.y * p.rows_per_chunk + threadIdx.x;
         r < min(p.R, (static_cast<int>(blockIdx.y) + 1) * p.rows_per_chunk); r += kThreads)
      p.alpha[static_cast<size_t>(r) * p.blocks + blockIdx.x] = 1.f;
  }
  if (mat_q == nullptr) return;
  float beta[VPL];
#pragma unroll
  for (int i = 0; i < VPL; ++i) beta[i] = s_beta[lane * VPL + i];
  const int my_row = 2 * (lane >> 4) + ((lane >> 3) & 1);
  const int r_end = min(p.R, (static_cast<int>(blockIdx.y) + 1) * p.rows_per_chunk);
  for (int r0 = blockIdx.y * p.rows_per_chunk + warp * kRowsAtOnce; r0 < r_end; r0 += kWarps * kRowsAtOnce) {
    float w[kRowsAtOnce][VPL], m[kRowsAtOnce];
    const int row_l = min(r0 + my_row, r_end - 1);
    const float a_l = p.option != OPT_COLUMN ? p.alpha[static_cast<size_t>(row_l) * p.blocks + blockIdx.x] : 1.f;
#pragma unroll
    for (int j = 0; j < kRowsAtOnce; ++j) {
      const int r = min(r0 + j, r_end - 1);
      load_cols<VPL>(p.w + static_cast<size_t>(r) * p.C + c0 + lane * VPL, w[j]);
      const float a = from_row(a_l, j);
      m[j] = 0.f;
#pragma unroll
      for (int i = 0; i < VPL; ++i) {
        w[j][i] = __fmul_rn(__fmul_rn(a, w[j][i]), beta[i]);
        m[j] = max_nan(m[j], fabsf(w[j][i]));
      }
    }
    const float s_l = max_nan(reduce_rows_max(m, lane), 1e-8f) / p.qmax;
    const float back_l = p.option != OPT_COLUMN ? store_format(1.0f / a_l, p.scale_format) : 1.f;
#pragma unroll
    for (int j = 0; j < kRowsAtOnce; ++j) {
      const float s = from_row(s_l, j), back = from_row(back_l, j);
      if (r0 + j < r_end) {
        float o[VPL];
#pragma unroll
        for (int i = 0; i < VPL; ++i)
          o[i] = __fmul_rn(back, __fmul_rn(code_of(__fdiv_rn(w[j][i], s), p.qmin, p.qmax), s));
        float* dst = mat_q + static_cast<size_t>(r0 + j) * p.C + c0 + lane * VPL;
        if constexpr (VPL % 4 == 0) {
#pragma unroll
          for (int i = 0; i < VPL; i += 4) *reinterpret_cast<float4*>(dst + i) = make_float4(o[i], o[i + 1], o[i + 2], o[i + 3]);
        } else {
#pragma unroll
          for (int i = 0; i < VPL; ++i) dst[i] = o[i];
        }
      }
    }
  }
}

template <int VPL>
static int search(Params p, int iters, float* mat_q, float* column_scales, cudaStream_t s) {
  const dim3 grid(static_cast<unsigned>(p.blocks), static_cast<unsigned>(p.chunks)), block(kThreads);
  const size_t smem = static_cast<size_t>(kWarps) * 2 * 32 * VPL * sizeof(float);
  float* buf[2] = {p.partials, p.partials + static_cast<size_t>(p.chunks) * 2 * p.C};
  if (p.option != OPT_ROW && p.col_init != COL_ONE) DQ_CHECK_CUDA(launch_pdl(column_stat_kernel<VPL>, grid, block, smem, s, p));
  for (int i = 0; i < iters; ++i) {
    if (i == 0)
      DQ_CHECK_CUDA(launch_pdl(iteration_kernel<VPL, true>, grid, block, smem, s, p, buf[0], buf[1]));
    else
      DQ_CHECK_CUDA(launch_pdl(iteration_kernel<VPL, false>, grid, block, smem, s, p, buf[i & 1], buf[(i + 1) & 1]));
  }
  DQ_CHECK_CUDA(launch_pdl(finish_kernel<VPL>, grid, block, 0, s, p, buf[iters & 1], mat_q, column_scales));
  return DQ_OK;
}

// Row chunks: enough CTAs for a few blocks of columns to fill the chip, few enough that adding up the partial sums
// stays small beside reading the rows; whole groups of the rows a CTA works on at once.
static int chunk_rows(int R) {
  const int unit = kWarps * kRowsAtOnce;
  return ((R + kMaxChunks - 1) / kMaxChunks + unit - 1) / unit * unit;
}

}  // namespace bcd
}  // namespace dq

using namespace dq;

extern "C" size_t dq_dualquant_workspace_bytes(int R, int C) {
  if (R < 1 || C < 1) return 0;
  const int rows = bcd::chunk_rows(R);
  return static_cast<size_t>((R + rows - 1) / rows) * 4 * C * sizeof(float);
}

extern "C" int dq_dualquant_search(const float* w, int R, int C, int block_size, int num_iter, int scale_option,
                                   int row_init, int col_init, int scale_format, float qmin, float qmax, float* alpha,
                                   float* beta, float* mat_q, float* column_scales, void* workspace,
                                   size_t workspace_bytes, void* stream) {
  if (current_state() == nullptr) return DQ_ERR_NOT_INIT;
  DQ_REQUIRE(w != nullptr && alpha != nullptr && beta != nullptr && workspace != nullptr, DQ_ERR_NULL,
             "null w / alpha / beta / workspace");
  DQ_REQUIRE(block_size == 32 || block_size == 64 || block_size == 128 || block_size == 256, DQ_ERR_UNSUPPORTED,
             "block size %d has no kernel (32, 64, 128, 256)", block_size);
  DQ_REQUIRE(R >= 1 && C >= block_size && C % block_size == 0, DQ_ERR_SHAPE, "bad shape R=%d C=%d block %d", R, C,
             block_size);
  DQ_REQUIRE(num_iter >= 1, DQ_ERR_SHAPE, "num_iter must be at least 1 (got %d)", num_iter);
  DQ_REQUIRE(scale_option >= 0 && scale_option <= 2 && row_init >= 0 && row_init <= 1 && col_init >= 0 && col_init <= 3 &&
                 scale_format >= 0 && scale_format <= 2,
             DQ_ERR_UNSUPPORTED, "unknown option");
  DQ_REQUIRE(aligned(w, 16) && (mat_q == nullptr || aligned(mat_q, 16)), DQ_ERR_ALIGN, "w and mat_q must be 16-byte aligned");
  DQ_REQUIRE(workspace_bytes >= dq_dualquant_workspace_bytes(R, C), DQ_ERR_WORKSPACE, "workspace too small");
  bcd::Params p;
  p.w = w;
  p.R = R;
  p.C = C;
  p.blocks = C / block_size;
  p.rows_per_chunk = bcd::chunk_rows(R);
  p.chunks = (R + p.rows_per_chunk - 1) / p.rows_per_chunk;
  p.option = scale_option;
  p.row_init = row_init;
  p.col_init = col_init;
  p.scale_format = scale_format;
  p.qmin = qmin;
  p.qmax = qmax;
  p.alpha = alpha;
  p.beta = beta;
  p.partials = static_cast<float*>(workspace);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (block_size) {
    case 32: return bcd::search<1>(p, num_iter, mat_q, column_scales, s);
    case 64: return bcd::search<2>(p, num_iter, mat_q, column_scales, s);
    case 128: return bcd::search<4>(p, num_iter, mat_q, column_scales, s);
    default: return bcd::search<8>(p, num_iter, mat_q, column_scales, s);
  }
}
