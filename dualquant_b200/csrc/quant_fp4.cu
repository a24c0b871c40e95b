// Block-scaled FP4 quantisers for sm_100a: MXFP4 (E2M1 elements, blocks of 32, E8M0 scale) and
// NVFP4 (E2M1 elements, blocks of 16, E4M3 block scale over a second-level fp32 scale).
//
//   x32 = float(x) * a[k]                       (a optional)
//   MXFP4: e = floor(log2(absmax_block)) - 2 clamped to [-127, 127] (-127 for a zero block);
//          q = e2m1(x32 * 2^-e)                 scale byte = e + 127
//   NVFP4: ts = absmax_row / (6 * 448) (1 for a zero row), or a given per-tensor value;
//          bs = e4m3(clamp(absmax_block / 6 / ts, 2^-6, 448));    q = e2m1(x32 / (ts * bs))
// Element and scale conversions use the hardware converters (cvt.rn.satfinite.e2m1x2.f32 /
// .e4m3x2.f32: round to nearest even, saturating).  Codes and scale bytes are those of IEEE divisions; the quotients are
// estimated with an approximate reciprocal, and only those near a rounding boundary are divided (nvfp4_scale_byte,
// fp4_emit_vector).  One CTA per row, the row in registers, 8 consecutive elements per thread; a block spans 2 (NVFP4) or
// 4 (MXFP4) lanes.  2 bytes in, 0.5 byte + scale out per element.
#include "dq_common.h"
#include "dq_ptx.cuh"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

namespace dq {

enum { FP4_MODE_CODES = 0, FP4_MODE_FAKE = 1 };
constexpr int kFp4ManyRows = 512;  // from here on the chip is full of rows: fewer threads per row, more rows per SM

// Eight values -> eight E2M1 codes in one word, the first in the lowest nibble.
__device__ __forceinline__ uint32_t e2m1x8(const float* v) {
  uint32_t out;
  asm("{\n"
      ".reg .b8 t0, t1, t2, t3;\n"
      "cvt.rn.satfinite.e2m1x2.f32 t0, %2, %1;\n"
      "cvt.rn.satfinite.e2m1x2.f32 t1, %4, %3;\n"
      "cvt.rn.satfinite.e2m1x2.f32 t2, %6, %5;\n"
      "cvt.rn.satfinite.e2m1x2.f32 t3, %8, %7;\n"
      "mov.b32 %0, {t0, t1, t2, t3};\n"
      "}\n"
      : "=r"(out)
      : "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]));
  return out;
}
// The eight values times f, two per instruction.
__device__ __forceinline__ void mul8(const float* v, float f, float* out) {
#pragma unroll
  for (int k = 0; k < 8; k += 2) {
    const float2 t = __fmul2_rn(make_float2(v[k], v[k + 1]), make_float2(f, f));
    out[k] = t.x;
    out[k + 1] = t.y;
  }
}
// 1 / x to one unit in the last place, subnormals flushed
__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ float e2m1_value(uint32_t code) {
  // 1 sign, 2 exponent, 1 mantissa bit: 0, 0.5, then (1 + m/2) * 2^(e-1)
  const uint32_t e = (code >> 1) & 3u, m = code & 1u;
  const float frac = 1.0f + 0.5f * static_cast<float>(m);
  const float v = (e == 0) ? 0.5f * static_cast<float>(m) : frac * __uint_as_float((126u + e) << 23);
  return (code & 8u) ? -v : v;
}

__device__ __forceinline__ uint32_t e4m3_byte_of(float v) {
  uint16_t out;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(out) : "f"(0.f), "f"(v));
  return out & 0xFFu;  // second operand lands in the low byte
}

// Scale bytes of an NVFP4 block: want = bmax / 6 / ts, clamped to the normal range of E4M3 [2^-6, 448] before the cast, as
// the reference's scale quantiser does (scale_formats.py:39-45): an all-zero or tiny block gets the scale 2^-6.  The
// quotient is estimated with a product (inv6ts = 1 / 6 / ts, within 2^-21); where both ends of that interval convert to
// the same byte, so does the quotient, and the two IEEE divisions are left to the blocks on a rounding boundary.
__device__ __forceinline__ uint32_t nvfp4_scale_byte(float bmax, float ts, float inv6ts) {
  const float w = __fmul_rn(bmax, inv6ts);
  const float lo = fmaxf(fminf(__fmul_rn(w, 0.99999904632568359375f), 448.0f), 0.015625f);  // 1 - 2^-20
  const float hi = fmaxf(fminf(__fmul_rn(w, 1.00000095367431640625f), 448.0f), 0.015625f);  // 1 + 2^-20
  unsigned short two;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(two) : "f"(hi), "f"(lo));
  const uint32_t b = two & 0xFFu;
  if (b == static_cast<uint32_t>(two >> 8) && inv6ts >= 1e-30f && inv6ts <= 1e30f) return b;
  const float want = __fdiv_rn(__fdiv_rn(bmax, 6.0f), ts);
  return e4m3_byte_of(fmaxf(fminf(want, 448.0f), 0.015625f));
}

__device__ __forceinline__ void fp4_load8(const __nv_bfloat16* p, float* v) {
  const uint4 raw = *reinterpret_cast<const uint4*>(p);
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[2 * i] = __uint_as_float(w[i] << 16);
    v[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
  }
}
__device__ __forceinline__ void fp4_load8(const float* p, float* v) {
  const float4 a = *reinterpret_cast<const float4*>(p);
  const float4 b = *reinterpret_cast<const float4*>(p + 4);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

// One vector of 8 consecutive elements (already scaled by the column scale) whose block absmax is
// known: block scale, element codes, stores.  sf_off = where this vector's block scale byte goes
// (used by the first vector of a block only).
__device__ __forceinline__ void fp4_emit_vector(const float* v, float bmax, float ts, float inv6ts, int fmt, int mode,
                                                int row, int K, int idx, int blk, int64_t sf_off,
                                                uint8_t* __restrict__ codes, uint8_t* __restrict__ sf,
                                                float* __restrict__ out) {
    float q[8];
    float deq_scale;
    uint32_t sf_byte, packed;
    if (fmt == DQ_FP4_MXFP4) {
      int e = -127;
      if (bmax != 0.f) {
        e = static_cast<int>((__float_as_uint(bmax) >> 23) & 0xFFu) - 127 - 2;
        e = max(-127, min(127, e));
      }
      sf_byte = static_cast<uint32_t>(e + 127);
      // 2^-e and 2^e by their bits (subnormal at the far end): one multiplication rounds exactly like scalbnf(v, -e)
      const float down = __uint_as_float(e == 127 ? 0x00400000u : static_cast<uint32_t>(127 - e) << 23);
      deq_scale = __uint_as_float(e == -127 ? 0x00400000u : static_cast<uint32_t>(127 + e) << 23);
      mul8(v, down, q);
      packed = e2m1x8(q);
    } else {
      sf_byte = nvfp4_scale_byte(bmax, ts, inv6ts);
      const float bs = __uint_as_float((sf_byte << 20) + (120u << 23));  // a normal E4M3 number, by its bits
      const float denom = __fmul_rn(ts, bs);
      deq_scale = denom;
      if (mode == FP4_MODE_FAKE) deq_scale = bs;  // applied as (q * bs) * ts below
      if (denom == 0.f) {
        packed = 0;
      } else {
        // v / denom rounded to E2M1 without eight IEEE divisions: t = v * rcp(denom) is within 2^-21.4 |t| of the
        // quotient; if t (1 - 2^-20) and t (1 + 2^-20) convert to the same codes, so does everything between them, the
        // correctly rounded quotient included.  Otherwise (an element sits on a rounding boundary, or the reciprocal
        // left its range) the thread takes the exact divisions, in a branch of its own.
        const float inv = rcp_approx(denom);
        float t[8], lo[8], hi[8];
        mul8(v, inv, t);
        mul8(t, 0.99999904632568359375f, lo);  // 1 - 2^-20
        mul8(t, 1.00000095367431640625f, hi);  // 1 + 2^-20
        packed = e2m1x8(lo);
        if (packed != e2m1x8(hi) || !(inv >= 1e-30f && inv <= 1e30f && __fmul_rn(bmax, inv) <= 1e30f)) {
#pragma unroll
          for (int k = 0; k < 8; ++k) q[k] = __fdiv_rn(v[k], denom);
          packed = e2m1x8(q);
        }
      }
    }
    if (mode == FP4_MODE_CODES) {
      *reinterpret_cast<uint32_t*>(codes + static_cast<int64_t>(row) * (K / 2) + idx / 2) = packed;
      if ((idx % blk) == 0) sf[sf_off] = static_cast<uint8_t>(sf_byte);
    } else {
      float o[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float qv = e2m1_value((packed >> (4 * k)) & 0xFu);
        o[k] = (fmt == DQ_FP4_MXFP4) ? __fmul_rn(qv, deq_scale) : __fmul_rn(__fmul_rn(qv, deq_scale), ts);
      }
      float* orow = out + static_cast<int64_t>(row) * K + idx;
      *reinterpret_cast<float4*>(orow) = make_float4(o[0], o[1], o[2], o[3]);
      *reinterpret_cast<float4*>(orow + 4) = make_float4(o[4], o[5], o[6], o[7]);
    }
}

// Eight input elements as loaded (bf16: one 16-byte vector; fp32: two).
template <typename XT>
struct Fp4Raw;
template <>
struct Fp4Raw<__nv_bfloat16> {
  uint4 r;
  __device__ __forceinline__ void load(const __nv_bfloat16* p) { r = *reinterpret_cast<const uint4*>(p); }
  __device__ __forceinline__ void expand(float* v) const {
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[2 * i] = __uint_as_float(w[i] << 16);
      v[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
    }
  }
};
template <>
struct Fp4Raw<float> {
  float v8[8];
  __device__ __forceinline__ void load(const float* p) { fp4_load8(p, v8); }
  __device__ __forceinline__ void expand(float* v) const {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = v8[i];
  }
};

// One CTA per row, the row in registers in its input width: all of a row's loads are in flight at once, and it is read
// from memory once although NVFP4 needs the row's absmax before its first block scale.  The column scale is applied
// again in the second pass (from L1).  PER_SM CTAs' worth of registers.
template <int THREADS, int VPT, int PER_SM, typename XT>
__global__ void __launch_bounds__(THREADS, PER_SM)
quant_fp4_kernel(const XT* x, int64_t ldx, const float* a, int K, int fmt,
                 const float* tensor_scale, uint8_t* __restrict__ codes,
                 uint8_t* __restrict__ sf, float* __restrict__ row_scale, float* __restrict__ out,
                 int mode, int M, int sf_atoms, int activations) {
  // THREADS bounds the launch; the CTA may be smaller (a multiple of 32): vectors are dealt out
  // with the launched size as the stride, so that a row of K/8 vectors leaves few idle slots.
  __shared__ float red[THREADS / 32];
  // x comes from the kernel before this one.  As the first half of a linear (activations = 1) the GEMM behind it may
  // start at once and fetch its weights; a stand-alone call may be making those weights.  Linears of up to 16 rows gain
  // 10 to 20 % by it; of 1024 to 8192 rows, in a chain of linears MXFP4 ones 2 % and NVFP4 ones nothing, called one by one
  // on a cold L2 neither (within 0.5 % either way over twelve shapes; 4096 x 18944 -> 3584 as NVFP4 273.5 us both ways).
  if (activations) grid_dep_launch_dependents();
  grid_dep_wait();
  const int nthreads = static_cast<int>(blockDim.x);
  const int row = blockIdx.x;
  // sf_atoms: the scale bytes go straight into the order the GEMM streams,
  // [row tile of 128][k / (4 blocks)][(r % 32) * 16 + (r / 32) * 4 + block % 4]; the grid then
  // covers the rows up to the next multiple of 128 and the CTAs past M write zero scales.
  const int lg_blk = (fmt == DQ_FP4_MXFP4) ? 5 : 4;
  const int nsf = K >> lg_blk;
  const int rr = row & 127;
  uint8_t* sf_row = sf + (sf_atoms ? static_cast<int64_t>(row >> 7) * (nsf >> 2) * 512 + (rr & 31) * 16 + (rr >> 5) * 4
                                   : static_cast<int64_t>(row) * nsf);
  auto sf_offset = [&](int ksf) -> int64_t { return sf_atoms ? (ksf >> 2) * 512 + (ksf & 3) : ksf; };
  if (row >= M) {
    for (int ksf = threadIdx.x; ksf < nsf; ksf += nthreads) sf_row[sf_offset(ksf)] = 0;
    return;
  }
  const XT* xr = x + static_cast<int64_t>(row) * ldx;
  Fp4Raw<XT> raw[VPT];
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int idx = (i * nthreads + threadIdx.x) * 8;
    if (idx < K) raw[i].load(xr + idx);
  }
  auto scaled = [&](int i, int idx, float* v) {
    raw[i].expand(v);
    if (a != nullptr) {
      float av[8];
      fp4_load8(a + idx, av);
#pragma unroll
      for (int e = 0; e < 8; e += 2) {
        const float2 t = __fmul2_rn(make_float2(v[e], v[e + 1]), make_float2(av[e], av[e + 1]));
        v[e] = t.x;
        v[e + 1] = t.y;
      }
    }
  };
  auto absmax8 = [&](const float* v) -> float {
    float m = fabsf(v[0]);
#pragma unroll
    for (int e = 1; e < 8; ++e) m = fmaxf(m, fabsf(v[e]));
    return m;
  };
  float ts = 1.f, inv6ts = 1.f;
  if (fmt == DQ_FP4_NVFP4) {
    if (tensor_scale != nullptr) {
      ts = *tensor_scale;
    } else {
      float rmax = 0.f;
#pragma unroll
      for (int i = 0; i < VPT; ++i) {
        const int idx = (i * nthreads + threadIdx.x) * 8;
        if (idx < K) {
          float v[8];
          scaled(i, idx, v);
          rmax = fmaxf(rmax, absmax8(v));
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) rmax = fmaxf(rmax, __shfl_xor_sync(0xffffffffu, rmax, o));
      if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = rmax;
      __syncthreads();
      float m = red[0];
      for (int i = 1; i < nthreads / 32; ++i) m = fmaxf(m, red[i]);
      ts = (m == 0.f) ? 1.f : __fdiv_rn(m, 2688.0f);
    }
    if (threadIdx.x == 0 && row_scale != nullptr) row_scale[row] = ts;
    inv6ts = __fmul_rn(rcp_approx(ts), 0.16666667163372039794921875f);
  }
#pragma unroll
  for (int i = 0; i < VPT; ++i) {  // every lane runs every vector: the shuffles need the warp
    const int idx = (i * nthreads + threadIdx.x) * 8;
    float v[8], bmax = 0.f;
    if (idx < K) {
      scaled(i, idx, v);
      bmax = absmax8(v);
    }
    // block absmax: 16 elements = 2 adjacent lanes, 32 elements = 4 adjacent lanes
    bmax = fmaxf(bmax, __shfl_xor_sync(0xffffffffu, bmax, 1));
    if (fmt == DQ_FP4_MXFP4) bmax = fmaxf(bmax, __shfl_xor_sync(0xffffffffu, bmax, 2));
    if (idx < K)
      fp4_emit_vector(v, bmax, ts, inv6ts, fmt, mode, row, K, idx, 1 << lg_blk, sf_offset(idx >> lg_blk), codes, sf_row, out);
  }
}

// Per-tensor second-level NVFP4 scale: absmax(x) / (6 * 448), 1 for an all-zero tensor.
template <typename XT>
__global__ void absmax_kernel(const XT* __restrict__ x, int64_t n, unsigned int* __restrict__ bits) {
  float m = 0.f;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    m = fmaxf(m, fabsf(static_cast<float>(x[i])));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(bits, __float_as_uint(m));  // order-preserving for m >= 0
}
__global__ void nvfp4_scale_finalize_kernel(float* scale) {
  const float m = *scale;  // holds the absmax bit pattern
  *scale = (m == 0.f) ? 1.f : __fdiv_rn(m, 2688.0f);
}

template <typename XT>
static int launch_fp4(const XT* x, int64_t ldx, const float* a, int M, int K, int fmt,
                      const float* tensor_scale, uint8_t* codes, uint8_t* sf, float* row_scale,
                      float* out, int mode, cudaStream_t stream, int sf_atoms = 0, int activations = 0) {
  DQ_REQUIRE(fmt == DQ_FP4_MXFP4 || fmt == DQ_FP4_NVFP4, DQ_ERR_UNSUPPORTED, "unknown FP4 format %d", fmt);
  DQ_REQUIRE(x != nullptr, DQ_ERR_NULL, "x is null");
  const int blk = (fmt == DQ_FP4_MXFP4) ? 32 : 16;
  DQ_REQUIRE(M >= 0 && K >= blk && K % blk == 0, DQ_ERR_SHAPE, "K=%d must be a multiple of the block size %d", K, blk);
  DQ_REQUIRE(K <= 32768, DQ_ERR_UNSUPPORTED, "K=%d exceeds 32768", K);
  DQ_REQUIRE(ldx >= K && ldx % 8 == 0, DQ_ERR_ALIGN, "ldx=%lld must be >= K and a multiple of 8", (long long)ldx);
  DQ_REQUIRE(aligned(x, 16) && (a == nullptr || aligned(a, 16)), DQ_ERR_ALIGN, "x and a must be 16-byte aligned");
  DQ_REQUIRE((codes == nullptr || aligned(codes, 4)) && (out == nullptr || aligned(out, 16)), DQ_ERR_ALIGN,
             "outputs misaligned");
  if (M == 0) return DQ_OK;
  DQ_REQUIRE(!sf_atoms || (K / blk) % 4 == 0, DQ_ERR_SHAPE,
             "scale factors in GEMM order need K %% %d == 0 (K=%d)", 4 * blk, K);
  const int vec = K / 8;
  const int rows = sf_atoms ? (M + 127) / 128 * 128 : M;
  // T bounds the CTA, V = vectors of 8 per thread, P = CTAs per SM the registers are limited for; the CTA launched is the
  // smallest multiple of 32 threads that covers the row with V vectors each.  Few rows: many threads per row, one or two
  // vectors each, because latency counts.  Many rows: eight (fp32: four) vectors per thread, so that an SM holds three
  // rows of 18944 and has their 110 KB in flight.
#define DQ_FP4_LAUNCH(T, V, P)                                                                                           \
  DQ_CHECK_CUDA(launch_pdl(quant_fp4_kernel<T, V, P, XT>, dim3(rows), dim3(((vec + (V) - 1) / (V) + 31) / 32 * 32), 0,   \
                           stream, x, ldx, a, K, fmt, tensor_scale, codes, sf, row_scale, out, mode, M, sf_atoms, activations))
  constexpr int kMany = sizeof(XT) == 2 ? 8 : 4;
  if (M >= kFp4ManyRows && vec > 256) {
    if (vec <= 128 * kMany) DQ_FP4_LAUNCH(128, kMany, 7);
    else if (vec <= 320 * kMany) DQ_FP4_LAUNCH(320, kMany, 3);
    else if (vec <= 512 * kMany) DQ_FP4_LAUNCH(512, kMany, 2);
    else DQ_FP4_LAUNCH(1024, kMany, 1);
  } else if (vec <= 128) DQ_FP4_LAUNCH(128, 1, 1);
  else if (vec <= 256) DQ_FP4_LAUNCH(256, 1, 1);
  else if (vec <= 512) DQ_FP4_LAUNCH(512, 1, 1);
  else if (vec <= 1024) DQ_FP4_LAUNCH(512, 2, 1);
  else if (vec <= 2048) DQ_FP4_LAUNCH(1024, 2, 1);
  else DQ_FP4_LAUNCH(1024, 4, 1);
#undef DQ_FP4_LAUNCH
  DQ_CHECK_CUDA(cudaGetLastError());
  return DQ_OK;
}

// The activation half of a linear: dq_quant_fp4_atoms whose GEMM may start early.
int quant_fp4_activations(const void* x, int x_is_f32, int64_t ldx, const float* a, int M, int K, int fmt, uint8_t* codes,
                          uint8_t* sf_atoms, float* row_scale, cudaStream_t s) {
  if (x_is_f32)
    return launch_fp4(static_cast<const float*>(x), ldx, a, M, K, fmt, static_cast<const float*>(nullptr), codes, sf_atoms,
                      row_scale, nullptr, FP4_MODE_CODES, s, 1, 1);
  return launch_fp4(static_cast<const __nv_bfloat16*>(x), ldx, a, M, K, fmt, static_cast<const float*>(nullptr), codes,
                    sf_atoms, row_scale, nullptr, FP4_MODE_CODES, s, 1, 1);
}

}  // namespace dq

using namespace dq;

extern "C" int dq_quant_fp4(const void* x, int x_is_f32, int64_t ldx, const float* a, int M, int K,
                            int fmt, const float* tensor_scale, uint8_t* codes, uint8_t* sf,
                            float* row_scale, void* stream) {
  if (current_state() == nullptr) return DQ_ERR_NOT_INIT;
  if (M == 0) return DQ_OK;
  DQ_REQUIRE(codes != nullptr && sf != nullptr, DQ_ERR_NULL, "codes / sf is null");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (x_is_f32)
    return launch_fp4(static_cast<const float*>(x), ldx, a, M, K, fmt, tensor_scale, codes, sf,
                      row_scale, nullptr, FP4_MODE_CODES, s);
  return launch_fp4(static_cast<const __nv_bfloat16*>(x), ldx, a, M, K, fmt, tensor_scale, codes, sf,
                    row_scale, nullptr, FP4_MODE_CODES, s);
}

extern "C" int dq_quant_fp4_atoms(const void* x, int x_is_f32, int64_t ldx, const float* a, int M,
                                  int K, int fmt, const float* tensor_scale, uint8_t* codes,
                                  uint8_t* sf_atoms, float* row_scale, void* stream) {
  if (current_state() == nullptr) return DQ_ERR_NOT_INIT;
  if (M == 0) return DQ_OK;
  DQ_REQUIRE(codes != nullptr && sf_atoms != nullptr, DQ_ERR_NULL, "codes / sf_atoms is null");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (x_is_f32)
    return launch_fp4(static_cast<const float*>(x), ldx, a, M, K, fmt, tensor_scale, codes, sf_atoms,
                      row_scale, nullptr, FP4_MODE_CODES, s, 1);
  return launch_fp4(static_cast<const __nv_bfloat16*>(x), ldx, a, M, K, fmt, tensor_scale, codes,
                    sf_atoms, row_scale, nullptr, FP4_MODE_CODES, s, 1);
}

extern "C" int dq_fakequant_fp4(const void* x, int x_is_f32, int64_t ldx, const float* a, int M,
                                int K, int fmt, const float* tensor_scale, float* out,
                                void* stream) {
  if (current_state() == nullptr) return DQ_ERR_NOT_INIT;
  if (M == 0) return DQ_OK;
  DQ_REQUIRE(out != nullptr, DQ_ERR_NULL, "out is null");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (x_is_f32)
    return launch_fp4(static_cast<const float*>(x), ldx, a, M, K, fmt, tensor_scale, nullptr, nullptr,
                      nullptr, out, FP4_MODE_FAKE, s);
  return launch_fp4(static_cast<const __nv_bfloat16*>(x), ldx, a, M, K, fmt, tensor_scale, nullptr,
                    nullptr, nullptr, out, FP4_MODE_FAKE, s);
}

extern "C" int dq_nvfp4_tensor_scale(const void* x, int x_is_f32, int64_t numel, float* scale,
                                     void* stream) {
  if (current_state() == nullptr) return DQ_ERR_NOT_INIT;
  DQ_REQUIRE(x != nullptr && scale != nullptr && numel > 0, DQ_ERR_NULL, "null or empty input");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  DQ_CHECK_CUDA(cudaMemsetAsync(scale, 0, sizeof(float), s));
  const int blocks = static_cast<int>(numel / 4096 > 1184 ? 1184 : (numel + 4095) / 4096);
  if (x_is_f32)
    absmax_kernel<<<blocks, 256, 0, s>>>(static_cast<const float*>(x), numel,
                                         reinterpret_cast<unsigned int*>(scale));
  else
    absmax_kernel<<<blocks, 256, 0, s>>>(static_cast<const __nv_bfloat16*>(x), numel,
                                         reinterpret_cast<unsigned int*>(scale));
  nvfp4_scale_finalize_kernel<<<1, 1, 0, s>>>(scale);
  DQ_CHECK_CUDA(cudaGetLastError());
  return DQ_OK;
}
