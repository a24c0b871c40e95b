// W4A4 int4 dual-scale GEMM for large token counts (prefill) on the FP8 tensor-core path.
//
//   Y[m,n] = r[n] * sx[m] * sum_g sw[n,g] * ( sum_{k in group g} qx[m,k] * qw[n,k] )
//
// Same result, bit for bit, as the kind::i8 kernel (gemm_w4a4_int4.cu); what changes is how the
// per-group integer sums are formed.  Every int4 code (-8 .. 7) is an exact E4M3 number, products
// and 128-term sums of such codes are integers below 2^24, so tcgen05.mma kind::f8f6f4 with an
// fp32 accumulator delivers each group sum exactly - as a float.  That removes the two things that
// bound the integer kernel on the CUDA cores: the int32 -> fp32 conversion of every accumulator
// element (a quarter-rate instruction) and the nibble unpacking (the operands arrive as bytes,
// straight from TMA).  The epilogue is one packed FMA per two accumulator elements.
//
// Operands: weights and activation codes as E4M3 bytes, row-major [N, K] and [M, K]
// (dq_expand_w_int4_e4m3 makes the former from the packed int4 artefact, dq_codes_to_e4m3 the
// latter from the quantiser's int8 codes).  The 4-bit artefact stays the storage format; the byte
// form is a derived copy for token counts where the GEMM is compute-bound.
//
// The kernel (gemm_w4a4_int4_f8.cuh) works on tiles of 256 weight rows x TN tokens on a pair of CTAs; this file
// holds the operand conversions, the choice of TN and the C entry points.
#include "gemm_w4a4_int4_f8.cuh"
#include "expand_w_e4m3.cuh"

namespace dq {
namespace f8 {

cudaError_t run_out0(int tn, const Launch& l);
cudaError_t run_out1(int tn, const Launch& l);
cudaError_t run_out2(int tn, const Launch& l);
cudaError_t run_out3(int tn, const Launch& l);
cudaError_t run_out5(int tn, const Launch& l);
cudaError_t run_scatter(const Launch& l);
cudaError_t init_out0();
cudaError_t init_out1();
cudaError_t init_out2();
cudaError_t init_out3();
cudaError_t init_out5();

// the low nibbles of the four bytes of v, packed into bits 0-15
__device__ __forceinline__ uint32_t low_nibbles(uint32_t v) {
  return (v & 0xFu) | ((v >> 4) & 0xF0u) | ((v >> 8) & 0xF00u) | ((v >> 12) & 0xF000u);
}

// An expansion on its own: a thread per chunk.
constexpr int kExpandThreads = 256;
__global__ void __launch_bounds__(kExpandThreads) expand_w_e4m3_kernel(const WeightExpansion e) {
  grid_dep_launch_dependents();
  grid_dep_wait();
  expand_chunks<kExpandThreads, 1>(e, blockIdx.x);
}

// int8 codes (-8..7) [M, K] with row stride ld -> E4M3 bytes [M, K]; one thread per 16 codes
__global__ void __launch_bounds__(256) codes_to_e4m3_kernel(const int8_t* codes, int64_t ld, int M,
                                                            int K, uint8_t* __restrict__ x8) {
  grid_dep_launch_dependents();
  grid_dep_wait();
  const int vec = K / 16;
  const int64_t total = static_cast<int64_t>(M) * vec;
  for (int64_t u = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; u < total;
       u += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t m = u / vec;
    const int kv = static_cast<int>(u - m * vec);
    const uint4 raw = *reinterpret_cast<const uint4*>(codes + m * ld + kv * 16);
    uint4 o;
    o.x = e4m3x4_of_nibbles(low_nibbles(raw.x));
    o.y = e4m3x4_of_nibbles(low_nibbles(raw.y));
    o.z = e4m3x4_of_nibbles(low_nibbles(raw.z));
    o.w = e4m3x4_of_nibbles(low_nibbles(raw.w));
    *reinterpret_cast<uint4*>(x8 + m * K + kv * 16) = o;
  }
}

// Token tile: the one whose rounds of one tile per CTA pair cost least.  A wide tile is the most efficient per token
// (a group of 256 tokens costs 1.7 times a group of 96, below that a group costs what its weight tile costs), a narrower
// one leaves less of the last round empty, or spreads a small batch over the chip.  Group times: measured on B200 in
// long runs at the power cap.
static int pick_tile(int M, int row_pairs, int ng, int pairs, bool direct, float* cost_us = nullptr) {
  static const struct { int tn; float group_us; } kTiles[] = {{256, 0.57f}, {224, 0.53f}, {192, 0.46f}, {160, 0.41f},
                                                              {128, 0.36f}, {96, 0.33f},  {64, 0.31f},  {32, 0.30f}};
  const int forced = tuning(DQ_TUNE_F8_TILE);
  int best = 256;
  float best_cost = 1e30f;
  for (const auto& t : kTiles) {
    if (direct && t.tn != 256 && t.tn != 128 && t.tn != 32) continue;  // what the direct-store mode is built for
    if (forced == t.tn) return t.tn;
    const int64_t tiles = static_cast<int64_t>(row_pairs) * ((M + t.tn - 1) / t.tn);
    const int64_t rounds = (tiles + pairs - 1) / pairs;
    const float cost = rounds * (ng * t.group_us + 2.0f + t.tn / 256.0f);
    if (cost < best_cost) {
      best_cost = cost;
      best = t.tn;
    }
  }
  if (cost_us != nullptr) *cost_us = best_cost;
  return best;
}

}  // namespace f8

int init_gemm_int4_f8_kernels() {
  cudaError_t e = f8::init_out0();
  if (e == cudaSuccess) e = f8::init_out1();
  if (e == cudaSuccess) e = f8::init_out2();
  if (e == cudaSuccess) e = f8::init_out3();
  if (e == cudaSuccess) e = f8::init_out5();
  if (e != cudaSuccess)
    return set_error(DQ_ERR_CUDA, "cudaFuncSetAttribute(gemm_w4a4_e4m3) failed: %s", cudaGetErrorString(e));
  return DQ_OK;
}

// w8 / x8: E4M3 bytes, row-major [N, K] / [M, K]
static int launch_gemm_int4_e4m3_impl(const uint8_t* x8, const float* sx, const uint8_t* w8, const void* sw_t,
                                      const float* r, int M, int N, int K, void* y, int y_dtype, Addend add,
                                      cudaStream_t stream, DeviceState* st, const f8::ScatterDst* scatter) {
  f8::Launch l = {};
  // bf16 output (optionally with a residual) and fp32 output without one leave through tiled bulk stores (16-byte
  // aligned rows); anything else is stored directly
  const bool yb = y_dtype == DQ_DTYPE_BF16;
  int out = 0;
  if (scatter != nullptr) out = 4;
  else if (yb && N % 8 == 0 && aligned(y, 16) && (add.ld == 0 || aligned(add.p, 16)))
    out = add.p == nullptr ? 1 : add.ld == 0 ? 5 : 3;
  else if (!yb && add.p == nullptr && N % 4 == 0 && aligned(y, 16)) out = 2;
  l.row_pairs = (N + 2 * f8::kBN - 1) / (2 * f8::kBN);
  const int pairs = st->sm_count / 2;
  const int tn = out == 4 ? 256 : f8::pick_tile(M, l.row_pairs, K / kGroup, pairs, out == 0);
  int rc = make_tmap_2d_u8(&l.tm_w, w8, static_cast<uint64_t>(K), static_cast<uint64_t>(N), static_cast<uint64_t>(K),
                           128, f8::kBN, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != DQ_OK) return rc;
  rc = make_tmap_2d_u8(&l.tm_x, x8, static_cast<uint64_t>(K), static_cast<uint64_t>(M), static_cast<uint64_t>(K), 128,
                       static_cast<uint32_t>(tn / 2), CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != DQ_OK) return rc;
  if (out == 1 || out == 3 || out == 5) {
    rc = make_tmap_2d_out(&l.tm_y, y, 2, static_cast<uint64_t>(N), static_cast<uint64_t>(M), f8::kBN, tn);
    if (rc == DQ_OK && out == 3)
      rc = make_tmap_2d_out(&l.tm_res, add.p, 2, static_cast<uint64_t>(N), static_cast<uint64_t>(M), f8::kBN, tn);
  } else if (out == 2) {
    rc = make_tmap_2d_out(&l.tm_y, y, 4, static_cast<uint64_t>(N), static_cast<uint64_t>(M), f8::kBN, tn / 2);
  }
  if (rc != DQ_OK) return rc;
  l.tok_tiles = (M + tn - 1) / tn;
  const int64_t tiles = static_cast<int64_t>(l.row_pairs) * l.tok_tiles;
  l.ctas = 2 * static_cast<int>(tiles < pairs ? tiles : pairs);
  // activations of one block of token tiles: about 40 MB, so that they stay in L2 (126 MB) beside
  // the weight tiles in use while every row pair passes over them
  int64_t tok_block = (40ll << 20) / (static_cast<int64_t>(tn) * K);
  if (tok_block < 1) tok_block = 1;
  if (tok_block > l.tok_tiles) tok_block = l.tok_tiles;
  l.tok_block = static_cast<int>(tok_block);
  l.sw_t = static_cast<const __half*>(sw_t);
  l.r = r;
  l.sx = sx;
  l.y = y;
  l.y_bf16 = yb ? 1 : 0;
  l.add = add;
  l.M = M;
  l.N = N;
  l.K = K;
  l.status = st->status_dev;
  l.stream = stream;
  if (scatter != nullptr) l.sc = *scatter;
  const cudaError_t e = out == 4   ? f8::run_scatter(l)
                        : out == 5 ? f8::run_out5(tn, l)
                        : out == 3 ? f8::run_out3(tn, l)
                        : out == 2 ? f8::run_out2(tn, l)
                        : out == 1 ? f8::run_out1(tn, l)
                                   : f8::run_out0(tn, l);
  if (e != cudaSuccess) return set_error(DQ_ERR_CUDA, "gemm_w4a4_e4m3 launch failed: %s", cudaGetErrorString(e));
  return DQ_OK;
}

float gemm_int4_bytes_us(int M, int N, int K, int sm_count) {
  float us = 0.f;
  f8::pick_tile(M, (N + 2 * f8::kBN - 1) / (2 * f8::kBN), K / kGroup, sm_count / 2, false, &us);
  return us;
}

int launch_gemm_int4_e4m3(const uint8_t* x8, const float* sx, const uint8_t* w8, const void* sw_t, const float* r,
                          int M, int N, int K, void* y, int y_dtype, Addend add, cudaStream_t stream,
                          DeviceState* st) {
  return launch_gemm_int4_e4m3_impl(x8, sx, w8, sw_t, r, M, N, K, y, y_dtype, add, stream, st, nullptr);
}

int launch_expand_w_e4m3(const WeightExpansion& e, cudaStream_t stream) {
  DQ_CHECK_CUDA(launch_pdl(f8::expand_w_e4m3_kernel, dim3(static_cast<unsigned>(expand_ctas(e.N, e.K, f8::kExpandThreads))),
                           dim3(f8::kExpandThreads), 0, stream, e));
  return DQ_OK;
}

}  // namespace dq

using namespace dq;

extern "C" int dq_gemm_w4a4_int4_e4m3_scatter(const uint8_t* x8, const float* sx, const uint8_t* w8, const void* sw_t,
                                              const float* r, int M, int N, int K, int G, const dq_exchange_ctx* ctx,
                                              void* stream) {
  DeviceState* st = current_state();
  if (st == nullptr) return DQ_ERR_NOT_INIT;
  DQ_REQUIRE(x8 != nullptr && sx != nullptr && w8 != nullptr && sw_t != nullptr && ctx != nullptr, DQ_ERR_NULL,
             "null x8 / sx / w8 / sw_t / ctx");
  DQ_REQUIRE(G == kGroup, DQ_ERR_UNSUPPORTED, "weight group size must be %d (got %d)", kGroup, G);
  DQ_REQUIRE(ctx->world >= 1 && ctx->world <= 8 && ctx->rank >= 0 && ctx->rank < ctx->world, DQ_ERR_SHAPE,
             "bad exchange context (world %d, rank %d)", ctx->world, ctx->rank);
  DQ_REQUIRE(K >= kGroup && K % kGroup == 0 && N == ctx->hidden && N % f8::kBN == 0 &&
                 ctx->tokens_per_rank % 256 == 0 && static_cast<int64_t>(M) == ctx->world * ctx->tokens_per_rank,
             DQ_ERR_SHAPE, "scatter GEMM needs N == hidden (%d), N %% 128 == 0, tokens_per_rank %% 256 == 0 and "
             "M == world * tokens_per_rank (M=%d N=%d K=%d tokens_per_rank=%lld)", ctx->hidden, M, N, K,
             static_cast<long long>(ctx->tokens_per_rank));
  DQ_REQUIRE(aligned(x8, 16) && aligned(w8, 16), DQ_ERR_ALIGN, "x8 and w8 must be 16-byte aligned");
  f8::ScatterDst sc;
  memset(&sc, 0, sizeof(sc));
  for (int p = 0; p < ctx->world; ++p) {
    DQ_REQUIRE(ctx->part_ptrs[p] != nullptr && aligned(ctx->part_ptrs[p], 16), DQ_ERR_ALIGN,
               "partial buffer of rank %d is null or not 16-byte aligned", p);
    sc.part[p] = static_cast<unsigned short*>(ctx->part_ptrs[p]);
  }
  sc.rank = ctx->rank;
  sc.tq = static_cast<int>(ctx->tokens_per_rank);
  sc.rot = static_cast<int>(((ctx->rank + 1) % ctx->world) * (ctx->tokens_per_rank / 256));
  return launch_gemm_int4_e4m3_impl(x8, sx, w8, sw_t, r, M, N, K, nullptr, DQ_DTYPE_BF16, Addend{},
                                    static_cast<cudaStream_t>(stream), st, &sc);
}

extern "C" int dq_expand_w_int4_e4m3(const uint8_t* w_packed, int N, int K, int G, uint8_t* w8, void* stream) {
  DeviceState* st = current_state();
  if (st == nullptr) return DQ_ERR_NOT_INIT;
  DQ_REQUIRE(w_packed != nullptr && w8 != nullptr, DQ_ERR_NULL, "null w_packed / w8");
  DQ_REQUIRE(G == kGroup, DQ_ERR_UNSUPPORTED, "weight group size must be %d (got %d)", kGroup, G);
  DQ_REQUIRE(N >= 1 && K >= kGroup && K % kGroup == 0, DQ_ERR_SHAPE, "bad shape N=%d K=%d", N, K);
  DQ_REQUIRE(aligned(w_packed, 16) && aligned(w8, 16), DQ_ERR_ALIGN, "w_packed and w8 must be 16-byte aligned");
  return launch_expand_w_e4m3({w_packed, w8, N, K}, static_cast<cudaStream_t>(stream));
}

extern "C" int dq_codes_to_e4m3(const int8_t* codes, int64_t ld, int M, int K, uint8_t* x8, void* stream) {
  DeviceState* st = current_state();
  if (st == nullptr) return DQ_ERR_NOT_INIT;
  if (M == 0) return DQ_OK;
  DQ_REQUIRE(codes != nullptr && x8 != nullptr, DQ_ERR_NULL, "null codes / x8");
  DQ_REQUIRE(M >= 1 && K >= 16 && K % 16 == 0 && ld >= K && ld % 16 == 0, DQ_ERR_SHAPE, "bad shape M=%d K=%d ld=%lld", M,
             K, static_cast<long long>(ld));
  DQ_REQUIRE(aligned(codes, 16) && aligned(x8, 16), DQ_ERR_ALIGN, "codes and x8 must be 16-byte aligned");
  const int64_t vecs = static_cast<int64_t>(M) * (K / 16);
  int64_t blocks = (vecs + 255) / 256;
  if (blocks > st->sm_count * 16) blocks = st->sm_count * 16;
  DQ_CHECK_CUDA(launch_pdl(f8::codes_to_e4m3_kernel, dim3(static_cast<unsigned>(blocks)), dim3(256), 0,
                           static_cast<cudaStream_t>(stream), codes, ld, M, K, x8));
  return DQ_OK;
}

extern "C" int dq_gemm_w4a4_int4_e4m3(const uint8_t* x8, const float* sx, const uint8_t* w8, const void* sw_t,
                                      const float* r, int M, int N, int K, int G, void* y, int y_dtype,
                                      const void* residual, void* stream) {
  DeviceState* st = current_state();
  if (st == nullptr) return DQ_ERR_NOT_INIT;
  if (M == 0) return DQ_OK;
  DQ_REQUIRE(x8 != nullptr && sx != nullptr && w8 != nullptr && sw_t != nullptr && y != nullptr, DQ_ERR_NULL,
             "null x8 / sx / w8 / sw_t / y");
  DQ_REQUIRE(G == kGroup, DQ_ERR_UNSUPPORTED, "weight group size must be %d (got %d)", kGroup, G);
  DQ_REQUIRE(M >= 1 && N >= 1 && K >= kGroup && K % kGroup == 0, DQ_ERR_SHAPE, "bad shape M=%d N=%d K=%d", M, N, K);
  DQ_REQUIRE(y_dtype == DQ_DTYPE_F32 || y_dtype == DQ_DTYPE_BF16, DQ_ERR_UNSUPPORTED, "unknown y_dtype %d", y_dtype);
  DQ_REQUIRE(aligned(x8, 16) && aligned(w8, 16), DQ_ERR_ALIGN, "x8 and w8 must be 16-byte aligned");
  return launch_gemm_int4_e4m3(x8, sx, w8, sw_t, r, M, N, K, y, y_dtype, Addend{residual, N},
                               static_cast<cudaStream_t>(stream), st);
}
