// One-call PermLinear.forward on the real int4 path.  Decode batches (M <= 16, no online Hadamard)
// may run as ONE kernel that quantises in its prologue; everything else is activation quantiser +
// GEMM on the caller's stream with the intermediates in caller-provided scratch.  Prefill batches
// (expansion_pays) take the FP8 tensor-core path when the caller's scratch also has room for
// the byte form of the weight: quantiser (E4M3 codes) + weight expansion + GEMM.
#include "dq_common.h"

namespace {
inline size_t round_up(size_t v, size_t a) { return (v + a - 1) / a * a; }
}  // namespace

extern "C" size_t dq_linear_w4a4_int4_scratch_bytes(int M, int N, int K) {
  (void)N;
  if (M < 0 || K < 0) return 0;
  return round_up(static_cast<size_t>(M) * static_cast<size_t>(K), 256) +
         round_up(static_cast<size_t>(M) * sizeof(float), 256);
}

// Whether a linear does best on the FP8-path GEMM with the weight's byte form, at extra_us for making it: never under 256
// tokens, always from 1024, between by the GEMMs' estimates - the FP8-path GEMM does not split K and loses where K is long
// and the row tiles few.  Its estimate, whose group times are those of long runs at the power cap, is high for wide outputs,
// hence the margin there.  Microseconds with the quantiser; packed, byte form expanded by the call, byte form kept:
//   4096 -> 4096     256 tokens  17  27  21    512 tokens  26  30  24     768 tokens   44   34   28    1024 tokens   43   34   29
//   4096 -> 28672                80  87  52               132 117  86                 179  139  106                224  161  131
//   14336 -> 4096                45  84  63                73  91  71                 121  100   81                140  111   92
//   14336 -> 1392                29  58  51                46  64  57                  51   68   61                 80   78   69
// Over 150 shapes of 256 to 1200 tokens the choice costs 0.4 % on average and 18 % at worst with a byte form expanded by the
// call, 0.7 and 24 % with one kept.
static bool byte_form_pays(int M, int N, int K, float extra_us) {
  if (M < 256 || N < 1 || K < dq::kGroup || K % dq::kGroup != 0) return false;
  if (M >= 1024) return true;
  const dq::DeviceState* st = dq::current_state();
  const int sms = st != nullptr ? st->sm_count : 148;  // (a size asked for before dq_init)
  return dq::gemm_int4_packed_us(M, N, K, sms) >=
         (M > 384 && N >= 6144 ? 0.75f : 1.0f) * (dq::gemm_int4_bytes_us(M, N, K, sms) + extra_us);
}
// The expansion is a launch and 1.5 bytes per weight: 4096 -> 4096 5.4 us, 14336 -> 4096 20, 4096 -> 28672 33.
static bool expansion_pays(int M, int N, int K) {
  return byte_form_pays(M, N, K, 2.5f + 0.31e-6f * static_cast<float>(N) * static_cast<float>(K));
}

extern "C" int dq_linear_w4a4_int4_byte_form_pays(int M, int N, int K) { return byte_form_pays(M, N, K, 0.f) ? 1 : 0; }

extern "C" size_t dq_linear_w4a4_int4_prefill_scratch_bytes(int M, int N, int K) {
  const size_t base = dq_linear_w4a4_int4_scratch_bytes(M, N, K);
  if (!expansion_pays(M, N, K)) return base;
  return base + round_up(static_cast<size_t>(N) * static_cast<size_t>(K), 256);
}

// Quantiser and GEMM with the codes and token scales in the scratch.  The FP8-path GEMM runs with the caller's byte form of
// the weight (w8), or where it pays with one expanded behind the token scales if the scratch has room for it.
static int quant_and_gemm(const void* x_bf16, int64_t ldx, const float* a, const dq_hadamard_desc* had,
                          const uint8_t* w_packed, const uint8_t* w8, const void* sw_t, const float* r, const void* bias,
                          int M, int N, int K, int G, void* y, int y_dtype, int scale_fp16, void* scratch,
                          size_t scratch_bytes, void* stream) {
  uint8_t* base = static_cast<uint8_t*>(scratch);
  int8_t* codes = static_cast<int8_t*>(scratch);
  float* sx = reinterpret_cast<float*>(base + round_up(static_cast<size_t>(M) * K, 256));
  const dq::Addend add = {bias, 0};
  if (w8 == nullptr && G == dq::kGroup && (scale_fp16 & ~0xFF) == 0 && expansion_pays(M, N, K) &&
      scratch_bytes >= dq_linear_w4a4_int4_prefill_scratch_bytes(M, N, K)) {
    uint8_t* expanded = base + dq_linear_w4a4_int4_scratch_bytes(M, N, K);
    DQ_REQUIRE(w_packed != nullptr, DQ_ERR_NULL, "w_packed is null");
    DQ_REQUIRE(dq::aligned(w_packed, 16), DQ_ERR_ALIGN, "w_packed must be 16-byte aligned");
    const int rc = dq::quant_act_int4_and_expand(x_bf16, ldx, a, had, M, K, codes, sx, scale_fp16 | DQ_CODES_E4M3,
                                                 {w_packed, expanded, N, K}, static_cast<cudaStream_t>(stream));
    if (rc != DQ_OK) return rc;
    w8 = expanded;
  } else {
    const int rc = dq_quant_act_int4(x_bf16, ldx, a, had, M, K, codes, sx,
                                     scale_fp16 | (w8 != nullptr ? DQ_CODES_E4M3 : 0), stream);
    if (rc != DQ_OK) return rc;
  }
  if (w8 == nullptr)
    return dq::gemm_w4a4_int4_addend(codes, sx, w_packed, sw_t, r, add, M, N, K, G, y, y_dtype, stream);
  dq::DeviceState* st = dq::current_state();
  if (st == nullptr) return DQ_ERR_NOT_INIT;
  DQ_REQUIRE(sw_t != nullptr && y != nullptr, DQ_ERR_NULL, "null sw_t / y");
  DQ_REQUIRE(G == dq::kGroup, DQ_ERR_UNSUPPORTED, "weight group size must be %d (got %d)", dq::kGroup, G);
  DQ_REQUIRE(N >= 1 && K >= dq::kGroup && K % dq::kGroup == 0, DQ_ERR_SHAPE, "bad shape N=%d K=%d", N, K);
  DQ_REQUIRE(y_dtype == DQ_DTYPE_F32 || y_dtype == DQ_DTYPE_BF16, DQ_ERR_UNSUPPORTED, "unknown y_dtype %d", y_dtype);
  DQ_REQUIRE(dq::aligned(w8, 16), DQ_ERR_ALIGN, "w8 must be 16-byte aligned");
  return dq::launch_gemm_int4_e4m3(reinterpret_cast<const uint8_t*>(codes), sx, w8, sw_t, r, M, N, K, y, y_dtype, add,
                                   static_cast<cudaStream_t>(stream), st);
}

extern "C" int dq_linear_w4a4_int4(const void* x_bf16, int64_t ldx, const float* a,
                                   const dq_hadamard_desc* had, const uint8_t* w_packed,
                                   const void* sw_t, const float* r, int M, int N, int K, int G,
                                   void* y, int y_dtype, int scale_fp16, void* scratch,
                                   size_t scratch_bytes, void* stream) {
  DQ_REQUIRE(scratch != nullptr, DQ_ERR_NULL, "scratch is null");
  DQ_REQUIRE(dq::aligned(scratch, 256), DQ_ERR_ALIGN, "scratch must be 256-byte aligned");
  DQ_REQUIRE(scratch_bytes >= dq_linear_w4a4_int4_scratch_bytes(M, N, K), DQ_ERR_WORKSPACE,
             "scratch of %zu bytes is smaller than the %zu required", scratch_bytes,
             dq_linear_w4a4_int4_scratch_bytes(M, N, K));
  if (M == 0) return DQ_OK;
  // Decode batches without an online Hadamard: one launch, the quantiser runs inside the GEMM
  // kernel and the scratch stays untouched.  Same codes, scales and sums as the two launches below.
  if ((had == nullptr || had->kind == DQ_HAD_NONE) && G == dq::kGroup &&
      dq::tuning(dq::DQ_TUNE_LINEAR_FUSED) != 0) {
    dq::DeviceState* st = dq::current_state();
    if (st == nullptr) return DQ_ERR_NOT_INIT;
    if (dq::gemv_fused_covers(M, N, K, st)) {
      DQ_REQUIRE(y_dtype == DQ_DTYPE_F32 || y_dtype == DQ_DTYPE_BF16, DQ_ERR_UNSUPPORTED,
                 "unknown y_dtype %d", y_dtype);
      return dq::launch_gemv_fused(x_bf16, ldx, a, w_packed, r, M, N, K, y, y_dtype, scale_fp16,
                                   static_cast<cudaStream_t>(stream), st);
    }
  }
  return quant_and_gemm(x_bf16, ldx, a, had, w_packed, nullptr, sw_t, r, nullptr, M, N, K, G, y, y_dtype, scale_fp16, scratch,
                        scratch_bytes, stream);
}

extern "C" int dq_linear_w4a4_int4_bias(const void* x_bf16, int64_t ldx, const float* a, const dq_hadamard_desc* had,
                                        const uint8_t* w_packed, const uint8_t* w8, const void* sw_t, const float* r,
                                        const void* bias, int M, int N, int K, int G, void* y, int y_dtype,
                                        int scale_fp16, void* scratch, size_t scratch_bytes, void* stream) {
  DQ_REQUIRE(scratch != nullptr, DQ_ERR_NULL, "scratch is null");
  DQ_REQUIRE(dq::aligned(scratch, 256), DQ_ERR_ALIGN, "scratch must be 256-byte aligned");
  DQ_REQUIRE(scratch_bytes >= dq_linear_w4a4_int4_scratch_bytes(M, N, K), DQ_ERR_WORKSPACE,
             "scratch of %zu bytes is smaller than the %zu required", scratch_bytes,
             dq_linear_w4a4_int4_scratch_bytes(M, N, K));
  DQ_REQUIRE(dq::aligned(bias, y_dtype == DQ_DTYPE_BF16 ? 2 : 4), DQ_ERR_ALIGN, "misaligned bias");
  if (M == 0) return DQ_OK;
  return quant_and_gemm(x_bf16, ldx, a, had, w_packed, w8, sw_t, r, bias, M, N, K, G, y, y_dtype, scale_fp16, scratch,
                        scratch_bytes, stream);
}

// ---------------------------------------------------------------------------------------------
// Allocation-free variant
// ---------------------------------------------------------------------------------------------
// Scratch for dq_linear_w4a4_int4_static lives in the library image itself, so the caller never
// has to obtain device memory.  Every GPU that loads the library carries these bytes until the
// process exits.  The array name below is only a host-side handle: the device address that
// kernels can use is looked up once per device with cudaGetSymbolAddress.
#define DQ_STATIC_SCRATCH_BYTES (2u * 1024u * 1024u + 16u * 1024u)
static __device__ __align__(256) unsigned char g_static_scratch[DQ_STATIC_SCRATCH_BYTES];
static void* g_static_scratch_addr[dq::kMaxDevices] = {nullptr};

extern "C" size_t dq_linear_w4a4_int4_static_max_bytes(void) { return DQ_STATIC_SCRATCH_BYTES; }

extern "C" int dq_linear_w4a4_int4_static(const void* x_bf16, int64_t ldx, const float* a,
                                          const dq_hadamard_desc* had, const uint8_t* w_packed,
                                          const void* sw_t, const float* r, int M, int N, int K,
                                          int G, void* y, int y_dtype, int scale_fp16,
                                          void* stream) {
  DQ_REQUIRE(M >= 0 && N >= 1 && K >= 1, DQ_ERR_SHAPE, "bad shape M=%d N=%d K=%d", M, N, K);
  const size_t need = dq_linear_w4a4_int4_scratch_bytes(M, N, K);
  DQ_REQUIRE(need <= DQ_STATIC_SCRATCH_BYTES, DQ_ERR_WORKSPACE,
             "M=%d x K=%d needs %zu bytes of scratch; the built-in scratch holds %u "
             "(use dq_linear_w4a4_int4 with caller-provided scratch for larger batches)",
             M, K, need, DQ_STATIC_SCRATCH_BYTES);
  int dev = -1;
  DQ_CHECK_CUDA(cudaGetDevice(&dev));
  DQ_REQUIRE(dev >= 0 && dev < dq::kMaxDevices, DQ_ERR_SHAPE, "device index %d out of range", dev);
  if (g_static_scratch_addr[dev] == nullptr) {
    // one-time set-up for this device (it is the current one): symbol -> device address
    void* ptr = nullptr;
    DQ_CHECK_CUDA(cudaGetSymbolAddress(&ptr, g_static_scratch));
    DQ_REQUIRE(ptr != nullptr, DQ_ERR_CUDA, "cudaGetSymbolAddress returned a null address");
    g_static_scratch_addr[dev] = ptr;
  }
  return dq_linear_w4a4_int4(x_bf16, ldx, a, had, w_packed, sw_t, r, M, N, K, G, y, y_dtype,
                             scale_fp16, g_static_scratch_addr[dev], DQ_STATIC_SCRATCH_BYTES,
                             stream);
}
