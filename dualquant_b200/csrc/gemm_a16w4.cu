// A16W4 dual-scale linear for sm_100a: 16-bit activations against the int4 weight artefact,
//
//   Y[m,n] = r[n] * sum_k fp16(x[m,k] * a[k]) * fp16(qw[n,k] * sw[n, k/128])
//
// the computation of the reference's fused-beta Triton kernel
// (vendor/dualscale_kernel_benchmark/fused_dual_scale_kernel.py:55-149: beta multiplied into the
// activation tile on its way in, nibbles de-quantised with the group scale, floating-point dot
// product) on the tensor cores of this GPU: tcgen05.mma kind::f16 with fp16 operands and fp32
// accumulators in tensor memory over the whole K (the group scale is folded into the fp16 weight,
// so nothing has to be drained per group).  fp16 rather than bf16 operands: with 8-bit mantissas
// the reference's own acceptance check (mean relative error below 1 % against the fp32 formulation,
// fused_dual_scale_kernel.py:269-308) fails at 1.4-5.7 %, with 11-bit mantissas it passes at
// 0.25-0.4 %; the group scales are fp16 already, so code * scale is one exactly rounded product.
// Activations beyond the fp16 range saturate at +-65504.
//
// Tile: 256 weight rows x TN tokens on a pair of CTAs (tcgen05 cta_group::2); a CTA holds 128 of the rows and half of
// the tokens' activations.  The weight operand goes to the tensor core from TENSOR MEMORY: a set of eight of the sixteen
// unpack warps reads the packed tile (8 KB codes + 256 B scales per group of 128 k), expands the nibbles to fp16
// code * scale, a weight row per thread, and stores them with tcgen05.st (lane = weight row, column = two k).  Shared memory
// then carries only the packed tile and the activations: 80 KB per group of a 256-token tile, in 1024 cycles of UMMAs.
// 4096 -> 28672: 16 tokens 25 us, 512 tokens 92, 8192 tokens 1212 (1.6 PFLOPS).  (A single-CTA 128 x 128 tile with the
// expanded weights in shared memory moved 144 KB in 512 and was bound by that port: 50, 209, 2820 us.)
//   warps 0-15   unpack, two sets of eight that take groups in turn: warp w owns TMEM lanes 32 (w & 3) .. and
//                k 64 ((w >> 2) & 1) .. of a group.  A nibble pair becomes half2 by bit tricks: (w >> s) & 0x000F000F
//                picks two two's-complement nibbles, ^ 0x64086408 turns them into the fp16 numbers 1032 + code, a packed
//                subtract gives code exactly, a packed multiply by the fp16 group scale the weight.  The nibbles picked
//                together are k and k + 2; the pre-pass below writes the activations in that order, so nothing has to be
//                shuffled here.
//   warps 16-19  epilogue: accumulator -> registers -> shared memory (32 tokens at a time) -> bulk store
//   warps 20, 23 producers: two tiled copies of activations, one bulk copy of packed weights per group.  (One producer
//                for both, with the tile and ring positions divided out of a group counter, took 0.9 us per group.)
//   warps 21-22  UMMA issue (of the even CTA, for both); tiles of up to 64 tokens: two warps take alternate groups into
//                an accumulator each, because issuing a group takes one warp longer than executing it.  They alternate over
//                all groups of the CTA, not from a tile's first: a ring slot then stays with one warp also where a tile
//                has an odd number of groups
// Persistent CTAs; where the tiles leave the chip idle (decode batches) K is split over the pairs of a larger cluster
// instead, and the partial tiles are summed in rank order through distributed shared memory.  Every wait is bounded.
//
// The activation scale and the conversion to fp16 run as a small separate pass
// (xs = fp16(x * a), caller scratch) so that the GEMM can stage activations with TMA.
#include "dq_common.h"
#include "dq_ptx.cuh"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

namespace dq {
namespace a16 {

constexpr int kBN = 128;                 // weight rows per CTA; a pair works on 256
constexpr int kSets = 2;  // sets of eight unpack warps, taking groups in turn: one set needs 0.42 us for a group, two 0.33
constexpr int kUnpackWarps = 8, kEpiWarp = kSets * 8, kEpiWarps = 4, kProducerWarp = kEpiWarp + 4, kIssuerWarp = kEpiWarp + 5,
              kWeightWarp = kEpiWarp + 7;
constexpr int kThreads = (kEpiWarp + 8) * 32;
constexpr int kACols = 64;               // TMEM columns of one expanded group: 128 fp16
constexpr int kOutChunk = 32 * kBN * 4;  // 32 tokens x 128 rows of fp32 (bf16 uses half)

enum { ASITE_TMA = 51, ASITE_UNPACK = 52, ASITE_MMA = 53, ASITE_EPI = 54, ASITE_ALIGN = 55 };

template <int TN>
struct Cfg {
  static constexpr int kIssuers = (TN <= 64) ? 2 : 1;           // accumulators per tile
  static constexpr int kAccTiles = (TN <= 192) ? 2 : 1;         // tiles whose accumulators fit
  static constexpr int kAccCols = TN * kIssuers * kAccTiles;
  static constexpr int NA = (512 - kAccCols) / kACols < 4 ? (512 - kAccCols) / kACols : 4;  // expanded groups
  static constexpr int kXAtom = TN / 2 * 128;                   // this CTA's tokens x 64 k
  static constexpr int kXStage = 2 * kXAtom;
  static constexpr int SP = 6;                                  // packed-tile stages
  static constexpr int kFixed = SP * kTileBytes + 2 * kOutChunk + 512;
  static constexpr int kFit = (227 * 1024 - kFixed) / kXStage;
  static constexpr int SX = kFit < 8 ? kFit : 8;                // activation stages
  static constexpr int kOffX = 0;
  static constexpr int kOffOut = SX * kXStage;
  static constexpr int kOffP = kOffOut + 2 * kOutChunk;
  static constexpr int kOffBar = kOffP + SP * kTileBytes;
  static constexpr int kNumBars = 2 * SP + 2 * SX + 2 * NA + 2 * kAccTiles;
  static constexpr int kSmemBytes = kOffBar + kNumBars * 8 + 16;
  static_assert(kSmemBytes <= 227 * 1024 && SX >= 3 && NA >= 2, "rings");
  // Waits are by phase parity, so a warp must not be a whole phase ahead of a barrier's previous user: where warps take
  // groups in turn, every slot of a ring they wait on belongs to one of them.
  static_assert(SP % kSets == 0 && NA % kSets == 0, "packed tiles and expanded groups: a set of unpack warps per slot");
  static_assert(NA % kIssuers == 0 && SX % kIssuers == 0, "expanded groups and activations: an issuer per slot");
  static_assert(kXAtom % 1024 == 0, "swizzle atoms on 1 KB boundaries");
  static_assert(TN > 64 || TN * kBN * 4 <= kOffP, "split-K exchange tile");
};

// Instruction descriptor, kind::f16: fp16 A and B (both K-major), fp32 accumulator.
//   [4,6) D format (1 = F32)  [7,10) A format (0 = F16)  [10,13) B format (0 = F16)
//   [17,23) N >> 3  [24,29) M >> 4
__host__ __device__ constexpr uint32_t idesc_f16(int m, int n) {
  return (1u << 4) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}

// D[tmem of both CTAs] (+)= A[tmem of both] * B[smem of both]
__device__ __forceinline__ void umma_f16_pair(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                              uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n"
      "}\n" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// two two's-complement nibbles (bits 0-3 and 16-19 of t) -> half2 (code * scale)
__device__ __forceinline__ uint32_t nib2_to_f16x2(uint32_t t, __half2 s2) {
  const uint32_t biased = (t & 0x000F000Fu) ^ 0x64086408u;  // fp16 numbers 1024 + 8 + code
  __half2 v = *reinterpret_cast<const __half2*>(&biased);
  const uint32_t k1032 = 0x64086408u;
  v = __hsub2(v, *reinterpret_cast<const __half2*>(&k1032));  // exact: small integers
  v = __hmul2(v, s2);                                          // one rounding: fp16(code * scale)
  return *reinterpret_cast<const uint32_t*>(&v);
}

template <int TN>
__global__ void __launch_bounds__(kThreads, 1)
gemm_a16w4_kernel(const uint8_t* __restrict__ w_packed, const __grid_constant__ CUtensorMap tm_x,
                  const __grid_constant__ CUtensorMap tm_y, int bulk_store, const float* r,
                  void* __restrict__ y, int y_bf16, int M, int N, int K, int row_pairs, int tok_tiles, int tok_block,
                  int split, int groups_per_split, int* status) {
  using C = Cfg<TN>;
  constexpr int kIssuers = C::kIssuers;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* full_p = reinterpret_cast<uint64_t*>(smem + C::kOffBar);
  uint64_t* empty_p = full_p + C::SP;
  uint64_t* full_x = empty_p + C::SP;      // (even CTA) both CTAs' activations of a group have landed
  uint64_t* empty_x = full_x + C::SX;
  uint64_t* a_full = empty_x + C::SX;      // (even CTA) both CTAs' weights of a group are expanded
  uint64_t* a_free = a_full + C::NA;
  uint64_t* acc_full = a_free + C::NA;
  uint64_t* acc_empty = acc_full + C::kAccTiles;  // (even CTA)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + C::kAccTiles);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int lane = tid & 31;
  const uint32_t crank = cluster_ctarank();
  const uint32_t even = crank & ~1u;                 // the pair's even CTA
  const int rank = static_cast<int>(crank & 1u);
  const int total_groups = K / kGroup;
  // split == 1: persistent pairs over the tiles; else one tile per cluster, pair s of it takes a slice of K
  const int pair = split == 1 ? static_cast<int>(blockIdx.x) >> 1 : static_cast<int>(blockIdx.x) / (2 * split);
  const int pairs = split == 1 ? static_cast<int>(gridDim.x) >> 1 : static_cast<int>(gridDim.x) / (2 * split);
  const int g_begin = split == 1 ? 0 : static_cast<int>(crank >> 1) * groups_per_split;
  int ng = total_groups - g_begin;
  if (ng > groups_per_split) ng = groups_per_split;
  if (ng < 0) ng = 0;
  const int row_tiles = (N + kBN - 1) / kBN;
  const int total_tiles = row_pairs * tok_tiles;
  const int my_tiles = (total_tiles - pair + pairs - 1) / pairs;
  // token tiles in blocks whose activations stay in L2 while every row pair passes over them, tokens fastest
  const int full_block = tok_block * row_pairs;
  auto tile_of = [&](int it, int& row, int& tok) {
    const int t = pair + it * pairs;
    const int b = t / full_block, rem = t - b * full_block;
    const int width = (tok_tiles - b * tok_block < tok_block) ? (tok_tiles - b * tok_block) : tok_block;
    const int rp = rem / width;
    tok = b * tok_block + (rem - rp * width);
    row = 2 * rp + rank;
  };

  if (tid == 0) {
    for (int i = 0; i < C::SP; ++i) { mbar_init(&full_p[i], 1); mbar_init(&empty_p[i], kUnpackWarps); }
    for (int i = 0; i < C::SX; ++i) { mbar_init(&full_x[i], 1); mbar_init(&empty_x[i], 1); }
    for (int i = 0; i < C::NA; ++i) { mbar_init(&a_full[i], 2 * kUnpackWarps); mbar_init(&a_free[i], 1); }
    for (int i = 0; i < C::kAccTiles; ++i) { mbar_init(&acc_full[i], kIssuers); mbar_init(&acc_empty[i], 2 * kEpiWarps); }
    *abort_flag = (smem_u32(smem) & 1023u) != 0 ? ASITE_ALIGN : 0;  // the swizzle needs 1 KB boundaries: nothing runs then
    fence_mbar_init();
  }
  if (warp == kIssuerWarp) {
    tmem_alloc_pair(tmem_slot, 512);
    tmem_relinquish_pair();
  }
  if (warp == kProducerWarp && lane == 0) {
    tma_prefetch_desc(&tm_x);
    if (bulk_store) tma_prefetch_desc(&tm_y);
  }
  // The next kernel starts early at any number of tokens: in a chain of linears that is worth 7 to 17 % up to 16 tokens
  // (4096 -> 4096 11.2 -> 9.3 us) and 0 to 3 % from 128 to 4096 (4096 -> 28672 at 512 tokens 89.8 us either way):
  // the CTAs that wait during the K loop are those of the next pre-pass, at most eight per SM.
  grid_dep_launch_dependents();
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the peers' barriers are initialised before anything arrives on them
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  const uint32_t a_base = tmem_base + C::kAccCols;
  const bool live = *abort_flag == 0;

  if (warp < kEpiWarp) {
    // ------------------------------------------------------------------ unpack
    const int q = warp & 3, h = (warp >> 2) & 1;
    const int row = q * 32 + lane;
    const uint32_t t_lane = a_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(h * 32);
    const uint32_t a_full_addr = dsmem_map(smem_u32(a_full), even);
    const int total = live ? my_tiles * ng : 0;
    // chunk positions inside the packed row are swizzled by (row >> 1) & 3
    const int at0 = row * 64 + (((2 * h) ^ ((row >> 1) & 3)) << 4), at1 = row * 64 + (((2 * h + 1) ^ ((row >> 1) & 3)) << 4);
    for (int gi = warp >> 3; gi < total; gi += kSets) {
      const int sp = gi % C::SP, ab = gi % C::NA;
      if (!mbar_wait(&full_p[sp], (gi / C::SP) & 1, abort_flag, ASITE_UNPACK)) break;
      const uint8_t* tile = smem + C::kOffP + sp * kTileBytes;
      const uint4 w0 = *reinterpret_cast<const uint4*>(tile + at0), w1 = *reinterpret_cast<const uint4*>(tile + at1);
      const __half2 s2 = __half2half2(reinterpret_cast<const __half*>(tile + kTileCodeBytes)[row]);
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty_p[sp]);
      uint32_t v[32];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const uint4 w = c ? w1 : w0;
        const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          // low nibbles: k = 4 j + {0, 2}, {1, 3} of the chunk's first half; high nibbles: of its second
          v[16 * c + 2 * j] = nib2_to_f16x2(ww[j], s2);
          v[16 * c + 2 * j + 1] = nib2_to_f16x2(ww[j] >> 8, s2);
          v[16 * c + 8 + 2 * j] = nib2_to_f16x2(ww[j] >> 4, s2);
          v[16 * c + 8 + 2 * j + 1] = nib2_to_f16x2(ww[j] >> 12, s2);
        }
      }
      if (!mbar_wait(&a_free[ab], ((gi / C::NA) & 1) ^ 1, abort_flag, ASITE_UNPACK)) break;
      tc_fence_after();
      tmem_st_x32(t_lane + static_cast<uint32_t>(ab * kACols), v);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(a_full_addr + static_cast<uint32_t>(ab) * 8u);
    }
  } else if (warp < kProducerWarp) {
    // ------------------------------------------------------------------ epilogue
    const int q = warp & 3;
    const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
    const uint32_t acc_empty_addr = dsmem_map(smem_u32(acc_empty), even);
    const bool leader = warp == kEpiWarp && lane == 0;
    const bool second = kIssuers == 2 && ng > 1;  // both issuers had groups of a tile to add up
    int chunk_no = 0;
    grid_dep_wait();  // what last used y may still be running
    for (int it = 0; it < my_tiles && live; ++it) {
      int row_tile, tok_tile;
      tile_of(it, row_tile, tok_tile);
      const int n = row_tile * kBN + q * 32 + lane, t0 = tok_tile * TN;
      const int cols = M - t0 < TN ? (M - t0 + 31) & ~31 : TN;
      const float rn = (n < N && r != nullptr) ? r[n] : 1.f;
      const int set = it % C::kAccTiles;
      const int only = (kIssuers == 2 && ng == 1) ? it & 1 : 0;  // a tile's only group is in the accumulator of its issuer
      if (TN <= 64 ? !mbar_wait(&acc_full[set], (it / C::kAccTiles) & 1, abort_flag, ASITE_EPI)
                   : !mbar_wait_relaxed(&acc_full[set], (it / C::kAccTiles) & 1, abort_flag, ASITE_EPI))
        break;
      tc_fence_after();
#pragma unroll 1
      for (int c0 = 0; c0 < cols; c0 += 32) {
        float v[32];
        {
          uint32_t u[32];
          const uint32_t at = t_lane + static_cast<uint32_t>((set * kIssuers + only) * TN + c0);
          tmem_ld_x32(at, u);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = ng > 0 ? __uint_as_float(u[j]) : 0.f;
          if (second) {
#pragma unroll
            for (int b = 0; b < 32; b += 16) {
              uint32_t u2[16];
              tmem_ld_x16(at + TN + b, u2);
              tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 16; ++j) v[b + j] += __uint_as_float(u2[j]);
            }
          }
        }
        if (c0 + 32 >= cols) {  // the accumulator goes back before its last columns are stored
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(acc_empty_addr + static_cast<uint32_t>(set) * 8u);
        }
        if (split > 1) {
          // partial tile -> this CTA's exchange buffer [token][row] over the idle activation ring
          float* red = reinterpret_cast<float*>(smem);
#pragma unroll
          for (int j = 0; j < 32; ++j) red[(c0 + j) * kBN + q * 32 + lane] = v[j];
        } else if (bulk_store) {
          uint8_t* buf = smem + C::kOffOut + (chunk_no & 1) * kOutChunk;
          ++chunk_no;
          // at most one store is outstanding, so the buffer of the chunk before the last has been read
          if (leader) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
          asm volatile("bar.sync 1, 128;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            if (y_bf16)
              reinterpret_cast<__nv_bfloat16*>(buf)[j * kBN + q * 32 + lane] = __float2bfloat16_rn(v[j] * rn);
            else
              reinterpret_cast<float*>(buf)[j * kBN + q * 32 + lane] = v[j] * rn;
          }
          fence_proxy_async_smem();
          asm volatile("bar.sync 1, 128;" ::: "memory");
          if (leader) {
            if (row_tile < row_tiles) tma_store_2d(&tm_y, buf, row_tile * kBN, t0 + c0);
            bulk_commit_group();
          }
        } else if (n < N) {
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (t0 + c0 + j < M) store_y(y, Addend{}, y_bf16, t0 + c0 + j, n, N, v[j] * rn);
        }
      }
    }
    if (leader) bulk_wait_group_read0();
  } else if (warp == kProducerWarp) {
    // ------------------------------------------------------------------ activations (both CTAs)
    // An elected lane, here and for the weights: descriptors and barrier arithmetic stay in uniform registers.  Against a
    // test of the lane number, us before / after: 8 x 4096 -> 4096 9.0 / 8.5, 16 x 4096 -> 28672 24.3 / 22.8, 100 x 4096 ->
    // 6144 15.9 / 15.0, 300 x 4096 -> 4096 19.4 / 19.5; from 512 tokens on, at the power cap, equal.
    if (live && elect_one()) {
      const uint64_t pol_x = l2_policy_evict_last();
      const uint32_t full_x_addr = dsmem_map(smem_u32(full_x), even);
      grid_dep_wait();
      int sx = 0;
      uint32_t ph = 1;
      bool ok = true;
      for (int it = 0; it < my_tiles && ok; ++it) {
        int row_tile, tok_tile;
        tile_of(it, row_tile, tok_tile);
        const int t0 = tok_tile * TN + rank * (TN / 2);
        for (int i = 0; i < ng; ++i) {
          if (!mbar_wait(&empty_x[sx], ph, abort_flag, ASITE_TMA)) { ok = false; break; }
          if (rank == 0) mbar_expect_tx(&full_x[sx], 2 * C::kXStage);
          uint8_t* xs = smem + C::kOffX + sx * C::kXStage;
          const int kx = (g_begin + i) * 256;
          tma_load_2d_pair(xs, &tm_x, kx, t0, full_x_addr + static_cast<uint32_t>(sx) * 8u, pol_x);
          tma_load_2d_pair(xs + C::kXAtom, &tm_x, kx + 128, t0, full_x_addr + static_cast<uint32_t>(sx) * 8u, pol_x);
          if (++sx == C::SX) { sx = 0; ph ^= 1u; }
        }
      }
    }
  } else if (warp == kWeightWarp) {
    // ------------------------------------------------------------------ packed weights (both CTAs): they do not depend
    // on the kernel before this one, so the ring fills while that one is still running
    if (live && elect_one()) {
      const uint64_t pol_w = tok_tiles == 1 ? l2_policy_evict_first() : l2_policy_evict_last();
      int sp = 0;
      uint32_t ph = 1;
      bool ok = true;
      for (int it = 0; it < my_tiles && ok; ++it) {
        int row_tile, tok_tile;
        tile_of(it, row_tile, tok_tile);
        if (row_tile >= row_tiles) row_tile = row_tiles - 1;  // computed and not stored
        const uint8_t* src = w_packed + (static_cast<size_t>(row_tile) * total_groups + g_begin) * kTileBytes;
        for (int i = 0; i < ng; ++i, src += kTileBytes) {
          if (!mbar_wait(&empty_p[sp], ph, abort_flag, ASITE_TMA)) { ok = false; break; }
          mbar_expect_tx(&full_p[sp], kTileBytes);
          bulk_load_1d(smem + C::kOffP + sp * kTileBytes, src, kTileBytes, &full_p[sp], pol_w);
          if (++sp == C::SP) { sp = 0; ph ^= 1u; }
        }
      }
    }
  } else if (warp < kIssuerWarp + kIssuers && rank == 0 && live) {
    // ------------------------------------------------------------------ UMMA issue, for both CTAs (whole warp, one lane acts)
    constexpr uint32_t idesc = idesc_f16(2 * kBN, TN);
    const int mine = warp - kIssuerWarp;
    bool ok = true;
    for (int it = 0; it < my_tiles && ok; ++it) {
      const int set = it % C::kAccTiles;
      const uint32_t d_tmem = tmem_base + static_cast<uint32_t>((set * kIssuers + mine) * TN);
      ok = __all_sync(0xffffffffu, mbar_wait(&acc_empty[set], ((it / C::kAccTiles) & 1) ^ 1, abort_flag, ASITE_MMA));
      const int first = (mine + it * ng) & (kIssuers - 1);  // of this warp's groups in the tile: gi & 1 == mine
      for (int i = first; i < ng && ok; i += kIssuers) {
        const int gi = it * ng + i, ab = gi % C::NA, sx = gi % C::SX;
        ok = mbar_wait(&full_x[sx], (gi / C::SX) & 1, abort_flag, ASITE_MMA) &&
             mbar_wait(&a_full[ab], (gi / C::NA) & 1, abort_flag, ASITE_MMA);
        ok = __all_sync(0xffffffffu, ok);  // the warp leaves the loop together
        if (!ok) break;
        tc_fence_after();
        if (elect_one()) {
          const uint64_t db = umma_desc_k_sw128(smem_u32(smem + C::kOffX + sx * C::kXStage));
          const uint32_t at = a_base + static_cast<uint32_t>(ab * kACols);
#pragma unroll
          for (int j = 0; j < 8; ++j)  // eight K = 16 steps: 8 columns of A, 32 bytes along K of B inside an atom
            umma_f16_pair(d_tmem, at + 8 * j, db + (j >> 2) * (C::kXAtom >> 4) + 2 * (j & 3), idesc,
                          (i != first || j > 0) ? 1u : 0u);
          umma_commit_pair(&a_free[ab], even);
          umma_commit_pair(&empty_x[sx], even);
        }
        __syncwarp();
      }
      if (ok && elect_one()) umma_commit_pair(&acc_full[set], even);
      __syncwarp();
    }
  }

  __syncwarp();
  // ---------------------------------------------------------------------- split-K reduction
  if (split > 1) {
    cluster_sync_all();
    const int si = static_cast<int>(crank >> 1);
    int row_tile, tok_tile;
    tile_of(0, row_tile, tok_tile);
    const int t0 = tok_tile * TN, c4 = lane;
    const uint32_t red_base = smem_u32(smem);
    for (int tl = si + split * warp; tl < TN && t0 + tl < M; tl += split * (kThreads / 32)) {
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      const uint32_t off = static_cast<uint32_t>((tl * kBN + c4 * 4) * 4);
      for (int p = 0; p < split; ++p) {
        const float4 v = dsmem_ld_f4(dsmem_map(red_base + off, static_cast<uint32_t>(2 * p + rank)));
        acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
      }
      const float vals[4] = {acc.x, acc.y, acc.z, acc.w};
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int n = row_tile * kBN + c4 * 4 + u;
        if (n < N) store_y(y, Addend{}, y_bf16, t0 + tl, n, N, vals[u] * (r != nullptr ? r[n] : 1.f));
      }
    }
    __syncwarp();
  }
  // The CTAs leave together: until here a peer may read this CTA's operands or exchange tile and arrive on its barriers.
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == kIssuerWarp) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
  if (tid == 0 && *abort_flag != 0) atomicCAS(status, 0, *abort_flag);
}

// xs[m, k] = fp16(float(x[m, k]) * a[k]) (a may be null), saturating at the fp16 range; inside every four k the order is
// 0, 2, 1, 3 (see the unpack warps)
__global__ void __launch_bounds__(256) scale_cols_f16_kernel(const __nv_bfloat16* x, int64_t ldx,
                                                             const float* a, int M, int K,
                                                             __half* __restrict__ xs) {
  grid_dep_launch_dependents();
  grid_dep_wait();
  const int vec = K / 8;
  const int64_t total = static_cast<int64_t>(M) * vec;
  for (int64_t u = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; u < total;
       u += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int m = static_cast<int>(u / vec), kv = static_cast<int>(u % vec);
    const uint4 raw = *reinterpret_cast<const uint4*>(x + static_cast<int64_t>(m) * ldx + kv * 8);
    float av[8] = {1.f, 1.f, 1.f, 1.f, 1.f, 1.f, 1.f, 1.f};
    if (a != nullptr) {
      const float4 a0 = *reinterpret_cast<const float4*>(a + kv * 8);
      const float4 a1 = *reinterpret_cast<const float4*>(a + kv * 8 + 4);
      av[0] = a0.x; av[1] = a0.y; av[2] = a0.z; av[3] = a0.w;
      av[4] = a1.x; av[5] = a1.y; av[6] = a1.z; av[7] = a1.w;
    }
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
    float v[8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[2 * i] = fminf(fmaxf(__fmul_rn(__uint_as_float(w[i] << 16), av[2 * i]), -65504.f), 65504.f);
      v[2 * i + 1] = fminf(fmaxf(__fmul_rn(__uint_as_float(w[i] & 0xFFFF0000u), av[2 * i + 1]), -65504.f), 65504.f);
    }
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int k = 4 * (i >> 1) + (i & 1);  // (0, 2), (1, 3), (4, 6), (5, 7)
      const __half2 p = __floats2half2_rn(v[k], v[k + 2]);
      o[i] = *reinterpret_cast<const uint32_t*>(&p);
    }
    *reinterpret_cast<uint4*>(xs + static_cast<int64_t>(m) * K + kv * 8) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

template <int TN>
static int launch(const void* xs, const uint8_t* w_packed, const float* r, int M, int N, int K, void* y, int y_dtype,
                  int split, cudaStream_t stream, DeviceState* st) {
  CUtensorMap tm_x, tm_y;
  int rc = make_tmap_2d_u8(&tm_x, xs, static_cast<uint64_t>(K) * 2, M, static_cast<uint64_t>(K) * 2, 128, TN / 2,
                           CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != DQ_OK) return rc;
  const int esz = y_dtype == DQ_DTYPE_BF16 ? 2 : 4;
  const int bulk = split == 1 && (static_cast<size_t>(N) * esz) % 16 == 0 && aligned(y, 16) ? 1 : 0;
  tm_y = tm_x;  // a valid map is passed either way
  if (bulk) {
    rc = make_tmap_2d_out(&tm_y, y, esz, static_cast<uint64_t>(N), static_cast<uint64_t>(M), kBN, 32);
    if (rc != DQ_OK) return rc;
  }
  const int row_pairs = (N + 2 * kBN - 1) / (2 * kBN), tok_tiles = (M + TN - 1) / TN;
  const int tiles = row_pairs * tok_tiles, pairs = st->sm_count / 2;
  const int ng = K / kGroup, gps = (ng + split - 1) / split;
  int tok_block = static_cast<int>((40ll << 20) / (static_cast<int64_t>(TN) * K * 2));
  if (tok_block < 1) tok_block = 1;
  if (tok_block > tok_tiles) tok_block = tok_tiles;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * (split > 1 ? tiles * split : (tiles < pairs ? tiles : pairs)), 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = Cfg<TN>::kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2 * split;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_a16w4_kernel<TN>, w_packed, tm_x, tm_y, bulk, r, y,
                                           y_dtype == DQ_DTYPE_BF16 ? 1 : 0, M, N, K, row_pairs, tok_tiles, tok_block,
                                           split, gps, st->status_dev);
  if (e != cudaSuccess)
    return set_error(DQ_ERR_CUDA, "gemm_a16w4 launch failed (TN=%d split=%d): %s", TN, split, cudaGetErrorString(e));
  return DQ_OK;
}

// Token tile and split of K: the cheapest in rounds of one tile per CTA pair.  Group times measured on B200, the wide
// tiles' in long runs at the power cap (a 256-token tile has one accumulator and waits for its drain once per tile; up to
// 64 tokens a group costs what its nibbles cost to expand).
struct Shape {
  int tn, split;
};
static Shape pick_shape(int M, int row_pairs, int ng, int sm_count) {
  static const struct { int tn; float group_us; } kTiles[] = {{256, 0.82f}, {192, 0.60f}, {128, 0.45f}, {64, 0.335f}, {32, 0.33f}};
  const int forced = tuning(DQ_TUNE_A16_TILE);
  Shape best = {256, 1};
  float best_cost = 1e30f;
  for (const auto& t : kTiles) {
    if (forced != 0 && forced % 1000 != t.tn) continue;
    const int tiles = row_pairs * ((M + t.tn - 1) / t.tn);
    for (int split = 1; split <= (t.tn <= 64 ? 4 : 1); split *= 2) {
      if (split > 1 && ng / split < 2) break;
      if (forced >= 1000 && forced / 1000 != split) continue;
      // a cluster needs its CTAs in one GPC, which leaves some SMs unused: 33 clusters of four run together, 15 of eight
      const int fit = split == 1 ? sm_count / 2 : sm_count * 17 / 20 / (2 * split);
      const int rounds = (tiles + fit - 1) / fit;
      const float cost = rounds * ((ng + split - 1) / split * t.group_us + (t.tn == 256 ? 2.0f : 1.0f) + (split > 1 ? 1.5f : 0.0f));
      if (cost < best_cost) {
        best_cost = cost;
        best = {t.tn, split};
      }
    }
  }
  return best;
}

}  // namespace a16

int init_gemm_a16w4_kernels() {
  cudaError_t e = cudaFuncSetAttribute(a16::gemm_a16w4_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       a16::Cfg<32>::kSmemBytes);
#define DQ_A16_ATTR(TN)                                                                                     \
  if (e == cudaSuccess)                                                                                     \
    e = cudaFuncSetAttribute(a16::gemm_a16w4_kernel<TN>, cudaFuncAttributeMaxDynamicSharedMemorySize,       \
                             a16::Cfg<TN>::kSmemBytes);
  DQ_A16_ATTR(64) DQ_A16_ATTR(128) DQ_A16_ATTR(192) DQ_A16_ATTR(256)
#undef DQ_A16_ATTR
  if (e != cudaSuccess)
    return set_error(DQ_ERR_CUDA, "cudaFuncSetAttribute(gemm_a16w4) failed: %s", cudaGetErrorString(e));
  return DQ_OK;
}

}  // namespace dq

using namespace dq;

extern "C" size_t dq_linear_a16w4_scratch_bytes(int M, int N, int K) {
  (void)N;
  if (M < 0 || K < 0) return 0;
  return (static_cast<size_t>(M) * static_cast<size_t>(K) * 2 + 255) / 256 * 256;
}

extern "C" int dq_linear_a16w4(const void* x_bf16, int64_t ldx, const float* a, const uint8_t* w_packed,
                               const float* r, int M, int N, int K, int G, void* y, int y_dtype,
                               void* scratch, size_t scratch_bytes, void* stream) {
  DeviceState* st = current_state();
  if (st == nullptr) return DQ_ERR_NOT_INIT;
  if (M == 0) return DQ_OK;
  DQ_REQUIRE(x_bf16 != nullptr && w_packed != nullptr && y != nullptr, DQ_ERR_NULL, "null x / w_packed / y");
  DQ_REQUIRE(G == kGroup, DQ_ERR_UNSUPPORTED, "weight group size must be %d (got %d)", kGroup, G);
  DQ_REQUIRE(M >= 1 && N >= 1 && K >= kGroup && K % kGroup == 0, DQ_ERR_SHAPE, "bad shape M=%d N=%d K=%d", M, N, K);
  DQ_REQUIRE(y_dtype == DQ_DTYPE_F32 || y_dtype == DQ_DTYPE_BF16, DQ_ERR_UNSUPPORTED, "unknown y_dtype %d", y_dtype);
  DQ_REQUIRE(aligned(x_bf16, 16) && aligned(w_packed, 16) && ldx % 8 == 0 && ldx >= K, DQ_ERR_ALIGN,
             "x and w_packed must be 16-byte aligned, ldx a multiple of 8 and >= K");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  DQ_REQUIRE(a == nullptr || aligned(a, 16), DQ_ERR_ALIGN, "a must be 16-byte aligned");
  DQ_REQUIRE(scratch != nullptr && aligned(scratch, 256), DQ_ERR_ALIGN, "scratch must be non-null and 256-byte aligned");
  DQ_REQUIRE(scratch_bytes >= dq_linear_a16w4_scratch_bytes(M, N, K), DQ_ERR_WORKSPACE,
             "scratch of %zu bytes is smaller than the %zu required", scratch_bytes,
             dq_linear_a16w4_scratch_bytes(M, N, K));
  const int64_t vecs = static_cast<int64_t>(M) * (K / 8);
  int blocks = static_cast<int>((vecs + 255) / 256);
  if (blocks > st->sm_count * 8) blocks = st->sm_count * 8;
  DQ_CHECK_CUDA(launch_pdl(a16::scale_cols_f16_kernel, dim3(blocks), dim3(256), 0, s,
                           static_cast<const __nv_bfloat16*>(x_bf16), ldx, a, M, K,
                           static_cast<__half*>(scratch)));
  const a16::Shape shape = a16::pick_shape(M, (N + 2 * a16::kBN - 1) / (2 * a16::kBN), K / kGroup, st->sm_count);
  switch (shape.tn) {
    case 32: return a16::launch<32>(scratch, w_packed, r, M, N, K, y, y_dtype, shape.split, s, st);
    case 64: return a16::launch<64>(scratch, w_packed, r, M, N, K, y, y_dtype, shape.split, s, st);
    case 128: return a16::launch<128>(scratch, w_packed, r, M, N, K, y, y_dtype, shape.split, s, st);
    case 192: return a16::launch<192>(scratch, w_packed, r, M, N, K, y, y_dtype, shape.split, s, st);
    default: return a16::launch<256>(scratch, w_packed, r, M, N, K, y, y_dtype, shape.split, s, st);
  }
}
