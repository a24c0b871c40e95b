// Block-scaled FP4 W4A4 GEMM for prefill-size batches: the persistent form of gemm_fp4_kernel, on CTA pairs.
//
//   Y[m,n] = r[n] * tw * tx[m] * sum_k ( qx[m,k] * sfx[m, k/B] ) * ( qw[n,k] * sfw[n, k/B] )
//
// Tile: 256 weight rows x 256 tokens on a pair of CTAs (tcgen05 cta_group::2, kind::mxf4nvf4.block_scale, K = 64 a UMMA).
// Each CTA holds 128 of the rows and fetches HALF of the tokens' codes, so that a stage of 256 k is 38 KB instead of the
// 54 KB of a CTA on its own: less to move through shared memory, and four or five stages in flight instead of three.  A
// stage's round trip - copies, scale factors to tensor memory, UMMAs, refill - takes about 1.9 us, and with three of them
// it was the copies in flight that set the pace (0.62 us a stage where the UMMAs take 0.28).  The sums are formed by the
// same instructions in the same order as in the one-tile-per-CTA kernel; results are equal.
// Against single CTAs with three stages (bf16 out, cold L2, us): MXFP4 4096 x 3584 -> 37888 260 -> 211 (5.3 PFLOPS), 4096 x
// 18944 -> 3584 144 -> 109; NVFP4 147 -> 114, 8192 x 3584 -> 18944 341 -> 223.  Long runs of it meet the 1 kW power cap.
//
// One CTA per SM walks over tiles; the producer, the scale-factor copiers and the rings they feed never stop at a tile
// boundary, so the next tile's operands are in shared memory while the accumulator of the finished one is drained (eight
// epilogue warps: tensor memory -> registers -> [token][row] chunks in shared memory -> tiled bulk stores).
//
//   warp 0       TMA producer (one lane), both CTAs; the bytes of both are counted on the even CTA's barrier
//   warp 1       UMMA issue for the pair (one lane of the even CTA); owns the tensor-memory allocation in each CTA
//   warps 2, 3   even CTA: scale factors shared -> tensor memory of both CTAs (tcgen05.cp), half of the copies each (a copy
//                costs its thread ~70 cycles of issue)
//   warps 4-11   epilogue, two teams of four (one warp per TMEM lane quarter), alternate 32-token chunks; a warp first moves
//                all its columns to registers and hands the accumulator back, then converts and stores while the next
//                tile's UMMAs run
// Every barrier wait is bounded.
#include "dq_common.h"
#include "dq_ptx.cuh"
#include "gemm_fp4.cuh"

#include <cuda_bf16.h>
#include <string.h>

namespace dq {
namespace fp4p {

constexpr int kTok = 256;
constexpr int kBBytes = kTok / 2 * 128;  // this CTA's half of the tokens
constexpr int kMaxStages = 5;
constexpr int kThreads = 384;  // twelve warps: registers are granted to warps in fours, 168 per thread at this size
constexpr int kSfColsStage = 48;  // 16 columns of weight scale factors, 2 x 16 of activation scale factors
constexpr int kSfColBase = kTok;
constexpr uint32_t kTmemCols = 512;
constexpr int kNumBars = 3 * kMaxStages + 2;
static_assert(kSfColBase + kMaxStages * kSfColsStage <= 512, "tensor memory columns");

// bf16 output: a chunk of 32 tokens takes 8 KB of the store buffers instead of 16, which is room for a fifth stage
template <bool BF16>
struct PCfg {
  static constexpr int kStages = BF16 ? 5 : 4;
  static constexpr int kOffA = 0;
  static constexpr int kOffB = kOffA + kStages * kFTileBytes;
  static constexpr int kOffSFA = kOffB + kStages * kBBytes;
  static constexpr int kOffSFB = kOffSFA + kStages * 2048;
  static constexpr int kOffOut = kOffSFB + kStages * 2 * 2048;
  static constexpr int kOutBuf = 32 * kFBN * (BF16 ? 2 : 4);  // one chunk: 32 tokens x 128 rows
  static constexpr int kOffBar = kOffOut + 4 * kOutBuf;
  static constexpr int kSmemBytes = kOffBar + kNumBars * 8 + 16;
  static_assert(kSmemBytes <= 227 * 1024 && kStages <= kMaxStages, "shared memory");
  static_assert(kOffB % 1024 == 0 && kOffOut % 1024 == 0, "operand tiles on 1 KB boundaries");
};

enum { PSITE_TMA = 71, PSITE_MMA = 72, PSITE_SF = 73, PSITE_EPI = 74, PSITE_ACC = 75, PSITE_ALIGN = 76 };

__device__ __forceinline__ void bulk_wait_group_read1() {
  asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
}

__device__ __forceinline__ void tma_load_3d_pair(void* smem_dst, const CUtensorMap* tm, int x, int y, int z,
                                                 uint32_t bar_addr, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2.L2::cache_hint"
      " [%0], [%1, {%2, %3, %4}], [%5], %6;" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(tm)), "r"(x), "r"(y), "r"(z), "r"(bar_addr), "l"(policy)
      : "memory");
}
// One scale-factor atom from the shared memory of each CTA of the pair to its tensor memory (same offsets in both)
__device__ __forceinline__ void tmem_cp_pair(uint32_t taddr, uint64_t sdesc) {
  asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(sdesc) : "memory");
}
// Completes `bar` of this CTA once the copies issued so far by this thread have finished in both CTAs
__device__ __forceinline__ void umma_commit_pair_here(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
template <int NVFP4>
__device__ __forceinline__ void umma_fp4_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t sfa,
                                              uint32_t sfb, uint32_t accumulate) {
  if constexpr (NVFP4) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %6, 0;\n"
        "tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], %1, %2, %3, [%4], [%5], p;\n}\n" ::
            "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(sfa), "r"(sfb), "r"(accumulate)
        : "memory");
  } else {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %6, 0;\n"
        "tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.scale_vec::2X [%0], %1, %2, %3, [%4], [%5], p;\n}\n" ::
            "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(sfa), "r"(sfb), "r"(accumulate)
        : "memory");
  }
}

// The tiles of a launch: `full` tiles of 256 tokens, then, where the last round would keep few of the pairs busy, its
// tiles as halves of 128 tokens on twice as many pairs.  Token tiles in blocks of tok_block; inside a block all row pairs,
// tokens fastest: the pairs running at one time share a few weight tiles and a block's activations stay in L2.
struct Tiles {
  int row_pairs, tok_tiles, tok_block, full, units;
};

// BIAS is a template parameter: tested at run time in the epilogue it made the kernel 6 % (MXFP4) to 19 % (NVFP4) slower.
template <int NVFP4, bool BIAS, bool BF16>
__global__ void __launch_bounds__(kThreads, 1) __cluster_dims__(2, 1, 1)
gemm_fp4_persist_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x,
                        const __grid_constant__ CUtensorMap tm_y, const __grid_constant__ CUtensorMap tm_sfw,
                        const __grid_constant__ CUtensorMap tm_sfx, const float* r,
                        const float* w_scale, const float* x_scale, const void* bias,
                        int M, int N, int K, const Tiles tiles, int* status) {
  using C = PCfg<BF16>;
  constexpr int kStages = C::kStages;
  constexpr int kAtoms = NVFP4 ? 4 : 2;  // scale-factor atoms per operand block per stage
  constexpr uint32_t kSfBytes = kAtoms * 512;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + C::kOffBar);  // (even CTA) both CTAs' copies of a stage have landed
  uint64_t* empty = full + kMaxStages;        // the stage's UMMAs have finished
  uint64_t* sf_ready = empty + kMaxStages;    // (even CTA) the stage's scale factors are in both tensor memories
  uint64_t* acc_full = sf_ready + kMaxStages;
  uint64_t* acc_empty = acc_full + 1;         // (even CTA) both CTAs' epilogues have read the accumulator
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = static_cast<int>(cluster_ctarank());
  const int pair = static_cast<int>(blockIdx.x) >> 1, pairs = static_cast<int>(gridDim.x) >> 1;
  const int nst = K / kFKStage;
  const int my_tiles = (tiles.units - pair + pairs - 1) / pairs;
  const int full_block = tiles.tok_block * tiles.row_pairs;
  auto tile_of = [&](int it, int& row, int& t0, int& toks) {
    int t = pair + it * pairs, half = 0;
    toks = kTok;
    if (t >= tiles.full) {
      const int h = t - tiles.full;
      t = tiles.full + (h >> 1);
      half = h & 1;
      toks = kTok / 2;
    }
    const int b = t / full_block, rem = t - b * full_block;
    const int left = tiles.tok_tiles - b * tiles.tok_block, width = left < tiles.tok_block ? left : tiles.tok_block;
    const int rp = rem / width;
    row = 2 * rp + rank;
    t0 = (b * tiles.tok_block + (rem - rp * width)) * kTok + half * (kTok / 2);
  };

  if (tid == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
      mbar_init(&sf_ready[i], 2);
    }
    mbar_init(acc_full, 1);
    mbar_init(acc_empty, 16);  // the eight epilogue warps of both CTAs
    *abort_flag = (smem_u32(smem) & 1023u) != 0 ? PSITE_ALIGN : 0;  // the swizzle needs 1 KB boundaries: nothing runs then
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, kTmemCols);
    tmem_relinquish_pair();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tm_w);
    tma_prefetch_desc(&tm_x);
    tma_prefetch_desc(&tm_y);
    tma_prefetch_desc(&tm_sfw);
    tma_prefetch_desc(&tm_sfx);
  }
  // No early start for the kernel behind this one: the next quantiser's CTAs, resident and waiting during the K loop, cost
  // more than the launch they hide (NVFP4 linears on single CTAs, us with / without: 3294 x 4096 -> 11968 131 / 126, 8192 x
  // 3584 -> 18944 362 / 341, 8192 x 3584 -> 37888 667 / 616; on pairs, chains of linears at 640 to 1000 tokens: up to 10 %
  // slower, 1.5 % on average, NVFP4 1000 x 4096 -> 4096 26.0 / 23.7).  Up to 511 tokens it would gain 3 to 6 % on average (MXFP4
  // 256 x 4096 -> 4096 11.6 / 12.8) and lose 4 % at worst.
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the peer's barriers are initialised before anything arrives on them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const bool live = *abort_flag == 0;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (both CTAs)
    if (elect_one() && live) {
      const uint64_t pol = l2_policy_evict_last();
      const uint32_t full_addr = dsmem_map(smem_u32(full), 0);  // the even CTA's
      grid_dep_wait();  // the activation codes and scale factors come from the kernel before this one
      int s = 0;
      uint32_t ph = 1;
      bool ok = true;
      for (int it = 0; it < my_tiles && ok; ++it) {
        int row_tile, t0, toks;
        tile_of(it, row_tile, t0, toks);
        const int n0 = row_tile * kFBN, x0 = t0 + rank * (toks / 2);
        for (int i = 0; i < nst; ++i) {
          if (!mbar_wait(&empty[s], ph, abort_flag, PSITE_TMA)) { ok = false; break; }
          // the boxes are whole (a half tile uses half of them; what lies outside the tensors arrives as zeros and counts)
          if (rank == 0) mbar_expect_tx(&full[s], 2 * (kFTileBytes + kBBytes + 3 * kSfBytes));
          const uint32_t bar = full_addr + static_cast<uint32_t>(s) * 8u;
          tma_load_2d_pair(smem + C::kOffA + s * kFTileBytes, &tm_w, i * 128, n0, bar, pol);
          tma_load_2d_pair(smem + C::kOffB + s * kBBytes, &tm_x, i * 128, x0, bar, pol);
          tma_load_3d_pair(smem + C::kOffSFA + s * 2048, &tm_sfw, 0, i * kAtoms, row_tile, bar, pol);
          tma_load_3d_pair(smem + C::kOffSFB + s * 4096, &tm_sfx, 0, i * kAtoms, t0 / kFTN, bar, pol);
          if (++s == kStages) { s = 0; ph ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ UMMA issue, for both CTAs
    if (rank == 0 && elect_one() && live) {
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int it = 0; it < my_tiles && ok; ++it) {
        int row_tile, t0, toks;
        tile_of(it, row_tile, t0, toks);
        // the accumulator of the previous tile has been read by the epilogue warps of both CTAs
        if (!mbar_wait(acc_empty, (it & 1) ^ 1, abort_flag, PSITE_ACC)) break;
        for (int i = 0; i < nst; ++i) {
          if (!mbar_wait(&full[s], ph, abort_flag, PSITE_MMA)) { ok = false; break; }
          if (!mbar_wait(&sf_ready[s], ph, abort_flag, PSITE_MMA)) { ok = false; break; }
          tc_fence_after();
          const uint32_t sfa_t = tmem_base + kSfColBase + s * kSfColsStage;
          const uint32_t sfb_t = sfa_t + 16;
          const uint64_t da = umma_desc_k_sw128(smem_u32(smem + C::kOffA + s * kFTileBytes));
          const uint64_t db = umma_desc_k_sw128(smem_u32(smem + C::kOffB + s * kBBytes));
#pragma unroll
          for (int j = 0; j < 4; ++j) {  // four K = 64 UMMAs: +32 bytes along K each
            const int atom = NVFP4 ? j : (j >> 1);
            const uint32_t sf_id = NVFP4 ? 0u : static_cast<uint32_t>((j & 1) * 2);
            const uint32_t idesc = umma_idesc_fp4(2 * kFBN, toks, NVFP4 ? 0 : 1, sf_id);
            umma_fp4_pair<NVFP4>(tmem_base, da + 2 * j, db + 2 * j, idesc, sfa_t + 4 * atom, sfb_t + 8 * atom,
                                 (i > 0 || j > 0) ? 1u : 0u);
          }
          umma_commit_pair(&empty[s]);
          if (i == nst - 1) umma_commit_pair(acc_full);
          if (++s == kStages) { s = 0; ph ^= 1u; }
        }
      }
    }
  } else if (warp < 4) {
    // ------------------------------------------------------------------ scale-factor copiers, for both CTAs
    // warp 2: weights and the first half of activation rows 0-127; warp 3: the other half and activation rows 128-255
    if (rank == 0 && elect_one() && live) {
      const bool second = (warp == 3);
      const int total = my_tiles * nst;
      int s = 0;
      uint32_t ph = 0;
      for (int gi = 0; gi < total; ++gi) {
        if (!mbar_wait(&full[s], ph, abort_flag, PSITE_SF)) break;
        tc_fence_after();
        const uint32_t sf_t = tmem_base + kSfColBase + s * kSfColsStage;
        const uint64_t src_a = sf_atom_desc(smem_u32(smem + C::kOffSFA + s * 2048));
        const uint64_t src_b = sf_atom_desc(smem_u32(smem + C::kOffSFB + s * 4096));
        // (descriptor addresses count 16 bytes: an atom is 32 of them, a block of 128 tokens kAtoms atoms)
        if (!second) {
#pragma unroll
          for (int at = 0; at < kAtoms; ++at) tmem_cp_pair(sf_t + 4 * at, src_a + 32 * at);
#pragma unroll
          for (int at = 0; at < kAtoms / 2; ++at) tmem_cp_pair(sf_t + 16 + 8 * at, src_b + 32 * at);
        } else {
#pragma unroll
          for (int at = kAtoms / 2; at < kAtoms; ++at) tmem_cp_pair(sf_t + 16 + 8 * at, src_b + 32 * at);
#pragma unroll
          for (int at = 0; at < kAtoms; ++at) tmem_cp_pair(sf_t + 16 + 8 * at + 4, src_b + 32 * (kAtoms + at));
        }
        umma_commit_pair_here(&sf_ready[s]);
        if (++s == kStages) { s = 0; ph ^= 1u; }
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue
    const int team = (warp - 4) >> 2;  // 0: warps 4-7, 1: warps 8-11
    const int q = warp & 3;            // TMEM lane quarter
    const bool leader = (warp & 3) == 0 && lane == 0;
    const uint32_t acc_empty_addr = dsmem_map(smem_u32(acc_empty), 0);  // the even CTA's
    int chunk_no = 0;                  // chunks this team has staged so far (buffer parity)
    grid_dep_wait();  // the token scales come from the kernel before this one
    for (int it = 0; it < my_tiles && live; ++it) {
      int row_tile, t0, toks;
      tile_of(it, row_tile, t0, toks);
      const int n0 = row_tile * kFBN;
      const int n = n0 + q * 32 + lane;
      int tok_cols = M - t0;
      if (tok_cols > toks) tok_cols = toks;
      // (past the last token, or the odd CTA past the last row: the accumulator is handed back, nothing is stored)
      const int col_end = (tok_cols > 0 && n0 < N) ? (tok_cols + 31) & ~31 : 0;
      float rn = 0.f;
      if (n < N) {
        rn = (r != nullptr) ? r[n] : 1.f;
        if (w_scale != nullptr) rn *= *w_scale;
      }
      const float bias_n = BIAS && n < N ? bias_value(bias, BF16, n) : 0.f;
      if (!mbar_wait(acc_full, it & 1, abort_flag, PSITE_EPI)) break;
      tc_fence_after();
      // all of this warp's columns (up to four chunks of 32) to registers, then the accumulator
      // goes back to the tensor core
      uint32_t v[4][32];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int c0 = team * 32 + k * 64;
        if (c0 < col_end) tmem_ld_x32(tmem_base + (static_cast<uint32_t>(q * 32) << 16) + c0, v[k]);
      }
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(acc_empty_addr);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int c0 = team * 32 + k * 64;
        if (c0 < col_end) {  // uniform over the team
          uint8_t* buf = smem + C::kOffOut + (2 * team + (chunk_no & 1)) * C::kOutBuf;
          ++chunk_no;
          // the store that last used this buffer (two chunks ago) has finished reading it
          if (leader) bulk_wait_group_read1();
          if (team == 0) asm volatile("bar.sync 1, 128;" ::: "memory");
          else asm volatile("bar.sync 2, 128;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const int m = t0 + c0 + j;
            const float tx = (x_scale != nullptr && m < M) ? x_scale[m] : 1.f;
            const float val = __uint_as_float(v[k][j]) * (rn * tx);
            if constexpr (BF16)
              reinterpret_cast<__nv_bfloat16*>(buf)[j * kFBN + q * 32 + lane] = bf16_with_bias(val, BIAS ? bias : nullptr, bias_n);
            else
              reinterpret_cast<float*>(buf)[j * kFBN + q * 32 + lane] = BIAS ? __fadd_rn(val, bias_n) : val;
          }
          fence_proxy_async_smem();
          if (team == 0) asm volatile("bar.sync 1, 128;" ::: "memory");
          else asm volatile("bar.sync 2, 128;" ::: "memory");
          if (leader) {
            tma_store_2d(&tm_y, buf, n0, t0 + c0);
            bulk_commit_group();
          }
        }
      }
    }
    if (leader) bulk_wait_group_read0();
  }

  // Both CTAs leave together: until here the peer may read this CTA's operands and arrive on its barriers.
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, kTmemCols);
  }
  if (tid == 0 && *abort_flag != 0) atomicCAS(status, 0, *abort_flag);
}

}  // namespace fp4p

template <typename F>
static cudaError_t for_each_persist(F&& f) {
  cudaError_t e = f(fp4p::gemm_fp4_persist_kernel<0, false, false>, fp4p::PCfg<false>::kSmemBytes);
  if (e == cudaSuccess) e = f(fp4p::gemm_fp4_persist_kernel<1, false, false>, fp4p::PCfg<false>::kSmemBytes);
  if (e == cudaSuccess) e = f(fp4p::gemm_fp4_persist_kernel<0, true, false>, fp4p::PCfg<false>::kSmemBytes);
  if (e == cudaSuccess) e = f(fp4p::gemm_fp4_persist_kernel<1, true, false>, fp4p::PCfg<false>::kSmemBytes);
  if (e == cudaSuccess) e = f(fp4p::gemm_fp4_persist_kernel<0, false, true>, fp4p::PCfg<true>::kSmemBytes);
  if (e == cudaSuccess) e = f(fp4p::gemm_fp4_persist_kernel<1, false, true>, fp4p::PCfg<true>::kSmemBytes);
  if (e == cudaSuccess) e = f(fp4p::gemm_fp4_persist_kernel<0, true, true>, fp4p::PCfg<true>::kSmemBytes);
  if (e == cudaSuccess) e = f(fp4p::gemm_fp4_persist_kernel<1, true, true>, fp4p::PCfg<true>::kSmemBytes);
  return e;
}

int init_gemm_fp4_persist_kernels() {
  const cudaError_t e = for_each_persist([](auto kernel, int smem) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  });
  if (e != cudaSuccess)
    return set_error(DQ_ERR_CUDA, "cudaFuncSetAttribute(gemm_fp4_persist) failed: %s", cudaGetErrorString(e));
  return DQ_OK;
}

// Prefill-size batches whose output the copy engine can address; the caller has validated the operands.
int launch_gemm_fp4_persist(const uint8_t* x_codes, const uint8_t* x_sf_atoms, const float* x_scale,
                            const uint8_t* w_codes, const uint8_t* w_sf_atoms, const float* w_scale, const float* r,
                            const void* bias, int M, int N, int K, int nvfp4, void* y, int y_dtype, cudaStream_t stream,
                            DeviceState* st) {
  CUtensorMap tm_w, tm_x, tm_y, tm_sfw, tm_sfx;
  int rc = make_tmap_2d_u8(&tm_w, w_codes, static_cast<uint64_t>(K) / 2, N, static_cast<uint64_t>(K) / 2, 128, kFBN,
                           CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != DQ_OK) return rc;
  rc = make_tmap_2d_u8(&tm_x, x_codes, static_cast<uint64_t>(K) / 2, M, static_cast<uint64_t>(K) / 2, 128, fp4p::kTok / 2,
                       CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != DQ_OK) return rc;
  const bool bf = y_dtype == DQ_DTYPE_BF16;
  rc = make_tmap_2d_out(&tm_y, y, bf ? 2 : 4, static_cast<uint64_t>(N), static_cast<uint64_t>(M), kFBN, 32);
  if (rc != DQ_OK) return rc;
  const int stage_atoms = nvfp4 ? 4 : 2, tile_atoms = K / kFKStage * stage_atoms;
  rc = make_tmap_sf_atoms(&tm_sfw, w_sf_atoms, tile_atoms, (N + 127) / 128, stage_atoms, 1);
  if (rc != DQ_OK) return rc;
  rc = make_tmap_sf_atoms(&tm_sfx, x_sf_atoms, tile_atoms, (M + 127) / 128, stage_atoms, 2);
  if (rc != DQ_OK) return rc;
  fp4p::Tiles t;
  t.row_pairs = (N + 2 * kFBN - 1) / (2 * kFBN);
  t.tok_tiles = (M + fp4p::kTok - 1) / fp4p::kTok;
  const int pairs = st->sm_count / 2, all = t.row_pairs * t.tok_tiles, rest = all % pairs;
  // few tiles in the last round: twice as many half ones, in about 0.65 of the time (a half tile's copies are a whole one's)
  const bool halves = rest > 0 && 2 * rest <= pairs;
  t.full = halves ? all - rest : all;
  t.units = halves ? all + rest : all;
  // a block of token tiles whose packed activations (K / 2 bytes per token) take about 40 MB of L2
  t.tok_block = static_cast<int>((40ll << 20) / (static_cast<int64_t>(fp4p::kTok) * (K / 2)));
  if (t.tok_block < 1) t.tok_block = 1;
  if (t.tok_block > t.tok_tiles) t.tok_block = t.tok_tiles;
  const int grid = 2 * (t.units < pairs ? t.units : pairs);
#define DQ_FP4P(NV, BI, BF)                                                                                                \
  launch_pdl(fp4p::gemm_fp4_persist_kernel<NV, BI, BF>, dim3(grid), dim3(fp4p::kThreads), fp4p::PCfg<BF>::kSmemBytes,      \
             stream, tm_w, tm_x, tm_y, tm_sfw, tm_sfx, r, w_scale, x_scale, bias, M, N, K, t, st->status_dev)
#define DQ_FP4P_OUT(NV, BI) (bf ? DQ_FP4P(NV, BI, true) : DQ_FP4P(NV, BI, false))
  const cudaError_t e = nvfp4 ? (bias != nullptr ? DQ_FP4P_OUT(1, true) : DQ_FP4P_OUT(1, false))
                              : (bias != nullptr ? DQ_FP4P_OUT(0, true) : DQ_FP4P_OUT(0, false));
#undef DQ_FP4P_OUT
#undef DQ_FP4P
  if (e != cudaSuccess) return set_error(DQ_ERR_CUDA, "gemm_fp4_persist launch failed: %s", cudaGetErrorString(e));
  return DQ_OK;
}

}  // namespace dq
