// The FP8-path int4 GEMM kernel (see gemm_w4a4_int4_f8.cu for the arithmetic, the operands and the dispatch), as a
// template over the token tile and the output mode.
//
// Tile: 256 weight rows x TN tokens on a PAIR of CTAs (tcgen05 cta_group::2).  Each CTA holds 128 of the rows (UMMA M
// = 256: 128 TMEM lanes in either CTA), fetches those rows of the weight and HALF of the tokens' codes, and keeps a
// TN-column accumulator for its rows.  What this buys: per weight group (128 k) a CTA moves 16 KB + TN / 2 x 128 B
// through its shared memory, once in and once out, against 16 KB + TN x 128 B for a CTA on its own (at TN = 256: 64
// instead of 96 KB a group for 512 cycles of UMMAs), and twice the rows share a fetch of the codes from L2.  Bound: in
// a long run the 1 kW power cap (8192 x 14336 -> 4096: 1.41 GHz, about 820 cycles per group, 450 us; the single-CTA
// kernel 1.53 GHz, 980 cycles, 483 us), in a short one the loop accumulator -> drain -> next UMMAs (404 us).
//
// Persistent CTAs, one per SM.  Per group: two tiled TMA copies per CTA (their bytes are counted on the even CTA's
// barrier), four UMMAs of K = 32 issued by the even CTA into accumulator g % kAccs, drained in both CTAs by eight
// epilogue warps (warp w: lanes 32 (w & 3) .., columns TN / 2 (w >> 2) ..) while the next group's UMMAs run.
//   warps 0-7   epilogue: tcgen05.ld in batches of up to 64 columns, run += acc * sw[n,g]; at the end of the tile
//               Y = run * r[n] * sx[m], see OUT below
//   warp 8      TMA producer (one lane)
//   warps 9-10  UMMA issue (one lane each, of the even CTA): alternate groups.  Waits, four UMMAs and a commit are a
//               chain of some 700 cycles for one thread, longer than the UMMAs of a group; warp 9 owns the allocation
//   warp 11     idle: registers are re-balanced per warpgroup (epilogue 232, the rest 40)
// Every barrier wait is bounded (the register re-balancing cannot block: its budgets are checked at compile time).
#pragma once
#include "dq_common.h"
#include "dq_ptx.cuh"

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <string.h>

namespace dq {
namespace f8 {

constexpr int kBN = 128;        // weight rows per CTA; a pair works on 256
constexpr int kEpiWarps = 8, kProducerWarp = 8, kIssuerWarp = 9, kIssuers = 2;
constexpr int kThreads = 384;   // padded to whole warpgroups
// setmaxnreg.inc waits (without bound) until the CTA's pool holds the registers it asks for, and the pool is what the
// launch granted (threads x registers per thread) minus what the other warps keep: the two budgets must fit into it.
constexpr int kLaunchRegs = (65536 / kThreads) / 8 * 8;
constexpr int kEpiRegs = 232, kAuxRegs = 40;
static_assert(kEpiWarps * 32 * kEpiRegs + 128 * kAuxRegs <= kThreads * kLaunchRegs, "register pool of the CTA");

constexpr int pow2_at_least(int v) { return v <= 32 ? 32 : v <= 64 ? 64 : v <= 128 ? 128 : v <= 256 ? 256 : 512; }

template <int TN>
struct Cfg {
  static_assert(TN % 32 == 0 && TN >= 32 && TN <= 256, "token tile");
  static constexpr int kABytes = kBN * kGroup;              // this CTA's 128 weight rows of one group
  static constexpr int kBBytes = TN / 2 * kGroup;           // this CTA's half of the tokens
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kOutBytes = TN * kBN * 2;            // output tile (bf16), or half of it (fp32)
  static constexpr int kFixedBytes = kOutBytes + 2 * TN * 4 + 256;
  static constexpr int kFit = (227 * 1024 - kFixedBytes) / kStageBytes;
  static constexpr int kStages = kFit < 10 ? kFit : 10;
  // accumulators: as many as fit in tensor memory, because a short tile's group takes the tensor core less time than
  // the round trip issue -> drain -> hand back
  static constexpr int kAccStride = pow2_at_least(TN);
  static constexpr int kAccs = 512 / kAccStride < 8 ? 512 / kAccStride : 8;
  static_assert(kAccs <= kStages, "see the done barriers");
  static constexpr int kTmemCols = kAccs * kAccStride;
  static constexpr int kCPW = TN / 2;                       // accumulator columns per epilogue warp
  static constexpr int kOffOut = kStages * kStageBytes;
  static constexpr int kOffSx = kOffOut + kOutBytes;        // token scales of the tile, double-buffered
  static constexpr int kOffBar = kOffSx + 2 * TN * 4;
  static constexpr int kNumBars = 2 * kStages + kAccs + 5;
  static constexpr int kSmemBytes = kOffBar + kNumBars * 8 + 16;
  static_assert(kSmemBytes <= 227 * 1024, "shared memory");
  static_assert(kStages >= 3 && kABytes % 1024 == 0 && kBBytes % 1024 == 0, "stages");
};

enum { FSITE_TMA = 61, FSITE_MMA_FULL = 62, FSITE_MMA_ACC = 63, FSITE_EPI = 64, FSITE_ALIGN = 65, FSITE_OUT = 66 };

// Instruction descriptor, kind::f8f6f4: E4M3 A and B (format code 0, both K-major), fp32 accumulator.
//   [4,6) D format (1 = F32)  [7,10) A format  [10,13) B format  [17,23) N >> 3  [24,29) M >> 4
__host__ __device__ constexpr uint32_t idesc_e4m3(int m, int n) {
  return (1u << 4) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}

__device__ __forceinline__ void umma_f8_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Destinations of the scatter output mode (OUT = 4): the partial-output buffer of every rank,
// [world][tq][N] bf16, where slot `rank` of the owner of a tile's tokens receives the tile.
struct ScatterDst {
  unsigned short* part[8];
  int rank, tq, rot;  // rot: token tiles are visited starting at tile `rot`, so that the ranks start on different owners
};

// OUT: how the output tile leaves - 0 direct stores (any shape, fp32 or bf16, optional residual or bias),
// 1 bf16 through shared memory and one tiled bulk store, 3 the same with the residual added, 5 with a bias, 2 fp32
// through shared memory in two halves, 4 bf16 through shared memory and then 16-byte stores into the partial
// buffer of the rank that owns the tile's tokens (peer memory; tensor-parallel prompt pass).  A template
// parameter: with all three epilogues in one kernel the K loop's code ran 20-25 % slower.
template <int TN, int OUT>
__global__ void __launch_bounds__(kThreads, 1) __cluster_dims__(2, 1, 1)
gemm_w4a4_e4m3_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x,
                      const __grid_constant__ CUtensorMap tm_y, const __grid_constant__ CUtensorMap tm_res,
                      const __half* __restrict__ sw_t, const float* r,
                      const float* sx, void* __restrict__ y, int y_bf16,
                      const Addend add, int M, int N, int K, int row_pairs, int tok_tiles,
                      int tok_block, int* status, const __grid_constant__ ScatterDst sc) {
  using C = Cfg<TN>;
  constexpr int bulk_out = (OUT == 3 || OUT == 5) ? 1 : OUT;  // non-zero: the tile is staged in shared memory
  constexpr int kTN = TN, kCPW = C::kCPW, kStages = C::kStages, kAccs = C::kAccs;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kOffBar);
  uint64_t* full = bars;                 // (even CTA) both CTAs' copies of a stage have landed
  // The UMMAs of the stage's group have finished: the producer may refill the stage, the epilogue may read the
  // accumulator.  One barrier for both: a group's UMMAs wait for the drain of the group kAccs before, so with kAccs <=
  // kStages no epilogue warp is a whole phase behind.
  uint64_t* done = full + kStages;
  uint64_t* acc_empty = done + kStages;    // (even CTA) both CTAs' epilogues have drained the accumulator
  uint64_t* out_free = acc_empty + kAccs;  // the output tile may be overwritten and the token scales are in place
  uint64_t* out_ready = out_free + 1;   // the output tile is written
  uint64_t* res_full = out_ready + 1;   // the residual tile has landed in the output buffer (bf16 output);
                                        // fp32 output: the first half's store has left the buffer
  uint64_t* half_ready = res_full + 1;  // [2]: fp32 output, first / second half of the tile's tokens are written
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(half_ready + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const int ng = K / kGroup;
  const int rank = static_cast<int>(cluster_ctarank());
  const int pair = static_cast<int>(blockIdx.x) >> 1, pairs = static_cast<int>(gridDim.x) >> 1;
  const int row_tiles = (N + kBN - 1) / kBN;  // of 128 rows; the last pair's odd CTA may be past them
  const int total_tiles = row_pairs * tok_tiles;
  const int my_tiles = (total_tiles - pair + pairs - 1) / pairs;
  // Tile order: token tiles in blocks of tok_block; inside a block all row pairs, tokens fastest.  The
  // CTAs running at one time then share a few weight tiles, and a block's activations (sized by the
  // host to fit in L2 next to them) are read from HBM once.
  const int full_block = tok_block * row_pairs;
  auto tile_of = [&](int it, int& row, int& tok) {
    const int t = pair + it * pairs;
    const int b = t / full_block, rem = t - b * full_block;
    const int width = (tok_tiles - b * tok_block < tok_block) ? (tok_tiles - b * tok_block) : tok_block;
    const int rp = rem / width;
    tok = b * tok_block + (rem - rp * width);
    row = 2 * rp + rank;
    if constexpr (OUT == 4) {
      tok += sc.rot;
      if (tok >= tok_tiles) tok -= tok_tiles;
    }
  };
  if (tid == 0) {
    for (int i = 0; i < kStages; ++i) { mbar_init(&full[i], 1); mbar_init(&done[i], 1); }
    for (int i = 0; i < kAccs; ++i) mbar_init(&acc_empty[i], 2 * kEpiWarps);
    mbar_init(out_free, kEpiWarps);
    mbar_init(out_ready, kEpiWarps);
    mbar_init(res_full, 1);
    mbar_init(&half_ready[0], kEpiWarps / 2);
    mbar_init(&half_ready[1], kEpiWarps / 2);
    *abort_flag = (smem_u32(smem) & 1023u) != 0 ? FSITE_ALIGN : 0;  // the swizzle needs 1 KB boundaries: nothing runs then
    fence_mbar_init();
  }
  if (warp == kIssuerWarp) {
    tmem_alloc_pair(tmem_slot, C::kTmemCols);
    tmem_relinquish_pair();
  }
  if (warp == kProducerWarp && lane == 0) {
    tma_prefetch_desc(&tm_w);
    tma_prefetch_desc(&tm_x);
    if (bulk_out && OUT != 4) tma_prefetch_desc(&tm_y);
    if (OUT == 3) tma_prefetch_desc(&tm_res);
  }
  // The next kernel may start early for batches where its launch counts; with many tokens its CTAs, one per row, resident
  // and waiting during the K loop, cost more.  Linears in a chain, with / without: 14336 -> 4096 at 384 tokens 66 / 76 us,
  // 640 76 / 84, 1023 84 / 88, 1300 129 / 130, 2048 159 / 153, 8192 572 / 547; 14336 -> 1392 at 512 57 / 58, 1024 69 / 67,
  // 4096 194 / 181; with K = 4096 within 1 % up to 8192 tokens.
  if (M < 1024) grid_dep_launch_dependents();
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the peer's barriers are initialised before anything arrives on them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const bool live = *abort_flag == 0;

  if (warp < kEpiWarps) {
    // ------------------------------------------------------------------ epilogue
    setmaxnreg_inc<kEpiRegs>();
    const int q = warp & 3, h = warp >> 2;
    const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(h * kCPW);
    const uint32_t acc_empty_addr = dsmem_map(smem_u32(acc_empty), 0);  // the even CTA's
    float run[kCPW];
    constexpr int kScaleAhead = 4;
    unsigned short sq[kScaleAhead];
    const unsigned short* sw_row = nullptr;
    // Ring positions as addresses and phases that step along: per group the loop around the FMAs is then some forty
    // instructions (index arithmetic with remainders had made it ninety, and two warps share a scheduler).
    const uint32_t done_addr = smem_u32(done), done_end = done_addr + kStages * 8;
    uint32_t done_at = done_addr, done_ph = 0, acc = 0;
    // Batches of up to 64 columns under one wait: every wait costs a full tensor-memory round trip, so the fewer per
    // group the sooner the accumulator goes back to the tensor core.
    auto group_step = [&](float s) -> bool {
      if (!mbar_wait_addr(done_at, done_ph, abort_flag, FSITE_EPI)) return false;
      tc_fence_after();
      const uint32_t t0a = t_lane + acc * C::kAccStride;
#pragma unroll
      for (int c0 = 0; c0 < kCPW; c0 += 64) {
        uint32_t v[64];
        const int width = kCPW - c0 < 64 ? kCPW - c0 : 64;  // (a constant once unrolled)
        if (width >= 32) tmem_ld_x32(t0a + static_cast<uint32_t>(c0), v);
        if (width >= 64) tmem_ld_x32(t0a + static_cast<uint32_t>(c0 + 32), v + 32);
        if (width % 32 != 0) tmem_ld_x16(t0a + static_cast<uint32_t>(c0 + width - 16), v + (width - 16));
        tmem_ld_wait();
        if (c0 + 64 >= kCPW) {  // the accumulator is free once its last column has been read
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(acc_empty_addr + acc * 8u);
          acc = (acc + 1) & (kAccs - 1);
          done_at += 8;
          if (done_at == done_end) {
            done_at = done_addr;
            done_ph ^= 1u;
          }
        }
        // Scalar FMAs: packed ones read three register pairs, and whether their banks collide was up to the register
        // allocation - from one token tile, or one unrelated line of code, to the next the K loop took 1.0 or 1.5 times
        // as long (8192 x 4096 x 14336: 435 - 600 us).  The issue slots they would save are not short here.
#pragma unroll
        for (int j = 0; j < 64; ++j)
          if (j < width) run[c0 + j] = fmaf(__uint_as_float(v[j]), s, run[c0 + j]);
      }
      return true;
    };
    bool ok = live;
    unsigned short* out_sm = reinterpret_cast<unsigned short*>(smem + C::kOffOut);
    float* sx_sm = reinterpret_cast<float*>(smem + C::kOffSx);
    constexpr bool bulk_res = (OUT == 3);
    grid_dep_wait();  // the token scales come from the kernel before this one
    for (int it = 0; it < my_tiles && ok; ++it) {
      int row_tile, tok_tile;
      tile_of(it, row_tile, tok_tile);
      const int n = row_tile * kBN + q * 32 + lane;
      const int t0 = tok_tile * kTN;
      if (bulk_out && tid < kTN) sx_sm[(it & 1) * kTN + tid] = (t0 + tid < M) ? sx[t0 + tid] : 0.f;
#pragma unroll
      for (int j = 0; j < kCPW; ++j) run[j] = 0.f;
      // (a row tile past the last one is computed on zeros and not stored: any scales will do)
      sw_row = reinterpret_cast<const unsigned short*>(sw_t) +
               static_cast<size_t>(row_tile < row_tiles ? row_tile : 0) * ng * kBN + q * 32 + lane;
#pragma unroll
      for (int d = 0; d < kScaleAhead; ++d) sq[d] = (d < ng) ? __ldg(sw_row + static_cast<size_t>(d) * kBN) : 0;
      sw_row += kScaleAhead * kBN;
      const int res_at = (ng / 2) / kScaleAhead * kScaleAhead;  // a group well after the previous tile's store
      for (int i0 = 0; i0 < ng && ok; i0 += kScaleAhead) {
        if (bulk_res && i0 == res_at && tid == 0) {
          // residual tile -> the output buffer (the previous tile's store has left it long ago)
          bulk_wait_group_read0();
          mbar_expect_tx(res_full, C::kOutBytes);
          tma_load_2d(out_sm, &tm_res, row_tile * kBN, t0, res_full, l2_policy_evict_first());
        }
#pragma unroll
        for (int u = 0; u < kScaleAhead; ++u) {
          if (ok && i0 + u < ng) {
            const float s = __half2float(__ushort_as_half(sq[u]));
            if (i0 + u + kScaleAhead < ng) sq[u] = __ldg(sw_row + u * kBN);
            ok = group_step(s);
          }
        }
        sw_row += kScaleAhead * kBN;
      }
      if (!ok) break;
      if constexpr (OUT == 4) {
        // Y tile -> shared memory as [token][row] bf16, then every warp sends 32 tokens: 256 bytes per
        // token (16 lanes x 16 bytes) into slot sc.rank of the owner's partial buffer.  The host
        // guarantees whole tiles (N % 128 == 0, M % 256 == 0) and tiles that do not straddle owners.
        __syncwarp();
        if (lane == 0) mbar_arrive(out_free);  // this warp has read its share of the previous tile
        if (!mbar_wait(out_free, it & 1, abort_flag, FSITE_OUT)) break;
        const float rn = (r != nullptr && n < N) ? r[n] : 1.f;
        const float4* sx4 = reinterpret_cast<const float4*>(sx_sm + (it & 1) * kTN + h * kCPW);
        unsigned short* dst = out_sm + (h * kCPW) * kBN + q * 32 + lane;
#pragma unroll
        for (int j = 0; j < kCPW; j += 4) {
          const float4 sv = sx4[j >> 2];
          dst[(j + 0) * kBN] = __bfloat16_as_ushort(__float2bfloat16_rn(run[j + 0] * (rn * sv.x)));
          dst[(j + 1) * kBN] = __bfloat16_as_ushort(__float2bfloat16_rn(run[j + 1] * (rn * sv.y)));
          dst[(j + 2) * kBN] = __bfloat16_as_ushort(__float2bfloat16_rn(run[j + 2] * (rn * sv.z)));
          dst[(j + 3) * kBN] = __bfloat16_as_ushort(__float2bfloat16_rn(run[j + 3] * (rn * sv.w)));
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(out_ready);
        if (!mbar_wait(out_ready, it & 1, abort_flag, FSITE_OUT)) break;
        const int owner = t0 / sc.tq;
        unsigned short* base = sc.part[owner] +
                               (static_cast<size_t>(sc.rank) * sc.tq + (t0 - owner * sc.tq)) * static_cast<size_t>(N) +
                               row_tile * kBN;
        constexpr int kTokPerWarp = kTN / kEpiWarps;
#pragma unroll 4
        for (int u = 0; u < (row_tile < row_tiles ? kTokPerWarp / 2 : 0); ++u) {
          const int tok = warp * kTokPerWarp + 2 * u + (lane >> 4);
          const uint4 v16 = *reinterpret_cast<const uint4*>(out_sm + tok * kBN + (lane & 15) * 8);
          *reinterpret_cast<uint4*>(base + static_cast<size_t>(tok) * N + (lane & 15) * 8) = v16;
        }
      } else if constexpr (OUT == 1 || OUT == 3 || OUT == 5) {
        // Y tile -> shared memory as [token][row] bf16 (a warp's 32 rows of one token are 64
        // contiguous bytes), then one tiled bulk store; rows past N and tokens past M are clipped
        // by the copy.  With a residual, its tile was copied into the same buffer during the K loop.  Two-byte global stores from here would cost more than two groups' UMMAs.
        if (tid == 0) bulk_wait_group_read0();  // the previous tile's store has left the buffer
        __syncwarp();
        if (lane == 0) mbar_arrive(out_free);
        if (!mbar_wait(out_free, it & 1, abort_flag, FSITE_OUT)) break;
        if (bulk_res && !mbar_wait(res_full, it & 1, abort_flag, FSITE_OUT)) break;
        const float rn = (r != nullptr && n < N) ? r[n] : 1.f;
        const float4* sx4 = reinterpret_cast<const float4*>(sx_sm + (it & 1) * kTN + h * kCPW);
        unsigned short* dst = out_sm + (h * kCPW) * kBN + q * 32 + lane;
        // bf16(linear) [+ residual or bias, rounded again]: what a bf16 "x = x + linear(h)" computes
        float bias = 0.f;
        if (OUT == 5 && n < N)
          bias = __uint_as_float(static_cast<uint32_t>(reinterpret_cast<const unsigned short*>(add.p)[n]) << 16);
        auto put = [&](int j, float val) {
          unsigned short bits = __bfloat16_as_ushort(__float2bfloat16_rn(val));
          if (bulk_res) {
            const float lin = __uint_as_float(static_cast<uint32_t>(bits) << 16);
            const float res = __uint_as_float(static_cast<uint32_t>(dst[j * kBN]) << 16);
            bits = __bfloat16_as_ushort(__float2bfloat16_rn(__fadd_rn(lin, res)));
          }
          if (OUT == 5)
            bits = __bfloat16_as_ushort(
                __float2bfloat16_rn(__fadd_rn(__uint_as_float(static_cast<uint32_t>(bits) << 16), bias)));
          dst[j * kBN] = bits;
        };
#pragma unroll
        for (int j = 0; j < kCPW; j += 4) {
          const float4 sv = sx4[j >> 2];
          put(j + 0, run[j + 0] * (rn * sv.x));
          put(j + 1, run[j + 1] * (rn * sv.y));
          put(j + 2, run[j + 2] * (rn * sv.z));
          put(j + 3, run[j + 3] * (rn * sv.w));
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(out_ready);
        bool stored = true;
        if (tid == 0) {
          stored = mbar_wait(out_ready, it & 1, abort_flag, FSITE_OUT);
          if (stored && row_tile < row_tiles) {
            tma_store_2d(&tm_y, out_sm, row_tile * kBN, t0);
            bulk_commit_group();
          }
        }
        ok = __all_sync(0xffffffffu, stored ? 1 : 0) != 0;  // the warp leaves the loop together
      } else if constexpr (OUT == 2) {
        // fp32 output: the buffer holds half a tile, [TN / 2 tokens][128 rows] of fp32.  The four warps
        // with the first half of the tokens stage and store first; the other four follow once that store has been
        // read.  Each half is stored by a thread of its own team, which also waits for its copy
        // before the buffer is reused.
        
        if (lane == 0 && (warp == 0 || warp == 4)) bulk_wait_group_read0();
        __syncwarp();
        if (lane == 0) mbar_arrive(out_free);
        if (!mbar_wait(out_free, it & 1, abort_flag, FSITE_OUT)) break;
        if (h == 1 && !mbar_wait(res_full, it & 1, abort_flag, FSITE_OUT)) break;
        const float rn = (r != nullptr && n < N) ? r[n] : 1.f;
        const float4* sx4 = reinterpret_cast<const float4*>(sx_sm + (it & 1) * kTN + h * kCPW);
        float* dst = reinterpret_cast<float*>(out_sm) + q * 32 + lane;
#pragma unroll
        for (int j = 0; j < kCPW; j += 4) {
          const float4 sv = sx4[j >> 2];
          dst[(j + 0) * kBN] = run[j + 0] * (rn * sv.x);
          dst[(j + 1) * kBN] = run[j + 1] * (rn * sv.y);
          dst[(j + 2) * kBN] = run[j + 2] * (rn * sv.z);
          dst[(j + 3) * kBN] = run[j + 3] * (rn * sv.w);
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&half_ready[h]);
        bool stored = true;
        if (lane == 0 && (warp == 0 || warp == 4)) {
          stored = mbar_wait(&half_ready[h], it & 1, abort_flag, FSITE_OUT);
          if (stored) {
            if (row_tile < row_tiles && t0 + h * kCPW < M) {
              tma_store_2d(&tm_y, out_sm, row_tile * kBN, t0 + h * kCPW);
              bulk_commit_group();
            }
            if (h == 0) {
              bulk_wait_group_read0();
              mbar_arrive(res_full);  // the second half may overwrite the buffer
            }
          }
        }
        ok = __all_sync(0xffffffffu, stored ? 1 : 0) != 0;
      } else if (n < N) {  // OUT == 0
        const float rn = (r != nullptr) ? r[n] : 1.f;
        const int m0 = t0 + h * kCPW;
        const int cnt = (M - m0 < kCPW) ? (M - m0) : kCPW;
        const float* sxp = sx + m0;
        // A loop for each kind of result, with a pointer that steps: the address arithmetic and the tests of a common
        // one took 1.6 times the whole kernel (6124 x 2048 -> 18318, fp32: 551 us against 333).
        if (add.p != nullptr) {
#pragma unroll
          for (int j = 0; j < kCPW; ++j)
            if (j < cnt) store_y(y, add, y_bf16, m0 + j, n, N, run[j] * (rn * __ldg(sxp + j)));
        } else if (y_bf16) {
          __nv_bfloat16* yp = reinterpret_cast<__nv_bfloat16*>(y) + static_cast<size_t>(m0) * N + n;
#pragma unroll
          for (int j = 0; j < kCPW; ++j) {
            if (j < cnt) *yp = __float2bfloat16_rn(run[j] * (rn * __ldg(sxp + j)));
            yp += N;
          }
        } else {
          float* yp = reinterpret_cast<float*>(y) + static_cast<size_t>(m0) * N + n;
#pragma unroll
          for (int j = 0; j < kCPW; ++j) {
            if (j < cnt) *yp = run[j] * (rn * __ldg(sxp + j));
            yp += N;
          }
        }
      }
    }
    if constexpr (OUT == 4) __threadfence_system();  // this thread's stores to peers are performed before the kernel ends
    if (bulk_out && OUT != 4 && lane == 0 && (warp == 0 || warp == 4)) bulk_wait_group_read0();
  } else {
    setmaxnreg_dec<kAuxRegs>();
    if (warp == kProducerWarp) {
      // ---------------------------------------------------------------- TMA producer (both CTAs)
      if (elect_one()) {
        const uint64_t pol = l2_policy_evict_last();
        const uint32_t full_addr = dsmem_map(smem_u32(full), 0);  // the even CTA's
        grid_dep_wait();  // operands may come from the kernels just before this one
        bool ok = live;
        int gi = 0;
        for (int it = 0; it < my_tiles && ok; ++it) {
          int row_tile, tok_tile;
          tile_of(it, row_tile, tok_tile);
          const int n0 = row_tile * kBN, t0 = tok_tile * kTN + rank * (kTN / 2);
          for (int i = 0; i < ng; ++i, ++gi) {
            const int s = gi % kStages;
            if (!mbar_wait(&done[s], ((gi / kStages) & 1) ^ 1, abort_flag, FSITE_TMA)) { ok = false; break; }
            if (rank == 0) mbar_expect_tx(&full[s], 2 * C::kStageBytes);
            uint8_t* st = smem + s * C::kStageBytes;
            tma_load_2d_pair(st, &tm_w, i * kGroup, n0, full_addr + static_cast<uint32_t>(s) * 8u, pol);
            tma_load_2d_pair(st + C::kABytes, &tm_x, i * kGroup, t0, full_addr + static_cast<uint32_t>(s) * 8u, pol);
          }
        }
      }
    } else if (warp >= kIssuerWarp && warp < kIssuerWarp + kIssuers && rank == 0) {
      // ---------------------------------------------------------------- UMMA issue, for both CTAs
      if (elect_one() && live) {
        constexpr uint32_t idesc = idesc_e4m3(2 * kBN, kTN);
        const int my_groups = my_tiles * ng;
        for (int gi = warp - kIssuerWarp; gi < my_groups; gi += kIssuers) {
          const int s = gi % kStages, b = gi % kAccs;
          const uint32_t a_addr = smem_u32(smem + s * C::kStageBytes);
          const uint64_t da = umma_desc_k_sw128(a_addr);
          const uint64_t db = umma_desc_k_sw128(a_addr + C::kABytes);
          // operands first: they are there long before the accumulator comes back, on the critical path of a wide tile
          if (!mbar_wait(&full[s], (gi / kStages) & 1, abort_flag, FSITE_MMA_FULL)) break;
          if (!mbar_wait(&acc_empty[b], ((gi / kAccs) & 1) ^ 1, abort_flag, FSITE_MMA_ACC)) break;
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(b * C::kAccStride);
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) umma_f8_pair(d_tmem, da + 2 * kk, db + 2 * kk, idesc, kk > 0 ? 1u : 0u);
          umma_commit_pair(&done[s]);
        }
      }
    }
  }

  // Both CTAs leave together: until here the peer may read this CTA's operands and arrive on its barriers.
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == kIssuerWarp) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, C::kTmemCols);
  }
  if (tid == 0 && *abort_flag != 0) atomicCAS(status, 0, *abort_flag);
}

// Arguments of a launch, the same for every instantiation.
struct Launch {
  CUtensorMap tm_w, tm_x, tm_y, tm_res;
  const __half* sw_t;
  const float *r, *sx;
  void* y;
  int y_bf16;
  Addend add;
  int M, N, K, row_pairs, tok_tiles, tok_block;
  int* status;
  ScatterDst sc;
  int ctas;
  cudaStream_t stream;
};
template <int TN, int OUT>
cudaError_t run(const Launch& l) {
  return launch_pdl(gemm_w4a4_e4m3_kernel<TN, OUT>, dim3(l.ctas), dim3(kThreads), Cfg<TN>::kSmemBytes, l.stream, l.tm_w,
                    l.tm_x, l.tm_y, l.tm_res, l.sw_t, l.r, l.sx, l.y, l.y_bf16, l.add, l.M, l.N, l.K, l.row_pairs,
                    l.tok_tiles, l.tok_block, l.status, l.sc);
}
template <int TN, int OUT>
cudaError_t allow_smem() {
  return cudaFuncSetAttribute(gemm_w4a4_e4m3_kernel<TN, OUT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              Cfg<TN>::kSmemBytes);
}

}  // namespace f8
}  // namespace dq
