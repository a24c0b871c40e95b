// Packed int4 weight tiles -> E4M3 bytes, row-major [N, K]: the operand of the FP8-path GEMM.  Device code of the kernel that
// does only this (gemm_w4a4_int4_f8.cu) and of the activation quantisers that take it along (act_quant_int4.cu).
#pragma once
#include "dq_common.h"

namespace dq {

// Four two's-complement nibbles (bits 0-15 of sel) -> four E4M3 bytes of the same integers.
// Non-negative codes 0..7: 00 38 40 44 48 4A 4C 4E; negative codes -8..-1: D0 CE CC CA C8 C4 C0 B8.
// The byte permute takes the nibbles as selectors: its low three bits look up a magnitude, and where the fourth (the
// sign) is set it replicates the sign bit of the byte looked up - so one permute over bytes of 0x80 gives 0x80 for a
// non-negative code and 0xFF for a negative one, and that selects between the two tables and makes the sign bit.
__device__ __forceinline__ uint32_t e4m3x4_of_nibbles(uint32_t sel) {
  const uint32_t s3 = sel & 0x7777u;
  const uint32_t pos = __byte_perm(0x44403800u, 0x4E4C4A48u, s3);
  const uint32_t neg = __byte_perm(0x4A4C4E50u, 0x38404448u, s3);  // magnitudes
  uint32_t r;
  asm("prmt.b32 %0, %1, %1, %2;" : "=r"(r) : "r"(0x80808080u), "r"(sel));
  return (pos & ~r) | (neg & r & 0x7F7F7F7Fu) | ((r << 7) & 0x80808080u);
}
// A packed word of the artefact (low nibbles: four consecutive k, high nibbles: the four sixteen further on) -> both fours
__device__ __forceinline__ void e4m3_of_word(uint32_t w, uint32_t& lo, uint32_t& hi) {
  const uint32_t a = e4m3x4_of_nibbles(w), b = e4m3x4_of_nibbles(w >> 16);  // lo0 hi0 lo1 hi1 | lo2 hi2 lo3 hi3
  lo = __byte_perm(a, b, 0x6420);
  hi = __byte_perm(a, b, 0x7531);
}

// A CTA of THREADS expands THREADS * AHEAD 16-byte chunks (32 codes each), AHEAD in flight per thread.
template <int THREADS, int AHEAD>
__device__ __forceinline__ void expand_chunks(const WeightExpansion& e, uint32_t block) {
  const uint32_t groups = static_cast<uint32_t>(e.K / kGroup);
  const int64_t total = static_cast<int64_t>((e.N + 127) / 128) * groups * 512;
  const int64_t c0 = static_cast<int64_t>(block) * (THREADS * AHEAD) + threadIdx.x;
  uint4 raw[AHEAD];
#pragma unroll
  for (int i = 0; i < AHEAD; ++i) {
    const int64_t c = c0 + i * THREADS;
    if (c < total) raw[i] = *reinterpret_cast<const uint4*>(e.w_packed + (c >> 9) * kTileBytes + (c & 511) * 16);
  }
#pragma unroll
  for (int i = 0; i < AHEAD; ++i) {
    const int64_t c = c0 + i * THREADS;
    const uint32_t r = static_cast<uint32_t>(c >> 2) & 127, ch = (static_cast<uint32_t>(c) & 3) ^ ((r >> 1) & 3);
    const uint32_t tg = static_cast<uint32_t>(c >> 9), tile = tg / groups, g = tg - tile * groups;
    const int64_t row = static_cast<int64_t>(tile) * 128 + r;
    if (c >= total || row >= e.N) continue;
    const uint32_t w[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w};
    uint32_t lo[4], hi[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) e4m3_of_word(w[j], lo[j], hi[j]);  // k = 4j .. 4j+3 of the chunk, k = 16 + 4j ..
    uint8_t* dst = e.w8 + row * e.K + (g * 4 + ch) * 32;
    *reinterpret_cast<uint4*>(dst) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    *reinterpret_cast<uint4*>(dst + 16) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
  }
}
inline int64_t expand_ctas(int N, int K, int chunks_per_cta) {
  return (static_cast<int64_t>((N + 127) / 128) * (K / kGroup) * 512 + chunks_per_cta - 1) / chunks_per_cta;
}

// A quantiser's launch of `rows` CTAs with an expansion taken along: `ctas` more of them.  Long quantiser CTAs that all find a
// place at once (up to `resident`) come first, spread over the SMs as on their own (28 * P with the Hadamard, linears, us: 1100 x
// 1792 -> 4096 28.6 -> 25.5, 1024 x 1792 -> 2048 19.5 -> 16.7, 1100 x 3584 -> 4096 40.3 -> 37.4); else the others lie evenly
// between them: of the first b CTAs floor(b * share / 2^32) expand.  share is ctas * 2^32 / (rows + ctas) rounded up, so that with rows >= 1 it
// fits 32 bits and is not 0, no CTA counts twice, and the whole grid (fewer than 2^32 CTAs: the rounding adds less than one) has
// exactly `ctas` of them.
struct ExpansionShare {
  WeightExpansion e;
  uint32_t rows, share;  // share 0: the quantiser's CTAs first
};
constexpr int kShareAhead = 4;
inline unsigned take_along(const WeightExpansion& e, int threads, int64_t rows, int64_t resident, ExpansionShare* s) {
  const int64_t ctas = expand_ctas(e.N, e.K, threads * kShareAhead), total = rows + ctas;
  s->e = e;
  s->rows = static_cast<uint32_t>(rows);
  s->share = rows <= resident ? 0
                              : static_cast<uint32_t>(((static_cast<uint64_t>(ctas) << 32) + static_cast<uint64_t>(total) - 1) /
                                                      static_cast<uint64_t>(total));
  return static_cast<unsigned>(total);
}
// This CTA's index among the quantiser's; or, after its part of the expansion, -1.
template <int THREADS>
__device__ __forceinline__ int quantiser_cta(const ExpansionShare& s) {
  uint32_t before = __umulhi(blockIdx.x, s.share);
  bool expands = __umulhi(blockIdx.x + 1, s.share) != before;
  if (s.share == 0) {
    expands = blockIdx.x >= s.rows;
    if (expands) before = blockIdx.x - s.rows;
  }
  if (!expands) return static_cast<int>(blockIdx.x - before);
  expand_chunks<THREADS, kShareAhead>(s.e, before);
  return -1;
}

}  // namespace dq
