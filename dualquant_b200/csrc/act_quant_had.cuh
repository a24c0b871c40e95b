// The fast online-Hadamard quantiser kernels and their dispatch, as templates over the input type.
// Included by one translation unit per input type (act_quant_had_bf16.cu, act_quant_had_f32.cu):
// every unit has its own copy of the constant-bank factor table and of the upload cache, and only
// launches its own kernels, so the copies never have to agree.
#pragma once
#include "act_quant_common.cuh"
#include "act_quant_had28.cuh"

namespace dq {
namespace {

constexpr int kHadFastMaxSmem = 200 * 1024;

// ---------------------------------------------------------------------------------------------
// fast online Hadamard: warp-shuffle butterflies inside segments, one thread per column across
// ---------------------------------------------------------------------------------------------
// The row is viewed as S segments of P contiguous elements (S <= 32, P = 32 * R).
//   phase A (wht_inner): Walsh-Hadamard of length P inside every segment; a warp owns a segment,
//            lane l holds elements l + 32 r: stages h < 32 exchange registers with lane ^ h, stages
//            h >= 32 are register butterflies.  Same stage order and operand order as
//            the reference loop (h = 1, 2, 4, ...; (a, b) -> (a + b, a - b)), so bit-identical.
//   phase B: per column c (0..P-1) across the S segments:
//            matrix mode   out[i] = sum_j H[i][j] * (v[j] * scale), j ascending  (had_K @ x)
//            butterfly mode  remaining Walsh-Hadamard stages over the segment index, then * scale
// Full transform of size 28 * 512: A + matrix.  Full power-of-two size: A + butterflies.
// Partial (across heads) transform: butterflies only, segments = heads.
// Stages h = 1, 2, 4 on eight adjacent elements, where the row is loaded: in registers they cost an addition each, behind
// the shared memory a shuffle more.
__device__ __forceinline__ void wht8(float (&v)[8]) {
#pragma unroll
  for (int h = 1; h < 8; h <<= 1) {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      if ((e & h) == 0) {
        const float u = v[e], w = v[e + h];
        v[e] = __fadd_rn(u, w);
        v[e + h] = __fsub_rn(u, w);
      }
    }
  }
}

// Eight adjacent elements of thread t at p = base + 8 t, two 16-byte accesses; lanes 4 .. 7 of every eight take the halves
// in the other order, so that eight lanes touch all banks once.
__device__ __forceinline__ void row_store8(float* p, const float (&v)[8]) {
  const bool swap = (threadIdx.x & 4) != 0;
  const float4 lo = make_float4(v[0], v[1], v[2], v[3]), hi = make_float4(v[4], v[5], v[6], v[7]);
  *reinterpret_cast<float4*>(p + (swap ? 4 : 0)) = swap ? hi : lo;
  *reinterpret_cast<float4*>(p + (swap ? 0 : 4)) = swap ? lo : hi;
}
__device__ __forceinline__ void row_load8(const float* p, float (&v)[8]) {
  const bool swap = (threadIdx.x & 4) != 0;
  const float4 f = *reinterpret_cast<const float4*>(p + (swap ? 4 : 0));
  const float4 g = *reinterpret_cast<const float4*>(p + (swap ? 0 : 4));
  const float4 lo = swap ? g : f, hi = swap ? f : g;
  v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w;
  v[4] = hi.x; v[5] = hi.y; v[6] = hi.z; v[7] = hi.w;
}

// The stages from h = 8 on.
template <int R>
__device__ __forceinline__ void wht_segment_warp(float* seg, int lane, float post = 1.0f) {
  // lane l holds elements l + 32 r (r < R): conflict-free shared-memory access; stages h < 32
  // pair lanes (shuffle), stages h >= 32 pair registers r and r + h/32.  Stage order h = 1, 2, ...
  float v[R];
#pragma unroll
  for (int r = 0; r < R; ++r) v[r] = seg[lane + 32 * r];
  // the lane with bit m clear keeps a + b, its partner a - b: other + sign * own, one FMA either
  // way (the product with +-1 is exact, so the FMA rounds exactly like the addition / subtraction)
#pragma unroll
  for (int m = 8; m < 32; m <<= 1) {
    const float sign = (lane & m) != 0 ? -1.0f : 1.0f;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float other = __shfl_xor_sync(0xffffffffu, v[r], m);
      v[r] = __fmaf_rn(v[r], sign, other);
    }
  }
#pragma unroll
  for (int h = 1; h < R; h <<= 1) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if ((r & h) == 0) {
        const float u = v[r], w = v[r + h];
        v[r] = __fadd_rn(u, w);
        v[r + h] = __fsub_rn(u, w);
      }
    }
  }
  // `post`: the transform's scale when a matrix stage follows (it multiplies every value once, here,
  // instead of once per thread that reads the value there); 1 otherwise, an exact identity
#pragma unroll
  for (int r = 0; r < R; ++r) seg[lane + 32 * r] = __fmul_rn(v[r], post);
}

// The K x K +-1 matrix of the "full" transform, in constant memory so that an FMA takes its
// coefficient as an immediate constant-bank operand (one instruction per term instead of a
// shared-memory load plus an FMA).  Every entry is stored twice, (h, h): the matrix stage works on
// two columns at a time with packed fp32 FMAs, each half of which rounds like the scalar fmaf.
// Refreshed by the host when a call brings a different matrix.
__constant__ float2 c_had_mat2[32 * 32];
__device__ float2 g_had_stage[32 * 32];  // the table is assembled here, then copied to the constant bank

__global__ void __launch_bounds__(1024) had_table_kernel(const float* __restrict__ had_mat, int S) {
  const int t = threadIdx.x, i = t >> 5, j = t & 31;
  const float h = (i < S && j < S) ? had_mat[i * S + j] : 0.f;  // rows and columns padded to 32 with zeros
  g_had_stage[t] = make_float2(h, h);
}

// Output rows QI, QI + G, ... of the matrix stage for one column pair, fully unrolled (see the
// call site); matrix_rows_dispatch selects the copy for a run-time qi in [0, G).
template <int HN, int G, int QI>
__device__ __forceinline__ void matrix_rows_static(const float2* v, float* row, int P, int c, int S, float& amax) {
#pragma unroll
  for (int i = QI; i < HN; i += G) {
    if (i < S) {  // (kept as a run-time test also for a known order: without it the short-row shapes ran 10-25 % slower)
      float2 acc = make_float2(0.f, 0.f);
#pragma unroll
      for (int j = 0; j < HN; ++j) acc = __ffma2_rn(c_had_mat2[i * 32 + j], v[j], acc);
      *reinterpret_cast<float2*>(row + i * P + c) = acc;
      amax = fmaxf(amax, fmaxf(fabsf(acc.x), fabsf(acc.y)));
    }
  }
}
template <int HN, int G, int QI = 0>
__device__ __forceinline__ void matrix_rows_dispatch(int qi, const float2* v, float* row, int P, int c, int S,
                                                     float& amax) {
  if constexpr (QI < G) {
    if (qi == QI) matrix_rows_static<HN, G, QI>(v, row, P, c, S, amax);
    else matrix_rows_dispatch<HN, G, QI + 1>(qi, v, row, P, c, S, amax);
  }
}

// THREADS = 512: one CTA per SM, the shortest time per row (decode batches, one row per SM at most).
// THREADS = 256: three CTAs per SM; with many rows one row's load, barrier and store phases overlap
// another row's arithmetic (two CTAs per SM with more registers each measured 30 % slower).
// HS: order of the +-1 factor where it is known (28 for 28672 = 28 * 1024; shorter rows of that order have a kernel of their
// own, act_quant_had28.cuh), so that the matrix stage has no padded terms; 0 = any order up to 32.
template <int R, typename XT, int THREADS, int HS = 0>
__global__ void __launch_bounds__(THREADS, THREADS == 256 ? 3 : 1)
act_quant_had_fast_kernel(const XT* x, const XT* up, int64_t ldx,
                          const float* a, int K,
                          int S, int inner, int matrix, float had_scale, int8_t* __restrict__ codes,
                          float* __restrict__ sx, float* __restrict__ out, int mode, int scale_fp16) {
  extern __shared__ float sm_row[];
  __shared__ float red[THREADS / 32];
  float* row = sm_row;
  grid_dep_launch_dependents();
  grid_dep_wait();
  const int P = K / S;
  const int rr = blockIdx.x;
  const XT* xr = x + static_cast<int64_t>(rr) * ldx;
  const XT* ur = (up != nullptr) ? up + static_cast<int64_t>(rr) * ldx : nullptr;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  // four pieces of x (and up) in flight per thread: one at a time, a row of 14336 waited for seven memory round trips
  // before its arithmetic (8192 gated rows: 470 -> 424 us, 306 without the gate; seven in flight: 445)
  constexpr int kAhead = 4;
  for (int base = threadIdx.x * 8; base < K; base += kAhead * THREADS * 8) {
    Raw8<XT> xw[kAhead], uw[kAhead];
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      const int idx = base + i * THREADS * 8;
      if (idx < K) {
        xw[i].load(xr + idx);
        if (ur != nullptr) uw[i].load(ur + idx);
      }
    }
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      const int idx = base + i * THREADS * 8;
      if (idx < K) {
        float v[8];
        if (ur != nullptr) gated8(xw[i], uw[i], v);
        else xw[i].expand(v);
        if (a != nullptr) {
          float av[8];
          load8(a + idx, av);
#pragma unroll
          for (int e = 0; e < 8; ++e) v[e] = __fmul_rn(v[e], av[e]);
        }
        if (inner) wht8(v);
        row_store8(row + idx, v);
      }
    }
  }
  __syncthreads();

  if (inner) {
    for (int sgm = warp; sgm < S; sgm += THREADS / 32)
      wht_segment_warp<R>(row + sgm * P, lane, matrix ? had_scale : 1.0f);
    __syncthreads();
  }
  const bool scale_here = !inner;  // no Walsh-Hadamard phase: the matrix stage scales its own inputs

  float amax = 0.f;
  if (matrix) {
    // two adjacent columns per thread (P is even): packed loads, packed FMAs
    constexpr int HN = (HS > 0) ? HS : 32;  // factor order known at compile time, or padded to 32
    constexpr int pairs = 16 * R;  // P = 32 R
    if constexpr (pairs < THREADS) {
      // Short segments (rows of 28 * 64 ... 28 * 256 values, the shards of a row-parallel linear):
      // fewer column pairs than threads.  G = THREADS / pairs threads share one pair, each holding
      // its S inputs in registers and forming the output rows i = qi, qi + G, ...; every sum is the
      // same j-ascending chain as below.  (pairs is a power of two, so G is whole; qi is the same for
      // all lanes of a warp once a segment has 64 values, which keeps the coefficient loads uniform.)
      constexpr int G = THREADS / pairs;
      const int c = 2 * (static_cast<int>(threadIdx.x) & (pairs - 1)), qi = static_cast<int>(threadIdx.x) / pairs;
      float2 v[HN];
#pragma unroll
      for (int j = 0; j < HN; ++j)
        v[j] = (j < S) ? *reinterpret_cast<const float2*>(row + j * P + c) : make_float2(0.f, 0.f);
      if (scale_here) {
#pragma unroll
        for (int j = 0; j < HN; ++j) {
          v[j].x = __fmul_rn(v[j].x, had_scale);
          v[j].y = __fmul_rn(v[j].y, had_scale);
        }
      }
      __syncthreads();  // every thread holds its inputs before the first output row replaces them
      if constexpr (G <= 8) {
        // the thread's output rows are known once qi is: one fully unrolled copy per value of qi, so
        // that every coefficient is a constant-bank operand of its FMA (HN x HN FMAs of code in all)
        matrix_rows_dispatch<HN, G>(qi, v, row, P, c, S, amax);
      } else
      for (int i = qi; i < S; i += 2 * G) {  // two independent chains in flight
        const int i2 = i + G;
        const bool second = i2 < S;
        const float2* h0 = c_had_mat2 + i * 32;
        const float2* h1 = c_had_mat2 + (second ? i2 : i) * 32;
        float2 acc0 = make_float2(0.f, 0.f), acc1 = make_float2(0.f, 0.f);
#pragma unroll
        for (int j = 0; j < HN; ++j) {
          acc0 = __ffma2_rn(h0[j], v[j], acc0);
          acc1 = __ffma2_rn(h1[j], v[j], acc1);
        }
        *reinterpret_cast<float2*>(row + i * P + c) = acc0;
        amax = fmaxf(amax, fmaxf(fabsf(acc0.x), fabsf(acc0.y)));
        if (second) {
          *reinterpret_cast<float2*>(row + i2 * P + c) = acc1;
          amax = fmaxf(amax, fmaxf(fabsf(acc1.x), fabsf(acc1.y)));
        }
      }
    } else
    for (int c = 2 * threadIdx.x; c < P; c += 2 * THREADS) {
      float2 v[HN];
#pragma unroll
      for (int j = 0; j < HN; ++j)
        v[j] = (HS > 0 || j < S) ? *reinterpret_cast<const float2*>(row + j * P + c) : make_float2(0.f, 0.f);
      if (scale_here) {
#pragma unroll
        for (int j = 0; j < HN; ++j) {
          v[j].x = __fmul_rn(v[j].x, had_scale);
          v[j].y = __fmul_rn(v[j].y, had_scale);
        }
      }
      // the known order is fully unrolled, so that every coefficient is a constant-bank operand of
      // its FMA and the independent accumulation chains can be interleaved; the generic form keeps
      // two output rows in flight (a fully unrolled 32 x 32 stage in every instantiation is most of
      // this file's compile time)
      constexpr int kUnrollRows = (HS > 0) ? HN : 2;
#pragma unroll kUnrollRows
      for (int i = 0; i < HN; ++i) {
        if (HS > 0 || i < S) {  // a known order is the factor's order: no padded rows
          float2 acc = make_float2(0.f, 0.f);
#pragma unroll
          for (int j = 0; j < HN; ++j)  // H entries are +-1 (0 in the padding): same as acc + H*v, j ascending
            acc = __ffma2_rn(c_had_mat2[i * 32 + j], v[j], acc);
          *reinterpret_cast<float2*>(row + i * P + c) = acc;
          amax = fmaxf(amax, fmaxf(fabsf(acc.x), fabsf(acc.y)));
        }
      }
    }
  } else {
  for (int c = threadIdx.x; c < P; c += THREADS) {
    float v[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = (j < S) ? row[j * P + c] : 0.f;
    {
#pragma unroll
      for (int hb = 0; hb < 5; ++hb) {
        constexpr int kOne = 1;
        const int h = kOne << hb;
        if (h < S) {
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            if ((j & h) == 0) {
              const float u = v[j], w = v[j + h];
              v[j] = __fadd_rn(u, w);
              v[j + h] = __fsub_rn(u, w);
            }
          }
        }
      }
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        if (j < S) {
          const float o = __fmul_rn(v[j], had_scale);
          row[j * P + c] = o;
          amax = fmaxf(amax, fabsf(o));
        }
      }
    }
  }
  }
  TokenQuant tq = {1.f, 1.f, false};
  if (mode != MODE_RAW) {
    amax = block_max(amax, red, THREADS / 32);
    tq = token_quant(amax, token_scale(amax, scale_fp16));
    if (threadIdx.x == 0 && sx != nullptr) sx[rr] = tq.s;
  } else {
    __syncthreads();
  }
  int8_t* crow = (codes != nullptr) ? codes + static_cast<int64_t>(rr) * K : nullptr;
  float* orow = out_row_ptr(out, rr, K, mode);
  for (int idx = threadIdx.x * 8; idx < K; idx += THREADS * 8) {
    float v[8];
    row_load8(row + idx, v);
    emit8(v, tq, mode, crow, orow, idx, scale_fp16);
  }
}

// ---------------------------------------------------------------------------------------------
// the same transform for a handful of rows: one thread-block cluster per row
// ---------------------------------------------------------------------------------------------
// At decode sizes (a few token rows) the fast kernel is one CTA per row on a few SMs and its phases
// - load (+ SiLU * up), Walsh-Hadamard inside the segments, the S x S stage across them, absmax,
// codes - are a serial chain.  Here four CTAs share a row: CTA c loads and transforms segments
// [c S/4, (c+1) S/4), then computes the matrix stage for columns [c P/4, (c+1) P/4) of every
// segment; the row absmax is exchanged through distributed shared memory.  The columns of the other
// CTAs' segments are copied over once, 16 bytes per load: read from there by every thread that needs
// them, a value at a time, they were 448 warp-wide remote loads per CTA at some 20 cycles each.
// Every sum is formed exactly as in the fast kernel (same Walsh-Hadamard routine, j ascending fp32
// FMAs with the factor's entry as coefficient), so scales and codes are bit-identical.  The factor is
// read from the caller's matrix, not from the constant bank: nothing has to be uploaded between the
// kernels of a decode step.  Needs S % 4 == 0.
constexpr int kHadClusterCtas = 4;
constexpr int kHadClusterThreads = 512;
constexpr int kHadClusterMaxRows = 64;

template <int R, typename XT>
__global__ void __launch_bounds__(kHadClusterThreads, 1)
act_quant_had_cluster_kernel(const XT* x, const XT* up, int64_t ldx,
                             const float* a, int S, float had_scale, const float* had_mat,
                             int8_t* __restrict__ codes, float* __restrict__ sx, float* __restrict__ out, int mode,
                             int scale_fp16) {
  constexpr int P = 32 * R;                   // segment length
  constexpr int PC = P / kHadClusterCtas;     // columns of the matrix stage per CTA
  constexpr int G = kHadClusterThreads / PC;  // threads per column: output rows i = qi, qi + G, ...
  extern __shared__ float sm_row[];
  __shared__ float red[kHadClusterThreads / 32];
  __shared__ float pmax[kHadClusterCtas];
  const int SQ = S / kHadClusterCtas;         // segments per CTA
  const int K = S * P;
  float* seg = sm_row;                        // [SQ][P]: this CTA's segments (read by its peers)
  float* colv = sm_row + SQ * P;              // [S][PC]: this CTA's columns of all segments, then its slice of the result
  float* coef = colv + S * PC;                // [S][32]: the factor, rows padded with zeros
  grid_dep_launch_dependents();
  grid_dep_wait();
  const int rank = static_cast<int>(cluster_ctarank());
  const int rr = blockIdx.x / kHadClusterCtas;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t base = static_cast<int64_t>(rr) * ldx + static_cast<int64_t>(rank) * SQ * P;
  const XT* xr = x + base;
  const XT* ur = (up != nullptr) ? up + base : nullptr;
  const float* ar = (a != nullptr) ? a + static_cast<int64_t>(rank) * SQ * P : nullptr;
  // the factor's loads are issued first and the row's three operands together: one memory round trip in all
  constexpr int kCoefs = 1024 / kHadClusterThreads;  // S <= 32
  float cf[kCoefs];
#pragma unroll
  for (int u = 0; u < kCoefs; ++u) {
    const int i = tid + u * kHadClusterThreads, j = i & 31;
    cf[u] = (i < S * 32 && j < S) ? had_mat[(i >> 5) * S + j] : 0.f;
  }
  for (int idx = tid * 8; idx < SQ * P; idx += kHadClusterThreads * 8) {
    Raw8<XT> xw, uw;
    float v[8], av[8];
    xw.load(xr + idx);
    if (ur != nullptr) uw.load(ur + idx);
    if (ar != nullptr) load8(ar + idx, av);
    if (ur != nullptr) gated8(xw, uw, v);
    else xw.expand(v);
    if (ar != nullptr) {
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = __fmul_rn(v[e], av[e]);
    }
    wht8(v);
    row_store8(seg + idx, v);
  }
#pragma unroll
  for (int u = 0; u < kCoefs; ++u) {
    const int i = tid + u * kHadClusterThreads;
    if (i < S * 32) coef[i] = cf[u];
  }
  __syncthreads();
  for (int sgm = warp; sgm < SQ; sgm += kHadClusterThreads / 32) wht_segment_warp<R>(seg + sgm * P, lane, had_scale);
  cluster_sync_all();  // every CTA's segments are transformed (and scaled) and visible to its peers
  {
    const uint32_t seg_addr = smem_u32(seg);
    for (int u = tid; u < S * (PC / 4); u += kHadClusterThreads) {
      const int j = u / (PC / 4), c4 = u - j * (PC / 4);
      const int owner = j / SQ;
      const uint32_t from = seg_addr + static_cast<uint32_t>(((j - owner * SQ) * P + rank * PC + c4 * 4) * 4);
      *reinterpret_cast<float4*>(colv + j * PC + c4 * 4) = dsmem_ld_f4(dsmem_map(from, static_cast<uint32_t>(owner)));
    }
  }
  __syncthreads();

  const int col = tid % PC, qi = tid / PC;
  float v[32];
#pragma unroll
  for (int j = 0; j < 32; ++j) v[j] = j < S ? colv[j * PC + col] : 0.f;
  __syncthreads();  // every thread holds its inputs before the first result replaces them
  float amax = 0.f;
  for (int i = qi; i < S; i += G) {  // i is the same for every lane of a warp
    const float4* h4 = reinterpret_cast<const float4*>(coef + i * 32);
    float acc = 0.f;
#pragma unroll
    for (int j = 0; j < 32; j += 4) {
      const float4 h = h4[j >> 2];
      acc = fmaf(h.x, v[j], acc);
      acc = fmaf(h.y, v[j + 1], acc);
      acc = fmaf(h.z, v[j + 2], acc);
      acc = fmaf(h.w, v[j + 3], acc);
    }
    colv[i * PC + col] = acc;
    amax = fmaxf(amax, fabsf(acc));
  }
  TokenQuant tq = {1.f, 1.f, false};
  amax = block_max_once(amax, red, kHadClusterThreads / 32);  // (also orders the colv writes before their reads below)
  if (tid < kHadClusterCtas)
    dsmem_store_f32(dsmem_map(smem_u32(&pmax[rank]), static_cast<uint32_t>(tid)), amax);
  cluster_sync_all();  // the four partial maxima have landed everywhere; no remote access after this point
  if (mode != MODE_RAW) {
    float full = pmax[0];
#pragma unroll
    for (int c = 1; c < kHadClusterCtas; ++c) full = fmaxf(full, pmax[c]);
    tq = token_quant(full, token_scale(full, scale_fp16));
    if (rank == 0 && tid == 0 && sx != nullptr) sx[rr] = tq.s;
  }
  int8_t* crow = (codes != nullptr) ? codes + static_cast<int64_t>(rr) * K : nullptr;
  float* orow = out_row_ptr(out, rr, K, mode);
  for (int u = tid; u < S * (PC / 8); u += kHadClusterThreads) {
    const int i = u / (PC / 8), piece = u - i * (PC / 8);
    float e8[8];
    row_load8(colv + i * PC + piece * 8, e8);
    emit8(e8, tq, mode, crow, orow, i * P + rank * PC + piece * 8, scale_fp16);
  }
}

// ---------------------------------------------------------------------------------------------
// the across-heads transform (o_proj input): registers only
// ---------------------------------------------------------------------------------------------
// Row = S heads of 128 values, Walsh-Hadamard over the head index for each of the 128 lanes of a head.  A decode batch
// is bound by the chain load -> stages -> absmax -> codes of one row, so a row gets as many threads as keep the chain
// short: a thread owns two columns of at most eight heads (sixteen values), the head groups sit 8 (S = 32) or 16 (S = 16)
// lanes apart, where the last stages are shuffles, and a row costs one barrier; up to four heads a row is one warp, four
// columns to a lane, and costs none.  Many rows are bound by instruction issue: a CTA walks rows gridDim.x apart with
// the activation scale in registers and the next row's loads in flight.  Same stage order and operand order as above.
// Codes only (int8 or E4M3, fp32 or fp16 scale), no gate.
// Against one lane for eight columns of sixteen heads (64 rows up; one CTA with two shared-memory passes below), us at
// 32 heads: 8 rows 3.7 -> 2.6, 64 rows 9.0 -> 2.7, 1000 rows 10.7 -> 7.5, 16384 rows 150 -> 74 (2.7 TB/s).
template <int S>
struct HeadsRow {
  static constexpr int kHeads = (S < 8) ? S : 8;          // heads per thread
  static constexpr int kGroups = S / kHeads;              // head groups
  static constexpr int kCols = (S <= 4) ? 4 : 2;          // columns per thread
  static constexpr int kLanes = 32 / kGroups;             // column sets per warp
  static constexpr int kWarps = 128 / (kLanes * kCols);   // warps per row
  static constexpr int kRows = (S <= 4) ? 4 : 1;          // rows per CTA
  static constexpr int kThreads = 32 * kWarps * kRows;
  // CTAs per SM: 64 registers a thread hold eight heads of two columns, their scales and the next row
  static constexpr int kCtas = (S == 2 ? 1280 : 1024) / kThreads;
};

template <int S, typename XT, bool E4M3>
__global__ void __launch_bounds__(HeadsRow<S>::kThreads, HeadsRow<S>::kCtas)
act_quant_had_heads_kernel(const XT* x, int64_t ldx, const float* a, int M, float had_scale,
                           int8_t* __restrict__ codes, float* __restrict__ sx, int scale_fp16) {
  using H = HeadsRow<S>;
  constexpr int HL = H::kHeads, C = H::kCols, CL = H::kLanes;
  __shared__ float red[2][H::kWarps];  // of alternate rows: one barrier per row
  grid_dep_launch_dependents();
  grid_dep_wait();
  const int lane = threadIdx.x & 31;
  const int warp = (H::kRows > 1) ? 0 : threadIdx.x >> 5;  // warp of the row
  const int row_in_cta = (H::kRows > 1) ? threadIdx.x >> 5 : 0;
  const int at = (lane / CL) * HL * 128 + (warp * CL + (lane & (CL - 1))) * C;  // first head's columns
  constexpr int kWords = C * sizeof(XT) / 4;
  uint32_t raw[HL][kWords];
  auto load = [&](int64_t row) {
#pragma unroll
    for (int j = 0; j < HL; ++j) {
      const XT* p = x + row * ldx + at + j * 128;
      if constexpr (kWords == 1) {
        raw[j][0] = *reinterpret_cast<const uint32_t*>(p);
      } else {
#pragma unroll
        for (int e = 0; e < kWords; e += 2) {
          const uint2 w = *reinterpret_cast<const uint2*>(reinterpret_cast<const uint32_t*>(p) + e);
          raw[j][e] = w.x;
          raw[j][e + 1] = w.y;
        }
      }
    }
  };
  const int64_t step = static_cast<int64_t>(gridDim.x) * H::kRows;
  int64_t row = static_cast<int64_t>(blockIdx.x) * H::kRows + row_in_cta;
  if (row < M) load(row);
  float av[HL][C];
  if (a != nullptr) {
#pragma unroll
    for (int j = 0; j < HL; ++j) {
#pragma unroll
      for (int e = 0; e < C; e += 2) {
        const float2 w = *reinterpret_cast<const float2*>(a + at + j * 128 + e);
        av[j][e] = w.x;
        av[j][e + 1] = w.y;
      }
    }
  }
  int buf = 0;
  for (; row < M; row += step, buf ^= 1) {  // (a row's warps leave the loop together)
    float v[HL][C];
#pragma unroll
    for (int j = 0; j < HL; ++j) {
#pragma unroll
      for (int e = 0; e < C; ++e) {
        if constexpr (sizeof(XT) == 2)
          v[j][e] = __uint_as_float((e & 1) ? raw[j][e / 2] & 0xFFFF0000u : raw[j][e / 2] << 16);
        else
          v[j][e] = __uint_as_float(raw[j][e]);
      }
    }
    if (row + step < M) load(row + step);
    if (a != nullptr) {
#pragma unroll
      for (int j = 0; j < HL; ++j) {
#pragma unroll
        for (int e = 0; e < C; ++e) v[j][e] = __fmul_rn(v[j][e], av[j][e]);
      }
    }
#pragma unroll
    for (int h = 1; h < HL; h <<= 1) {
#pragma unroll
      for (int j = 0; j < HL; ++j) {
        if ((j & h) == 0) {
#pragma unroll
          for (int e = 0; e < C; ++e) {
            const float u = v[j][e], w = v[j + h][e];
            v[j][e] = __fadd_rn(u, w);
            v[j + h][e] = __fsub_rn(u, w);
          }
        }
      }
    }
#pragma unroll
    for (int o = CL; o < 32; o <<= 1) {  // heads HL * (o / CL) apart
      const float sign = (lane & o) != 0 ? -1.0f : 1.0f;  // a + b below, a - b above: other + sign * own, rounded once
#pragma unroll
      for (int j = 0; j < HL; ++j) {
#pragma unroll
        for (int e = 0; e < C; ++e) {
          const float other = __shfl_xor_sync(0xffffffffu, v[j][e], o);
          v[j][e] = __fmaf_rn(v[j][e], sign, other);
        }
      }
    }
    float amax = 0.f;
#pragma unroll
    for (int j = 0; j < HL; ++j) {
#pragma unroll
      for (int e = 0; e < C; ++e) {
        v[j][e] = __fmul_rn(v[j][e], had_scale);
        amax = fmaxf(amax, fabsf(v[j][e]));
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if constexpr (H::kWarps > 1) {
      if (lane == 0) red[buf][warp] = amax;
      __syncthreads();
#pragma unroll
      for (int i = 0; i < H::kWarps; ++i) amax = fmaxf(amax, red[buf][i]);
    }
    const TokenQuant tq = token_quant(amax, token_scale(amax, scale_fp16));
    if (warp == 0 && lane == 0 && sx != nullptr) sx[row] = tq.s;
    int8_t* crow = codes + row * (S * 128) + at;
    constexpr int kQ = 8 / C;  // heads per eight values
#pragma unroll
    for (int j = 0; j < HL; j += kQ) {
      float in[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) in[e] = v[j + e / C][e % C];
      const uint2 packed = quant_pack8(in, tq, E4M3);
#pragma unroll
      for (int p = 0; p < 8; p += 4) {
        const uint32_t w = p == 0 ? packed.x : packed.y;
        if constexpr (C == 4) {
          *reinterpret_cast<uint32_t*>(crow + (j + p / 4) * 128) = w;
        } else {
          *reinterpret_cast<uint16_t*>(crow + (j + p / 2) * 128) = static_cast<uint16_t>(w);
          *reinterpret_cast<uint16_t*>(crow + (j + p / 2 + 1) * 128) = static_cast<uint16_t>(w >> 16);
        }
      }
    }
  }
}

// Copies a device-resident S x S matrix into c_had_mat2 (rows padded to 32) when it is not the
// one already there.  The matrix behind a given pointer is assumed immutable (it is the constant
// Hadamard factor of a layer); the copy is a stream-ordered device-to-device memcpy.
static int upload_had_matrix(const float* had_mat, int S, cudaStream_t stream) {
  static const float* cached[kMaxDevices] = {nullptr};
  static int cached_s[kMaxDevices] = {0};
  int dev = 0;
  DQ_CHECK_CUDA(cudaGetDevice(&dev));
  // While the stream is being captured the copy is always recorded, so that a replayed graph
  // carries its own matrix whatever was uploaded between capture and replay.  Outside capture
  // the copy is skipped when the same pointer was uploaded last; the upload is ordered on the
  // caller's stream only, so calls that bring a Hadamard matrix must share one stream per
  // device (or be ordered by the caller).
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  DQ_CHECK_CUDA(cudaStreamIsCapturing(stream, &cap));
  const bool capturing = cap != cudaStreamCaptureStatusNone;
  // Once an upload sits inside a graph, a replay can rewrite the table at any time behind the
  // back of this cache: from then on every call uploads.
  static bool seen_capture[kMaxDevices] = {false};
  if (capturing) seen_capture[dev] = true;
  if (!seen_capture[dev] && cached[dev] == had_mat && cached_s[dev] == S) return DQ_OK;
  void* sym = nullptr;
  void* stage = nullptr;
  DQ_CHECK_CUDA(cudaGetSymbolAddress(&sym, c_had_mat2));
  DQ_CHECK_CUDA(cudaGetSymbolAddress(&stage, g_had_stage));
  had_table_kernel<<<1, 1024, 0, stream>>>(had_mat, S);
  DQ_CHECK_CUDA(cudaGetLastError());
  DQ_CHECK_CUDA(cudaMemcpyAsync(sym, stage, sizeof(float2) * 32 * 32, cudaMemcpyDeviceToDevice, stream));
  // a captured copy has not run yet: whatever is cached no longer describes the table
  cached[dev] = capturing ? nullptr : had_mat;
  cached_s[dev] = capturing ? 0 : S;
  return DQ_OK;
}

// Picks the segmentation for the fast kernel; returns false when the shape is outside its range.
struct HadPlan {
  int S, R, inner, matrix;
};
static bool plan_fast_hadamard(const dq_hadamard_desc* had, int K, HadPlan* plan) {
  auto pow2 = [](int v) { return v > 0 && (v & (v - 1)) == 0; };
  if (had->kind == DQ_HAD_FULL && had->had_k > 1) {
    const int P = K / had->had_k;
    if (had->had_k > 32 || !pow2(P) || P < 32 || P > 1024) return false;
    *plan = {had->had_k, P / 32, 1, 1};
    return true;
  }
  if (had->kind == DQ_HAD_FULL) {  // pure Walsh-Hadamard of length K
    if (!pow2(K) || K < 64) return false;
    int P = K / 32 < 32 ? 32 : K / 32;   // S = K / P <= 32
    if (P > 1024) return false;
    *plan = {K / P, P / 32, 1, 0};
    return true;
  }
  if (had->kind == DQ_HAD_PARTIAL) {
    const int H = K / had->had_dim;
    if (H > 32 || !pow2(H)) return false;
    *plan = {H, 1, 0, 0};
    return true;
  }
  return false;
}

template <typename XT>
int init_had_fast_t() {
  constexpr int kHadMaxSmem = kHadFastMaxSmem;
  cudaError_t e = cudaSuccess;
#define DQ_HAD_ATTR(R)                                                                        \
  if (e == cudaSuccess)                                                                       \
    e = cudaFuncSetAttribute(act_quant_had_fast_kernel<R, XT, 512>,                             \
                             cudaFuncAttributeMaxDynamicSharedMemorySize, kHadMaxSmem);        \
  if (e == cudaSuccess)                                                                       \
    e = cudaFuncSetAttribute(act_quant_had_fast_kernel<R, XT, 256>,                             \
                             cudaFuncAttributeMaxDynamicSharedMemorySize, kHadMaxSmem);
  DQ_HAD_ATTR(1) DQ_HAD_ATTR(2) DQ_HAD_ATTR(4) DQ_HAD_ATTR(8) DQ_HAD_ATTR(16) DQ_HAD_ATTR(32)
#undef DQ_HAD_ATTR
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(act_quant_had_fast_kernel<32, XT, 512, 28>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kHadMaxSmem);
#define DQ_HAD_ATTRC(R)                                                                       \
  if (e == cudaSuccess)                                                                       \
    e = cudaFuncSetAttribute(act_quant_had_cluster_kernel<R, XT>,                               \
                             cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
  DQ_HAD_ATTRC(4) DQ_HAD_ATTRC(8) DQ_HAD_ATTRC(16) DQ_HAD_ATTRC(32)
#undef DQ_HAD_ATTRC
#define DQ_HAD_ATTR_28(P)                                                                     \
  if (e == cudaSuccess)                                                                       \
    e = cudaFuncSetAttribute(act_quant_had28_kernel<P, XT>, cudaFuncAttributeMaxDynamicSharedMemorySize, Had28<P>::kSmem); \
  if (e == cudaSuccess)                                                                       \
    e = cudaFuncSetAttribute(act_quant_had28_kernel<P, XT, sizeof(XT) == 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                             Had28<P>::kSmem);
  DQ_HAD_ATTR_28(64) DQ_HAD_ATTR_28(128) DQ_HAD_ATTR_28(256) DQ_HAD_ATTR_28(512)
#undef DQ_HAD_ATTR_28
  if (e != cudaSuccess)
    return set_error(DQ_ERR_CUDA, "cudaFuncSetAttribute(act_quant_had fast) failed: %s", cudaGetErrorString(e));
  return DQ_OK;
}

// Runs the fast (or, for a handful of rows, the cluster) kernel when the transform is one they cover;
// *taken tells the caller whether a launch was made.
template <typename XT>
int launch_had_fast_t(const XT* x, const XT* up, int64_t ldx, const float* a, const dq_hadamard_desc* had, int M, int K,
                      size_t smem, int8_t* codes, float* sx, float* out, int mode, int scale_fp16,
                      cudaStream_t stream, bool* taken, Along* along) {
  *taken = false;
    HadPlan plan;
    if (plan_fast_hadamard(had, K, &plan)) {
      *taken = true;
      // across 2 ... 32 heads of 128 values: the register-only kernel
      if (had->kind == DQ_HAD_PARTIAL && had->had_dim == 128 && plan.S >= 2 && up == nullptr && mode == MODE_CODES &&
          codes != nullptr && (scale_fp16 & 0xFF) != 2) {
        DeviceState* st = current_state();
        if (st == nullptr) return DQ_ERR_NOT_INIT;
#define DQ_HAD_HEADS(SS)                                                                                            \
  {                                                                                                                 \
    using H = HeadsRow<SS>;                                                                                         \
    const int ctas = (M + H::kRows - 1) / H::kRows, most = H::kCtas * st->sm_count;                                 \
    const dim3 grid(ctas < most ? ctas : most);                                                                     \
    if ((scale_fp16 & kCodesE4M3) != 0)                                                                             \
      DQ_CHECK_CUDA(launch_pdl(act_quant_had_heads_kernel<SS, XT, true>, grid, dim3(H::kThreads), 0, stream, x,     \
                               ldx, a, M, had->scale, codes, sx, scale_fp16));                                      \
    else                                                                                                            \
      DQ_CHECK_CUDA(launch_pdl(act_quant_had_heads_kernel<SS, XT, false>, grid, dim3(H::kThreads), 0, stream, x,    \
                               ldx, a, M, had->scale, codes, sx, scale_fp16));                                      \
  }
        switch (plan.S) {
          case 2: DQ_HAD_HEADS(2); break;
          case 4: DQ_HAD_HEADS(4); break;
          case 8: DQ_HAD_HEADS(8); break;
          case 16: DQ_HAD_HEADS(16); break;
          default: DQ_HAD_HEADS(32); break;
        }
#undef DQ_HAD_HEADS
        return DQ_OK;
      }
      // a handful of rows (decode): four CTAs per row
      if (plan.matrix && plan.inner && plan.S % kHadClusterCtas == 0 && M <= kHadClusterMaxRows && plan.R >= 4) {
        const int P = 32 * plan.R;
        const size_t csmem = static_cast<size_t>(plan.S / kHadClusterCtas * P + plan.S * (P / kHadClusterCtas) + plan.S * 32) * 4;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(kHadClusterCtas * M, 1, 1);
        cfg.blockDim = dim3(kHadClusterThreads, 1, 1);
        cfg.dynamicSmemBytes = csmem;
        cfg.stream = stream;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = kHadClusterCtas;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 2;
#define DQ_HAD_CLUSTER(RR)                                                                                  \
  DQ_CHECK_CUDA(cudaLaunchKernelEx(&cfg, act_quant_had_cluster_kernel<RR, XT>, x, up, ldx, a, plan.S, had->scale, \
                                   had->had_mat, codes, sx, out, mode, scale_fp16))
        switch (plan.R) {
          case 4: DQ_HAD_CLUSTER(4); break;
          case 8: DQ_HAD_CLUSTER(8); break;
          case 16: DQ_HAD_CLUSTER(16); break;
          default: DQ_HAD_CLUSTER(32); break;
        }
#undef DQ_HAD_CLUSTER
        return DQ_OK;
      }
      // 28 * 64 ... 28 * 512 values and more rows than the cluster kernel takes (28 * 64: any number): from the first row on
      // it is the faster one (14336, us: 65 rows 14.7 -> 8.1, 300 rows 22.9 -> 15.0; 1792: 70 rows 9.3 -> 7.3)
      if (plan.matrix && plan.inner && plan.S == 28 && plan.R >= 2 && plan.R <= 16) {
#define DQ_HAD28(P)                                                                                                    \
  {                                                                                                                    \
    constexpr bool kExpand = sizeof(XT) == 2;                                                                          \
    ExpansionShare ex = {};                                                                                            \
    const bool both = kExpand && along != nullptr;                                                                     \
    const int ctas = (M + Had28<P>::kRows - 1) / Had28<P>::kRows;                                                      \
    const unsigned grid = both ? along->take(kHad28Threads, ctas, 3, &ex) : static_cast<unsigned>(ctas);               \
    DQ_CHECK_CUDA(launch_pdl(both ? act_quant_had28_kernel<P, XT, kExpand> : act_quant_had28_kernel<P, XT>,            \
                             dim3(grid), dim3(kHad28Threads), Had28<P>::kSmem, stream, x, up, ldx, a, M, had->scale,   \
                             had->had_mat, codes, sx, out, mode, scale_fp16, ex));                                     \
  }
        switch (plan.R) {
          case 2: DQ_HAD28(64); break;
          case 4: DQ_HAD28(128); break;
          case 8: DQ_HAD28(256); break;
          default: DQ_HAD28(512); break;
        }
#undef DQ_HAD28
        return DQ_OK;
      }
      if (plan.matrix) {
        int rc2 = upload_had_matrix(had->had_mat, plan.S, stream);
        if (rc2 != DQ_OK) return rc2;
      }
      // many rows: smaller CTAs, several per SM (the row must leave room for three of them)
      const DeviceState* dst = current_state();
      const bool small_cta = dst != nullptr && M > 2 * dst->sm_count && smem <= 72 * 1024;
#define DQ_HAD_FAST_T(RR, TT, HH)                                                                      \
  DQ_CHECK_CUDA(launch_pdl(act_quant_had_fast_kernel<RR, XT, TT, HH>, dim3(M), dim3(TT), smem, stream, x, up, \
                           ldx, a, K, plan.S, plan.inner, plan.matrix, had->scale, codes, sx,   \
                           out, mode, scale_fp16))
#define DQ_HAD_FAST(RR)                                            \
  if (small_cta) {                                                 \
    DQ_HAD_FAST_T(RR, 256, 0);                                     \
  } else {                                                         \
    DQ_HAD_FAST_T(RR, 512, 0);                                     \
  }
      switch (plan.R) {
        case 1: DQ_HAD_FAST(1); break;
        case 2: DQ_HAD_FAST(2); break;
        case 4: DQ_HAD_FAST(4); break;
        case 8: DQ_HAD_FAST(8); break;
        case 16: DQ_HAD_FAST(16); break;
        default:
          if (plan.matrix && plan.S == 28) DQ_HAD_FAST_T(32, 512, 28);
          else DQ_HAD_FAST(32);
          break;
      }
#undef DQ_HAD_FAST
#undef DQ_HAD_FAST_T
      return DQ_OK;
    }
  return DQ_OK;
}

}  // namespace
}  // namespace dq
