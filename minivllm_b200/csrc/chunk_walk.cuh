// The walk over a sequence's chunks (state_chunk.cuh) on tcgen05, the state in tensor memory.
//
// Everything is transposed: tensor memory's 128 lanes are 128 value columns.  Per chunk of 64 tokens
//   O^T = S_0^T Q^T (+) V^T A^T        S_0 as a TMEM operand in two bf16 terms, V^T straight from rows of tokens (MN-major)
//   S^T = decay S_0^T + V^T K          accumulated onto the decayed state where it lies
// gla and time mixing (kMem false): Q, K and A come decayed and in two terms each from the preparing kernel, as one block of
// scratch that lies there as the swizzled tiles want it, so a chunk is one bulk copy and its V.  mLSTM (kMem): Q and K are the
// projection's rows; alpha is applied to O^T's first product, and w V is split into two terms here.
//
// 18 warps: 0-7 own the state (a thread has a value column and half of the channels: scales, splits and writes it back),
// 8-11 read O and store rows (and carry n and the denominators), 12-15 form w V, 16 issues the products, 17 loads.  The chain of a chunk
// is state -> update -> state; O's products run beside the next chunk's scaling and splitting.  Whole chunks
// come by TMA; a sequence's ragged last chunk is copied by warps 12-15 with zeros past its end, and so are all chunks of rows
// that are not made of whole slabs.
//
// A wait that runs out (or an error word that is set already) ends the CTA.  The warps that issue copies and products and those of
// the state leave their loops before they do anything more; the others go through the rest of theirs, which then changes shared
// memory and rows of a result that nobody may use.  (The warps that read O share a barrier; to agree there on leaving cost mLSTM
// 1.4 %.)  Nobody arrives at a barrier behind a wait that failed: who saw one fail has also seen s_abort.  (With such arrivals a
// launch failed, most likely where a warp's 32 met a barrier of 128 + 1, WB_EMPTY, that lacked one.)  Copies and products in flight
// are waited for, and no state is written.
//
// The roles' loops are rolled: unrolled, five of them pushed one another out of the instruction cache (a fourth of the stalls),
// and a chunk of mLSTM took 4.1 us instead of 3.6.
// Bound: gla and time mixing read 98 KB a chunk, two column blocks of a head the same 82 KB of it, at about 6 TB/s over all SMs
// (L2); mLSTM the chain of w V, state and update.  Before (register MMAs): 885 and 242 us for the two walks below.
//   1 x 16,384 tokens, 8 heads of 128 x 256 (gla, 9 segments): 38 us own states, 11 us join, 74 to 84 us walk
//   16 x 512-1536 tokens, 8 heads of 128 x 256 (mLSTM): 121 us
//
// More CTAs than SMs: the longest sequences go first (that mLSTM walk, 256 CTAs, took 138 us in the order of the batch; gla on the
// same, in all: 216 -> 191 us).
//
// A sequence's chunks take their time one after the other.  Where sequences, heads and column blocks are too few for the SMs,
// sequences are cut into segments: a pass over each segment from a zero state (kState: no O), a join that turns the segments'
// own states into the states in front of them, and the full pass over all segments at once.
#pragma once
#include <atomic>
#include "state_chunk.cuh"
#include "tcgen05.cuh"
#include "tmap.cuh"

namespace mv {

constexpr int kWalkThreads = 18 * 32, kWalkCols = 128;
constexpr int kSlab = kChunk * 128;                       // bytes of 64 rows of 64 bf16 values
constexpr int kWalkV = 2 * kSlab;

// Byte offset of element (row, col) in a tile of 64 rows, slabs of 64 columns, 128-byte swizzle.
__host__ __device__ constexpr int tile_at(int row, int col) {
  return (col >> 6) * kSlab + row * 128 + ((((col & 63) >> 3) ^ (row & 7)) << 4) + (col & 7) * 2;
}

extern std::atomic<int> g_walk_inject;                    // api.cu; the next launch's WalkParams::inject

// Scratch of a chunk and head.  kMem: [A hi, A lo, vectors]; else [Q hi, Q lo, K hi, K lo, A hi, A lo, decays].
template <int K, bool kMem> struct WalkBlob {
  static constexpr int kT = K / 64 * kSlab;               // bytes of a tile of 64 tokens x K
  static constexpr int kQ = 0, kK = 2 * kT, kA = kMem ? 0 : 4 * kT, kVec = kA + 2 * kSlab;
  static constexpr int kFloats = kMem ? 4 * kChunk + K + 4 : K;
  // vectors of kMem, in floats
  static constexpr int kAlpha = 0, kWrite = kChunk, kRow = 2 * kChunk, kFloor = 3 * kChunk, kSum = 4 * kChunk, kDecay = kSum + K;
  static constexpr int64_t kBytes = kVec + kFloats * 4;
};
// One stage of shared memory: the blob, then for kMem Q and K, then V, then for kMem w V in two terms.
template <int K, bool kMem> struct WalkStage {
  using B = WalkBlob<K, kMem>;
  static constexpr int kQ = (static_cast<int>(B::kBytes) + 1023) / 1024 * 1024, kK = kQ + (kMem ? B::kT : 0);
  static constexpr int kV = kK + (kMem ? B::kT : 0), kW = kV + kWalkV, kBytes = kW + (kMem ? 2 * kWalkV : 0);
  static constexpr int kSmem = 2 * kBytes + kChunk * kWalkCols * 2 + 1024;      // stages, rows of O, alignment
};

struct WalkParams {
  __nv_bfloat16* out; int64_t out_stride;
  float* den;                                             // kMem
  const __nv_bfloat16 *q, *k, *v; int64_t stride;         // q and k: kMem
  const int32_t *cu, *slots, *start;
  int num_seqs;
  float *state, *n_state; int num_slots, heads, K, V;
  const unsigned char* scratch;
  int seg_chunks;                                         // chunks of a segment, 0: sequences are whole
  float *seg_state, *seg_n, *seg_decay;                   // per segment and head: K x V, K (kMem), K
  int* error_word;
  bool tma;                                               // whole chunks by TMA
  int inject;                                             // test hook, normally 0.  1: the first CTA's first state warp withholds its
                                                          // second arrival, so that the product warp's bounded wait runs out
};

// Segment x of the batch: its sequence and its place in it.  Whole warp; false past the last.
__device__ __forceinline__ bool find_segment(const int32_t* cu, int num_seqs, int seg_chunks, int x, int& seq, int& seg) {
  const int lane = threadIdx.x & 31, tokens = seg_chunks * kChunk;
  int base = 0;
  for (int b = 0; b < num_seqs; b += 32) {
    const int s = b + lane, n = s < num_seqs ? (max(cu[s + 1] - cu[s], 0) + tokens - 1) / tokens : 0;
    int incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    const uint32_t past = __ballot_sync(0xffffffffu, base + incl > x);
    if (past) {
      const int at = __ffs(past) - 1;
      seq = b + at;
      seg = x - base - __shfl_sync(0xffffffffu, incl - n, at);
      return true;
    }
    base += __shfl_sync(0xffffffffu, incl, 31);
  }
  return false;
}
// The sequence that `rank` others of up to 32 are longer than (or as long and in front of).  Whole warp.
__device__ __forceinline__ int longest_sequence(const int32_t* cu, int num_seqs, int rank) {
  const int lane = threadIdx.x & 31, len = lane < num_seqs ? cu[lane + 1] - cu[lane] : 0;
  int before = 0;
  for (int i = 0; i < num_seqs; ++i) {
    const int other = __shfl_sync(0xffffffffu, len, i);
    before += other > len || (other == len && i < lane) ? 1 : 0;
  }
  return __ffs(__ballot_sync(0xffffffffu, lane < num_seqs && before == rank)) - 1;
}
__device__ __forceinline__ int segments_before(const int32_t* cu, int s, int seg_chunks) {
  int n = 0;
  for (int i = threadIdx.x & 31; i < s; i += 32) n += (max(cu[i + 1] - cu[i], 0) + seg_chunks * kChunk - 1) / (seg_chunks * kChunk);
  return __reduce_add_sync(0xffffffffu, n);
}

namespace tc {
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
// Four K = 16 steps, A and B in shared memory, by the elected lane of a converged warp; descriptors move by kA and kB units.
template <int kA, int kB>
__device__ __forceinline__ void mma_ss_4(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, bool accum) {
  const uint32_t acc = accum ? 1u : 0u;
  asm volatile(
      "{\n\t.reg .pred pe, pt, pf;\n\t.reg .b64 da, db;\n\t"
      "elect.sync _|pe, 0xffffffff;\n\t"
      "setp.eq.u32 pt, %3, %3;\n\t"
      "setp.ne.u32 pf, %4, 0;\n\t"
      "@pe tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, pf;\n\t"
      "add.s64 da, %1, %5;\n\tadd.s64 db, %2, %6;\n\t"
      "@pe tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, pt;\n\t"
      "add.s64 da, %1, %7;\n\tadd.s64 db, %2, %8;\n\t"
      "@pe tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, pt;\n\t"
      "add.s64 da, %1, %9;\n\tadd.s64 db, %2, %10;\n\t"
      "@pe tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, pt;\n\t}"
      ::"r"(d_tmem), "l"(a), "l"(b), "r"(idesc), "r"(acc), "n"(kA), "n"(kB), "n"(2 * kA), "n"(2 * kB), "n"(3 * kA), "n"(3 * kB)
      : "memory");
}
// The same with A in tensor memory, eight columns a step.
template <int kB>
__device__ __forceinline__ void mma_ts_4(uint32_t d_tmem, uint32_t a_tmem, uint64_t b, uint32_t idesc, bool accum) {
  const uint32_t acc = accum ? 1u : 0u;
  asm volatile(
      "{\n\t.reg .pred pe, pt, pf;\n\t.reg .b64 db;\n\t.reg .b32 ta;\n\t"
      "elect.sync _|pe, 0xffffffff;\n\t"
      "setp.eq.u32 pt, %3, %3;\n\t"
      "setp.ne.u32 pf, %4, 0;\n\t"
      "@pe tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, pf;\n\t"
      "add.u32 ta, %1, 8;\n\tadd.s64 db, %2, %5;\n\t"
      "@pe tcgen05.mma.cta_group::1.kind::f16 [%0], [ta], db, %3, pt;\n\t"
      "add.u32 ta, %1, 16;\n\tadd.s64 db, %2, %6;\n\t"
      "@pe tcgen05.mma.cta_group::1.kind::f16 [%0], [ta], db, %3, pt;\n\t"
      "add.u32 ta, %1, 24;\n\tadd.s64 db, %2, %7;\n\t"
      "@pe tcgen05.mma.cta_group::1.kind::f16 [%0], [ta], db, %3, pt;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b), "r"(idesc), "r"(acc), "n"(kB), "n"(2 * kB), "n"(3 * kB) : "memory");
}
}  // namespace tc

enum WalkBar { WB_BLOB = 0, WB_FULL = 2, WB_EMPTY = 4, WB_SREADY = 6, WB_SDONE, WB_ODONE, WB_OFREE, WB_DRAIN, WB_COUNT };

template <int K, bool kMem, bool kState>
__global__ void __launch_bounds__(kWalkThreads, 1)
chunk_walk_kernel(const WalkParams p, const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                  const __grid_constant__ CUtensorMap map_v) {
  using B = WalkBlob<K, kMem>;
  using St = WalkStage<K, kMem>;
  extern __shared__ unsigned char smem_raw[];
  __shared__ uint64_t s_bar[WB_COUNT];
  __shared__ uint32_t s_tmem;
  __shared__ volatile int s_abort;
  __shared__ int s_sticky;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int error = tid == 0 ? *reinterpret_cast<volatile int*>(p.error_word) : 0;
  // what this CTA walks
  int s, seg = 0, unit = blockIdx.x, h = blockIdx.y, block = blockIdx.z;
  if (!p.seg_chunks && p.num_seqs <= 32 && gridDim.x * gridDim.y * gridDim.z > kNumSMs) {      // longest sequences first
    const int per = gridDim.y * gridDim.z, at = unit + p.num_seqs * (h + static_cast<int>(gridDim.y) * block), rest = at % per;
    h = rest / static_cast<int>(gridDim.z);
    block = rest % static_cast<int>(gridDim.z);
    unit = s = longest_sequence(p.cu, p.num_seqs, at / per);
  } else if (p.seg_chunks) {
    if (!find_segment(p.cu, p.num_seqs, p.seg_chunks, unit, s, seg)) return;      // uniform: the grid is an upper bound
  } else {
    s = unit;
  }
  const int p0 = block * kWalkCols, pw = min(kWalkCols, p.V - p0);
  const int n_all = p.cu[s + 1] - p.cu[s];
  if (n_all <= 0) return;
  const int seq_chunks = (n_all + kChunk - 1) / kChunk, c0 = seg * p.seg_chunks;
  const int chunks = p.seg_chunks ? min(p.seg_chunks, seq_chunks - c0) : seq_chunks;
  const bool last_seg = c0 + chunks == seq_chunks;
  if (kState && last_seg) return;                          // nobody starts behind it
  const int first = p.cu[s] + c0 * kChunk, n_tok = n_all - c0 * kChunk;
  const int chunk0 = chunks_before(p.cu, s) + c0;
  const int slot = p.slots[s], st0 = p.start[s];
  const bool live = slot >= 0 && slot < p.num_slots && st0 >= 0;
  const int64_t pair = (static_cast<int64_t>(live ? slot : 0) * p.heads + h), seg_pair = static_cast<int64_t>(unit) * p.heads + h;

  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  unsigned char* smem = smem_raw + (base - smem_u32(smem_raw));
  auto bar = [&](int i) { return smem_u32(&s_bar[i]); };
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(bar(WB_BLOB + i), 1);
      tc::mbar_init(bar(WB_FULL + i), 128);
      tc::mbar_init(bar(WB_EMPTY + i), 1 + 128);
    }
    tc::mbar_init(bar(WB_SREADY), 256);
    tc::mbar_init(bar(WB_SDONE), 1);
    tc::mbar_init(bar(WB_ODONE), 1);
    tc::mbar_init(bar(WB_OFREE), 128);
    tc::mbar_init(bar(WB_DRAIN), 1);
    tc::mbar_fence_init();
    s_abort = 0;
    s_sticky = error;                                      // read once so that the whole CTA agrees
  }
  if (warp == 16) {
    tc::tmem_alloc(smem_u32(&s_tmem), 512);
    tc::tmem_relinquish();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = s_tmem;
  // columns: S, two buffers of [hi | lo], then O (kMem: its two products)
  const uint32_t tS = tmem, tHL = tmem + 128, tO = tmem + 384;
  auto wait = [&](int b, int parity, int where) { return tc::mbar_wait(bar(b), parity, &s_abort, p.error_word, where); };
  auto all = [](bool ok) { return __all_sync(0xffffffffu, ok) != 0; };
  auto aborted = [&] { return __any_sync(0xffffffffu, s_abort) != 0; };
  auto stage_at = [&](int i) { return (i & 1) * St::kBytes; };
  auto whole = [&](int i) { return p.tma && n_tok - i * kChunk >= kChunk; };    // chunk i comes by TMA

  if (s_sticky != 0) {
    // a wait ran out in a launch before: straight to the end, as prefill does
  } else if (warp < 8) {
    // ---------------------------------------------------------------- the state
    const int row = (warp & 3) * 32 + lane, ch0 = (warp >> 2) * (K / 2);
    const bool on = row < pw;
    const uint32_t lanes = static_cast<uint32_t>(warp & 3) << 21;
    const uint32_t own = tS + lanes + ch0;
    {
      const float* src = (p.seg_chunks ? p.seg_state + seg_pair * p.K * p.V : p.state + pair * p.K * p.V) + p0 + row;
      const bool has = !kState && on && (p.seg_chunks || (live && st0 > 0));
#pragma unroll 1
      for (int c = 0; c < K / 2; c += 16) {
        uint32_t x[16];
#pragma unroll
        for (int e = 0; e < 16; ++e)
          x[e] = has && ch0 + c + e < p.K ? __float_as_uint(src[static_cast<int64_t>(ch0 + c + e) * p.V]) : 0u;
        tc::tmem_st16(own + c, x);
      }
      tc::wait_st();
    }
    for (int i = 0; i < chunks; ++i) {
      const unsigned char* st = smem + stage_at(i);
      bool ok = i == 0 || wait(WB_SDONE, (i - 1) & 1, 1);
      ok = all(wait(WB_BLOB + (i & 1), (i >> 1) & 1, 2) && ok);
      if (!ok) break;
      tc::fence_after_sync();
      const float* vec = reinterpret_cast<const float*>(st + B::kVec);
      const uint32_t hl = tHL + (i & 1) * 128 + lanes + ch0 / 2;
#pragma unroll 1
      for (int c = 0; c < K / 2; c += 32) {
        uint32_t x[32];
        tc::tmem_ld32(own + c, x);
        tc::wait_ld();
#pragma unroll
        for (int half = 0; half < 32; half += 16) {
          if (!kState) {
            uint32_t hi[8], lo[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) split2(__uint_as_float(x[half + 2 * e]), __uint_as_float(x[half + 2 * e + 1]), hi[e], lo[e]);
            tc::tmem_st8(hl + (c + half) / 2, hi);
            tc::tmem_st8(hl + 64 + (c + half) / 2, lo);
          }
#pragma unroll
          for (int e = 0; e < 16; e += 4) {
            float4 d;
            if constexpr (kMem) d = make_float4(vec[B::kDecay], vec[B::kDecay], vec[B::kDecay], vec[B::kDecay]);
            else d = *reinterpret_cast<const float4*>(vec + ch0 + c + half + e);
            const float2 lo2 = mul_f32x2(make_float2(__uint_as_float(x[half + e]), __uint_as_float(x[half + e + 1])), make_float2(d.x, d.y));
            const float2 hi2 = mul_f32x2(make_float2(__uint_as_float(x[half + e + 2]), __uint_as_float(x[half + e + 3])), make_float2(d.z, d.w));
            x[half + e] = __float_as_uint(lo2.x); x[half + e + 1] = __float_as_uint(lo2.y);
            x[half + e + 2] = __float_as_uint(hi2.x); x[half + e + 3] = __float_as_uint(hi2.y);
          }
        }
        tc::tmem_st32(own + c, x);
      }
      tc::wait_st();
      tc::fence_before_sync();
      if (!(p.inject == 1 && i == 1 && warp == 0 && blockIdx.x + blockIdx.y + blockIdx.z == 0)) tc::mbar_arrive(bar(WB_SREADY));
    }
    wait(WB_SDONE, (chunks - 1) & 1, 3);
    tc::fence_after_sync();
    const bool keep = !aborted() && on && (kState || (last_seg && live));
    float* dst = (kState ? p.seg_state + seg_pair * p.K * p.V : p.state + pair * p.K * p.V) + p0 + row;
#pragma unroll 1
    for (int c = 0; c < K / 2; c += 16) {
      uint32_t x[16];
      tc::tmem_ld16(own + c, x);
      tc::wait_ld();
      if (keep) {
#pragma unroll
        for (int e = 0; e < 16; ++e)
          if (ch0 + c + e < p.K) dst[static_cast<int64_t>(ch0 + c + e) * p.V] = __uint_as_float(x[e]);
      }
    }
  } else if (warp < 12) {
    // ---------------------------------------------------------------- results
    const int t = tid - 256, lw = warp - 8, row = lw * 32 + lane;
    const uint32_t lanes = static_cast<uint32_t>(lw) << 21;
    const bool first_block = block == 0, keeps_n = kMem && first_block;
    constexpr int kPer = K / 32;
    float n[kPer], prod = 1.f;                             // channels lane * kPer ..; the segment's decay of channel t
    if constexpr (kMem) {
      const float* src = p.seg_chunks ? p.seg_n + seg_pair * p.K : p.n_state + pair * p.K;
#pragma unroll
      for (int e = 0; e < kPer; ++e) {
        const int ch = lane * kPer + e;
        n[e] = !kState && keeps_n && ch < p.K && (p.seg_chunks || (live && st0 > 0)) ? src[ch] : 0.f;
      }
    }
    __nv_bfloat16* rows = reinterpret_cast<__nv_bfloat16*>(smem + 2 * St::kBytes);
    for (int i = 0; i < chunks; ++i) {
      unsigned char* st = smem + stage_at(i);
      const float* vec = reinterpret_cast<const float*>(st + B::kVec);
      const int nt = min(kChunk, n_tok - i * kChunk);
      if (kState) {
        wait(WB_BLOB + (i & 1), (i >> 1) & 1, 7);
        if (first_block && t < K) prod *= kMem ? vec[B::kDecay] : vec[t];
      }
      if constexpr (kMem) {
        if (keeps_n) {
          if constexpr (!kState) {
            wait(WB_FULL + (i & 1), (i >> 1) & 1, 6);
#pragma unroll 2
            for (int r = 0; r < 16; r += 2) {              // two tokens at a time, each half of the warp ends with one
              float d[2];
#pragma unroll
              for (int x = 0; x < 2; ++x) {
                const unsigned char* qr = st + St::kQ + tile_at(lw * 16 + r + x, lane * kPer);
                d[x] = 0.f;
#pragma unroll
                for (int e = 0; e < kPer; e += 2) {
                  const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(qr + e * 2));
                  d[x] = fmaf(n[e + 1], f.y, fmaf(n[e], f.x, d[x]));
                }
              }
              float dot = (lane & 16 ? d[1] : d[0]) + __shfl_xor_sync(0xffffffffu, lane & 16 ? d[0] : d[1], 16);
#pragma unroll
              for (int o = 8; o >= 1; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
              const int tok = lw * 16 + r + (lane >> 4);
              if (!(lane & 15) && tok < nt)
                p.den[(static_cast<int64_t>(first) + i * kChunk + tok) * p.heads + h] =
                    fmaxf(fabsf(fmaf(vec[B::kAlpha + tok], dot, vec[B::kRow + tok])), vec[B::kFloor + tok]) + kMemFloor;
            }
          }
#pragma unroll
          for (int e = 0; e < kPer; ++e) n[e] = fmaf(vec[B::kDecay], n[e], vec[B::kSum + lane * kPer + e]);
        }
      }
      if constexpr (kState) {
        if (!s_abort) tc::mbar_arrive(bar(WB_EMPTY + (i & 1)));
        continue;
      }
      wait(WB_ODONE, i & 1, 4);
      __syncwarp();
      tc::fence_after_sync();
      asm volatile("bar.sync 1, 128;" ::: "memory");       // the rows of the chunk before are stored
#pragma unroll 1
      for (int c = 0; c < kChunk; c += 16) {
        uint32_t o[16];
        tc::tmem_ld16(tO + lanes + c, o);
        if constexpr (kMem) {
          uint32_t a[16];
          tc::tmem_ld16(tO + 64 + lanes + c, a);
          tc::wait_ld();
#pragma unroll
          for (int e = 0; e < 16; e += 2) {
            const float2 x = fma_f32x2(make_float2(__uint_as_float(o[e]), __uint_as_float(o[e + 1])), *reinterpret_cast<const float2*>(vec + B::kAlpha + c + e),
                                       make_float2(__uint_as_float(a[e]), __uint_as_float(a[e + 1])));
            o[e] = __float_as_uint(x.x);
            o[e + 1] = __float_as_uint(x.y);
          }
        } else {
          tc::wait_ld();
        }
#pragma unroll
        for (int e = 0; e < 16; ++e) rows[(c + e) * kWalkCols + row] = __float2bfloat16_rn(__uint_as_float(o[e]));
      }
      tc::fence_before_sync();
      if (!s_abort) {
        tc::mbar_arrive(bar(WB_EMPTY + (i & 1)));          // the stage's vectors and Q are read
        tc::mbar_arrive(bar(WB_OFREE));
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");
      __nv_bfloat16* dst = p.out + (static_cast<int64_t>(first) + i * kChunk) * p.out_stride + static_cast<int64_t>(h) * p.V + p0;
#pragma unroll 2
      for (int j = 0; j < 8; ++j) {
        const int r = j * 8 + (t >> 4), c = (t & 15) * 8;
        if (r < nt && c < pw)
          *reinterpret_cast<uint4*>(dst + static_cast<int64_t>(r) * p.out_stride + c) = *reinterpret_cast<const uint4*>(rows + r * kWalkCols + c);
      }
    }
    const bool ok = !aborted();
    if (kState && ok && first_block && t < p.K) p.seg_decay[seg_pair * p.K + t] = prod;
    if constexpr (kMem) {
      if (ok && keeps_n && lw == 0 && (kState || (last_seg && live))) {
        float* dst = kState ? p.seg_n + seg_pair * p.K : p.n_state + pair * p.K;
#pragma unroll
        for (int e = 0; e < kPer; ++e)
          if (lane * kPer + e < p.K) dst[lane * kPer + e] = n[e];
      }
    }
  } else if (warp < 16) {
    // ---------------------------------------------------------------- w V, ragged chunks
    const int t = tid - 384;
    const __nv_bfloat16* v = p.v + static_cast<int64_t>(h) * p.V + p0;
    auto copy = [&](int i) {
      const int s2 = i & 1, nt = min(kChunk, n_tok - i * kChunk);
      const uint32_t st = base + stage_at(i);
      if (i >= 2) wait(WB_EMPTY + s2, ((i >> 1) - 1) & 1, 5);
      const int64_t row0 = static_cast<int64_t>(first) + i * kChunk;
#pragma unroll 2
      for (int j = 0; j < 8; ++j) {
        const int r = j * 8 + (t >> 4), c = (t & 15) * 8;
        const bool ok = r < nt && c < pw;
        cp_async16(st + St::kV + tile_at(r, c), ok ? v + (row0 + r) * p.stride + c : p.v, ok ? 16 : 0);
      }
      if constexpr (kMem) {
#pragma unroll 2
        for (int j = t; j < kChunk * (K / 8); j += 128) {
          const int r = j / (K / 8), c = (j % (K / 8)) * 8;
          const bool ok = r < nt && c < p.K;
          const int64_t off = ok ? (row0 + r) * p.stride + h * p.K + c : 0;
          if (!kState) cp_async16(st + St::kQ + tile_at(r, c), p.q + off, ok ? 16 : 0);
          cp_async16(st + St::kK + tile_at(r, c), p.k + off, ok ? 16 : 0);
        }
      }
    };
    if (!whole(0)) copy(0);
    cp_async_commit();
    for (int i = 0; i < chunks; ++i) {
      if (i + 1 < chunks && !whole(i + 1)) copy(i + 1);
      cp_async_commit();
      cp_async_wait<1>();                                  // empty groups where chunks come by TMA
      wait(WB_BLOB + (i & 1), (i >> 1) & 1, 12);
      if constexpr (kMem) {
        unsigned char* st = smem + stage_at(i);
        const float* vec = reinterpret_cast<const float*>(st + B::kVec);
#pragma unroll 2
        for (int j = 0; j < 8; ++j) {                      // w V; a thread takes the pieces that it may have copied
          const int r = j * 8 + (t >> 4), at = tile_at(r, (t & 15) * 8);
          const float w = vec[B::kWrite + r];
          const uint4 x = *reinterpret_cast<const uint4*>(st + St::kV + at);
          const uint32_t xs[4] = {x.x, x.y, x.z, x.w};
          uint32_t hi[4], lo[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&xs[e]));
            const float2 y = mul_f32x2(f, make_float2(w, w));
            split2(y.x, y.y, hi[e], lo[e]);
          }
          *reinterpret_cast<uint4*>(st + St::kW + at) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
          *reinterpret_cast<uint4*>(st + St::kW + kWalkV + at) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        }
      }
      tc::fence_async_proxy();
      if (!s_abort) tc::mbar_arrive(bar(WB_FULL + (i & 1)));
    }
    cp_async_wait<0>();
  } else if (warp == 17) {
    // ---------------------------------------------------------------- loads
    if (lane == 0) {
      int i = 0;
      for (; i < chunks; ++i) {
        const uint32_t st = base + stage_at(i), b = bar(WB_BLOB + (i & 1));
        const bool rows = whole(i);
        if (i >= 2 && !wait(WB_EMPTY + (i & 1), ((i >> 1) - 1) & 1, 13)) break;
        const unsigned char* src = p.scratch + (static_cast<int64_t>(chunk0 + i) * p.heads + h) * B::kBytes;
        constexpr uint32_t kBlob = kState ? (kMem ? 0 : 2 * B::kT) + B::kFloats * 4 : static_cast<uint32_t>(B::kBytes);
        constexpr uint32_t kRows = kWalkV + (kMem ? (kState ? 1 : 2) * B::kT : 0);
        tc::mbar_expect_tx(b, kBlob + (rows ? kRows : 0));
        if (kState) {
          if (!kMem) tc::bulk_load(st + B::kK, src + B::kK, 2 * B::kT, b);
          tc::bulk_load(st + B::kVec, src + B::kVec, B::kFloats * 4, b);
        } else {
          tc::bulk_load(st, src, static_cast<uint32_t>(B::kBytes), b);
        }
        if (rows) {
          const int row0 = first + i * kChunk;
#pragma unroll
          for (int c = 0; c < kWalkCols; c += 64) tc::tma_load_3d(st + St::kV + c / 64 * kSlab, &map_v, h * p.V + p0 + c, row0, 0, b);
          if constexpr (kMem) {
#pragma unroll
            for (int c = 0; c < K; c += 64) {
              if (!kState) tc::tma_load_3d(st + St::kQ + c / 64 * kSlab, &map_q, h * p.K + c, row0, 0, b);
              tc::tma_load_3d(st + St::kK + c / 64 * kSlab, &map_k, h * p.K + c, row0, 0, b);
            }
          }
        }
      }
      // Nobody may be left to wait for the copies of the last two chunks asked for (an empty stage says that those before have
      // landed): they must not find the CTA gone.
      for (int j = max(0, i - 2); j < i; ++j) tc::mbar_wait_timed(bar(WB_BLOB + (j & 1)), (j >> 1) & 1);
    }
    __syncwarp();
  } else {
    // ---------------------------------------------------------------- products
    constexpr uint32_t kMN = 1u << 15;                     // A is MN-major
    constexpr uint32_t kUpdate = tc::instr_desc_f16(1, 1, true, 128, K) | kMN, kRead = tc::instr_desc_f16(1, 1, false, 128, kChunk),
                       kLocal = kRead | kMN;
    auto mn = [&](uint32_t at) { return tc::desc64(tc::desc_lo(at, kSlab), tc::kDescHiSw128Sbo1024); };
    auto km = [&](uint32_t at) { return tc::desc64(tc::desc_lo(at, 16), tc::kDescHiSw128Sbo1024); };
    for (int i = 0; i < chunks; ++i) {
      const uint32_t st = base + stage_at(i);
      if (!all(wait(WB_BLOB + (i & 1), (i >> 1) & 1, 8) && wait(WB_FULL + (i & 1), (i >> 1) & 1, 9) && wait(WB_SREADY, i & 1, 10))) break;
      tc::fence_after_sync();
      if constexpr (kMem) {
        tc::mma_ss_4<128, 128>(tS, mn(st + St::kW), mn(st + St::kK), kUpdate, true);
        tc::mma_ss_4<128, 128>(tS, mn(st + St::kW + kWalkV), mn(st + St::kK), kUpdate, true);
      } else {
        tc::mma_ss_4<128, 128>(tS, mn(st + St::kV), mn(st + B::kK), kUpdate, true);
        tc::mma_ss_4<128, 128>(tS, mn(st + St::kV), mn(st + B::kK + B::kT), kUpdate, true);
      }
      if constexpr (kState) {
        tc::commit_elected(bar(WB_SDONE), bar(WB_EMPTY + (i & 1)), true);
      } else {
        tc::commit_elected(bar(WB_SDONE), 0, false);
        if (i > 0 && !all(wait(WB_OFREE, (i - 1) & 1, 11))) break;
        tc::fence_after_sync();
        const uint32_t hi = tHL + (i & 1) * 128, lo = hi + 64, q = kMem ? st + St::kQ : st + B::kQ;
#pragma unroll
        for (int k = 0; k < K / 64; ++k) {
          tc::mma_ts_4<2>(tO, hi + k * 32, km(q + k * kSlab), kRead, k > 0);
          tc::mma_ts_4<2>(tO, lo + k * 32, km(q + k * kSlab), kRead, true);
          if (!kMem) tc::mma_ts_4<2>(tO, hi + k * 32, km(q + B::kT + k * kSlab), kRead, true);
        }
        const uint32_t o2 = kMem ? tO + 64 : tO;
        tc::mma_ss_4<128, 2>(o2, mn(st + St::kV), km(st + B::kA), kLocal, !kMem);
        tc::mma_ss_4<128, 2>(o2, mn(st + St::kV), km(st + B::kA + kSlab), kLocal, true);
        tc::commit_elected(bar(WB_ODONE), bar(WB_EMPTY + (i & 1)), true);
      }
    }
    __syncwarp();
    if (aborted()) {                                       // nobody may have waited for the last products: they must have run
      tc::commit_elected(bar(WB_DRAIN), 0, false);         // before tensor memory is freed
      tc::mbar_wait_timed(bar(WB_DRAIN), 0);
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 16) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, 512);
  }
}

// The segments' own states become the states in front of them, a thread per element of a sequence's and head's state; kMem: n
// behind them.  Loads of eight segments are in flight at a time.
constexpr int kJoinThreads = 256, kJoinBatch = 8;
template <bool kMem>
__global__ void __launch_bounds__(kJoinThreads) chunk_join_kernel(const WalkParams p) {
  const int s = blockIdx.x, h = blockIdx.y, at = blockIdx.z * kJoinThreads + threadIdx.x, size = p.K * p.V;
  const int n_tok = p.cu[s + 1] - p.cu[s];
  if (n_tok <= 0) return;
  const int per = p.seg_chunks * kChunk, segs = (n_tok + per - 1) / per, u0 = segments_before(p.cu, s, p.seg_chunks);
  if (at >= size + (kMem ? p.K : 0)) return;
  const int slot = p.slots[s], st0 = p.start[s];
  const bool has = slot >= 0 && slot < p.num_slots && st0 > 0, in_n = at >= size;
  const int64_t pair = static_cast<int64_t>(has ? slot : 0) * p.heads + h, unit = static_cast<int64_t>(u0) * p.heads + h;
  const int ch = in_n ? at - size : at / p.V;
  float* own_at = in_n ? p.seg_n + unit * p.K + ch : p.seg_state + unit * size + at;
  const int64_t step = static_cast<int64_t>(p.heads) * (in_n ? p.K : size);
  const float* decay = p.seg_decay + unit * p.K + ch;
  float x = !has ? 0.f : in_n ? p.n_state[pair * p.K + ch] : p.state[pair * size + at];
  for (int g0 = 0; g0 < segs; g0 += kJoinBatch) {
    float own[kJoinBatch], d[kJoinBatch];
#pragma unroll
    for (int j = 0; j < kJoinBatch; ++j) {
      const bool ok = g0 + j < segs - 1;
      own[j] = ok ? own_at[(g0 + j) * step] : 0.f;
      d[j] = ok ? decay[static_cast<int64_t>(g0 + j) * p.heads * p.K] : 0.f;
    }
#pragma unroll
    for (int j = 0; j < kJoinBatch; ++j)
      if (g0 + j < segs) {
        own_at[(g0 + j) * step] = x;
        x = fmaf(x, d[j], own[j]);
      }
  }
}

// Chunks of a segment, or 0 for whole sequences.  A segment costs a second, lighter pass and the join, so sequences are cut only
// where that brings at least three times as many CTAs, none shorter than four chunks, all of them within one wave, and where the mean
// sequence has more than three (mLSTM, whose chunks take twice as long: two) segments' chunks.  One sequence, 4 heads of 128 x 128:
// gla 8 chunks 31.3 us whole and 37.6 in segments, 16 chunks 45.6 and 38.2; mLSTM 8 chunks 36.3 and 38.3, 16 chunks 62.7 and 37.8.
inline int walk_segment(bool mem, int64_t tokens, int num_seqs, int heads, int V) {
  const int64_t blocks = static_cast<int64_t>(heads) * ((V + kWalkCols - 1) / kWalkCols);
  const int64_t all = kNumSMs / blocks;                     // segments there is room for
  if (num_seqs <= 0 || all < 3 * num_seqs) return 0;
  const int64_t room = num_seqs > 1 ? all - num_seqs : all; // each sequence's last segment may be a short one
  const int64_t chunks = (tokens + kChunk - 1) / kChunk, per = std::max<int64_t>(4, (chunks + room - 1) / room);
  return chunks > (mem ? 2 : 3) * per * num_seqs ? static_cast<int>(per) : 0;
}
// Whether the walk takes a call; the register form keeps narrow heads, where most of 128 lanes would idle, and short work, where
// setting the walk up (2 us) is not paid back.  us, walk and register form:
//   gla, 32 of 32 tokens, 16 heads of 64 x 128 44.0 and 40.7, 128 of 64 160 and 164; 8 heads of 64 x 72, 64 of 17 40.0 and 37.9,
//     16 of 128 19.9 and 21.0; heads of 128 x 256, 16 of 32 32.9 and 33.8
//   mLSTM, heads of 128: 4 x 128, 16 of 64 14.3 and 13.3, 64 of 64 24.9 and 27.5; 8 x 256, 32 of 32 42.4 and 40.6, 64 of 64 70.0 and 74.7
//     heads of 64: 16 x 128, 64 of 64 67.9 and 62.9, 16 of 128 31.8 and 33.8, 4 of 256 23.4 and 23.0, 16 of 256 46.4 and 53.8;
//     8 x 72, 64 of 128 55.7 and 54.2, 16 of 256 26.6 and 28.2; 4 x 128, 16 of 512 36.4 and 36.8, 1 of 512 33.9 and 31.7
//     heads that are not made of slabs, whose q and k four warps copy: 8 x 48 (96), 8 of 1024 79.8 and 66.1
inline bool walk_takes(bool mem, int64_t tokens, int num_seqs, int heads, int K, int V) {
  if (K <= 32 || V <= 64) return false;
  if (num_seqs <= 0 || walk_segment(mem, tokens, num_seqs, heads, V)) return true;
  const int64_t mean = tokens / num_seqs, pairs = static_cast<int64_t>(num_seqs) * heads, ctas = pairs * ((V + kWalkCols - 1) / kWalkCols);
  if (!mem) return K > 64 || mean > kChunk || (V % kWalkCols == 0 && pairs > 512);
  if (K % 64) return false;
  if (K > 64) return mean > kChunk || (ctas >= kNumSMs && (V <= kWalkCols || mean > kChunk / 2 || pairs > 256));
  return ctas >= 128 ? mean >= (V % kWalkCols ? 256 : 96) : ctas >= 48 && mean >= 512;
}
inline int64_t walk_segments(int64_t tokens, int num_seqs, int per) { return per ? tokens / (per * kChunk) + std::min<int64_t>(num_seqs, tokens) : 0; }
// Floats of the segments' states, n and decays.
inline int64_t walk_segment_floats(bool mem, int64_t tokens, int num_seqs, int heads, int K, int V) {
  return walk_segments(tokens, num_seqs, walk_segment(mem, tokens, num_seqs, heads, V)) * heads * (static_cast<int64_t>(K) * V + 2 * K);
}

// scratch holds the chunks' blobs, `segments` (16-byte aligned) walk_segment_floats.
template <int K, bool kMem>
int run_walk(const char* what, WalkParams p, int64_t tokens, float* segments, cudaStream_t st) {
  p.inject = g_walk_inject.exchange(0);                    // one call only
  p.seg_chunks = walk_segment(kMem, tokens, p.num_seqs, p.heads, p.V);
  const int64_t units = p.seg_chunks ? walk_segments(tokens, p.num_seqs, p.seg_chunks) : p.num_seqs;
  p.seg_state = segments;
  p.seg_n = segments + units * p.heads * p.K * p.V;
  p.seg_decay = p.seg_n + units * p.heads * p.K;
  constexpr int smem = WalkStage<K, kMem>::kSmem;
  static_assert(smem + 256 <= 227 * 1024, "a CTA's shared memory");
  const dim3 grid(static_cast<unsigned>(units), p.heads, (p.V + kWalkCols - 1) / kWalkCols);
  CUtensorMap maps[3] = {};
  p.tma = !kMem || p.K % 64 == 0;                          // a box of 64 columns of q or k stays within its head
  const __nv_bfloat16* from[3] = {kMem ? p.q : p.v, kMem ? p.k : p.v, p.v};
  for (int i = 0; i < 3 && p.tma; ++i) {
    const int64_t cols = static_cast<int64_t>(p.heads) * (i < 2 && kMem ? p.K : p.V);
    const int rc = make_tmap_bf16(&maps[i], from[i], cols, tokens, 1, p.stride, p.stride * tokens, kChunk, 1, what);
    if (rc) return rc;
  }
  auto launch = [&](auto kernel, dim3 g) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return fail(MV_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
    kernel<<<g, kWalkThreads, smem, st>>>(p, maps[0], maps[1], maps[2]);
    return check_launch(what);
  };
  if (p.seg_chunks) {
    int rc = launch(chunk_walk_kernel<K, kMem, true>, grid);
    if (rc) return rc;
    chunk_join_kernel<kMem><<<dim3(p.num_seqs, p.heads, (p.K * (p.V + (kMem ? 1 : 0)) + kJoinThreads - 1) / kJoinThreads), kJoinThreads, 0, st>>>(p);
    rc = check_launch(what);
    if (rc) return rc;
  }
  return launch(chunk_walk_kernel<K, kMem, false>, grid);
}

}  // namespace mv
