// The persistent prefill kernel on tcgen05: causal attention over packed sequences or a paged cache (prefill_varlen.cu), or with a
// sliding window, a bias per distance and a sink per head over packed keys (kWin; latent_prefill.cu).  Tensor memory and arithmetic
// as in prefill_varlen.cu; sixteen softmax warps and the roles below.
#pragma once
#include "mma.cuh"
#include "tcgen05.cuh"
#include <cuda.h>
#include <algorithm>
#include <atomic>
#include <type_traits>

namespace mv {

constexpr int kPfTile = 128;         // query rows and KV columns per tile
constexpr int kPfD = 128;
constexpr int kPfHalfBytes = kPfTile * 128;                 // one 64-element half of a 128-row tile
constexpr int kPfTileBytes = 2 * kPfHalfBytes;              // 32 KB
constexpr int kPfStages = 2;
constexpr int kPfSmemBytes = 2 * kPfTileBytes + 2 * kPfStages * kPfTileBytes + 1024;  // Q(2 heads) + K ring + V ring + align
constexpr float kRescaleThreshold = 8.f;                    // of a row's maximum, log2 units

struct PrefillParams {
  void* out;
  int64_t out_stride_tok;  // elements
  int out_align32;         // output rows start on 32-byte boundaries
  int inject;              // test hook, normally 0.  1: head A of tile 0 withholds its first "P ready" arrival,
                           // so that the MMA warp's bounded wait runs out and the abort path is exercised
  const int32_t* cu_seqlens;
  int num_seqs, num_heads, num_kv_heads, group, pairs;  // pairs = ceil(group / 2)
  float scale_log2;
  int fmt;          // 0 fp16, 1 bf16
  int* error_word;
  // Paged mode (prefix hit / chunked prefill): K and V are read from the paged cache through the block
  // tables, and sequence s has cu_seqlens_k-many keys of which the first (keys - queries) are already cached.
  int paged;
  const int32_t* cu_seqlens_k;
  const int32_t* block_tables;
  int64_t bt_stride;
  int max_blocks, block_size, box_rows;   // box_rows = min(block_size, 128): rows of one TMA box of the cache
  int sched_slot;                         // persistent form: which work counter this launch uses
  // Windowed form: packed keys (cu_seqlens_k), a bias (heads, distances) fp32 or null, a sink per head or null.
  int window, distances;
  const float* bias;
  int64_t bias_stride;
  const __nv_bfloat16* sink;
};

#ifdef MV_PF_TRACE
// Timeline probe (debug builds only, -DMV_PF_TRACE): one thread of each role of ONE CTA writes clock64()
// stamps per KV step, so that the phases of the pipeline can be read off without a profiler.
// Buffer (long long, 2048 entries, set with mv_debug_prefill_trace): entry ((role * 32 + i) * 8 + k) is stamp k
// of role `role` at index i.  One CTA per tile: i = KV step.  Persistent kernel: i = the CTA's unit number,
// roles 0 producer, 1 MMA warp, 2 / 3 first softmax warp of head A / B (entry k = 7 of role 0 holds the unit's
// number of KV steps); PF_STEP adds, from entry 1024 on, per-step stamps of the CTA's fourth unit
// ((role * 8 + step) * 8 + k; roles 0 MMA warp, 1 / 2 softmax A / B).
static __device__ long long* g_pf_trace = nullptr;
static __device__ int g_pf_trace_cta = -1;
// pf_tr is read once per thread at kernel start: a stamp is then one predicated store, cheap enough not to
// distort the warp it measures.
#define PF_STAMP(role, j, k)                                                      \
  do {                                                                            \
    if (pf_tr && (j) < 32) pf_tr[((role) * 32 + (j)) * 8 + (k)] = clock64();      \
  } while (0)
#define PF_TRACE_INIT() \
  long long* const pf_tr = (static_cast<int>(blockIdx.x) == g_pf_trace_cta && blockIdx.y == 0) ? g_pf_trace : nullptr
#define PF_STEP(unit, role, j, k)                                                              \
  do {                                                                                          \
    if (pf_tr && (unit) == 3 && (j) < 8) pf_tr[1024 + ((role) * 8 + (j)) * 8 + (k)] = clock64(); \
  } while (0)
#else
#define PF_STEP(unit, role, j, k) do {} while (0)
#define PF_STAMP(role, j, k) do {} while (0)
#define PF_TRACE_INIT() do {} while (0)
#endif

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// ---------------------------------------------------------------------------------------------
// Persistent form of the same kernel: one CTA per SM works through units (query tile x head pair).  The first
// unit of a CTA is its block index, further ones come from a counter in device memory (whoever is free takes
// the next; the KV loops of the units differ in length by up to the number of tiles of a sequence).  Tensor
// memory and the mbarriers are set up once; every role treats its units as one continuous stream of KV steps
// (ring stages and barrier phases run on across units), so the producer's loads and the first S = Q K^T of the
// next unit are under way while the softmax warps write the current unit's output, and nothing is torn down
// or set up between units.
//   Units: the producer warp looks a unit up (binary search in the tiles-before-sequence prefix sums, which
//   live in shared memory behind the tile buffers) and publishes what the other roles need of it in a ring of
//   descriptors (UFULL / UEMPTY), one unit ahead of the MMA warp.
//   Q buffer: QEMPTY is committed behind the unit's last QK, the producer waits for it before the next Q.
//   O accumulators: OFREE[t] gets an arrival of each of head t's softmax warps when it has read O in the epilogue;
//   the MMA warp waits for it before the first PV of head t's next unit.
//   Softmax: eight warps a head, 16 rows each.  With four a head and a whole row a thread, the first tile of a unit took
//   2,900 cycles behind its QK and the epilogue 2,000 during which the tensor cores idled: 4.3 us a unit beside its steps.  A
//   warpgroup of its own for the epilogue was measured too: it takes issue slots from the softmax and gained half as much.
//   Output: rows leave by TMA through each warp's staging buffer (a thread storing its own row makes 32 lines per
//   instruction, and the stores of one unit then hold up every shared-memory access of the SM for about 2,000 cycles).
//   32/8 heads, bf16, a graph of six launches on one input: 32 sequences of 128 to 2048 tokens 422 -> 396 us; 16 portions behind
//   cached halves 278 -> 243; 64 x 512 tokens 306 -> 229 us.  Inputs that change from call to call: 492 -> 464 and 307 -> 277.
//   Long sequences run at the power limit (56 % of the tensor cycles at 1.5 GHz, 1.2 PFLOP/s).
//   Code size: the MMA warp shares an instruction cache with the large softmax loop.  Its waits are the compact
//   form (rolled spin, the long-wait part a call) and the two warps with few registers keep their loops small;
//   with unrolled waits the same kernel was 25 % slower on the 32-sequence benchmark.
// ---------------------------------------------------------------------------------------------
enum { PB_Q = 0, PB_QEMPTY = 1, PB_KFULL = 2, PB_KEMPTY = 4, PB_VFULL = 6, PB_VEMPTY = 8, PB_SFULL = 10, PB_PREADY = 12,
       PB_ODONE = 14, PB_OFREE = 16, PB_SPARE = 18, PB_DRAIN = 19, PB_UFULL = 20, PB_UEMPTY = 24, PB_BFULL = 28, PB_BFREE = 30,
       PB_COUNT = 32 };
constexpr int kPpSoftWarps = 16, kPpThreads = kPpSoftWarps * 32 + 128;      // registers: 512 x 104 + 128 x 64, launched with 640 x 96
// Output staging of one softmax warp: 16 rows x 64 outputs, or 8 rows where bias tables need the room.
template <bool kWin> struct PfOut {
  static constexpr int kRows = kWin ? 8 : 16, kWarpBytes = kRows * 128, kBytes = kPpSoftWarps * kWarpBytes;
};
// Bias table of a head in the windowed form: an entry per distance with -inf where it is not visible, from -kPfBefore on (the
// first row to the last key of its tile) to kPfAfter past the last one that has a bias of its own.
constexpr int kPfBefore = 256, kPfAfter = 256, kPfMaxDistances = 512;
__device__ __forceinline__ void st_matrix4(uint32_t addr, const uint32_t (&r)[4]) {       // four 8 x 8 matrices of 16-bit values
  asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
}
__device__ __forceinline__ uint4 ld_shared16(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
constexpr int kPfSortSeqs = 8;      // sequences up to which units are sorted: a lookup goes through them, several times where they
                                    // have few tiles (at 32 sequences, 128 to 2048 tokens, one input, 421 us instead of 395)
constexpr int kPfUnitRing = 4;      // units handed from the producer warp to the other roles ahead of time
// Work counters of the persistent launches: [slot][0] = units handed out beyond the first one per CTA, [slot][1] = CTAs that have
// finished.  Zero between launches: the last CTA of a launch clears its slot.  Launches take the first kPfSchedSlots in turn, one
// sequence for the table whatever the instantiation, so that as many may be in flight.  A captured launch keeps its slot for as long
// as its graph is replayed, beside any number of others: those have slots of their own, each handed out once.
constexpr int kPfSchedSlots = 1024, kPfGraphSlots = 4096;
static __device__ unsigned int g_pf_sched[kPfSchedSlots + kPfGraphSlots][2];
static std::atomic<unsigned> g_pf_next{0};
static std::atomic<int> g_pf_graph_next{0};
static std::atomic<int> g_pf_last{-1};      // what the last launch was given, for tests
// -1: captured launches have taken all of theirs; the caller has a form without counters.
static int pf_take_slot(cudaStream_t st) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &status) != cudaSuccess) {
    cudaGetLastError();
    status = cudaStreamCaptureStatusNone;
  }
  int slot = -1;
  if (status == cudaStreamCaptureStatusNone) {
    slot = static_cast<int>(g_pf_next.fetch_add(1) % kPfSchedSlots);
  } else {
    int n = g_pf_graph_next.load();
    while (n < kPfGraphSlots && !g_pf_graph_next.compare_exchange_weak(n, n + 1)) {}
    if (n < kPfGraphSlots) slot = kPfSchedSlots + n;
  }
  g_pf_last.store(slot);
  return slot;
}

template <typename T, bool kWin>
__global__ void __launch_bounds__(kPpThreads, 1)
prefill_persistent_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                          const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_o, const PrefillParams p) {
  constexpr int kOutRows = PfOut<kWin>::kRows;
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bars[PB_COUNT];
  __shared__ uint32_t s_tmem_base;
  __shared__ int s_scan[kPpThreads / 32];
  __shared__ int s_base[kPfSortSeqs];                    // KV tiles of a sequence's cached keys
  __shared__ int s_abort;
  __shared__ int s_sticky;
  __shared__ __align__(16) int s_unit[kPfUnitRing][8];   // unit descriptors, see UnitDesc

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  PF_TRACE_INIT();
  if (tid == 0) PF_STAMP(0, 31, 0);
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t q_smem = smem_base;                                  // [head 2][half 2][128][128B]
  const uint32_t k_smem = q_smem + 2 * kPfTileBytes;                  // [stage][half][128][128B]
  const uint32_t v_smem = k_smem + kPfStages * kPfTileBytes;
  // output staging of the softmax warps, then the tiles before sequence i (num_seqs + 1)
  const uint32_t o_smem = v_smem + kPfStages * kPfTileBytes;
  int* s_pref = reinterpret_cast<int*>(smem_raw + (smem_base - smem_u32(smem_raw)) + 2 * kPfTileBytes +
                                       2 * kPfStages * kPfTileBytes + PfOut<kWin>::kBytes);
  const int table = kPfBefore + p.distances + kPfAfter;
  float* s_table = reinterpret_cast<float*>(s_pref + (p.num_seqs + 4) / 4 * 4);       // kWin: [unit parity][head] bias tables
  const uint32_t bar0 = smem_u32(bars);
  auto bar = [&](int i) { return bar0 + 8u * i; };
  volatile int* abort_flag = &s_abort;

  if (tid == 0) {
    s_abort = 0;
    s_sticky = *reinterpret_cast<volatile int*>(p.error_word);  // read once so that the whole CTA agrees
    s_pref[0] = 0;
  }
  __syncthreads();
  {  // block-wide inclusive scan of the tiles per sequence
    int carry = 0;
    for (int base = 0; base < p.num_seqs; base += kPpThreads) {
      const int s = base + tid;
      int n = 0;
      if (s < p.num_seqs) {
        const int len = p.cu_seqlens[s + 1] - p.cu_seqlens[s];
        n = len > 0 ? (len + kPfTile - 1) / kPfTile : 0;
        if (s < kPfSortSeqs) s_base[s] = kWin || p.paged ? (max(p.cu_seqlens_k[s + 1] - p.cu_seqlens_k[s] - len, 0) + kPfTile - 1) / kPfTile : 0;
      }
      int incl = n;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += v;
      }
      if (lane == 31) s_scan[warp] = incl;
      __syncthreads();
      int wofs = 0, tot = 0;
#pragma unroll
      for (int w2 = 0; w2 < kPpThreads / 32; ++w2) {
        const int v = s_scan[w2];
        if (w2 < warp) wofs += v;
        tot += v;
      }
      if (s < p.num_seqs) s_pref[s + 1] = carry + wofs + incl;
      carry += tot;
      __syncthreads();
    }
  }
  if (tid == 0) PF_STAMP(0, 31, 1);
  const int n_tiles = s_pref[p.num_seqs];
  const int ydim = p.num_kv_heads * p.pairs;
  const long long total_units = static_cast<long long>(n_tiles) * ydim;
  // A wait that ran out anywhere (this launch or an earlier one) leaves the error word set: return at once.
  unsigned int* sched = g_pf_sched[p.sched_slot];
  auto cta_done = [&]() {   // one thread: count this CTA; the last one leaves the slot zeroed for its next launch
    if (atomicAdd(&sched[1], 1u) == gridDim.x - 1) {
      sched[0] = 0;
      sched[1] = 0;
      __threadfence();
    }
  };
  if (s_sticky != 0 || static_cast<long long>(blockIdx.x) >= total_units) {   // uniform over the CTA
    if (tid == 0) cta_done();
    return;
  }

  // Units are (head pair y, query tile) and a CTA's first one is its block index; further ones come from a counter (whoever
  // is free takes the next: the KV loops differ in length by up to the number of tiles of a sequence, and any fixed
  // assignment leaves some SMs idle at the end).  Up to kPfSortSeqs sequences: longest KV loop first, so that what is left at
  // the end is short.  A tile's place in that order is its level, the number of KV steps up to its diagonal; a sequence has
  // one tile for each level from base + 1 on (base: KV tiles of its cached keys), so the tiles of a level are found by going
  // through the sequences.  Head pairs are taken in as many groups as still leave the last group work for twice the
  // longest loop on every SM: a group's K and V then stay in L2.  7 sequences of 5,142 tokens, 4/1 heads, bf16: 210 -> 181 us;
  // one of 3,000, 32/8 heads: 99 -> 83 us.
  // More sequences: y outermost, the tiles of a sequence in descending order (their loops are short against the whole).
  struct Unit {
    int seq, seq_start, seq_len, q0, first_pos, n_kv, kvh, head_a, k_row;
    bool has_b, split_p;
  };
  const bool sorted = p.num_seqs <= kPfSortSeqs && total_units > gridDim.x && total_units <= 0x7fffffff;
  auto tiles_of = [&](int q) { return s_pref[q + 1] - s_pref[q]; };
  auto in_level = [&](int q, int level) { return level > s_base[q] && level <= s_base[q] + tiles_of(q); };
  struct Order {                                       // where the producer is in the sorted order
    int top;
    unsigned groups;
    int group, y0, ys, level, above, here;
  };
  auto get_unit = [&](long long u, Order& o) {
    Unit w;
    int y, qtile, lo = 0;
    if (sorted) {
      y = static_cast<int>(static_cast<unsigned>(u) / static_cast<unsigned>(n_tiles));
      auto enter = [&](int level) {
        o.level = level;
        o.here = 0;
        for (int q = 0; q < p.num_seqs; ++q) o.here += in_level(q, level) ? 1 : 0;
      };
      const int group = static_cast<int>((static_cast<unsigned>(y + 1) * o.groups - 1) / static_cast<unsigned>(ydim));   // ydim < 2^16
      if (group != o.group) {
        o.group = group;
        o.y0 = static_cast<int>(static_cast<unsigned>(group) * ydim / o.groups);
        o.ys = static_cast<int>(static_cast<unsigned>(group + 1) * ydim / o.groups) - o.y0;
        o.above = 0;
        enter(o.top);
      }
      const unsigned v = static_cast<unsigned>(u) - static_cast<unsigned>(o.y0) * n_tiles;
      const int x = static_cast<int>(v / static_cast<unsigned>(o.ys));
      y = o.y0 + static_cast<int>(v - static_cast<unsigned>(x) * o.ys);
      while (x >= o.above + o.here && o.level > 1) {
        o.above += o.here;
        enter(o.level - 1);
      }
      int k = x - o.above;                             // the k-th sequence with a tile of this level
      for (int q = 0; q < p.num_seqs; ++q)
        if (in_level(q, o.level) && k-- == 0) lo = q;
      qtile = o.level - 1 - s_base[lo];
    } else {
      y = static_cast<int>(u / n_tiles);
      const int x = static_cast<int>(u - static_cast<long long>(y) * n_tiles);
      int hi = p.num_seqs - 1;                         // last sequence with s_pref[seq] <= x
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (s_pref[mid] <= x) lo = mid; else hi = mid - 1;
      }
      qtile = tiles_of(lo) - 1 - (x - s_pref[lo]);
    }
    w.seq = lo;
    w.kvh = y / p.pairs;
    const int pair = y - w.kvh * p.pairs;
    w.head_a = w.kvh * p.group + 2 * pair;
    w.has_b = 2 * pair + 1 < p.group;
    w.seq_start = p.cu_seqlens[lo];
    w.seq_len = p.cu_seqlens[lo + 1] - w.seq_start;
    w.q0 = qtile * kPfTile;
    int n_cached = kWin || p.paged ? (p.cu_seqlens_k[lo + 1] - p.cu_seqlens_k[lo]) - w.seq_len : 0;
    if (kWin) n_cached = max(n_cached, 0);               // tables have entries from -kPfBefore on
    w.first_pos = n_cached + w.q0;
    w.n_kv = (n_cached + min(w.q0 + kPfTile, w.seq_len) + kPfTile - 1) / kPfTile;
    w.split_p = !kWin && std::is_same<T, __nv_bfloat16>::value && w.first_pos < kPfTile;
    if (kWin) {                                          // positions and steps count from the first tile that a row can see
      w.n_kv = max(w.n_kv, 1);
      const int first = min(max(w.first_pos - p.window + 1, 0) / kPfTile, w.n_kv - 1);
      w.n_kv -= first;
      w.first_pos -= first * kPfTile;
      w.k_row = p.cu_seqlens_k[lo] + first * kPfTile;
    }
    return w;
  };
  // What the producer warp publishes for unit k of this CTA (slot k % kPfUnitRing): all the other roles need to
  // know about it, so that none of them has the lookup above on its critical path; n_kv = 0 says there is no
  // more work.  Every other warp says when it no longer needs the slot (UEMPTY, one arrival per warp): the MMA
  // warp once it has read the step count, a softmax warp behind its last KV step, where it reads the output rows' place (not
  // before: four registers fewer across the KV loop), ahead of its epilogue.
  // What the MMA warp needs of a unit, in one register (the warp runs on 64): the number of KV steps and two flags.
  constexpr int kUnitHasB = 1 << 30, kUnitSplitP = 1 << 29, kUnitSteps = (1 << 29) - 1;
  auto next_unit_steps = [&](int kk) {
    const int slot = kk % kPfUnitRing;
    tc::mbar_wait_compact<true>(bar(PB_UFULL + slot), (kk / kPfUnitRing) & 1, abort_flag, p.error_word, 13);
    const int d = s_unit[slot][7];
    __syncwarp();
    if (lane == 0) tc::mbar_arrive(bar(PB_UEMPTY + slot));
    return *abort_flag ? 0 : d;
  };

  if (tid == 0) {
    tc::mbar_init(bar(PB_Q), 1);
    tc::mbar_init(bar(PB_QEMPTY), 1);
    for (int s = 0; s < kPfStages; ++s) {
      tc::mbar_init(bar(PB_KFULL + s), 1);
      tc::mbar_init(bar(PB_KEMPTY + s), 1);
      tc::mbar_init(bar(PB_VFULL + s), 1);
      tc::mbar_init(bar(PB_VEMPTY + s), 1);
    }
    for (int t = 0; t < 2; ++t) {
      tc::mbar_init(bar(PB_SFULL + t), 1);
      tc::mbar_init(bar(PB_PREADY + t), kPpSoftWarps / 2);
      tc::mbar_init(bar(PB_ODONE + t), 1);
      tc::mbar_init(bar(PB_OFREE + t), kPpSoftWarps / 2);
    }
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(bar(PB_BFULL + i), 2);
      tc::mbar_init(bar(PB_BFREE + i), kPpSoftWarps);
    }
    tc::mbar_init(bar(PB_SPARE), 1);   // takes commits that nobody waits for
    tc::mbar_init(bar(PB_DRAIN), 1);
    for (int i = 0; i < kPfUnitRing; ++i) {
      tc::mbar_init(bar(PB_UFULL + i), 1);
      tc::mbar_init(bar(PB_UEMPTY + i), 1 + kPpSoftWarps + (kWin ? 2 : 0));   // the MMA warp, the softmax warps, the table warps
    }
    tc::mbar_fence_init();
  }
  if (warp == kPpSoftWarps) {
    tc::tmem_alloc(smem_u32(&s_tmem_base), 512);
    tc::tmem_relinquish();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = s_tmem_base;
  if (tid == 0) PF_STAMP(0, 31, 2);

  if (warp >= kPpSoftWarps) {
    tc::setmaxnreg_dec_64();
    if (warp == kPpSoftWarps) {
      // ------------------------------ TMA producer ------------------------------
      Order order = {1, 1u, -1, 0, 1, 0, 0, 0};
      if (sorted) {
        float steps = 0.f;
        for (int q = lane; q < p.num_seqs; q += 32) {
          const int n = tiles_of(q);
          order.top = max(order.top, n > 0 ? s_base[q] + n : 1);
          steps += static_cast<float>(n) * (static_cast<float>(s_base[q]) + 0.5f * static_cast<float>(n + 1));
        }
        order.top = __reduce_max_sync(0xffffffffu, order.top);
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) steps += __shfl_xor_sync(0xffffffffu, steps, o);
        const float fit = steps * static_cast<float>(ydim) / (2.f * static_cast<float>(gridDim.x) * static_cast<float>(order.top));
        order.groups = static_cast<unsigned>(max(1, min(p.num_kv_heads, static_cast<int>(fminf(fit, 65536.f)))));
      }
      if (lane == 0) {
        tc::tma_prefetch_desc(&tmap_q);
        tc::tma_prefetch_desc(&tmap_k);
        tc::tma_prefetch_desc(&tmap_v);
        int gk = 0, k = 0;          // KV steps and units so far: ring stages and phases run on across units
        long long u = blockIdx.x;   // first unit; later ones from the counter
        for (;; ++k) {
          // publish unit k (or the end) for the other roles; the index of the one after it is claimed further
          // down, two KV steps before this unit's loads end
          const int slot = k % kPfUnitRing;
          if (k >= kPfUnitRing) tc::mbar_wait_compact<true>(bar(PB_UEMPTY + slot), ((k / kPfUnitRing) - 1) & 1, abort_flag, p.error_word, 14);
          const bool live = u < total_units && !*abort_flag;
          Unit w;
          if (live) {
            w = get_unit(u, order);
            *reinterpret_cast<int4*>(&s_unit[slot][0]) = make_int4(w.n_kv, w.first_pos, w.seq_start, w.seq_len);
            *reinterpret_cast<int4*>(&s_unit[slot][4]) = make_int4(w.q0, w.head_a, (w.has_b ? 1 : 0) | (w.split_p ? 2 : 0),
                                                                         w.n_kv | (w.has_b ? kUnitHasB : 0) | (w.split_p ? kUnitSplitP : 0));
          } else {
            s_unit[slot][0] = 0;
            s_unit[slot][7] = 0;
          }
          tc::mbar_arrive(bar(PB_UFULL + slot));     // release: the stores above are visible to whoever sees the phase
          if (!live) break;
          PF_STAMP(0, k, 0);
          PF_STAMP(0, k, 1);
          tc::mbar_wait_compact<true>(bar(PB_QEMPTY), (k & 1) ^ 1, abort_flag, p.error_word, 11);   // passes at once for k = 0
          PF_STAMP(0, k, 2);
          const int row0 = w.seq_start + w.q0;
          tc::mbar_expect_tx(bar(PB_Q), (w.has_b ? 2 : 1) * kPfTileBytes);
          for (int t = 0; t < (w.has_b ? 2 : 1); ++t)
            for (int h = 0; h < 2; ++h)
              tc::tma_load_3d(q_smem + t * kPfTileBytes + h * kPfHalfBytes, &tmap_q, 64 * h, w.head_a + t, row0, bar(PB_Q));
          PF_STAMP(0, k, 3);
          auto load_kv_tile = [&](const CUtensorMap* tm, uint32_t dst, int j, uint32_t full_bar) {
            if (kWin || !p.paged) {
              for (int h = 0; h < 2; ++h)
                tc::tma_load_3d(dst + h * kPfHalfBytes, tm, 64 * h, w.kvh, (kWin ? w.k_row : w.seq_start) + j * kPfTile, full_bar);
              return;
            }
            const int32_t* table = p.block_tables + static_cast<int64_t>(w.seq) * p.bt_stride;
            for (int r = 0; r < kPfTile / p.box_rows; ++r) {
              const int pos = j * kPfTile + r * p.box_rows;
              const int blk = pos / p.block_size, off = pos - blk * p.block_size;
              const int phys = blk < p.max_blocks ? table[blk] : -1;
              const int slot = phys >= 0 ? phys * p.block_size + off : 0;
              for (int h = 0; h < 2; ++h)
                tc::tma_load_3d(dst + h * kPfHalfBytes + r * p.box_rows * 128, tm, 64 * h, w.kvh, slot, full_bar);
            }
          };
          for (int j = 0; j < w.n_kv; ++j, ++gk) {
            if (*abort_flag) break;                  // behind a wait that ran out, anyone's, no further step is asked for
            // Take the next unit as late as its latency allows (it passes under the waits of this unit's last
            // loads, and the MMA warp wants the unit by this unit's last step): a unit claimed earlier is one
            // that an idle SM cannot take at the end of the launch.
            if (j == max(w.n_kv - 2, 0)) u = static_cast<long long>(gridDim.x) + atomicAdd(&sched[0], 1u);
            const int s = gk % kPfStages;
            const uint32_t ph = ((gk / kPfStages) & 1) ^ 1;
            tc::mbar_wait_compact<true>(bar(PB_KEMPTY + s), ph, abort_flag, p.error_word, 1);
            tc::mbar_expect_tx(bar(PB_KFULL + s), kPfTileBytes);
            load_kv_tile(&tmap_k, k_smem + s * kPfTileBytes, j, bar(PB_KFULL + s));
            tc::mbar_wait_compact<true>(bar(PB_VEMPTY + s), ph, abort_flag, p.error_word, 2);
            tc::mbar_expect_tx(bar(PB_VFULL + s), kPfTileBytes);
            load_kv_tile(&tmap_v, v_smem + s * kPfTileBytes, j, bar(PB_VFULL + s));
            if (j == 0) PF_STAMP(0, k, 4);
          }
          PF_STAMP(0, k, 5);
#ifdef MV_PF_TRACE
          if (pf_tr && k < 32) pf_tr[(0 * 32 + k) * 8 + 7] = w.n_kv;
#endif
        }
        // After an abort nobody may be left to consume the loads already issued: give them time to land before
        // the CTA (and its shared memory) goes away.  A full barrier completes its phase when its bytes arrive.
        if (*abort_flag) {
          if (k > 0) tc::mbar_wait_timed(bar(PB_Q), (k - 1) & 1);
          for (int g2 = max(gk - kPfStages, 0); g2 < gk; ++g2) {
            tc::mbar_wait_timed(bar(PB_KFULL + g2 % kPfStages), (g2 / kPfStages) & 1);
            tc::mbar_wait_timed(bar(PB_VFULL + g2 % kPfStages), (g2 / kPfStages) & 1);
          }
        }
      }
    } else if (warp == kPpSoftWarps + 1) {
      // ------------------------------- MMA issuer -------------------------------
      const uint32_t idesc_qk = tc::instr_desc_f16(p.fmt, p.fmt, false, 128, 128);
      const uint32_t idesc_pv = tc::instr_desc_f16(p.fmt, p.fmt, true, 128, 128);
      const uint32_t desc_hi = tc::kDescHiSw128Sbo1024;
      const uint32_t q_lo0 = tc::desc_lo(q_smem, 16);
      const uint32_t k_lo0 = tc::desc_lo(k_smem, 16);
      const uint32_t v_lo0 = tc::desc_lo(v_smem, kPfHalfBytes);
      auto issue_qk = [&](int t, int s) {   // S_t = Q_t K(stage s)^T, then commit to SFULL[t]
        tc::mma_ss_k128_commit(tmem + t * 128, tc::desc64(q_lo0 + t * (kPfTileBytes >> 4), desc_hi),
                               tc::desc64(k_lo0 + s * (kPfTileBytes >> 4), desc_hi), idesc_qk, bar(PB_SFULL + t));
      };
      auto issue_pv = [&](int t, int s, bool accum, int p_col, uint32_t commit_bar) {
        tc::mma_ts_k128_commit(tmem + 256 + t * 128, tmem + t * 128 + p_col,
                               tc::desc64(v_lo0 + s * (kPfTileBytes >> 4), desc_hi), idesc_pv, accum, commit_bar);
      };
      int gk = 0, k = 0;             // KV steps and units so far
      // Barrier phases in one register (this warp runs on 64): bit t = parity of the steps so far of head t
      // (PREADY), bit 2 + t = parity of the units it has finished (OFREE), bit 4 + t = it has finished one.
      uint32_t phases = 0;
      // First QK of a unit whose first KV step has ring index g0.  With a single KV step it is also the last use
      // of the unit's Q tile.
      // PV of head t over V stage s (after the softmax warps' PREADY; at a unit's first step also after the
      // previous unit's O of this head has been read), commit to ODONE[t].
      auto pv_step = [&](int t, int s, bool first, bool split_p) {
        tc::mbar_wait_compact<true>(bar(PB_PREADY + t), (phases >> t) & 1u, abort_flag, p.error_word, 7);
        if (first && ((phases >> (4 + t)) & 1u))
          tc::mbar_wait_compact<true>(bar(PB_OFREE + t), ((phases >> (2 + t)) & 1u) ^ 1u, abort_flag, p.error_word, 12);
        tc::fence_after_sync();
        if (split_p) {
          issue_pv(t, s, !first, 0, bar(PB_SPARE));
          issue_pv(t, s, true, 64, bar(PB_ODONE + t));
        } else {
          issue_pv(t, s, !first, 0, bar(PB_ODONE + t));
        }
        phases ^= 1u << t;
      };
      int cur = next_unit_steps(0);
      if (cur != 0) {
        if (lane == 0) PF_STAMP(1, 0, 0);
        tc::mbar_wait_compact<true>(bar(PB_Q), 0, abort_flag, p.error_word, 3);
        tc::mbar_wait_compact<true>(bar(PB_KFULL + 0), 0, abort_flag, p.error_word, 4);
        tc::fence_after_sync();
        issue_qk(0, 0);
        if (cur & kUnitHasB) issue_qk(1, 0);
        // K stage is free once QK(0) of both heads has run; with a single KV step so is the Q buffer
        tc::commit_elected(bar(PB_KEMPTY + 0), bar(PB_QEMPTY), (cur & kUnitSteps) == 1);
      }
      while (cur != 0) {
        const int n_kv = cur & kUnitSteps;
        const bool has_b = (cur & kUnitHasB) != 0, split_p = (cur & kUnitSplitP) != 0;
        // ---- all steps but the last: PV(j) and QK(j + 1) of each head in turn ----
        for (int j = 0; j + 1 < n_kv; ++j, ++gk) {
          const int s = gk % kPfStages, s1 = s ^ 1;
          tc::mbar_wait_compact<true>(bar(PB_VFULL + s), (gk / kPfStages) & 1, abort_flag, p.error_word, 5);
          tc::mbar_wait_compact<true>(bar(PB_KFULL + s1), ((gk + 1) / kPfStages) & 1, abort_flag, p.error_word, 6);
          if (lane == 0) PF_STEP(k, 0, j, 0);
          pv_step(0, s, j == 0, split_p);
          if (lane == 0) PF_STEP(k, 0, j, 1);
          issue_qk(0, s1);
          if (lane == 0) PF_STEP(k, 0, j, 2);
          if (has_b) {
            pv_step(1, s, j == 0, split_p);
            if (lane == 0) PF_STEP(k, 0, j, 3);
            issue_qk(1, s1);
            if (lane == 0) PF_STEP(k, 0, j, 4);
          }
          // V stage s is free when both PV(j) have run, K stage s1 when both QK(j+1) have
          tc::commit_elected(bar(PB_VEMPTY + s), bar(PB_KEMPTY + s1), true);
          if (j + 2 == n_kv) tc::commit_elected(bar(PB_QEMPTY), 0, false);   // that was the unit's last QK
        }
        // ---- the last step: behind the unit's last PVs goes the first QK of the NEXT unit, so that its scores are
        // there when the softmax warps come back from storing this unit's output.  (Putting each head's QK
        // directly behind that head's PV was measured and is a few per cent slower.) ----
        {
          const int s = gk % kPfStages, s1 = s ^ 1;
          tc::mbar_wait_compact<true>(bar(PB_VFULL + s), (gk / kPfStages) & 1, abort_flag, p.error_word, 5);
          pv_step(0, s, n_kv == 1, split_p);
          if (has_b) pv_step(1, s, n_kv == 1, split_p);
          tc::commit_elected(bar(PB_VEMPTY + s), 0, false);   // V stage s is free when both PV have run
          if (lane == 0) PF_STAMP(1, k, 6);
          const int nxt = next_unit_steps(k + 1);
          if (nxt != 0) {
            if (lane == 0) PF_STAMP(1, k + 1, 0);
            tc::mbar_wait_compact<true>(bar(PB_Q), (k + 1) & 1, abort_flag, p.error_word, 3);
            if (lane == 0) PF_STAMP(1, k + 1, 1);
            tc::mbar_wait_compact<true>(bar(PB_KFULL + s1), ((gk + 1) / kPfStages) & 1, abort_flag, p.error_word, 4);
            if (lane == 0) PF_STAMP(1, k + 1, 2);
            tc::fence_after_sync();
            issue_qk(0, s1);
            if (lane == 0) PF_STAMP(1, k + 1, 5);
          }
          if (lane == 0) PF_STAMP(1, k + 1, 7);
          if (nxt & kUnitHasB) issue_qk(1, s1);
          // with a single KV step the next unit's first QK is also the last use of its Q tile
          if (nxt != 0) tc::commit_elected(bar(PB_KEMPTY + s1), bar(PB_QEMPTY), (nxt & kUnitSteps) == 1);
          if (lane == 0) PF_STAMP(1, k + 1, 3);
          ++gk;
          phases = (phases ^ (has_b ? 0xcu : 0x4u)) | (has_b ? 0x30u : 0x10u);
          cur = nxt;
          ++k;
        }
      }
      // After an abort nobody waits for the last MMAs: they must have run before tensor memory is freed.
      if (*abort_flag) {
        tc::commit_elected(bar(PB_DRAIN), 0, false);
        tc::mbar_wait_timed(bar(PB_DRAIN), 0);
      }
    } else if constexpr (kWin) {
      // ------------------------------ bias tables, a buffer per unit parity ------------------------------
      int held0 = -1, held1 = -1;                        // first head of the tables in each buffer
      for (int ku = 0;; ++ku) {
        const int slot = ku % kPfUnitRing, par = ku & 1;
        tc::mbar_wait_compact<true>(bar(PB_UFULL + slot), (ku / kPfUnitRing) & 1, abort_flag, p.error_word, 13);
        const int n_kv = *abort_flag ? 0 : s_unit[slot][0];
        if (n_kv == 0) break;
        const int head_a = s_unit[slot][5], heads = (s_unit[slot][6] & 1) ? 2 : 1;
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(bar(PB_UEMPTY + slot));
        if (ku >= 2) tc::mbar_wait_compact<true>(bar(PB_BFREE + par), ((ku >> 1) - 1) & 1, abort_flag, p.error_word, 16);
        if ((par ? held1 : held0) != head_a) {
          float* tab = s_table + par * 2 * table;
          for (int t = 0; t < heads; ++t)
            for (int i = (warp - kPpSoftWarps - 2) * 32 + lane; i < table; i += 64) {
              const int d = i - kPfBefore;
              tab[t * table + i] = d < 0 || d >= p.window ? -INFINITY
                                   : p.bias ? p.bias[(head_a + t) * p.bias_stride + min(d, p.distances - 1)] * 1.4426950408889634f : 0.f;
            }
          if (par) held1 = head_a;
          else held0 = head_a;
        }
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(bar(PB_BFULL + par));
      }
    }
  } else {
    // ------------------------------ softmax warps ------------------------------
    // Eight a head, two on each 32 lanes of tensor memory with 16 rows each, in the 16x256b layout: lane i holds columns
    // 8g + 2 (i & 3) + {0, 1} of rows i / 4 and i / 4 + 8 (a and b below), so that a row's maximum is two shuffles away and
    // nothing crosses warps.
    tc::setmaxnreg_inc_104();
    const int t = warp >> 3;                       // 0: head A, 1: head B
    const int row0w = (warp & 3) * 32 + ((warp >> 2) & 1) * 16;      // first row of the warp = TMEM lane
    const int row = row0w + (lane >> 2), colq = 2 * (lane & 3);
    const uint32_t lane_addr = static_cast<uint32_t>(row0w) << 16;
    const uint32_t s_addr = tmem + lane_addr + t * 128;
    const uint32_t o_addr = tmem + lane_addr + 256 + t * 128;
    const uint32_t o_stage = o_smem + warp * PfOut<kWin>::kWarpBytes;
    auto arrive = [&](int i) {                     // for the warp
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(bar(i));
    };
    int g = 0;                                     // KV steps of this head so far (barrier phases)
    for (int ku = 0;; ++ku) {
      const int slot = ku % kPfUnitRing;
      tc::mbar_wait_compact<false>(bar(PB_UFULL + slot), (ku / kPfUnitRing) & 1, abort_flag, p.error_word, 13);
      const int n_kv = *abort_flag ? 0 : s_unit[slot][0];
      if (n_kv == 0) break;
      if ((warp & 7) == 0 && lane == 0) PF_STAMP(2 + t, ku, 0);
      const int first_pos = s_unit[slot][1], flags = s_unit[slot][6];
      if constexpr (kWin) tc::mbar_wait_compact<false>(bar(PB_BFULL + (ku & 1)), (ku >> 1) & 1, abort_flag, p.error_word, 17);
      if (t == 1 && !(flags & 1)) {
        arrive(PB_UEMPTY + slot);
        if constexpr (kWin) arrive(PB_BFREE + (ku & 1));
        continue;
      }
      float m_a = -INFINITY, m_b = -INFINITY, l_a = 0.f, l_b = 0.f;
      for (int j = 0; j < n_kv; ++j) {
        tc::mbar_wait_compact<false>(bar(PB_SFULL + t), g & 1, abort_flag, p.error_word, 8);
        if ((warp & 7) == 0 && lane == 0 && j == 0) PF_STAMP(2 + t, ku, 2);
        if ((warp & 7) == 0 && lane == 0) PF_STEP(ku, 1 + t, j, 0);
        tc::fence_after_sync();
        uint32_t sv[2][32];                        // [half][4 group + {a, a, b, b}]
        tc::tmem_ld16x256_x8(s_addr, sv[0]);
        tc::tmem_ld16x256_x8(s_addr + 64, sv[1]);
        tc::wait_ld();
        // Keys of this tile sit at positions 128j + col, query row r at first_pos + r: a key is visible when
        // col <= r + shift.  Tiles that end at or before the first row's position need no mask at all.
        const int shift = first_pos - j * kPfTile;
        if constexpr (kWin) {
          // Distance of a row to a key: shift + row - col.  Scores leave here scaled, biased and masked.  One lookup masks and
          // biases; 34 of them serve a thread's 64 scores.
          const float* tab = s_table + ((ku & 1) * 2 + t) * table + kPfBefore;
          if (shift - (kPfTile - 1) < p.distances - 1) {
            tab += shift + row - colq;
            float b0 = tab[8], b1 = tab[7];        // row b sees in a group what row a sees in the one before
#pragma unroll
            for (int gr = 0; gr < 16; ++gr) {
              const float a0 = tab[-8 * gr], a1 = tab[-8 * gr - 1];
              uint32_t* x = &sv[gr >> 3][(gr & 7) * 4];
              x[0] = __float_as_uint(fmaf(__uint_as_float(x[0]), p.scale_log2, a0));
              x[1] = __float_as_uint(fmaf(__uint_as_float(x[1]), p.scale_log2, a1));
              x[2] = __float_as_uint(fmaf(__uint_as_float(x[2]), p.scale_log2, b0));
              x[3] = __float_as_uint(fmaf(__uint_as_float(x[3]), p.scale_log2, b1));
              b0 = a0;
              b1 = a1;
            }
          } else {
            const float2 sc = make_float2(p.scale_log2, p.scale_log2), far = make_float2(tab[p.distances - 1], tab[p.distances - 1]);
            const int gone = shift + row - colq - p.window;        // columns up to here lie in front of row a's window
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
              for (int i = 0; i < 32; i += 2) {
                const float2 x = tc::fma2(make_float2(__uint_as_float(sv[h][i]), __uint_as_float(sv[h][i + 1])), sc, far);
                sv[h][i] = __float_as_uint(x.x);
                sv[h][i + 1] = __float_as_uint(x.y);
              }
            if (shift + kPfTile - 1 >= p.window) {
#pragma unroll
              for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int i = 0; i < 32; ++i)
                  if (h * 64 + (i >> 2) * 8 + (i & 1) <= gone + ((i & 2) ? 8 : 0)) sv[h][i] = 0xff800000u;
            }
          }
        } else if (shift < kPfTile - 1) {
          const int vis = row + shift - colq;      // of row a; 8 more for row b
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (h * 64 + (i >> 2) * 8 + (i & 1) > vis + ((i & 2) ? 8 : 0)) sv[h][i] = 0xff800000u;  // -inf
        }
        float mxa[2], mxb[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          mxa[h] = mxb[h] = -INFINITY;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            mxa[h] = tc::max3(mxa[h], __uint_as_float(sv[h][4 * i]), __uint_as_float(sv[h][4 * i + 1]));
            mxb[h] = tc::max3(mxb[h], __uint_as_float(sv[h][4 * i + 2]), __uint_as_float(sv[h][4 * i + 3]));
          }
        }
        float xa = fmaxf(mxa[0], mxa[1]), xb = fmaxf(mxb[0], mxb[1]);
        xa = fmaxf(xa, __shfl_xor_sync(0xffffffffu, xa, 1));
        xb = fmaxf(xb, __shfl_xor_sync(0xffffffffu, xb, 1));
        xa = fmaxf(xa, __shfl_xor_sync(0xffffffffu, xa, 2));
        xb = fmaxf(xb, __shfl_xor_sync(0xffffffffu, xb, 2));
        if (!kWin) {
          xa *= p.scale_log2;                      // scale > 0, so max commutes with it
          xb *= p.scale_log2;
        }
        const bool grow_a = xa > m_a + kRescaleThreshold, grow_b = xb > m_b + kRescaleThreshold;
        if (j > 0 && __any_sync(0xffffffffu, grow_a || grow_b)) {
          // Rare: the reference maximum of some row of this warp moved.  PV of the previous step must have landed in O before
          // O is scaled; the next PV cannot start before this warp arrives at PREADY below.
          const float fa = grow_a ? ex2(m_a - xa) : 1.f, fb = grow_b ? ex2(m_b - xb) : 1.f;
          tc::mbar_wait_compact<false>(bar(PB_ODONE + t), (g - 1) & 1, abort_flag, p.error_word, 9);
          tc::fence_after_sync();
#pragma unroll 1
          for (int cc = 0; cc < 4; ++cc) {
            uint32_t ov[16];
            tc::tmem_ld16x256_x4(o_addr + cc * 32, ov);
            tc::wait_ld();
#pragma unroll
            for (int i = 0; i < 16; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * ((i & 2) ? fb : fa));
            tc::tmem_st16x256_x4(o_addr + cc * 32, ov);
          }
          l_a *= fa;
          l_b *= fb;
        }
        if (grow_a) m_a = xa;
        if (grow_b) m_b = xb;
        // exp2(s * scale - m) on packed pairs; one pair in eight goes to the FMA-pipe polynomial so that
        // the special-function unit does not see every exponential (of 0, 1/16, 1/8, 1/4 and 3/8 the best or within 1 %).  P lies over the first 64 columns of S: each warp's
        // rows of S are in its registers.  kSplit: rows with few keys, bf16, whose rounding residue goes behind P.
        // kWin: a row may see nothing of its first tiles
        const float na = kWin && m_a == -INFINITY ? 0.f : -m_a, nb = kWin && m_b == -INFINITY ? 0.f : -m_b;
        const float2 sc2 = make_float2(p.scale_log2, p.scale_log2), na2 = make_float2(na, na), nb2 = make_float2(nb, nb);
        float2 sum_a[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)}, sum_b[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        auto weights = [&](auto split) {
          constexpr bool kSplit = decltype(split)::value;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t pk[16], lo[kSplit ? 16 : 1];
#pragma unroll
            for (int i = 0; i < 16; ++i) {         // pair i: group i / 2, row a or b
              const float2 s2 = make_float2(__uint_as_float(sv[h][2 * i]), __uint_as_float(sv[h][2 * i + 1]));
              const float2 x = kWin ? tc::add2(s2, (i & 1) ? nb2 : na2) : tc::fma2(s2, sc2, (i & 1) ? nb2 : na2);
              float2 e;
              if ((i & 7) == 5 && !kSplit) {
                e = tc::ex2_poly2(x);
              } else {
                e.x = tc::ex2_mufu(x.x);
                e.y = tc::ex2_mufu(x.y);
              }
              float2& acc = (i & 1) ? sum_b[h] : sum_a[h];
              acc = tc::add2(acc, e);
              pk[i] = pack2<T>(e.x, e.y);
              if (kSplit) {
                const float2 hi = Elem<T>::to_f2(*reinterpret_cast<typename Elem<T>::T2*>(&pk[i]));
                lo[kSplit ? i : 0] = pack2<T>(e.x - hi.x, e.y - hi.y);
              }
            }
            tc::tmem_st16x128_x8(s_addr + h * 32, pk);
            if constexpr (kSplit) tc::tmem_st16x128_x8(s_addr + 64 + h * 32, lo);
          }
        };
        constexpr bool kMaySplit = !kWin && std::is_same<T, __nv_bfloat16>::value;
        if (kMaySplit && (flags & 2)) weights(std::integral_constant<bool, kMaySplit>{});
        else weights(std::false_type{});
        const float2 ta = tc::add2(sum_a[0], sum_a[1]), tb = tc::add2(sum_b[0], sum_b[1]);
        l_a += ta.x + ta.y;
        l_b += tb.x + tb.y;
        tc::wait_st();
        tc::fence_before_sync();
        if (!(p.inject == 1 && t == 0 && g == 0 && blockIdx.x == 0 && warp == 0)) arrive(PB_PREADY + t);
        if ((warp & 7) == 0 && lane == 0 && j == n_kv - 1) PF_STAMP(2 + t, ku, 3);
        if ((warp & 7) == 0 && lane == 0) PF_STEP(ku, 1 + t, j, 1);
        ++g;
      }

      if constexpr (kWin) arrive(PB_BFREE + (ku & 1));
      // ---- epilogue: O / l -> global, by TMA from this warp's staging buffer, 64 columns at a time ----
      l_a += __shfl_xor_sync(0xffffffffu, l_a, 1);
      l_b += __shfl_xor_sync(0xffffffffu, l_b, 1);
      l_a += __shfl_xor_sync(0xffffffffu, l_a, 2);
      l_b += __shfl_xor_sync(0xffffffffu, l_b, 2);
      const int seq_start = s_unit[slot][2], seq_len = s_unit[slot][3], row0 = s_unit[slot][4] + row0w, head = s_unit[slot][5] + t;
      float fa = 1.f, fb = 1.f;
      if (kWin && p.sink) {
        const float sk = __bfloat162float(p.sink[head]) * 1.4426950408889634f, ma = fmaxf(m_a, sk), mb = fmaxf(m_b, sk);
        fa = exp2f(m_a - ma);
        fb = exp2f(m_b - mb);
        l_a = l_a * fa + exp2f(sk - ma);
        l_b = l_b * fb + exp2f(sk - mb);
      }
      const float inv_a = l_a > 0.f ? fa / l_a : 0.f, inv_b = l_b > 0.f ? fb / l_b : 0.f;
      arrive(PB_UEMPTY + slot);
      tc::mbar_wait_compact<false>(bar(PB_ODONE + t), (g - 1) & 1, abort_flag, p.error_word, 10);
      if ((warp & 7) == 0 && lane == 0) PF_STAMP(2 + t, ku, 4);
      tc::fence_after_sync();
      uint32_t ov[2][32];
      tc::tmem_ld16x256_x8(o_addr, ov[0]);
      tc::tmem_ld16x256_x8(o_addr + 64, ov[1]);
      tc::wait_ld();
      tc::fence_before_sync();
      arrive(PB_OFREE + t);                        // the accumulator is read
      if ((warp & 7) == 0 && lane == 0) PF_STAMP(2 + t, ku, 5);
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int rr = 0; rr < 16; rr += kOutRows) {
          if (lane == 0) tc::bulk_wait_read();     // the copy before has left the buffer
          __syncwarp();
          // Four 8 x 8 blocks at a time: two groups of eight columns with their 16 rows, or four with rows rr .. rr + 7.  Lane i
          // gives the address of row i % 8 of block i / 8; swizzled as the tensor map has it.
#pragma unroll
          for (int i = 0; i < kOutRows / 4; ++i) {
            uint32_t x[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int gr = kOutRows == 16 ? 2 * i + (e >> 1) : 4 * i + e, second = kOutRows == 16 ? e & 1 : rr >> 3;
              const float f = second ? inv_b : inv_a;
              x[e] = pack2<T>(__uint_as_float(ov[h][4 * gr + 2 * second]) * f, __uint_as_float(ov[h][4 * gr + 2 * second + 1]) * f);
            }
            const int r = lane & (kOutRows - 1), ch = kOutRows == 16 ? 2 * i + (lane >> 4) : 4 * i + (lane >> 3);
            st_matrix4(o_stage + r * 128 + ((ch ^ (r & 7)) << 4), x);
          }
          if (row0 + rr + kOutRows <= seq_len) {
            tc::fence_async_proxy();
            __syncwarp();
            if (lane == 0) tc::tma_store_3d(&tmap_o, o_stage, h * 64, head, seq_start + row0 + rr);
          } else {                                 // the rows behind belong to the next sequence
            __syncwarp();
#pragma unroll
            for (int i = 0; i < kOutRows / 4; ++i) {       // eight lanes per row, four rows per instruction
              const int r = 4 * i + (lane >> 3), ch = lane & 7;
              const uint4 x = ld_shared16(o_stage + r * 128 + ((ch ^ (r & 7)) << 4));
              if (row0 + rr + r < seq_len)
                st_global16(static_cast<T*>(p.out) + static_cast<int64_t>(seq_start + row0 + rr + r) * p.out_stride_tok + static_cast<int64_t>(head) * kPfD + h * 64 + ch * 8, x);
            }
            __syncwarp();
          }
        }
      if ((warp & 7) == 0 && lane == 0) PF_STAMP(2 + t, ku, 6);
    }
    if (lane == 0) tc::bulk_wait_all();
  }
  // ---- teardown: everyone is done with tensor memory before it is freed ----
  tc::fence_before_sync();
  __syncthreads();
  if (warp == kPpSoftWarps) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, 512);
  }
  if (tid == 0) cta_done();
  if (tid == 0) PF_STAMP(0, 31, 3);
}

constexpr int kPfPersistentMaxSeqs = 320;   // the persistent form keeps num_seqs + 1 prefix sums in what shared
                                            // memory the tile buffers and the output staging leave

// p.sched_slot is taken; tmap_o's box is PfOut<kWin>::kRows rows.
template <typename T, bool kWin>
int launch_prefill_persistent(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& to, const PrefillParams& p,
                              int64_t max_tiles, int ydim, const char* what, cudaStream_t st) {
  constexpr int kPref = ((kPfPersistentMaxSeqs + 1) * 4 + 15) / 16 * 16, kBase = kPfSmemBytes + PfOut<kWin>::kBytes;
  constexpr int kMost = kBase + kPref + (kWin ? 4 * (kPfBefore + kPfMaxDistances + kPfAfter) * 4 : 0);
  static_assert(kMost + 640 <= 227 * 1024, "a CTA's shared memory");
  const int smem = kBase + ((p.num_seqs + 1) * 4 + 15) / 16 * 16 + (kWin ? 4 * (kPfBefore + p.distances + kPfAfter) * 4 : 0);
  static bool attr_done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !attr_done[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(prefill_persistent_kernel<T, kWin>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMost);
    if (e != cudaSuccess) {
      cudaGetLastError();
      return fail(MV_ERR_CUDA, "%s: cudaFuncSetAttribute: %s", what, cudaGetErrorString(e));
    }
    if (dev >= 0 && dev < 64) attr_done[dev] = true;
  }
  const unsigned grid = static_cast<unsigned>(std::min<int64_t>(max_tiles * ydim, kNumSMs));   // one CTA per SM
  prefill_persistent_kernel<T, kWin><<<grid, kPpThreads, smem, st>>>(tq, tk, tv, to, p);
  return check_launch(what);
}

}  // namespace mv
