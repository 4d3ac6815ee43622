// Sampling tail: row-wise argmax of the logits (greedy) or of the exponential-race scores (temperature),
// both mergeable across vocabulary shards.
//
// In the reference every tensor-parallel rank computes its vocabulary shard of
// the logits, rank 0 gathers the full (batch, 151,936) matrix
// (src/myvllm/layers/embedding_head.py:56-77) and the sampler works on that
// (src/myvllm/layers/sampler.py:15-19; greedy decoding is its temperature -> 0
// limit, the plain argmax).  Here a rank reduces its own shard to ONE 64-bit
// key per row -- the maximum logit in an order-preserving integer form in the
// high word, 2^32-1 minus the global column index in the low word -- so that
// the larger key is the larger logit and, between equal logits, the lower
// index.  Shards are merged by an integer MAX (an all-reduce of 8 bytes per
// row instead of a gather of the logits) and decoded to token ids.
// HBM-bound: one read of the logits, rows * cols * 2 bytes.
#include <climits>
#include <cooperative_groups.h>
#include "common.cuh"

namespace mv {

namespace cg = cooperative_groups;
constexpr int kArgmaxThreads = 256;
constexpr int kMaxRowCtas = 8;         // the portable cluster size

// float -> int32 whose signed order is the float order; NaN sorts above +inf (torch.argmax treats NaN as the
// maximum) and -0.0 maps to the key of +0.0 (they compare equal, so the lower index must win between them).
__device__ __forceinline__ int32_t orderable(float v) {
  if (v != v) return 0x7fffffff;
  const int32_t b = __float_as_int(v);
  if (b == static_cast<int32_t>(0x80000000u)) return 0;
  return b < 0 ? (b ^ 0x7fffffff) : b;
}
__device__ __forceinline__ long long make_key(float v, uint32_t index) {
  const unsigned long long hi = static_cast<uint32_t>(orderable(v));
  return static_cast<long long>((hi << 32) | static_cast<unsigned long long>(0xffffffffu - index));
}
__device__ __forceinline__ long long token_of_key(long long key) {
  return static_cast<long long>(0xffffffffu - static_cast<uint32_t>(key & 0xffffffffll));
}

// A thread walks its columns in increasing order and keeps the first maximum it meets (strict >), so equal logits resolve to the
// lowest index within a thread; across threads the keys do it.
// The best logit or score that a thread has met: the first maximum in visiting order, and a NaN is the maximum.
struct Best {
  float v = -INFINITY;
  bool nan = false, have = false;
  uint32_t idx = 0;
  __device__ __forceinline__ void offer(float x, uint32_t i) {
    if (nan) return;                            // a NaN already won: it is the maximum and came first
    const bool is_nan = x != x;
    if (is_nan || x > v || !have) {
      v = x;
      idx = i;
      nan = is_nan;
      have = true;
    }
  }
};

// A row belongs to the CTAs of a cluster (kOne: to one CTA, the numbers are constants); thread `at` of `threads` takes every
// threads-th piece.
template <bool kOne> struct RowShare {
  uint32_t at, threads, rank, ctas;
  __device__ __forceinline__ RowShare() {
    ctas = kOne ? 1 : cg::this_cluster().num_blocks();
    rank = kOne ? 0 : cg::this_cluster().block_rank();
    at = rank * kArgmaxThreads + threadIdx.x;
    threads = ctas * kArgmaxThreads;
  }
};

// The row's largest key from all threads of its cluster, written by its first CTA.
template <bool kOne>
__device__ __forceinline__ void finish_row(const Best& best, uint32_t index_offset, const RowShare<kOne>& my, int64_t row, long long* keys,
                                           long long* tokens) {
  long long key = best.have ? make_key(best.v, index_offset + best.idx) : LLONG_MIN;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const long long other = __shfl_xor_sync(0xffffffffu, key, off);
    key = other > key ? other : key;
  }
  __shared__ long long s_keys[kArgmaxThreads / 32], s_ctas[kMaxRowCtas];
  if ((threadIdx.x & 31) == 0) s_keys[threadIdx.x >> 5] = key;
  __syncthreads();
  if (threadIdx.x == 0)
#pragma unroll
    for (int w = 1; w < kArgmaxThreads / 32; ++w) key = s_keys[w] > key ? s_keys[w] : key;
  if (my.ctas > 1) {
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();                             // the first CTA has begun: its shared memory may be written
    if (threadIdx.x == 0) cluster.map_shared_rank(s_ctas, 0)[my.rank] = key;
    cluster.sync();
    if (my.rank == 0 && threadIdx.x == 0)
      for (uint32_t c = 1; c < my.ctas; ++c) key = s_ctas[c] > key ? s_ctas[c] : key;
  }
  if (my.rank == 0 && threadIdx.x == 0) {
    if (keys) keys[row] = key;
    if (tokens) tokens[row] = token_of_key(key);
  }
}

// The plain maximum over this thread's share of a row.  Per chunk of eight logits only its maximum is computed (packed 16-bit
// maxima, exact, NaN-propagating) and compared with the running one; the chunk that raised it is kept and searched for the
// position at the end.  Chunks are visited in increasing order and only a strictly larger maximum replaces the kept chunk,
// so the first of equal maxima survives.
template <typename T, bool kOne>
__device__ __forceinline__ void argmax_share(const T* row, int64_t cols, bool aligned, const RowShare<kOne>& my, Best& best) {
  // 16-byte chunks when every row starts on a 16-byte boundary
  const int64_t chunks = sizeof(T) == 2 && aligned ? cols / 8 : 0;
  if constexpr (sizeof(T) == 2) {
    using T2 = typename Elem<T>::T2;
    constexpr int kUnroll = 4;
    uint4 best_raw = make_uint4(0, 0, 0, 0);
    int64_t best_chunk = -1;
    float cbest = -INFINITY;
    bool cbest_nan = false;
    for (int64_t c0 = my.at; c0 < chunks; c0 += static_cast<int64_t>(my.threads) * kUnroll) {
      uint4 raw[kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int64_t c = c0 + static_cast<int64_t>(u) * my.threads;
        if (c < chunks) raw[u] = ld_stream16(row + c * 8);
      }
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int64_t c = c0 + static_cast<int64_t>(u) * my.threads;
        if (c < chunks && !cbest_nan) {
          const T2* p2 = reinterpret_cast<const T2*>(&raw[u]);
          const float m = Elem<T>::hmax_nan_f(Elem<T>::max2_nan(Elem<T>::max2_nan(p2[0], p2[1]),
                                                                Elem<T>::max2_nan(p2[2], p2[3])));
          const bool is_nan = m != m;
          if (is_nan || m > cbest || best_chunk < 0) {
            cbest = m;
            cbest_nan = is_nan;
            best_chunk = c;
            best_raw = raw[u];
          }
        }
      }
    }
    if (best_chunk >= 0) {   // position of the first maximum (or first NaN) inside the kept chunk
      const T2* p2 = reinterpret_cast<const T2*>(&best_raw);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = Elem<T>::to_f2(p2[j]);
        best.offer(f.x, static_cast<uint32_t>(best_chunk * 8 + 2 * j));
        best.offer(f.y, static_cast<uint32_t>(best_chunk * 8 + 2 * j + 1));
      }
    }
  }
  for (int64_t i = chunks * 8 + my.at; i < cols; i += my.threads)   // ragged tail, or rows that start anywhere
    best.offer(Elem<T>::to_f(row[i]), static_cast<uint32_t>(i));
}

constexpr int kArgmaxCtasPerSM = 5;
template <typename T, bool kOne>
__global__ void __launch_bounds__(kArgmaxThreads, kArgmaxCtasPerSM)
argmax_rows_kernel(const T* __restrict__ logits, int64_t row_stride, int64_t cols, uint32_t index_offset, bool aligned,
                   long long* __restrict__ keys, long long* __restrict__ tokens) {
  const RowShare<kOne> my;
  const int64_t r = blockIdx.x / my.ctas;
  Best best;
  argmax_share(logits + r * row_stride, cols, aligned, my, best);
  finish_row(best, index_offset, my, r, keys, tokens);
}

// ---------------------------------------------------------------------------------------------
// Temperature sampling: the reference's exponential race (src/myvllm/layers/sampler.py:15-19)
//   token = argmax_i softmax(logits / T)_i / E_i,   E_i ~ Exp(1)
// needs no normaliser: argmax_i p_i / E_i = argmax_i (logit_i / T - log E_i).  The score of a column depends
// only on that column, so the vocabulary shards of a tensor-parallel model reduce independently and merge by
// the same 64-bit MAX as the greedy keys -- provided every rank draws the SAME E_i for global column i.
// Hence a counter-based generator: Philox4x32-10 with key = seed and counter = (global column / 4, row, step),
// whose four 32-bit outputs serve columns 4g .. 4g+3.  u = (top 24 bits + 0.5) / 2^24, rounded to 32-bit floating point; E = -log(u).
// u is above 0, but the sum is rounded to even from 2^23 on, and its largest value, one column's in 2^24, to 2^24: u is 1 there, E
// is 0 and the score +inf (NaN for a logit of -inf), so that such a column wins its row.  The oracle has the same rounding.  Other
// E are at least 1e-7, so the reference's clamp at 1e-10 never binds.  A row with T == 0 is greedy.
// ---------------------------------------------------------------------------------------------
struct Philox {
  uint32_t x, y, z, w;
};
__host__ __device__ inline void philox_mulhilo(uint32_t a, uint32_t b, uint32_t& hi, uint32_t& lo) {
  const unsigned long long p = static_cast<unsigned long long>(a) * b;
  hi = static_cast<uint32_t>(p >> 32);
  lo = static_cast<uint32_t>(p);
}
__host__ __device__ inline Philox philox4x32_10(Philox c, uint32_t k0, uint32_t k1) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    uint32_t hi0, lo0, hi1, lo1;
    philox_mulhilo(0xD2511F53u, c.x, hi0, lo0);
    philox_mulhilo(0xCD9E8D57u, c.z, hi1, lo1);
    c = Philox{hi1 ^ c.y ^ k0, lo1, hi0 ^ c.w ^ k1, lo0};
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  return c;
}
// -log E for the 32 random bits of one column: Gumbel noise added to logit / T.
__device__ __forceinline__ float race_noise(uint32_t bits) {
  const float u = (static_cast<float>(bits >> 8) + 0.5f) * (1.0f / 16777216.0f);
  return -__logf(-logf(u));
}

// One thread takes the columns of kPiece / 4 Philox groups at a time: 16-byte loads of eight 16-bit or four 32-bit logits where
// rows and the shard start on such boundaries, else four single loads per group, so that a group's four words are drawn once
// in either case.
//
// Bound: instruction issue (a column's share of Philox is 15 slots).  A score is only formed where it can win.  With E = -log u
// >= 1 - u a score is at most v / T - log(1 - u), so a column whose 1 - u exceeds e^(v / T - best) is passed over for one
// ex2.approx instead of two logarithms; `best` is the warp's, which moves about ten times in a row.  The test errs on the side
// of forming the score: aim()'s slack covers the roundings of the exponent (a few 2^-23 of best, and those of the noise itself),
// kEdge those of u, and a NaN or an infinity fails the comparison.  Every score that is formed is the same as before, so are the
// tokens.  512 x 151,936 bf16: 236 us when every score was formed, 107 us now.
template <typename T, bool kVec>
__global__ void __launch_bounds__(kArgmaxThreads)
sample_rows_kernel(const T* __restrict__ logits, int64_t row_stride, int64_t cols, uint32_t index_offset, bool aligned,
                   const float* __restrict__ temperatures, unsigned long long seed, const long long* __restrict__ step_ptr,
                   long long* __restrict__ keys, long long* __restrict__ tokens) {
  const RowShare<false> my;
  const uint32_t rowi = blockIdx.x / my.ctas;
  const T* row = logits + static_cast<int64_t>(rowi) * row_stride;
  const float temp = temperatures[rowi];
  Best best;
  if (!(temp > 0.f)) {                           // a greedy row
    argmax_share(row, cols, aligned, my, best);
    finish_row(best, index_offset, my, rowi, keys, tokens);
    return;
  }
  const float inv_t = 1.0f / temp;
  const unsigned long long step = static_cast<unsigned long long>(*step_ptr);
  const uint32_t k0 = static_cast<uint32_t>(seed), k1 = static_cast<uint32_t>(seed >> 32);
  const uint32_t s0 = static_cast<uint32_t>(step), s1 = static_cast<uint32_t>(step >> 32);
  constexpr int kPiece = kVec && sizeof(T) == 2 ? 8 : 4;
  constexpr float kLog2 = 1.4426950408889634f, kEdge = 2.f - 0x1p-21f;
  const float slope = inv_t * kLog2;
  float shift = INFINITY;                        // (slack - best) in base 2
  // Piece p has the global columns base0 + p * kPiece and on; the first piece may begin before the shard, the last end behind it.
  // A thread meets its columns in increasing order, so that the first of equal scores is the one that it keeps: what the shard
  // has of a first piece that it begins inside goes to thread 0 before anything else.
  const uint32_t n_cols = static_cast<uint32_t>(cols), base0 = index_offset & ~3u, lead = index_offset - base0;
  const uint32_t skip = lead ? 1u : 0u, whole = (n_cols + lead) / kPiece, pieces = whole + ((n_cols + lead) % kPiece ? 1u : 0u);
  auto draw = [&](uint32_t p, uint32_t (&bits)[kPiece]) {
    const uint32_t group = (base0 >> 2) + p * (kPiece / 4);
#pragma unroll
    for (int q = 0; q < kPiece / 4; ++q) {
      const Philox a = philox4x32_10(Philox{group + q, rowi, s0, s1}, k0, k1);
      bits[4 * q] = a.x; bits[4 * q + 1] = a.y; bits[4 * q + 2] = a.z; bits[4 * q + 3] = a.w;
    }
  };
  auto aim = [&] {                               // the warp's best so far sets the test; a NaN leaves the others' maximum
    float top = best.v;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, off));
    // behind an infinite score only those that may be infinite too, and NaN, are looked at
    shift = top == INFINITY ? -3e38f : (0.02f + 4e-6f * fabsf(top) - top) * kLog2;
  };
  // The whole warp; lanes that are not `live` have nothing to offer, nor have columns outside the shard.
  auto consider = [&](const float (&v)[kPiece], uint32_t p, bool live, bool inside) {
    uint32_t bits[kPiece];
    draw(p, bits);
    float2 x[kPiece / 2];
    float most = -INFINITY;
#pragma unroll
    for (int j = 0; j < kPiece / 2; ++j) {
      x[j] = fma_f32x2(make_float2(v[2 * j], v[2 * j + 1]), make_float2(slope, slope), make_float2(shift, shift));
      x[j] = add_f32x2(make_float2(fast_exp2(x[j].x), fast_exp2(x[j].y)),
                       make_float2(__uint_as_float((bits[2 * j] >> 9) | 0x3f800000u), __uint_as_float((bits[2 * j + 1] >> 9) | 0x3f800000u)));
      most = max_nan(max_nan(most, x[j].x), x[j].y);
    }
    if (!__any_sync(0xffffffffu, live && !(most < kEdge))) return;
#pragma unroll
    for (int j = 0; j < kPiece; ++j) {
      const uint32_t i = p * kPiece + j - lead;
      if (live && !((j & 1 ? x[j / 2].y : x[j / 2].x) < kEdge) && (inside || i < n_cols)) best.offer(v[j] * inv_t + race_noise(bits[j]), i);
    }
    aim();
  };
  auto fetch = [&](uint32_t p, float (&v)[kPiece]) {       // a whole piece inside the shard
    const T* at = row + (p * kPiece - lead);
    if constexpr (kVec) {
      const uint4 raw = ld_stream16(at);
      if constexpr (sizeof(T) == 2) {
        const typename Elem<T>::T2* p2 = reinterpret_cast<const typename Elem<T>::T2*>(&raw);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = Elem<T>::to_f2(p2[j]);
          v[2 * j] = f.x;
          v[2 * j + 1] = f.y;
        }
      } else {
        const float4 f = *reinterpret_cast<const float4*>(&raw);
        v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
      }
    } else {
#pragma unroll
      for (int j = 0; j < kPiece; ++j) v[j] = Elem<T>::to_f(at[j]);
    }
  };
  if constexpr (!kVec) {
    if (skip && my.at == 0) {
      uint32_t bits[kPiece];
      draw(0, bits);
#pragma unroll
      for (uint32_t j = 1; j < 4; ++j)
        if (j >= lead && j - lead < n_cols) best.offer(Elem<T>::to_f(row[j - lead]) * inv_t + race_noise(bits[j]), j - lead);
    }
  }
  const uint32_t rounds = whole > skip ? (whole - skip) / my.threads : 0;
  uint32_t p = skip + my.at;
  if (rounds) {
    // one score per lane to begin with, so that the test has something to go by (the same column again is no gain over itself)
    float v[kPiece];
    uint32_t bits[kPiece];
    fetch(p, v);
    draw(p, bits);
    best.offer(v[0] * inv_t + race_noise(bits[0]), p * kPiece - lead);
    aim();
    for (uint32_t it = 0; it < rounds; ++it, p += my.threads) {
      float now[kPiece];
#pragma unroll
      for (int j = 0; j < kPiece; ++j) now[j] = v[j];
      if (it + 1 < rounds) fetch(p + my.threads, v);
      consider(now, p, true, true);
    }
  }
  // what is left: less than a round of whole pieces, and the one over the shard's end
  const uint32_t left = pieces - skip - rounds * my.threads;
  for (uint32_t it = 0; it * my.threads < left; ++it) {
    const uint32_t k = it * my.threads + my.at, q = skip + k + rounds * my.threads;
    const bool live = k < left;
    float v[kPiece];
#pragma unroll
    for (int j = 0; j < kPiece; ++j) {
      const uint32_t i = q * kPiece + j - lead;
      v[j] = live && i < n_cols ? Elem<T>::to_f(row[i]) : -INFINITY;
    }
    consider(v, q, live, false);
  }
  finish_row(best, index_offset, my, rowi, keys, tokens);
}

// keys (shards, rows) -> tokens (rows): the largest key of each row, decoded.
__global__ void argmax_decode_kernel(const long long* __restrict__ keys, int shards, int64_t rows,
                                     long long* __restrict__ tokens) {
  const int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (r >= rows) return;
  long long key = keys[r];
  for (int s = 1; s < shards; ++s) {
    const long long other = keys[static_cast<int64_t>(s) * rows + r];
    key = other > key ? other : key;
  }
  tokens[r] = token_of_key(key);
}

// A row's CTAs, one cluster.  Sampling, which is bound by issue, and logits that are read one by one: more of them while the rows
// alone would leave SMs with fewer than four, as long as each thread has two 16-byte pieces.
static unsigned row_ctas(int64_t rows, int64_t cols) {
  unsigned n = 1;
  while (n < kMaxRowCtas && rows * n < 4 * kNumSMs && cols >= static_cast<int64_t>(n) * 2 * kArgmaxThreads * 16) n *= 2;
  return n;
}
// Selection from 16-byte pieces is bound by memory and ends with a cluster's barriers: more CTAs only while all of them are
// resident at once, and while the row is long enough to pay for them.  bf16, a CTA a row against this rule: 151,936 columns 16
// rows 15.6 -> 5.5 us, 64 17.2 -> 7.9, 128 17.9 -> 10.7, 256 20.4 -> 17.3; from 512 rows on (27.8 us) one CTA, which two took 33.5
// for.  32,768 columns 64 rows 5.0 -> 4.2, 128 5.5 -> 5.3; 256 rows 6.4 with one, 6.8 with two.
static unsigned argmax_ctas(int64_t rows, int64_t cols) {
  const int64_t places = cols >= 65536 ? kArgmaxCtasPerSM * kNumSMs : kArgmaxCtasPerSM * kNumSMs / 2;
  unsigned n = 1;
  while (n < kMaxRowCtas && rows * n * 2 <= places && cols >= static_cast<int64_t>(n) * 16384) n *= 2;
  return n;
}

template <typename... P, typename... A>
static int launch_rows(const char* what, void (*kernel)(P...), int64_t rows, unsigned ctas, cudaStream_t st, A... args) {
  if (rows * ctas > 0x7fffffffLL) return fail(MV_ERR_LIMIT, "%s: too many rows", what);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(rows) * ctas);
  cfg.blockDim = dim3(kArgmaxThreads);
  cfg.stream = st;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = ctas;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = ctas > 1 ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
  return check_launch(what);
}

}  // namespace mv

extern "C" int mv_argmax_rows(const void* logits, int64_t row_stride, int64_t rows, int64_t cols,
                              int64_t index_offset, int64_t* keys, int64_t* tokens, int dtype, void* stream) {
  using namespace mv;
  if (dtype < MV_F16 || dtype > MV_F32) return fail(MV_ERR_DTYPE, "argmax_rows: dtype %d", dtype);
  if (rows < 0 || cols <= 0 || index_offset < 0) return fail(MV_ERR_SHAPE, "argmax_rows: negative or zero size");
  if (rows == 0) return MV_OK;
  if (!logits || (!keys && !tokens)) return fail(MV_ERR_NULL, "argmax_rows: null pointer");
  if (row_stride < cols) return fail(MV_ERR_SHAPE, "argmax_rows: row stride smaller than a row");
  const bool aligned = row_stride % 8 == 0 && aligned16(logits);   // otherwise element-wise loads
  if (index_offset + cols > 0xffffffffLL || rows > 0x7fffffffLL)
    return fail(MV_ERR_LIMIT, "argmax_rows: column index beyond 32 bits or too many rows");
  auto run = [&](auto zero) {
    using T = decltype(zero);
    const unsigned ctas = sizeof(T) == 2 && aligned ? argmax_ctas(rows, cols) : row_ctas(rows, cols);
    return launch_rows("argmax_rows_kernel", ctas == 1 ? argmax_rows_kernel<T, true> : argmax_rows_kernel<T, false>, rows, ctas, static_cast<cudaStream_t>(stream),
                       static_cast<const T*>(logits), row_stride, cols, static_cast<uint32_t>(index_offset), aligned,
                       reinterpret_cast<long long*>(keys), reinterpret_cast<long long*>(tokens));
  };
  return dtype == MV_F16 ? run(__half{}) : dtype == MV_F32 ? run(float{}) : run(__nv_bfloat16{});
}

extern "C" int mv_argmax_decode(const int64_t* keys, int shards, int64_t rows, int64_t* tokens, void* stream) {
  using namespace mv;
  if (shards <= 0 || rows < 0) return fail(MV_ERR_SHAPE, "argmax_decode: negative or zero size");
  if (rows == 0) return MV_OK;
  if (!keys || !tokens) return fail(MV_ERR_NULL, "argmax_decode: null pointer");
  const int threads = 128;
  const int64_t grid = (rows + threads - 1) / threads;
  if (grid > 0x7fffffffLL) return fail(MV_ERR_LIMIT, "argmax_decode: too many rows");
  argmax_decode_kernel<<<static_cast<unsigned>(grid), threads, 0, static_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const long long*>(keys), shards, rows, reinterpret_cast<long long*>(tokens));
  return check_launch("argmax_decode_kernel");
}

extern "C" int mv_sample_rows(const void* logits, int64_t row_stride, int64_t rows, int64_t cols, int64_t index_offset,
                              const float* temperatures, uint64_t seed, const int64_t* step, int64_t* keys,
                              int64_t* tokens, int dtype, void* stream) {
  using namespace mv;
  if (dtype < MV_F16 || dtype > MV_F32) return fail(MV_ERR_DTYPE, "sample_rows: dtype %d", dtype);
  if (rows < 0 || cols <= 0 || index_offset < 0) return fail(MV_ERR_SHAPE, "sample_rows: negative or zero size");
  if (rows == 0) return MV_OK;
  if (!logits || !temperatures || !step || (!keys && !tokens)) return fail(MV_ERR_NULL, "sample_rows: null pointer");
  if (row_stride < cols) return fail(MV_ERR_SHAPE, "sample_rows: row stride smaller than a row");
  if (index_offset + cols > 0xffffffffLL || rows > 0x7fffffffLL)
    return fail(MV_ERR_LIMIT, "sample_rows: column index beyond 32 bits or too many rows");
  auto run = [&](auto zero) {
    using T = decltype(zero);
    constexpr int kPiece = 16 / sizeof(T);
    const bool aligned = row_stride % 8 == 0 && aligned16(logits);
    const bool vec = row_stride % kPiece == 0 && aligned16(logits) && index_offset % kPiece == 0;
    return launch_rows("sample_rows_kernel", vec ? sample_rows_kernel<T, true> : sample_rows_kernel<T, false>, rows, row_ctas(rows, cols),
                       static_cast<cudaStream_t>(stream), static_cast<const T*>(logits), row_stride, cols,
                       static_cast<uint32_t>(index_offset), aligned, temperatures, static_cast<unsigned long long>(seed),
                       reinterpret_cast<const long long*>(step), reinterpret_cast<long long*>(keys),
                       reinterpret_cast<long long*>(tokens));
  };
  return dtype == MV_F16 ? run(__half{}) : dtype == MV_F32 ? run(float{}) : run(__nv_bfloat16{});
}

// The generator of mv_sample_rows on the host: the four 32-bit words for (seed, step, row, column group).
extern "C" int mv_philox4x32_10(uint64_t seed, uint64_t step, uint32_t row, uint32_t column_group, uint32_t* out4) {
  if (!out4) return mv::fail(MV_ERR_NULL, "philox: null output");
  const mv::Philox r = mv::philox4x32_10(mv::Philox{column_group, row, static_cast<uint32_t>(step), static_cast<uint32_t>(step >> 32)},
                                         static_cast<uint32_t>(seed), static_cast<uint32_t>(seed >> 32));
  out4[0] = r.x; out4[1] = r.y; out4[2] = r.z; out4[3] = r.w;
  return MV_OK;
}
