// Gated linear attention and time mixing in chunks of 64 tokens.  With b_t the running sums of the channels' log2 decays inside the chunk:
//   O = (q 2^b) S_0 + A V,      A[t, j] = sum_k q_t k_j 2^(b_t - b_j), j <= t
//   S = 2^b_last S_0 + (k 2^(b_last - b))^T V
// Time mixing (kTime) reads the state before the token's own decay: b_(t-1) in the place of b_t beside q, j < t in A, whose
// diagonal is q_t . (u k_t).
// gla_prepare_kernel  per chunk and head: b, both decayed operands, A.  A's 16 x 16 blocks are products of factors taken
//                     against b at one token, on tensor cores in two terms each.  Below the diagonal that is the last token
//                     before the block's rows, and every power of two is at most one.  On the diagonal it is the block's
//                     middle; a block in which some channel forgets more than 2^-60 is summed channel by channel instead.
// The walk over a sequence's chunks is chunk_walk.cuh's, or for narrow heads:
// gla_chunk_kernel    per sequence, head and block of value columns: see state_chunk.cuh
// V enters as the projection left it; the decayed operands, A and S in two terms.
#include "chunk_walk.cuh"

namespace mv {

constexpr int kGpThreads = 512;

struct GlaChunkParams {
  __nv_bfloat16* out; int64_t out_stride;
  const __nv_bfloat16 *q, *k, *v; int64_t stride;
  const __nv_bfloat16* z; int64_t z_stride;
  float inv_tau, q_scale;
  const float* zf; const __nv_bfloat16 *w0, *bonus;      // time mixing: z in fp32, its offset and the bonus (heads, K)
  const int32_t *cu, *slots, *start;
  int num_seqs;
  float* state; int num_slots, heads, K, V;
  unsigned char* scratch;                       // [chunk][head][Q hi, Q lo, K hi, K lo, A hi, A lo, 2^b_last]
  bool z_vec;                                   // z's rows are whole 16-byte pieces
};

template <int K> struct GlaScratch {
  static constexpr int64_t kVec = kChunk * K, kA = 4 * kVec, kDecay = kA + 2 * kChunk * kChunk;     // offsets in elements
  static constexpr int64_t kBytes = kDecay * 2 + K * 4;
};

// -log(sigmoid(z)) = max(-z, 0) + log(1 + e), e = e^-|z|, of two logits in packed 32-bit arithmetic.  e is 2^n e^r with Cody and
// Waite's reduction of the argument and a polynomial of degree 6 over |r| <= ln(2) / 2 (3e-9); log(1 + e) = e + e^2 P(e) with one
// of degree 8 over [0, 1] (5e-9); both are weighted least-squares fits with rounded coefficients.  Relative error against 64 bits
// over logits of N(3, 1) and N(0, 2): 3.8e-8 and 3.2e-8 rms, 1.0e-7 and 1.1e-7 at most; log1pf(expf(-z)) has 4.4e-8 and 3.8e-8,
// 1.3e-7 at most, and e from ex2.approx with a division 9.7e-8.  The kernel's time is that of the latter.
__device__ __forceinline__ float2 neg_log_sigmoid(float2 z) {
  constexpr float kRound = 0x1.8p23f, kLn2Hi = 0.693147182f, kLn2Lo = -1.90465421e-9f;
  auto both = [](float x) { return make_float2(x, x); };
  const float2 a = make_float2(fmaxf(-fabsf(z.x), -104.f), fmaxf(-fabsf(z.y), -104.f));
  const float2 m = fma_f32x2(a, both(1.44269502f), both(kRound)), n = add_f32x2(m, both(-kRound));     // m's low bits: n
  const float2 r = fma_f32x2(n, both(-kLn2Lo), fma_f32x2(n, both(-kLn2Hi), a));
  float2 x = fma_f32x2(r, both(0.001382069f), both(0.008368676f));
  x = fma_f32x2(x, r, both(0.041668266f));
  x = fma_f32x2(x, r, both(0.16666521f));
  x = fma_f32x2(x, r, both(0.49999994f));
  const float2 p = add_f32x2(fma_f32x2(mul_f32x2(r, r), x, r), both(1.f));
  const float2 scale = make_float2(__uint_as_float((__float_as_uint(m.x) + 151u) << 23), __uint_as_float((__float_as_uint(m.y) + 151u) << 23));
  const float2 e = mul_f32x2(mul_f32x2(p, scale), both(0x1p-24f));         // in two steps: down to 2^-149
  x = fma_f32x2(e, both(-0.0032904686f), both(0.020086242f));
  x = fma_f32x2(x, e, both(-0.05745723f));
  x = fma_f32x2(x, e, both(0.10661128f));
  x = fma_f32x2(x, e, both(-0.1534488f));
  x = fma_f32x2(x, e, both(0.19692102f));
  x = fma_f32x2(x, e, both(-0.24958019f));
  x = fma_f32x2(x, e, both(0.33330464f));
  x = fma_f32x2(x, e, both(-0.4999993f));
  return add_f32x2(fma_f32x2(mul_f32x2(e, e), x, e), make_float2(max_nan(-z.x, 0.f), max_nan(-z.y, 0.f)));
}

template <int K> struct GlaPrepShape {
  static constexpr int kRow = K + 8;                     // bf16 rows of q and k, then fp32 rows of k's factors in the same place
  // tables (block, channel): sum of a block's logarithms, and 2 to the power of what is in front of the block, of what follows it
  // up to the chunk's end, and of the ways from its edges to its middle
  enum { kTot, kFront, kBehind, kMidQ, kMidK, kTables };
  static constexpr int kBytes = 2 * kChunk * kRow * 2 + (kChunk + 1) * kRow * 4 + kTables * 4 * K * 4 + kChunk * 4;
};

// Two CTAs of 16 warps per SM.  A channel's two powers of a token, from the token to the edge of its block of 16, are formed once;
// everything else is products with a block's: the operands relative to the chunk's ends, and A's blocks.
// 1 x 16,384 tokens, 8 heads of 128: 168 us with powers formed per pair of blocks and logits read one by one, 105 us now
template <int K, bool kTime, bool kWalk>
__global__ void __launch_bounds__(kGpThreads, 2) gla_prepare_kernel(const GlaChunkParams p) {
  using Sh = GlaPrepShape<K>;
  using Sc = GlaScratch<K>;
  constexpr int R = Sh::kRow, kPairs = K / 16;           // pairs of channels per thread
  static_assert(kGpThreads == 512 && kChunk * K / 2 == kPairs * kGpThreads && 4 * K <= kGpThreads, "the split among threads");
  extern __shared__ __align__(16) unsigned char smem[];
  __nv_bfloat16 *sQ = reinterpret_cast<__nv_bfloat16*>(smem), *sK = sQ + kChunk * R;
  float* sKt = reinterpret_cast<float*>(smem);           // k 2^(end of its block - b), over sQ and sK
  float* sB = reinterpret_cast<float*>(sK + kChunk * R) + R;       // a row of zeros in front of token 0
  float* sQt = sB;                                       // q 2^(b - end of the block before), over sB
  float* sTab = sB + kChunk * R;
  float* sOwn = sTab + Sh::kTables * 4 * K;              // A's diagonal, time mixing
  auto tab = [&](int which, int blk) { return sTab + (which * 4 + blk) * K; };
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h = blockIdx.y;
  int seq, chunk;
  if (!find_chunk(p.cu, p.num_seqs, blockIdx.x, seq, chunk)) return;     // uniform: the grid is an upper bound
  const int64_t first = p.cu[seq] + static_cast<int64_t>(chunk) * kChunk;
  const int nt = min(kChunk, static_cast<int>(p.cu[seq + 1] - first));
  using Wb = WalkBlob<K, false>;
  constexpr int64_t kBlob = kWalk ? Wb::kBytes : Sc::kBytes, kABytes = kWalk ? Wb::kA : Sc::kA * 2;
  unsigned char* dst = p.scratch + (static_cast<int64_t>(blockIdx.x) * p.heads + h) * kBlob;
  // columns c and c + 1 of tile x (Q hi, Q lo, K hi, K lo), and of A's term x
  auto tile = [&](int x, int r, int c) -> uint32_t& {
    return *reinterpret_cast<uint32_t*>(dst + (kWalk ? x * Wb::kT + tile_at(r, c) : (x * Sc::kVec + r * K + c) * 2));
  };
  auto local = [&](int x, int r, int c) -> uint32_t& {
    return *reinterpret_cast<uint32_t*>(dst + kABytes + (kWalk ? x * kSlab + tile_at(r, c) : ((x * kChunk + r) * kChunk + c) * 2));
  };
  {
    const uint32_t qd = smem_u32(sQ), kd = smem_u32(sK);
    for (int i = tid; i < kChunk * (K / 8); i += kGpThreads) {
      const int r = i / (K / 8), c = (i % (K / 8)) * 8;
      const bool ok = r < nt && c < p.K;
      const int64_t off = ok ? (first + r) * p.stride + h * p.K + c : 0;
      cp_async16(qd + (r * R + c) * 2, p.q + off, ok ? 16 : 0);
      cp_async16(kd + (r * R + c) * 2, p.k + off, ok ? 16 : 0);
    }
    cp_async_commit();
  }
  auto log_decay = [&](float2 z, int c) {                // of channels c and c + 1
    if constexpr (kTime) {
      return make_float2(time_log_decay(z.x + __bfloat162float(p.w0[h * p.K + c])) * kLog2e,
                         time_log_decay(z.y + __bfloat162float(p.w0[h * p.K + c + 1])) * kLog2e);
    } else {
      return mul_f32x2(mul_f32x2(neg_log_sigmoid(z), make_float2(-p.inv_tau, -p.inv_tau)), make_float2(kLog2e, kLog2e));
    }
  };
  if (p.z_vec) {                                         // rows of z on 16-byte boundaries, K a multiple of eight
    for (int i = tid; i < kChunk * (K / 8); i += kGpThreads) {
      const int r = i / (K / 8), c = (i % (K / 8)) * 8;
      float b[8] = {};
      if (r < nt && c < p.K) {
        const int64_t at = (first + r) * p.z_stride + h * p.K + c;
        float z[8];
        if constexpr (kTime) {
          const float4 x = *reinterpret_cast<const float4*>(p.zf + at), y = *reinterpret_cast<const float4*>(p.zf + at + 4);
          z[0] = x.x; z[1] = x.y; z[2] = x.z; z[3] = x.w; z[4] = y.x; z[5] = y.y; z[6] = y.z; z[7] = y.w;
        } else {
          const uint4 raw = *reinterpret_cast<const uint4*>(p.z + at);
          const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[e]));
            z[2 * e] = f.x;
            z[2 * e + 1] = f.y;
          }
        }
#pragma unroll
        for (int e = 0; e < 8; e += 2) {
          const float2 x = log_decay(make_float2(z[e], z[e + 1]), c + e);
          b[e] = x.x;
          b[e + 1] = x.y;
        }
      }
      float4* to = reinterpret_cast<float4*>(sB + r * R + c);
      to[0] = make_float4(b[0], b[1], b[2], b[3]);
      to[1] = make_float4(b[4], b[5], b[6], b[7]);
    }
  } else {
    for (int i = tid; i < kChunk * (K / 2); i += kGpThreads) {
      const int r = i / (K / 2), c = (i % (K / 2)) * 2;    // p.K is a multiple of eight
      const int64_t at = (first + r) * p.z_stride + h * p.K + c;
      float2 b = make_float2(0.f, 0.f);
      if (r < nt && c < p.K)
        b = log_decay(kTime ? make_float2(p.zf[at], p.zf[at + 1]) : make_float2(__bfloat162float(p.z[at]), __bfloat162float(p.z[at + 1])), c);
      *reinterpret_cast<float2*>(sB + r * R + c) = b;
    }
  }
  for (int c = tid; c < R; c += kGpThreads) sB[c - R] = 0.f;
  __syncthreads();
  {                                                      // running sums: of 16 tokens, joined through the blocks' totals
    const int blk = tid / K, c = tid % K;
    float run[16], sum = 0.f;
    if (blk < 4) {
#pragma unroll
      for (int r = 0; r < 16; ++r) run[r] = sum += sB[(blk * 16 + r) * R + c];
      tab(Sh::kTot, blk)[c] = sum;
    }
    __syncthreads();
    if (blk < 4) {
      float front = 0.f, all = 0.f;
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const float t = tab(Sh::kTot, x)[c];
        if (x < blk) front += t;
        all += t;
      }
#pragma unroll
      for (int r = 0; r < 16; ++r) sB[(blk * 16 + r) * R + c] = front + run[r];
      const float end = front + sum;
      tab(Sh::kFront, blk)[c] = fast_exp2(front);
      tab(Sh::kBehind, blk)[c] = fast_exp2(all - end);
      tab(Sh::kMidQ, blk)[c] = fast_exp2(-run[7]);
      tab(Sh::kMidK, blk)[c] = fast_exp2(run[7] - sum);
      if (blk == 3) reinterpret_cast<float*>(dst + (kWalk ? Wb::kVec : Sc::kDecay * 2))[c] = fast_exp2(all);
    }
  }
  cp_async_wait<0>();
  __syncthreads();
  if (kTime) {
    for (int t = warp; t < kChunk; t += kGpThreads / 32) {
      float own = 0.f;
      for (int c = lane; c < p.K; c += 32)
        own = fmaf(__bfloat162float(sQ[t * R + c]) * __bfloat162float(p.bonus[h * p.K + c]), __bfloat162float(sK[t * R + c]), own);
      own = warp_sum(own);
      if (lane == 0) sOwn[t] = own;
    }
    __syncthreads();
  }
  const float* sE = kTime ? sB - R : sB;                 // exponents beside q
  auto put = [&](int t, int j, float x, float y) {
    uint32_t hi, lo;
    split2(x, y, hi, lo);
    local(0, t, j) = hi;
    local(1, t, j) = lo;
  };
  // Blocks 0 .. 5 of A below the diagonal, (1,0) (2,0) (2,1) (3,0) (3,1) (3,2), then the four on it: one per warp.
  const bool diag = warp >= 6;
  const int bi = diag ? warp - 6 : warp == 0 ? 1 : warp < 3 ? 2 : 3, bj = diag ? bi : warp - bi * (bi - 1) / 2;
  bool mine = warp < 10 && bi * 16 < nt;                 // rows of A past the sequence's end are nobody's
  if (mine && diag) {
    float least = 0.f;
    for (int c = lane; c < K; c += 32) least = fminf(least, tab(Sh::kTot, bi)[c]);
    if (__any_sync(0xffffffffu, least < -60.f)) {        // more than a block's factors can hold: channel by channel
      mine = false;
      for (int i = lane; i < 16 * 8; i += 32) {          // two neighbouring keys of one token
        const int t = bi * 16 + (i >> 3), j = bi * 16 + (i & 7) * 2;
        const int j_end = kTime ? t - 1 : t;
        float x = 0.f, y = 0.f;
        for (int c = 0; j <= j_end && c < K; ++c) {
          const float q = __bfloat162float(sQ[t * R + c]), bt = sE[t * R + c];
          x = fmaf(q * __bfloat162float(sK[j * R + c]), fast_exp2(bt - sB[j * R + c]), x);
          if (j + 1 <= j_end) y = fmaf(q * __bfloat162float(sK[(j + 1) * R + c]), fast_exp2(bt - sB[(j + 1) * R + c]), y);
        }
        if (kTime) {
          if (j == t) x = sOwn[t];
          if (j + 1 == t) y = sOwn[t];
        }
        put(t, j, x * p.q_scale, y * p.q_scale);
      }
    }
  }
  float2 qt[kPairs], kt[kPairs];
  // the rows of one step of a thread lie in one block of 16 when 512 threads cover 8 or 16 of them: its edges are read once
  constexpr int kRows = kGpThreads / (K / 2), kStep = kGpThreads % (K / 2) || kRows > 16 ? 1 : 16 / kRows;
#pragma unroll
  for (int m0 = 0; m0 < kPairs; m0 += kStep) {
    float2 ref, end, front, behind;
#pragma unroll
    for (int m = m0; m < m0 + kStep; ++m) {
      const int i = tid + m * kGpThreads, r = i / (K / 2), c = (i % (K / 2)) * 2;
      if (m == m0) {
        const int blk = r >> 4;
        ref = *reinterpret_cast<const float2*>(sB + (blk * 16 - 1) * R + c), end = *reinterpret_cast<const float2*>(sB + (blk * 16 + 15) * R + c);
        front = *reinterpret_cast<const float2*>(tab(Sh::kFront, blk) + c), behind = *reinterpret_cast<const float2*>(tab(Sh::kBehind, blk) + c);
        front.x *= p.q_scale; front.y *= p.q_scale;
      }
      const float2 b = *reinterpret_cast<const float2*>(sB + r * R + c), e = *reinterpret_cast<const float2*>(sE + r * R + c);
      const float2 q = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(sQ + r * R + c));
      const float2 k = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(sK + r * R + c));
      const float2 ex = add_f32x2(e, make_float2(-ref.x, -ref.y)), ey = add_f32x2(end, make_float2(-b.x, -b.y));
      qt[m] = mul_f32x2(q, make_float2(fast_exp2(ex.x), fast_exp2(ex.y)));
      kt[m] = mul_f32x2(k, make_float2(fast_exp2(ey.x), fast_exp2(ey.y)));
      uint32_t hi, lo;
      const float2 qo = mul_f32x2(qt[m], front), ko = mul_f32x2(kt[m], behind);
      split2(qo.x, qo.y, hi, lo);
      tile(0, r, c) = hi;
      tile(1, r, c) = lo;
      split2(ko.x, ko.y, hi, lo);
      tile(2, r, c) = hi;
      tile(3, r, c) = lo;
    }
  }
  if (kWalk) zero_upper(tid, kGpThreads, [&](int r, int c, int x) -> uint32_t& { return local(x, r, c); });
  __syncthreads();                                       // q, k and b are read
#pragma unroll
  for (int m = 0; m < kPairs; ++m) {
    const int i = tid + m * kGpThreads, r = i / (K / 2), c = (i % (K / 2)) * 2;
    *reinterpret_cast<float2*>(sQt + r * R + c) = qt[m];
    *reinterpret_cast<float2*>(sKt + r * R + c) = kt[m];
  }
  __syncthreads();
  if (!mine) return;
  const int g = lane >> 2, c2 = (lane & 3) * 2;
  const bool far = !diag && bj + 1 < bi;                 // blocks between the two
  float acc[2][4] = {};
#pragma unroll 2
  for (int kb = 0; kb < K; kb += 16) {
    uint32_t ah[4], al[4], bh[4], bl[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      // A: rows g, g + 8 of the block's tokens, channels c2 and c2 + 8;  B: n-tiles of eight keys each
      const int c = kb + c2 + (x >> 1) * 8, t = bi * 16 + g + (x & 1) * 8;
      float2 q = *reinterpret_cast<const float2*>(sQt + t * R + c);
      if (diag) {
        const float2 f = *reinterpret_cast<const float2*>(tab(Sh::kMidQ, bi) + c);
        q.x *= f.x; q.y *= f.y;
      } else if (far) {
        float2 f = *reinterpret_cast<const float2*>(tab(Sh::kTot, bi - 1) + c);
        if (bi - bj == 3) {
          const float2 f2 = *reinterpret_cast<const float2*>(tab(Sh::kTot, 1) + c);
          f.x += f2.x; f.y += f2.y;
        }
        q.x *= fast_exp2(f.x); q.y *= fast_exp2(f.y);
      }
      split2(q.x, q.y, ah[x], al[x]);
      const int cj = kb + c2 + (x & 1) * 8, j = bj * 16 + g + (x >> 1) * 8;
      float2 k = *reinterpret_cast<const float2*>(sKt + j * R + cj);
      if (diag) {
        const float2 f = *reinterpret_cast<const float2*>(tab(Sh::kMidK, bi) + cj);
        k.x *= f.x; k.y *= f.y;
      }
      split2(k.x, k.y, bh[x], bl[x]);
    }
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      Mma::run(acc[n], ah, bh[2 * n], bh[2 * n + 1]);
      Mma::run(acc[n], al, bh[2 * n], bh[2 * n + 1]);
      Mma::run(acc[n], ah, bl[2 * n], bl[2 * n + 1]);
    }
  }
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int t = bi * 16 + g + half * 8, j = bj * 16 + n * 8 + c2;
      float x = acc[n][2 * half], y = acc[n][2 * half + 1];
      if (kTime) {
        if (j == t) x = sOwn[t];
        if (j + 1 == t) y = sOwn[t];
      }
      put(t, j, j <= t ? x * p.q_scale : 0.f, j + 1 <= t ? y * p.q_scale : 0.f);
    }
}

template <int K> struct GlaChunkShape {
  static constexpr int kRow = K + 8;
  static constexpr int kVec = kChunk * kRow * 2, kTile = 2 * kChunk * kCkRow * 2;       // bytes
  static constexpr int stage(int pb) { return 4 * kVec + kChunk * (pb + 8) * 2 + kTile + K * 4; }
};

template <int K>
__global__ void __launch_bounds__(kChunkThreads, 1) gla_chunk_kernel(const GlaChunkParams p, int pb) {
  using Sh = GlaChunkShape<K>;
  using Sc = GlaScratch<K>;
  extern __shared__ __align__(16) unsigned char smem[];
  const int s = blockIdx.x, h = blockIdx.y, p0 = blockIdx.z * pb, pw = min(pb, p.V - p0);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, c2 = (lane & 3) * 2;
  const int vrow = pb + 8;
  const int first = p.cu[s], n_tok = p.cu[s + 1] - first;
  if (n_tok <= 0) return;
  const int chunk0 = chunks_before(p.cu, s), chunks = (n_tok + kChunk - 1) / kChunk;
  const int slot = p.slots[s], st0 = p.start[s];
  const bool live = slot >= 0 && slot < p.num_slots && st0 >= 0;
  float* gS = p.state + (static_cast<int64_t>(live ? slot : 0) * p.heads + h) * p.K * p.V;
  const int stage_bytes = Sh::stage(pb);
  const uint32_t base = smem_u32(smem);
  const __nv_bfloat16* v = p.v + static_cast<int64_t>(h) * p.V + p0;

  auto issue = [&](int c) {
    const uint32_t st = base + (c & 1) * stage_bytes;
    const int64_t row0 = static_cast<int64_t>(first) + c * kChunk;
    const int nt = min(kChunk, n_tok - c * kChunk);
    const __nv_bfloat16* src =
        reinterpret_cast<const __nv_bfloat16*>(p.scratch + (static_cast<int64_t>(chunk0 + c) * p.heads + h) * Sc::kBytes);
    for (int i = tid; i < 4 * kChunk * (K / 8); i += kChunkThreads) {
      const int r = i / (K / 8), cc = (i % (K / 8)) * 8;
      cp_async16(st + (r * Sh::kRow + cc) * 2, src + r * K + cc, 16);
    }
    const uint32_t vd = st + 4 * Sh::kVec, ad = vd + kChunk * vrow * 2;
    for (int i = tid; i < kChunk * (pb / 8); i += kChunkThreads) {
      const int r = i / (pb / 8), cc = (i % (pb / 8)) * 8;
      const bool ok = r < nt && cc < pw;
      cp_async16(vd + (r * vrow + cc) * 2, ok ? v + (row0 + r) * p.stride + cc : p.v, ok ? 16 : 0);
    }
    load_lower(ad, src + Sc::kA, tid, kChunkThreads);
    for (int i = tid; i < K / 4; i += kChunkThreads) cp_async16(ad + Sh::kTile + i * 16, src + Sc::kDecay + i * 8, 16);
    cp_async_commit();
  };
  issue(0);
  const bool work = warp * 16 < pw;
  ChunkState<K> S;
  S.load(gS, p0 + warp * 16, p0 + pw, p.V, p.K, lane, work && live && st0 > 0);
  const LaneAt at(lane);
  for (int c = 0; c < chunks; ++c) {
    cp_async_wait<0>();
    __syncthreads();                     // chunk c is here, and nobody reads the other stage any more
    if (c + 1 < chunks) issue(c + 1);
    if (!work) continue;
    unsigned char* stage = smem + (c & 1) * stage_bytes;
    const uint32_t st = base + (c & 1) * stage_bytes;
    const uint32_t vd = st + 4 * Sh::kVec, ad = vd + kChunk * vrow * 2;
    const float* decay = reinterpret_cast<const float*>(stage + 4 * Sh::kVec + kChunk * vrow * 2 + Sh::kTile);
    uint32_t va[4][4];                   // V^T, the A operand of two products
#pragma unroll
    for (int ib = 0; ib < 4; ++ib) ldmatrix_x4_trans(va[ib], vd + ((ib * 16 + at.row_b) * vrow + warp * 16 + at.col_b) * 2);
    float O[8][4] = {};
#pragma unroll
    for (int kb = 0; kb < K / 16; ++kb) {        // S_0^T Q^T
      uint32_t hi[4], lo[4];
      split_a(S.s[2 * kb], S.s[2 * kb + 1], hi, lo);
      const uint32_t qa = st + (at.row_b * Sh::kRow + kb * 16 + at.col_b) * 2;
#pragma unroll
      for (int np = 0; np < 4; np += 2) {
        uint32_t b[4], d[4];
        const uint32_t q0 = qa + np * 16 * Sh::kRow * 2, q1 = q0 + 16 * Sh::kRow * 2;
        ldmatrix_x4(b, q0);
        ldmatrix_x4(d, q1);
        Mma::run(O[2 * np], hi, b[0], b[1]);
        Mma::run(O[2 * np + 1], hi, b[2], b[3]);
        Mma::run(O[2 * np + 2], hi, d[0], d[1]);
        Mma::run(O[2 * np + 3], hi, d[2], d[3]);
        Mma::run(O[2 * np], lo, b[0], b[1]);
        Mma::run(O[2 * np + 1], lo, b[2], b[3]);
        Mma::run(O[2 * np + 2], lo, d[0], d[1]);
        Mma::run(O[2 * np + 3], lo, d[2], d[3]);
        ldmatrix_x4(b, q0 + Sh::kVec);
        ldmatrix_x4(d, q1 + Sh::kVec);
        Mma::run(O[2 * np], hi, b[0], b[1]);
        Mma::run(O[2 * np + 1], hi, b[2], b[3]);
        Mma::run(O[2 * np + 2], hi, d[0], d[1]);
        Mma::run(O[2 * np + 3], hi, d[2], d[3]);
      }
    }
#pragma unroll
    for (int ib = 0; ib < 4; ++ib) mma_lower<false>(O, va[ib], va[ib], ad, ib, at);
#pragma unroll
    for (int n = 0; n < K / 8; ++n) {
      const float2 d = *reinterpret_cast<const float2*>(decay + n * 8 + c2);
      S.s[n][0] *= d.x; S.s[n][1] *= d.y; S.s[n][2] *= d.x; S.s[n][3] *= d.y;
    }
#pragma unroll
    for (int term = 0; term < 2; ++term)
#pragma unroll
      for (int ib = 0; ib < 4; ++ib) {
        const uint32_t ka = st + (2 + term) * Sh::kVec + ((ib * 16 + at.row_t) * Sh::kRow + at.col_t) * 2;
#pragma unroll
        for (int np = 0; np < K / 16; ++np) {
          uint32_t b[4];
          ldmatrix_x4_trans(b, ka + np * 32);
          Mma::run(S.s[2 * np], va[ib], b[0], b[1]);
          Mma::run(S.s[2 * np + 1], va[ib], b[2], b[3]);
        }
      }
    const int64_t row0 = static_cast<int64_t>(first) + c * kChunk;
    store_out(O, reinterpret_cast<__nv_bfloat16*>(stage + 4 * Sh::kVec) + warp * 16, vrow,
              p.out + row0 * p.out_stride + static_cast<int64_t>(h) * p.V + p0 + warp * 16, p.out_stride,
              min(kChunk, n_tok - c * kChunk), pw - warp * 16, lane);
  }
  if (live && work) S.store(gS, p0 + warp * 16, p0 + pw, p.V, p.K, lane);
}

static int64_t gla_scratch_bytes(int K) {
  int64_t n = 0;
  chunk_dispatch(K, [&](auto kk) { n = GlaScratch<decltype(kk)::value>::kBytes; return 0; });
  return n;
}

}  // namespace mv

// Bytes of scratch for a step, or -1 when the kernels do not take the sizes.
extern "C" int64_t mv_gla_chunk_workspace_bytes(int64_t tokens, int num_seqs, int heads, int dim, int vdim) {
  using namespace mv;
  if (tokens < 0 || num_seqs < 0 || heads <= 0 || !chunk_takes(dim, vdim)) return -1;
  const int64_t chunks = chunk_bound(tokens, num_seqs) * heads;
  if (!walk_takes(false, tokens, num_seqs, heads, dim, vdim)) return chunks * gla_scratch_bytes(dim);
  return chunks * (dim <= 64 ? WalkBlob<64, false>::kBytes : WalkBlob<128, false>::kBytes) +
         walk_segment_floats(false, tokens, num_seqs, heads, dim, vdim) * 4;
}

// Both recurrences; kTime: p.zf, p.w0 and p.bonus, else p.z and p.inv_tau.
template <bool kTime>
static int run_chunks(const char* what, const mv::GlaChunkParams& p, int64_t tokens, int64_t workspace_bytes, int* error_word, cudaStream_t st) {
  using namespace mv;
  const int num_seqs = p.num_seqs, heads = p.heads, dim = p.K, vdim = p.V;
  if (num_seqs < 0 || tokens < 0 || heads <= 0 || heads > 65535 || !chunk_takes(dim, vdim))
    return fail(MV_ERR_SHAPE, "%s: heads %d, dim %d, vdim %d", what, heads, dim, vdim);
  if (num_seqs == 0 || tokens == 0) return MV_OK;
  if (!p.out || !p.q || !p.k || !p.v || !(kTime ? p.zf && p.w0 && p.bonus : p.z != nullptr) || !p.cu || !p.slots || !p.start || !p.state || !error_word)
    return fail(MV_ERR_NULL, "%s: null pointer", what);
  if (!vec8_ok(p.out, p.out_stride, 2) || !vec8_ok(p.q, p.stride, 2) || !vec8_ok(p.k, p.stride, 2) || !vec8_ok(p.v, p.stride, 2))
    return fail(MV_ERR_ALIGN, "%s: rows must start on 16-byte boundaries", what);
  const int64_t chunks = chunk_bound(tokens, num_seqs);
  if (!p.scratch || !aligned16(p.scratch) || workspace_bytes < mv_gla_chunk_workspace_bytes(tokens, num_seqs, heads, dim, vdim))
    return fail(MV_ERR_WORKSPACE, "%s: workspace", what);
  auto prepare = [&](auto kernel, int bytes) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return fail(MV_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
    kernel<<<dim3(static_cast<unsigned>(chunks), heads), kGpThreads, bytes, st>>>(p);
    return check_launch(what);
  };
  if (walk_takes(false, tokens, num_seqs, heads, dim, vdim)) {
    auto walk = [&](auto kk) {
      constexpr int K = decltype(kk)::value;
      const int rc = prepare(gla_prepare_kernel<K, kTime, true>, GlaPrepShape<K>::kBytes);
      if (rc) return rc;
      const WalkParams w{p.out, p.out_stride, nullptr, nullptr, nullptr, p.v, p.stride, p.cu, p.slots, p.start, num_seqs, p.state, nullptr,
                         p.num_slots, heads, dim, vdim, p.scratch, 0, nullptr, nullptr, nullptr, error_word, false};
      return run_walk<K, false>(what, w, tokens, reinterpret_cast<float*>(p.scratch + chunks * heads * WalkBlob<K, false>::kBytes), st);
    };
    return dim <= 64 ? walk(std::integral_constant<int, 64>{}) : walk(std::integral_constant<int, 128>{});
  }
  return chunk_dispatch(dim, [&](auto kk) {
    constexpr int K = decltype(kk)::value;
    const int rc = prepare(gla_prepare_kernel<K, kTime, false>, GlaPrepShape<K>::kBytes);
    if (rc) return rc;
    const int pb = chunk_columns(static_cast<int64_t>(num_seqs) * heads, vdim), smem = 2 * GlaChunkShape<K>::stage(pb);
    const cudaError_t e = cudaFuncSetAttribute(gla_chunk_kernel<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return fail(MV_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
    gla_chunk_kernel<K><<<dim3(num_seqs, heads, (vdim + pb - 1) / pb), kChunkThreads, smem, st>>>(p, pb);
    return check_launch(what);
  });
}

extern "C" int mv_gla_chunk_scan(void* out, int64_t out_stride, const void* q, const void* k, const void* v, int64_t stride,
                                 const void* z, int64_t z_stride, float tau, const int32_t* cu, int num_seqs,
                                 int64_t tokens, const int32_t* slots, const int32_t* start, float* state, int num_slots,
                                 int heads, int dim, int vdim, float q_scale, void* workspace, int64_t workspace_bytes,
                                 int* error_word, void* stream) {
  using namespace mv;
  if (!(tau > 0.f)) return fail(MV_ERR_SHAPE, "gla_chunk_scan: tau %f", tau);
  auto c = [](const void* x) { return static_cast<const __nv_bfloat16*>(x); };
  const GlaChunkParams p{static_cast<__nv_bfloat16*>(out), out_stride, c(q), c(k), c(v), stride, c(z), z_stride, 1.f / tau, q_scale,
                         nullptr, nullptr, nullptr,
                         cu, slots, start, num_seqs, state, num_slots, heads, dim, vdim, static_cast<unsigned char*>(workspace), vec8_ok(z, z_stride, 2)};
  return run_chunks<false>("gla_chunk_scan", p, tokens, workspace_bytes, error_word, static_cast<cudaStream_t>(stream));
}

extern "C" int mv_time_chunk_scan(void* out, int64_t out_stride, const void* r, const void* k, const void* v, int64_t stride,
                                  const float* z, int64_t z_stride, const void* w0, const void* bonus, const int32_t* cu,
                                  int num_seqs, int64_t tokens, const int32_t* slots, const int32_t* start, float* state,
                                  int num_slots, int heads, int dim, int vdim, void* workspace, int64_t workspace_bytes,
                                  int* error_word, void* stream) {
  using namespace mv;
  auto c = [](const void* x) { return static_cast<const __nv_bfloat16*>(x); };
  const GlaChunkParams p{static_cast<__nv_bfloat16*>(out), out_stride, c(r), c(k), c(v), stride, nullptr, z_stride, 1.f, 1.f,
                         z, c(w0), c(bonus),
                         cu, slots, start, num_seqs, state, num_slots, heads, dim, vdim, static_cast<unsigned char*>(workspace), vec8_ok(z, z_stride, 4)};
  return run_chunks<true>("time_chunk_scan", p, tokens, workspace_bytes, error_word, static_cast<cudaStream_t>(stream));
}
