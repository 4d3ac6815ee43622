// Paged decode attention over an int8 KV cache (per-token-per-head symmetric
// codes with fp16 scales, written by the quantising store_kvcache).
//
// Same plan, work items and warp-private cp.async rings as paged_decode.cu;
// what differs is the operand path.  Codes are dequantised in registers: a
// byte c is byte-permuted into the fp16 pattern 0x64xx = 1024 + (c ^ 0x80) =
// c + 1152 (exact), and the constant 1152 is NOT subtracted per element but
// taken out afterwards where it factors: S = Q.(C + 1152) - 1152 * rowsum(Q),
// O = P'.(C + 1152) - 1152 * rowsum(P'), the latter row sum coming from one
// extra MMA against a tile of ones so that it is exactly what the tensor core
// summed.  The MMAs run in fp16 with fp32 accumulation whatever the model
// dtype (q is converted), and the per-token scales are applied where they
// factor out: the K scale on the score column, the V scale on the
// probability column.  The k index of the
// QK^T MMAs and the n index of the PV MMAs are permuted so that every thread
// reads its operands with 16-byte shared-memory loads.
// HBM-bound: algorithmic bytes = sum(ctx) * num_kv_heads * (head_dim + 2) * 2.
#include "paged_decode.cuh"

namespace mv {

// A warp's loop iteration has a fixed latency (wait, dequantise, dependent MMAs, softmax shuffles) that is
// about the same for 16 or 32 tokens, and int8 rows are half as long as fp16 rows: 32-token tiles keep the
// bytes per iteration (8 KB) equal to the fp16 kernel's.
constexpr int kQTok = 32;     // tokens per warp tile
constexpr int kQStages = 3;
constexpr int kQD = 128;

struct Int8Smem {
  static constexpr int kRowBytes = kQD;                              // one row of codes
  static constexpr int kTileBytes = kQTok * kRowBytes;               // K or V codes of a tile
  static constexpr int kScaleBytes = 2 * kQTok * 4;                  // one 4-byte word per token, K then V
  static constexpr int kStageBytes = 2 * kTileBytes + kScaleBytes;
  static constexpr int kWarpBytes = kQStages * kStageBytes;
  static constexpr int kRingBytes = kDecWarps * kWarpBytes;
  static constexpr int kMergeStride = kQD + 8;
  static constexpr int kMergeBytes = kDecWarps * 16 * kMergeStride * 4 + kDecWarps * 16 * 2 * 4;
  static_assert(kMergeBytes <= kRingBytes, "merge buffer must fit in the ring");
};

__device__ __forceinline__ void cp_async4(uint32_t dst_smem, const void* src, int src_bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst_smem), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}
__device__ __forceinline__ float scale_of(uint32_t word, uint32_t odd) {
  return __half2float(__ushort_as_half(static_cast<unsigned short>(odd ? (word >> 16) : (word & 0xffffu))));
}

template <typename T>
__global__ void __launch_bounds__(kDecThreads, kDecCtasPerSM)
paged_decode_int8_kernel(const DecodeParams p) {
  using S = Int8Smem;
  constexpr int D = kQD;
  constexpr int KSTEPS = D / 16;
  constexpr int NT = D / 8;
  constexpr uint32_t kMagic = 0x64646464u, kBias = 0x80808080u;

  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ long long s_red[kDecWarps];
  __shared__ uint32_t s_mask[kDecWarps][kQStages][2];  // [0]: live rows of the tile, [1]: rows whose scale index is odd
  __shared__ int s_last;
  int* s_start = reinterpret_cast<int*>(smem + S::kRingBytes);

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;

  const DecodePlan plan = build_plan(p, s_start, s_red);
  if (p.arrivals == nullptr && blockIdx.x == 0) {
    for (int b = tid; b < p.batch; b += kDecThreads) p.binfo[b] = seq_items(s_start, plan, b);
  }
  zero_empty_sequences<T, D>(p, s_start);

  const int ydim = p.num_kv_heads * p.mtiles;
  const int n_units = plan.n_seg * ydim;
  const uint32_t ring = smem_u32(smem) + warp * S::kWarpBytes;
  const int8_t* kc = static_cast<const int8_t*>(p.k_cache);
  const int8_t* vc = static_cast<const int8_t*>(p.v_cache);
  const int bs = p.block_size;

  ItemWalk at;
  for (walk_start(p, s_start, plan, ydim, n_units, blockIdx.x, at); at.b >= 0;
       walk_next(p, s_start, plan, ydim, n_units, gridDim.x, at)) {
    const int kvh = at.y / p.mtiles, mt = at.y - kvh * p.mtiles;
    const DecodeItem di = piece_of(p, s_start, plan, at.b, at.seg);
    const int item = di.item, b = di.b, nsplit = di.nsplit, tok_begin = di.tok_begin, tok_end = di.tok_end;
    const int32_t* table = p.block_tables + static_cast<int64_t>(b) * p.bt_stride;
    const int rows_valid = min(16, p.group - mt * 16);
    const int h0 = kvh * p.group + mt * 16;

    const int span = tok_end - tok_begin;
    const int cta_tiles = span > 0 ? (span + kQTok - 1) / kQTok : 0;
    const int my_tiles = cta_tiles > warp ? (cta_tiles - warp + kDecWarps - 1) / kDecWarps : 0;

    auto issue = [&](int i) {
      if (i < my_tiles) {
        const int stage = i % kQStages;
        const int tok0 = tok_begin + (i * kDecWarps + warp) * kQTok;
        const int blk0 = tok0 / bs, off0 = tok0 - blk0 * bs;
        int off = off0 + lane, blk = blk0;           // lane r resolves row r of the tile
        while (off >= bs) { off -= bs; ++blk; }
        int slot = -1;
        if (tok0 + lane < tok_end) {
          const int pb = __ldg(table + blk);
          if (pb >= 0 && pb < p.num_blocks) slot = pb * bs + off;
        }
        const int64_t sidx = static_cast<int64_t>(slot) * p.num_kv_heads + kvh;  // scale index of my row
        const bool is_odd = slot >= 0 && (sidx & 1);
        const uint32_t live = __ballot_sync(0xffffffffu, slot >= 0);
        const uint32_t odd = __ballot_sync(0xffffffffu, is_odd);
        if (lane == 0) { s_mask[warp][stage][0] = live; s_mask[warp][stage][1] = odd; }
        const uint32_t kdst = ring + stage * S::kStageBytes;
        const uint32_t vdst = kdst + S::kTileBytes;
        const uint32_t sdst = vdst + S::kTileBytes;
        // scales: one aligned 4-byte word holding the fp16 (low or high half), K words then V words
        {
          const int64_t base = slot >= 0 ? (is_odd ? sidx - 1 : sidx) : 0;
          const int nbytes = slot >= 0 ? (is_odd ? 4 : 2) : 0;
          cp_async4(sdst + lane * 4, p.k_scale + base, nbytes);
          cp_async4(sdst + (kQTok + lane) * 4, p.v_scale + base, nbytes);
        }
        const int c = lane & 7, r0 = lane >> 3;
#pragma unroll
        for (int it = 0; it < kQTok / 4; ++it) {
          const int r = r0 + it * 4;
          const int s = __shfl_sync(0xffffffffu, slot, r);
          const int64_t boff = s >= 0 ? (static_cast<int64_t>(s) * p.num_kv_heads + kvh) * D + c * 16 : 0;
          const uint32_t doff = r * S::kRowBytes + ((c ^ (r & 7)) << 4);
          cp_async16(kdst + doff, kc + boff, s >= 0 ? 16 : 0);
          cp_async16(vdst + doff, vc + boff, s >= 0 ? 16 : 0);
        }
      }
      cp_async_commit();
    };

#pragma unroll
    for (int i = 0; i < kQStages - 1; ++i) issue(i);

    // Q fragments in fp16 with the permuted k index: k-step ks of thread t
    // covers head-dim elements 32t + 4ks .. 32t + 4ks + 3.
    uint32_t qa[KSTEPS][4];
    {
      const T* qbase = static_cast<const T*>(p.q) + (static_cast<int64_t>(b) * p.num_heads + h0) * D;
#pragma unroll
      for (int half_row = 0; half_row < 2; ++half_row) {
        const int row = g + 8 * half_row;
        const bool ok = row < rows_valid;
        const uint2* src = reinterpret_cast<const uint2*>(qbase + static_cast<int64_t>(row) * D + 32 * t);
#pragma unroll
        for (int ks = 0; ks < KSTEPS; ++ks) {
          uint2 raw = ok ? __ldg(src + ks) : make_uint2(0u, 0u);
          if constexpr (!std::is_same<T, __half>::value) {
            const float2 a = Elem<T>::to_f2(*reinterpret_cast<typename Elem<T>::T2*>(&raw.x));
            const float2 c2 = Elem<T>::to_f2(*reinterpret_cast<typename Elem<T>::T2*>(&raw.y));
            raw.x = pack2<__half>(a.x, a.y);
            raw.y = pack2<__half>(c2.x, c2.y);
          }
          qa[ks][half_row] = raw.x;       // k = 2t, 2t+1
          qa[ks][2 + half_row] = raw.y;   // k = 2t+8, 2t+9
        }
      }
    }

    // -1152 * sum over head_dim of q, per row: the bias of the un-subtracted codes in S
    float nbias0 = 0.f, nbias1 = 0.f;
#pragma unroll
    for (int ks = 0; ks < KSTEPS; ++ks) {
      const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&qa[ks][0]));
      const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&qa[ks][2]));
      const float2 c = __half22float2(*reinterpret_cast<const __half2*>(&qa[ks][1]));
      const float2 d = __half22float2(*reinterpret_cast<const __half2*>(&qa[ks][3]));
      nbias0 += (a.x + a.y) + (b.x + b.y);
      nbias1 += (c.x + c.y) + (d.x + d.y);
    }
    nbias0 += __shfl_xor_sync(0xffffffffu, nbias0, 1);
    nbias0 += __shfl_xor_sync(0xffffffffu, nbias0, 2);
    nbias1 += __shfl_xor_sync(0xffffffffu, nbias1, 1);
    nbias1 += __shfl_xor_sync(0xffffffffu, nbias1, 2);
    nbias0 *= -1152.f;
    nbias1 *= -1152.f;

    float o[NT][4];
#pragma unroll
    for (int j = 0; j < NT; ++j) { o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f; }
    float osum[4] = {0.f, 0.f, 0.f, 0.f};   // P' times a tile of ones: row sums of P' as the tensor core adds them
    float m0 = kNegBig, m1 = kNegBig, l0 = 0.f, l1 = 0.f;
    const uint32_t kOnes = 0x3c003c00u;     // fp16 (1, 1)

    for (int i = 0; i < my_tiles; ++i) {
      cp_async_wait<kQStages - 2>();
      __syncwarp();
      const int stage = i % kQStages;
      const uint32_t kbase = ring + stage * S::kStageBytes;
      const uint32_t vbase = kbase + S::kTileBytes;
      const uint32_t sbase = vbase + S::kTileBytes;
      const uint32_t live = s_mask[warp][stage][0], odd = s_mask[warp][stage][1];

      // ---- S = Q K^T on the codes: four n-tiles of 8 tokens ----
      float s[4][4];
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.f;
        const int row = 8 * n + g;
        const uint4 w0 = lds128(kbase + row * S::kRowBytes + (((2 * t) ^ (row & 7)) << 4));
        const uint4 w1 = lds128(kbase + row * S::kRowBytes + (((2 * t + 1) ^ (row & 7)) << 4));
        const uint32_t words[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
        for (int ks = 0; ks < KSTEPS; ++ks) {
          const uint32_t x = words[ks] ^ kBias;
          Mma16816<__half>::run(s[n], qa[ks], prmt(x, kMagic, 0x4140u), prmt(x, kMagic, 0x4342u));
        }
      }
      issue(i + kQStages - 1);

      // ---- K scales, mask, online softmax ----
      float mx0 = kNegBig, mx1 = kNegBig;
#pragma unroll
      for (int n = 0; n < 4; ++n) {
#pragma unroll
        for (int e2 = 0; e2 < 2; ++e2) {
          const int col = n * 8 + 2 * t + e2;
          const bool ok = (live >> col) & 1u;
          const float ks = scale_of(lds32(sbase + col * 4), (odd >> col) & 1u) * p.scale_log2;
          s[n][e2] = ok ? (s[n][e2] + nbias0) * ks : -INFINITY;
          s[n][2 + e2] = ok ? (s[n][2 + e2] + nbias1) * ks : -INFINITY;
        }
        mx0 = fmaxf(mx0, fmaxf(s[n][0], s[n][1]));
        mx1 = fmaxf(mx1, fmaxf(s[n][2], s[n][3]));
      }
      mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1));
      mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2));
      mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1));
      mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
      const float mn0 = fmaxf(m0, mx0), mn1 = fmaxf(m1, mx1);
      const float a0 = fast_exp2(m0 - mn0), a1 = fast_exp2(m1 - mn1);
      m0 = mn0; m1 = mn1;
      float ps0 = 0.f, ps1 = 0.f;
      uint32_t pa[2][4];   // A fragments of the two 16-token k-steps
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        const float p00 = fast_exp2(s[n][0] - mn0), p01 = fast_exp2(s[n][1] - mn0);
        const float p10 = fast_exp2(s[n][2] - mn1), p11 = fast_exp2(s[n][3] - mn1);
        ps0 += p00 + p01;
        ps1 += p10 + p11;
        // V scale of the two tokens of this column pair, folded into P
        const int col = n * 8 + 2 * t;
        const float vs0 = scale_of(lds32(sbase + (kQTok + col) * 4), (odd >> col) & 1u);
        const float vs1 = scale_of(lds32(sbase + (kQTok + col + 1) * 4), (odd >> (col + 1)) & 1u);
        const bool ok0 = (live >> col) & 1u, ok1 = (live >> (col + 1)) & 1u;
        pa[n >> 1][2 * (n & 1)] = pack2<__half>(ok0 ? p00 * vs0 : 0.f, ok1 ? p01 * vs1 : 0.f);
        pa[n >> 1][2 * (n & 1) + 1] = pack2<__half>(ok0 ? p10 * vs0 : 0.f, ok1 ? p11 * vs1 : 0.f);
      }
      l0 = l0 * a0 + ps0;
      l1 = l1 * a1 + ps1;

      // the running maximum rarely moves after the first tiles: rescale only when some row of the warp needs it
      if (__any_sync(0xffffffffu, a0 != 1.f || a1 != 1.f)) {
#pragma unroll
        for (int j = 0; j < NT; ++j) { o[j][0] *= a0; o[j][1] *= a0; o[j][2] *= a1; o[j][3] *= a1; }
        osum[0] *= a0; osum[1] *= a0; osum[2] *= a1; osum[3] *= a1;
      }
      // ---- O += P V on the codes; n-tile j of thread (g, t) is head-dim element 16*col + j ----
#pragma unroll
      for (int kk = 0; kk < 2; ++kk) {
        const int ra = 16 * kk + 2 * t, rb = ra + 1, rc = ra + 8, rd = ra + 9;
        const uint4 va = lds128(vbase + ra * S::kRowBytes + ((g ^ (ra & 7)) << 4));
        const uint4 vb = lds128(vbase + rb * S::kRowBytes + ((g ^ (rb & 7)) << 4));
        const uint4 vcx = lds128(vbase + rc * S::kRowBytes + ((g ^ (rc & 7)) << 4));
        const uint4 vd = lds128(vbase + rd * S::kRowBytes + ((g ^ (rd & 7)) << 4));
        const uint32_t wa[4] = {va.x, va.y, va.z, va.w}, wb[4] = {vb.x, vb.y, vb.z, vb.w};
        const uint32_t wc[4] = {vcx.x, vcx.y, vcx.z, vcx.w}, wd[4] = {vd.x, vd.y, vd.z, vd.w};
#pragma unroll
        for (int wi = 0; wi < 4; ++wi) {
          const uint32_t xa = wa[wi] ^ kBias, xb = wb[wi] ^ kBias, xc = wc[wi] ^ kBias, xd = wd[wi] ^ kBias;
          const uint32_t lo01 = prmt(xa, xb, 0x5140u), lo23 = prmt(xa, xb, 0x7362u);  // tokens ra, ra+1
          const uint32_t hi01 = prmt(xc, xd, 0x5140u), hi23 = prmt(xc, xd, 0x7362u);  // tokens ra+8, ra+9
          const uint32_t lo[4] = {prmt(lo01, kMagic, 0x4140u), prmt(lo01, kMagic, 0x4342u),
                                  prmt(lo23, kMagic, 0x4140u), prmt(lo23, kMagic, 0x4342u)};
          const uint32_t hi[4] = {prmt(hi01, kMagic, 0x4140u), prmt(hi01, kMagic, 0x4342u),
                                  prmt(hi23, kMagic, 0x4140u), prmt(hi23, kMagic, 0x4342u)};
#pragma unroll
          for (int jj = 0; jj < 4; ++jj) Mma16816<__half>::run(o[4 * wi + jj], pa[kk], lo[jj], hi[jj]);
        }
        Mma16816<__half>::run(osum, pa[kk], kOnes, kOnes);
      }
      __syncwarp();
    }
    cp_async_wait<0>();

    l0 += __shfl_xor_sync(0xffffffffu, l0, 1);
    l0 += __shfl_xor_sync(0xffffffffu, l0, 2);
    l1 += __shfl_xor_sync(0xffffffffu, l1, 1);
    l1 += __shfl_xor_sync(0xffffffffu, l1, 2);

    // every column of the ones tile carries the same row sum: take the bias of the V codes out of O
    {
      const float b0 = 1152.f * osum[0], b1 = 1152.f * osum[2];
#pragma unroll
      for (int j = 0; j < NT; ++j) { o[j][0] -= b0; o[j][1] -= b0; o[j][2] -= b1; o[j][3] -= b1; }
    }

    __syncthreads();
    float* sO = reinterpret_cast<float*>(smem);
    float* sML = sO + kDecWarps * 16 * S::kMergeStride;
    {
      float* mine = sO + warp * 16 * S::kMergeStride;
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        // accumulator column 2t+e of n-tile j holds head-dim element 16*(2t+e) + j
        mine[g * S::kMergeStride + 32 * t + j] = o[j][0];
        mine[g * S::kMergeStride + 32 * t + 16 + j] = o[j][1];
        mine[(g + 8) * S::kMergeStride + 32 * t + j] = o[j][2];
        mine[(g + 8) * S::kMergeStride + 32 * t + 16 + j] = o[j][3];
      }
      if (t == 0) {
        sML[(warp * 16 + g) * 2] = m0;
        sML[(warp * 16 + g) * 2 + 1] = l0;
        sML[(warp * 16 + g + 8) * 2] = m1;
        sML[(warp * 16 + g + 8) * 2 + 1] = l1;
      }
    }
    __syncthreads();
    merge_and_write<T, D>(p, sO, sML, S::kMergeStride, rows_valid, h0, b, item, nsplit);
    __syncthreads();
    combine_if_last<T, D>(p, s_start, plan, b, b * ydim + kvh * p.mtiles + mt, h0, rows_valid, nsplit, &s_last);
  }
}

// Groups of up to eight query heads: tokens on the M side of every product, heads on the N side, so that of a product's 16 x 8
// results half or more are wanted (with heads on M it was group / 16 of them).  That halves the products and the accumulators
// per cached byte, and the registers it frees hold twice the warps: eight a CTA, 16-token tiles, the same bytes in flight.
// The dequantised words are the same; K codes are the A operand of S^T = K Q^T, V codes, with tokens as the reduction, the A
// operand of O^T = V^T P^T, and P^T comes out of S^T's registers by two 8 x 8 transposes.  Bound: HBM, then issue (about 240
// slots per 4 KB tile and warp).
constexpr int kQ8Warps = 8, kQ8Tok = 16, kQ8Stages = 3;
struct Int8TokSmem {
  static constexpr int kRowBytes = kQD;
  static constexpr int kTileBytes = kQ8Tok * kRowBytes;
  static constexpr int kStageBytes = 2 * kTileBytes + 2 * kQ8Tok * 4;
  static constexpr int kWarpBytes = kQ8Stages * kStageBytes;
  static constexpr int kRingBytes = kQ8Warps * kWarpBytes;
  static constexpr int kMergeStride = kQD + 8;
  static_assert(kQ8Warps * 8 * (kMergeStride + 2) * 4 <= kRingBytes, "merge buffer must fit in the ring");
};
__device__ __forceinline__ uint32_t transpose8(uint32_t x) {       // an 8 x 8 matrix of 16-bit values, a row per four lanes
  uint32_t r;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(x));
  return r;
}

template <typename T>
__global__ void __launch_bounds__(kQ8Warps * 32, kDecCtasPerSM)
paged_decode_int8_tok_kernel(const DecodeParams p) {
  using S = Int8TokSmem;
  constexpr int D = kQD, KSTEPS = D / 16, MT = D / 16;
  constexpr uint32_t kMagic = 0x64646464u, kBias = 0x80808080u;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ long long s_red[kQ8Warps];
  __shared__ uint32_t s_mask[kQ8Warps][kQ8Stages][2];  // [0]: live rows of the tile, [1]: rows whose scale index is odd
  __shared__ int s_last;
  int* s_start = reinterpret_cast<int*>(smem + S::kRingBytes);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;

  const DecodePlan plan = build_plan<kQ8Warps>(p, s_start, s_red);
  if (p.arrivals == nullptr && blockIdx.x == 0) {
    for (int b = tid; b < p.batch; b += kQ8Warps * 32) p.binfo[b] = seq_items(s_start, plan, b);
  }
  zero_empty_sequences<T, D>(p, s_start);
  const int ydim = p.num_kv_heads;
  const int n_units = plan.n_seg * ydim;
  const uint32_t ring = smem_u32(smem) + warp * S::kWarpBytes;
  const int8_t* kc = static_cast<const int8_t*>(p.k_cache);
  const int8_t* vc = static_cast<const int8_t*>(p.v_cache);
  const int bs = p.block_size;

  ItemWalk at;
  for (walk_start(p, s_start, plan, ydim, n_units, blockIdx.x, at); at.b >= 0;
       walk_next(p, s_start, plan, ydim, n_units, gridDim.x, at)) {
    const int kvh = at.y;
    const DecodeItem di = piece_of(p, s_start, plan, at.b, at.seg);
    const int b = di.b, tok_begin = di.tok_begin, tok_end = di.tok_end;
    const int32_t* table = p.block_tables + static_cast<int64_t>(b) * p.bt_stride;
    const int rows_valid = p.group, h0 = kvh * p.group;
    const int span = tok_end - tok_begin;
    const int cta_tiles = span > 0 ? (span + kQ8Tok - 1) / kQ8Tok : 0;
    const int my_tiles = cta_tiles > warp ? (cta_tiles - warp + kQ8Warps - 1) / kQ8Warps : 0;

    auto issue = [&](int i) {
      if (i < my_tiles) {
        const int stage = i % kQ8Stages;
        const int tok0 = tok_begin + (i * kQ8Warps + warp) * kQ8Tok;
        const int blk0 = tok0 / bs, r_me = lane & 15;
        int off = tok0 - blk0 * bs + r_me, blk = blk0;   // lane r (r < 16) resolves row r of the tile; others mirror it
        while (off >= bs) { off -= bs; ++blk; }
        int slot = -1;
        if (tok0 + r_me < tok_end) {
          const int pb = __ldg(table + blk);
          if (pb >= 0 && pb < p.num_blocks) slot = pb * bs + off;
        }
        const int64_t sidx = static_cast<int64_t>(slot) * p.num_kv_heads + kvh;  // scale index of my row
        const bool is_odd = slot >= 0 && (sidx & 1);
        const uint32_t live = __ballot_sync(0xffffffffu, slot >= 0) & 0xffffu;
        const uint32_t odd = __ballot_sync(0xffffffffu, is_odd);
        if (lane == 0) { s_mask[warp][stage][0] = live; s_mask[warp][stage][1] = odd; }
        const uint32_t kdst = ring + stage * S::kStageBytes, vdst = kdst + S::kTileBytes, sdst = vdst + S::kTileBytes;
        // scales: one aligned 4-byte word holding the fp16 (low or high half); lanes 0-15 K's, 16-31 V's
        {
          const int64_t base = slot >= 0 ? (is_odd ? sidx - 1 : sidx) : 0;
          cp_async4(sdst + lane * 4, (lane < 16 ? p.k_scale : p.v_scale) + base, slot >= 0 ? (is_odd ? 4 : 2) : 0);
        }
        const int c = lane & 7, r0 = lane >> 3;
#pragma unroll
        for (int it = 0; it < kQ8Tok / 4; ++it) {
          const int r = r0 + it * 4;
          const int s = __shfl_sync(0xffffffffu, slot, r);
          const int64_t boff = s >= 0 ? (static_cast<int64_t>(s) * p.num_kv_heads + kvh) * D + c * 16 : 0;
          const uint32_t doff = r * S::kRowBytes + ((c ^ (r & 7)) << 4);
          cp_async16(kdst + doff, kc + boff, s >= 0 ? 16 : 0);
          cp_async16(vdst + doff, vc + boff, s >= 0 ? 16 : 0);
        }
      }
      cp_async_commit();
    };
#pragma unroll
    for (int i = 0; i < kQ8Stages - 1; ++i) issue(i);

    // Q^T as B operand, head g, with the permuted reduction index: step ks of thread t covers head-dim elements 32t + 4ks ..
    // 32t + 4ks + 3.  The codes are not un-biased: 1152 times a head's sum over q comes off its scores.
    uint32_t qb[KSTEPS][2];
    float qsum = 0.f;
    {
      const uint2* src = reinterpret_cast<const uint2*>(static_cast<const T*>(p.q) + (static_cast<int64_t>(b) * p.num_heads + h0 + g) * D + 32 * t);
#pragma unroll
      for (int ks = 0; ks < KSTEPS; ++ks) {
        uint2 raw = g < rows_valid ? __ldg(src + ks) : make_uint2(0u, 0u);
        const float2 x = Elem<T>::to_f2(*reinterpret_cast<typename Elem<T>::T2*>(&raw.x));
        const float2 y = Elem<T>::to_f2(*reinterpret_cast<typename Elem<T>::T2*>(&raw.y));
        qb[ks][0] = pack2<__half>(x.x, x.y);
        qb[ks][1] = pack2<__half>(y.x, y.y);
        const float2 xh = __half22float2(*reinterpret_cast<const __half2*>(&qb[ks][0]));
        const float2 yh = __half22float2(*reinterpret_cast<const __half2*>(&qb[ks][1]));
        qsum += (xh.x + xh.y) + (yh.x + yh.y);
      }
    }
    qsum += __shfl_xor_sync(0xffffffffu, qsum, 1);
    qsum += __shfl_xor_sync(0xffffffffu, qsum, 2);
    const float nbias0 = -1152.f * __shfl_sync(0xffffffffu, qsum, 8 * t);        // heads 2t and 2t + 1
    const float nbias1 = -1152.f * __shfl_sync(0xffffffffu, qsum, 8 * t + 4);

    float o[MT][4];
#pragma unroll
    for (int j = 0; j < MT; ++j) { o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f; }
    float osum[4] = {0.f, 0.f, 0.f, 0.f};   // ones times P': column sums of P' as the tensor core adds them
    const uint32_t ones[4] = {0x3c003c00u, 0x3c003c00u, 0x3c003c00u, 0x3c003c00u};
    float m0 = kNegBig, m1 = kNegBig, l0 = 0.f, l1 = 0.f;                        // heads 2t and 2t + 1

    for (int i = 0; i < my_tiles; ++i) {
      cp_async_wait<kQ8Stages - 2>();
      __syncwarp();
      const int stage = i % kQ8Stages;
      const uint32_t kbase = ring + stage * S::kStageBytes, vbase = kbase + S::kTileBytes, sbase = vbase + S::kTileBytes;
      const uint32_t live = s_mask[warp][stage][0], odd = s_mask[warp][stage][1];
      // ---- S^T: tokens g and g + 8, heads 2t and 2t + 1 ----
      float s[4] = {0.f, 0.f, 0.f, 0.f};
      {
        const uint4 a0 = lds128(kbase + g * S::kRowBytes + (((2 * t) ^ g) << 4)), a1 = lds128(kbase + g * S::kRowBytes + (((2 * t + 1) ^ g) << 4));
        const uint4 b0 = lds128(kbase + (g + 8) * S::kRowBytes + (((2 * t) ^ g) << 4)), b1 = lds128(kbase + (g + 8) * S::kRowBytes + (((2 * t + 1) ^ g) << 4));
        const uint32_t wa[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
        const uint32_t wb[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
        float s2[4] = {0.f, 0.f, 0.f, 0.f};             // two chains of products
#pragma unroll
        for (int ks = 0; ks < KSTEPS; ++ks) {
          const uint32_t x = wa[ks] ^ kBias, y = wb[ks] ^ kBias;
          const uint32_t a[4] = {prmt(x, kMagic, 0x4140u), prmt(y, kMagic, 0x4140u), prmt(x, kMagic, 0x4342u), prmt(y, kMagic, 0x4342u)};
          Mma16816<__half>::run(ks & 1 ? s2 : s, a, qb[ks][0], qb[ks][1]);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) s[e] += s2[e];
      }
      issue(i + kQ8Stages - 1);
      // ---- K scales, mask, online softmax ----
      const bool ok0 = (live >> g) & 1u, ok1 = (live >> (g + 8)) & 1u;
      const uint32_t od0 = (odd >> g) & 1u, od1 = (odd >> (g + 8)) & 1u;
      const float ks0 = scale_of(lds32(sbase + g * 4), od0) * p.scale_log2, ks1 = scale_of(lds32(sbase + (g + 8) * 4), od1) * p.scale_log2;
      s[0] = ok0 ? (s[0] + nbias0) * ks0 : -INFINITY;
      s[1] = ok0 ? (s[1] + nbias1) * ks0 : -INFINITY;
      s[2] = ok1 ? (s[2] + nbias0) * ks1 : -INFINITY;
      s[3] = ok1 ? (s[3] + nbias1) * ks1 : -INFINITY;
      // a running maximum rarely moves after the first tiles: one vote then instead of the reduction over tokens
      float mx0 = fmaxf(s[0], s[2]), mx1 = fmaxf(s[1], s[3]);
      if (__any_sync(0xffffffffu, mx0 > m0 || mx1 > m1)) {
#pragma unroll
        for (int off = 4; off < 32; off <<= 1) {
          mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, off));
          mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, off));
        }
        const float mn0 = fmaxf(m0, mx0), mn1 = fmaxf(m1, mx1);
        const float a0 = fast_exp2(m0 - mn0), a1 = fast_exp2(m1 - mn1);
        m0 = mn0; m1 = mn1;
        l0 *= a0; l1 *= a1;
        osum[0] *= a0; osum[1] *= a1;
#pragma unroll
        for (int j = 0; j < MT; ++j) { o[j][0] *= a0; o[j][1] *= a1; o[j][2] *= a0; o[j][3] *= a1; }
      }
      const float p00 = fast_exp2(s[0] - m0), p01 = fast_exp2(s[1] - m1), p10 = fast_exp2(s[2] - m0), p11 = fast_exp2(s[3] - m1);
      l0 += p00 + p10;
      l1 += p01 + p11;
      // V scales folded into P
      const float vs0 = ok0 ? scale_of(lds32(sbase + (kQ8Tok + g) * 4), od0) : 0.f, vs1 = ok1 ? scale_of(lds32(sbase + (kQ8Tok + g + 8) * 4), od1) : 0.f;
      const uint32_t pb0 = transpose8(pack2<__half>(p00 * vs0, p01 * vs0)), pb1 = transpose8(pack2<__half>(p10 * vs1, p11 * vs1));
      // ---- O^T += V^T P^T: row g of tile 2 wi + j is head-dim element 16 g + 4 wi + 2 j, row g + 8 the one behind it ----
      {
        const int ra = 2 * t, rb = ra + 1, rc = ra + 8, rd = ra + 9;
        const uint4 va = lds128(vbase + ra * S::kRowBytes + ((g ^ (ra & 7)) << 4)), vb = lds128(vbase + rb * S::kRowBytes + ((g ^ (rb & 7)) << 4));
        const uint4 vx = lds128(vbase + rc * S::kRowBytes + ((g ^ (rc & 7)) << 4)), vd = lds128(vbase + rd * S::kRowBytes + ((g ^ (rd & 7)) << 4));
        const uint32_t wa[4] = {va.x, va.y, va.z, va.w}, wb[4] = {vb.x, vb.y, vb.z, vb.w};
        const uint32_t wc[4] = {vx.x, vx.y, vx.z, vx.w}, wd[4] = {vd.x, vd.y, vd.z, vd.w};
#pragma unroll
        for (int wi = 0; wi < 4; ++wi) {
          const uint32_t xa = wa[wi] ^ kBias, xb = wb[wi] ^ kBias, xc = wc[wi] ^ kBias, xd = wd[wi] ^ kBias;
          const uint32_t lo01 = prmt(xa, xb, 0x5140u), lo23 = prmt(xa, xb, 0x7362u);  // tokens ra, ra+1
          const uint32_t hi01 = prmt(xc, xd, 0x5140u), hi23 = prmt(xc, xd, 0x7362u);  // tokens ra+8, ra+9
          const uint32_t a[4] = {prmt(lo01, kMagic, 0x4140u), prmt(lo01, kMagic, 0x4342u), prmt(hi01, kMagic, 0x4140u), prmt(hi01, kMagic, 0x4342u)};
          const uint32_t c[4] = {prmt(lo23, kMagic, 0x4140u), prmt(lo23, kMagic, 0x4342u), prmt(hi23, kMagic, 0x4140u), prmt(hi23, kMagic, 0x4342u)};
          Mma16816<__half>::run(o[2 * wi], a, pb0, pb1);
          Mma16816<__half>::run(o[2 * wi + 1], c, pb0, pb1);
        }
        Mma16816<__half>::run(osum, ones, pb0, pb1);
      }
      __syncwarp();
    }
    cp_async_wait<0>();
#pragma unroll
    for (int off = 4; off < 32; off <<= 1) {
      l0 += __shfl_xor_sync(0xffffffffu, l0, off);
      l1 += __shfl_xor_sync(0xffffffffu, l1, off);
    }
    __syncthreads();                          // the ring is idle now
    float* sO = reinterpret_cast<float*>(smem);
    float* sML = sO + kQ8Warps * 8 * S::kMergeStride;
    {
      const float b0 = 1152.f * osum[0], b1 = 1152.f * osum[1];      // the bias of the V codes
      float* mine = sO + (warp * 8 + 2 * t) * S::kMergeStride + 16 * g;
#pragma unroll
      for (int j = 0; j < MT; ++j) {
        *reinterpret_cast<float2*>(mine + 2 * j) = make_float2(o[j][0] - b0, o[j][2] - b0);
        *reinterpret_cast<float2*>(mine + S::kMergeStride + 2 * j) = make_float2(o[j][1] - b1, o[j][3] - b1);
      }
      if (g == 0) {
        sML[(warp * 8 + 2 * t) * 2] = m0;
        sML[(warp * 8 + 2 * t) * 2 + 1] = l0;
        sML[(warp * 8 + 2 * t + 1) * 2] = m1;
        sML[(warp * 8 + 2 * t + 1) * 2 + 1] = l1;
      }
    }
    __syncthreads();
    merge_and_write<T, D, kQ8Warps>(p, sO, sML, S::kMergeStride, rows_valid, h0, b, di.item, di.nsplit, 8);
    __syncthreads();
    combine_if_last<T, D>(p, s_start, plan, b, b * ydim + kvh, h0, rows_valid, di.nsplit, &s_last);
  }
}

template <typename T>
int launch_decode_int8(const DecodeParams& p, cudaStream_t st) {
  // Heads on M where a group has more than eight of them (and no more than 16 per product).
  const size_t plan = static_cast<size_t>(p.batch + 1) * sizeof(int);
  const bool tok = p.group <= 8 && Int8TokSmem::kRingBytes + plan + 512 <= 227 * 1024;
  const size_t smem = (tok ? Int8TokSmem::kRingBytes : Int8Smem::kRingBytes) + plan;
  constexpr size_t kStaticSmem = 256;
  if (smem + kStaticSmem > 227 * 1024)
    return fail(MV_ERR_LIMIT, "paged_decode(int8): batch %d needs %zu bytes of shared memory", p.batch, smem);
  const auto kernel = tok ? paged_decode_int8_tok_kernel<T> : paged_decode_int8_kernel<T>;
  static size_t attr_bytes[2][64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || attr_bytes[tok][dev] < smem) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) {
      cudaGetLastError();
      return fail(MV_ERR_CUDA, "paged_decode(int8): cudaFuncSetAttribute(%zu): %s", smem, cudaGetErrorString(e));
    }
    if (dev >= 0 && dev < 64) attr_bytes[tok][dev] = smem;
  }
  kernel<<<decode_grid(p), (tok ? kQ8Warps : kDecWarps) * 32, smem, st>>>(p);
  return check_launch("paged_decode_int8_kernel");
}

template int launch_decode_int8<__half>(const DecodeParams&, cudaStream_t);
template int launch_decode_int8<__nv_bfloat16>(const DecodeParams&, cudaStream_t);

}  // namespace mv
