// out = x w^T for up to 16 rows of x (a decode step of as many sequences), fp16 or bf16, fp32 accumulation; or, gated, the SwiGLU
// of such a product whose weight is [gate; up].
//
// A step reads every weight once and does nothing else worth the time, so the weights go straight from memory to registers as
// 16-byte pieces of their rows, and the products are register MMAs: 16 tokens on the M side, 8 features on the N side, the
// reduction index permuted so that a thread's piece is its operand of two steps.  A CTA owns 8 kTiles features and its warps
// take 64-wide blocks of the reduction in turn, which puts a matrix of a few megabytes in flight at once; sums of the warps
// are added in order in shared memory.  Bound: memory, and the latency of one trip to it where the matrix is small.  us for 16 rows,
// bf16, and of the library's product: 1,024 features of 3,072 4.0 (8.3), 1,024 of 2,048 3.5 (6.5), 4,096 of 1,024 3.9 (4.8), gated
// 3,072 of 1,024 5.3 (7.5 with the activation), 4,096 of 12,288 21.4 (22.3).  The library is ahead where the features are more than
// CTAs are resident for (6,144 of 4,096: 15.1 against 13.0) or the reduction is very deep: layers/linear.py has the lines.
#include "mma.cuh"

namespace mv {

template <typename T, int kTiles, int kWarps, bool kGated>
__global__ void __launch_bounds__(kWarps * 32, kWarps == 16 ? 1 : 2)
few_rows_kernel(T* __restrict__ out, const T* __restrict__ x, int64_t x_stride, const T* __restrict__ w, int rows, int n, int k) {
  constexpr int kAll = kGated ? 2 * kTiles : kTiles, kAhead = kAll == 2 ? 2 : 4;      // blocks fetched together
  __shared__ float s_sum[kWarps][kAll][32][4];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int f0 = blockIdx.x * 8 * kTiles, blocks = k / 64;
  const bool two = rows > 8;                               // rows 8 .. 15
  const T* wrow[kAll];
  bool on[kAll];
#pragma unroll
  for (int j = 0; j < kAll; ++j) {
    const int f = f0 + (j % kTiles) * 8;
    on[j] = f < n;                                         // n is a multiple of eight
    wrow[j] = w + static_cast<int64_t>((on[j] ? f + g : 0) + (j / kTiles) * n) * k + 8 * t;
  }
  const T* xa = x + static_cast<int64_t>(g < rows ? g : 0) * x_stride + 8 * t;
  const T* xb = x + static_cast<int64_t>(g + 8 < rows ? g + 8 : 0) * x_stride + 8 * t;
  const bool has_a = g < rows, has_b = g + 8 < rows;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  float acc[kAll][4] = {};
  for (int b0 = warp; b0 < blocks; b0 += kWarps * kAhead) {
    uint4 wv[kAhead][kAll][2], av[kAhead][2], bv[kAhead][2];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int b = b0 + u * kWarps, at = b * 64;
      const bool ok = b < blocks;
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int j = 0; j < kAll; ++j) wv[u][j][h] = ok && on[j] ? ld_stream16(wrow[j] + at + h * 32) : zero;
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int b = b0 + u * kWarps, at = b * 64;
      const bool ok = b < blocks;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        av[u][h] = ok && has_a ? __ldg(reinterpret_cast<const uint4*>(xa + at + h * 32)) : zero;
        bv[u][h] = two && ok && has_b ? __ldg(reinterpret_cast<const uint4*>(xb + at + h * 32)) : zero;
      }
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t a0[4] = {av[u][h].x, bv[u][h].x, av[u][h].y, bv[u][h].y}, a1[4] = {av[u][h].z, bv[u][h].z, av[u][h].w, bv[u][h].w};
#pragma unroll
        for (int j = 0; j < kAll; ++j) {
          Mma16816<T>::run(acc[j], a0, wv[u][j][h].x, wv[u][j][h].y);
          Mma16816<T>::run(acc[j], a1, wv[u][j][h].z, wv[u][j][h].w);
        }
      }
  }
#pragma unroll
  for (int j = 0; j < kAll; ++j) *reinterpret_cast<float4*>(s_sum[warp][j][lane]) = make_float4(acc[j][0], acc[j][1], acc[j][2], acc[j][3]);
  __syncthreads();
  for (int i = threadIdx.x; i < rows * 8 * kTiles; i += kWarps * 32) {
    const int r = i / (8 * kTiles), c = i - r * 8 * kTiles, j = c >> 3, from = (r & 7) * 4 + ((c & 7) >> 1), e = (r >> 3) * 2 + (c & 1);
    if (f0 + c >= n) continue;
    float y = 0.f;
#pragma unroll
    for (int v = 0; v < kWarps; ++v) y += s_sum[v][j][from][e];
    if (kGated) {
      float up = 0.f;
#pragma unroll
      for (int v = 0; v < kWarps; ++v) up += s_sum[v][kAll - kTiles + j][from][e];
      y = Elem<T>::to_f(Elem<T>::from_f(y));               // both rounded, as the product alone would leave them
      up = Elem<T>::to_f(Elem<T>::from_f(up));
      y = __fdividef(y, 1.0f + __expf(-y)) * up;
    }
    out[static_cast<int64_t>(r) * n + f0 + c] = Elem<T>::from_f(y);
  }
}

template <typename T, bool kGated>
static int launch_few_rows(void* out, const void* x, int64_t x_stride, const void* w, int rows, int n, int k, cudaStream_t st) {
  auto go = [&](auto kernel, int tiles, int warps) {
    kernel<<<(n / 8 + tiles - 1) / tiles, warps * 32, 0, st>>>(static_cast<T*>(out), static_cast<const T*>(x), x_stride,
                                                              static_cast<const T*>(w), rows, n, k);
    return check_launch("few_rows");
  };
  // Up to eight features an SM: 16 warps on a CTA's reduction; two such CTAs: eight each; more: 16 features a CTA, which is one
  // round of two CTAs an SM up to 4,736 of them and reads x half as often.
  const int units = n / 8;
  if (units <= kNumSMs) return go(few_rows_kernel<T, 1, 16, kGated>, 1, 16);
  if constexpr (!kGated) {
    if (units > 2 * kNumSMs) return go(few_rows_kernel<T, 2, 8, false>, 2, 8);
  }
  return go(few_rows_kernel<T, 1, 8, kGated>, 1, 8);
}

}  // namespace mv

extern "C" int mv_few_rows(void* out, const void* x, int64_t x_stride, const void* w, int rows, int n, int k, int gated, int dtype,
                           void* stream) {
  using namespace mv;
  if (dtype != MV_F16 && dtype != MV_BF16) return fail(MV_ERR_DTYPE, "few_rows: dtype %d", dtype);
  if (rows < 0 || rows > 16 || n <= 0 || k <= 0 || n % 8 || k % 64 || x_stride < k)
    return fail(MV_ERR_SHAPE, "few_rows: %d rows, %d x %d (at most 16 rows, multiples of 8 and 64)", rows, n, k);
  if (rows == 0) return MV_OK;
  if (!out || !x || !w) return fail(MV_ERR_NULL, "few_rows: null pointer");
  if (!aligned16(x) || !aligned16(w) || x_stride % 8) return fail(MV_ERR_ALIGN, "few_rows: rows must start on 16-byte boundaries");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (dtype == MV_F16)
    return gated ? launch_few_rows<__half, true>(out, x, x_stride, w, rows, n, k, st) : launch_few_rows<__half, false>(out, x, x_stride, w, rows, n, k, st);
  return gated ? launch_few_rows<__nv_bfloat16, true>(out, x, x_stride, w, rows, n, k, st)
               : launch_few_rows<__nv_bfloat16, false>(out, x, x_stride, w, rows, n, k, st);
}
