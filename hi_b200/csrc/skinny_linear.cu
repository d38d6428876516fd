// Dense products of few tokens: out[t, n] = sum_k x[t, k] w[n, k] (+ bias[n]), bfloat16 with float32 sums. A decode step's
// time is its weights' way out of HBM; the library's kernels for such shapes (clusters of split tiles fed by TMA) reach half
// the copy rate on the 4 to 64 MB matrices of a layer.
//
// A block takes 16 rows of w, its warps take turns over K in steps of 32: a lane loads 16 bytes of rows g and g + 8
// (four lanes: 64 neighbouring bytes) straight into mma.sync fragments, several steps ahead; the product's k order is the
// lanes' own (any order of k gives the same sum), so neither w nor x passes through shared memory. The warps' sums meet in
// shared memory at the end, in a fixed order. What bounds it: HBM for the large matrices, the launch and one trip to memory
// for the small ones. (32 rows a block were slower at every size but one.)
#include "api.h"
#include "common.cuh"
#include "mma.cuh"

namespace {

// NT: tiles of 8 tokens; U: steps in flight; THREADS / 32 warps share K
template <int NT, int U, int THREADS>
__global__ void __launch_bounds__(THREADS) skinny_linear_kernel(
    const __nv_bfloat16* __restrict__ x, long long x_ld, const __nv_bfloat16* __restrict__ w,
    const __nv_bfloat16* __restrict__ bias, void* __restrict__ out, int out_f32, int tokens, int n_out, int K) {
  constexpr int WARPS = THREADS / 32, TILE = 16 * NT * 8;
  __shared__ float red[WARPS * TILE];            // [warp][token][row]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q4 = lane & 3;
  const int row0 = blockIdx.x * 16;
  const __nv_bfloat16* wp[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) wp[i] = w + (size_t)min(row0 + g + 8 * i, n_out - 1) * K + q4 * 8;
  const __nv_bfloat16* xp[NT];
#pragma unroll
  for (int i = 0; i < NT; ++i) xp[i] = x + (size_t)min(g + 8 * i, tokens - 1) * x_ld + q4 * 8;
  float acc[NT][2][4];
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[n][e >> 2][e & 3] = 0.f;
  const int steps = (K + 31) / 32;
  uint4 wv[U][2], xv[U][NT];
  auto load = [&](int u, int s) {
    const bool in = s < steps && s * 32 + q4 * 8 < K;          // K is a multiple of 8
#pragma unroll
    for (int i = 0; i < 2; ++i)
      wv[u][i] = in ? __ldcs(reinterpret_cast<const uint4*>(wp[i] + (size_t)s * 32)) : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int i = 0; i < NT; ++i)
      xv[u][i] = in ? __ldg(reinterpret_cast<const uint4*>(xp[i] + (size_t)s * 32)) : make_uint4(0, 0, 0, 0);
  };
#pragma unroll
  for (int u = 0; u < U; ++u) load(u, warp + u * WARPS);
  for (int s0 = warp; s0 < steps; s0 += U * WARPS) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint4 lo = wv[u][0], hi = wv[u][1];
      const unsigned a0[4] = {lo.x, hi.x, lo.y, hi.y}, a1[4] = {lo.z, hi.z, lo.w, hi.w};
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        hb::mma_bf16(acc[n][0], a0, xv[u][n].x, xv[u][n].y);
        hb::mma_bf16(acc[n][1], a1, xv[u][n].z, xv[u][n].w);
      }
      load(u, s0 + (u + U) * WARPS);
    }
  }
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e)
      red[warp * TILE + (n * 8 + 2 * q4 + (e & 1)) * 16 + g + 8 * (e >> 1)] = acc[n][0][e] + acc[n][1][e];
  __syncthreads();
  for (int i = threadIdx.x; i < TILE; i += THREADS) {
    const int t = i / 16, row = row0 + i % 16;
    if (t >= tokens || row >= n_out) continue;
    float sum = 0.f;
#pragma unroll
    for (int k = 0; k < WARPS; ++k) sum += red[k * TILE + i];
    if (bias) sum += __bfloat162float(bias[row]);
    const size_t at = (size_t)t * n_out + row;
    if (out_f32) reinterpret_cast<float*>(out)[at] = sum;
    else reinterpret_cast<__nv_bfloat16*>(out)[at] = __float2bfloat16_rn(sum);
  }
}

template <int NT, int U, int THREADS>
int launch_skinny(const void* x, long long x_ld, const void* w, const void* bias, void* out, int out_f32, int tokens, int n_out,
                  int K, cudaStream_t stream) {
  skinny_linear_kernel<NT, U, THREADS><<<(n_out + 15) / 16, THREADS, 0, stream>>>(
      (const __nv_bfloat16*)x, x_ld, (const __nv_bfloat16*)w, (const __nv_bfloat16*)bias, out, out_f32, tokens, n_out, K);
  HB_LAUNCH_CHECK();
  return HB_OK;
}

}  // namespace

// x [tokens, K] with rows x_ld elements apart, w [n_out, K] contiguous, bias [n_out] or null, all bfloat16; out [tokens, n_out]
// contiguous, float32 or bfloat16. K and x_ld multiples of 8, x and w on 16 bytes, and sizes at which this kernel is the
// faster one (below); else HB_ERR_UNSUPPORTED.
extern "C" int hb_skinny_linear(const void* x, long long x_ld, const void* w, const void* bias, void* out, int out_dtype,
                                int tokens, int n_out, int K, cudaStream_t stream) {
  if (!x || !w || !out || tokens < 0 || n_out < 0 || K < 0 || (out_dtype != HB_DTYPE_F32 && out_dtype != HB_DTYPE_BF16))
    return HB_ERR_BAD_ARG;
  if (K == 0 || K % 8 || x_ld % 8 || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15))
    return HB_ERR_UNSUPPORTED;
  if (tokens == 0 || n_out == 0) return HB_OK;
  const int f = out_dtype == HB_DTYPE_F32;
  // As many warps a block as keep an SM's loads going with the blocks it gets; microseconds (w out of HBM, behind the norm that
  // makes x, in a graph), the library's first, for 1 and 8 tokens of n_out x K (2 and 8 where one token is the library's):
  //   512 threads, up to a block an SM: 2048 x 8192 22.0 / 9.7 and 19.7 / 9.7, 2048 x 2048 8.4 / 4.2 and 7.3 / 4.3, 2048 x 512 3.6 / 2.9
  //   and 4.0 / 2.7
  //   512 threads, up to two: 4096 x 8192 23.4 / 15.0 and 21.5 / 15.3, 4096 x 1024 6.1 / 4.0 and 5.8 / 4.1, but 3072 x 14336 19.6 / 21.2
  //   and 19.7 / 21.5: longer rows than 8,192 are the library's
  //   256 threads: 5120 x 8192 18.8 / 17.3 and 18.9 / 17.5, 6656 x 2048 7.1 / 6.1 and 6.8 / 6.3
  //   128 threads: 8192 x 2048 8.2 / 7.6 and 8.2 / 8.0, 8192 x 8192 25.0 / 23.6 and 25.0 / 24.0, but 8192 x 14336 38.7 / 37.8 and 38.1 / 39.3;
  //   14336 x 5120 27.0 / 24.7 and 25.7 / 25.1, 10240 x 4096 17.8 / 17.9 and 17.9 / 18.4, but 10240 x 8192 31.5 / 33.1 and 31.8 / 35.3,
  //   14336 x 1024 6.9 / 7.4 and 6.9 / 7.5;
  //   16384 x 5120 29.5 / 27.3 and 29.7 / 27.8, 32000 x 2048 24.3 / 20.6 and 25.1 / 21.4, 28672 x 4096 41.3 / 39.2 and 41.3 / 40.1, but
  //   16384 x 512 5.5 / 5.9 and 5.6 / 6.1, 28672 x 14336 123.0 / 124.6 and 123.8 / 128.0;
  //   128256 x 5120 192.0 / 184.9 and 191.2 / 187.6, but x 4096 156.2 / 164.3 and 158.9 / 167.2, x 8192 306.7 / 309.2 and 306.4 / 314.3
  // In a whole step the library's kernels can cost more than that: three layers' 8192 x 2048 products for 5 tokens, 13 us a step.
  // (the other way for 8 tokens of 7168 x 5120: 0.3 % of a decode step of eight Scout-sized layers)
  // For 9 to 16 tokens the library's wide kernels are the faster ones (8192 x 2048 8.4 / 9.9), its narrow ones are not
  // (2048 x 8192 13.2 / 10.9, 2048 x 2048 5.6 / 4.6, 64 x 2048 4.6 / 3.7).
  // One token of wide rows of 4,096 and more: even alone, and beside the expert kernels of a step of one request the library
  // is the faster one (Scout-sized, eight layers: 1.451 ms a step against 1.459). With 8 tokens it is the other way (routed
  // experts beside the shared one of 16384 x 5120 and 5120 x 8192: 304 us against 328 with the library). In decode steps of eight
  // Scout-sized layers: 2 requests 1,093 tokens/s with the kernel, 1,083 with the library alone, 4 requests 1,675 and 1,670; 8 requests
  // 2,330 and 2,345 on a card at its power limit, the same on one below it.
  const bool narrow = n_out <= 148 * 16;
  auto faster = [&] {
    if (narrow) return true;
    if (tokens > 8 || (tokens == 1 && n_out > 296 * 16 && K >= 4096)) return false;
    if (n_out <= 296 * 16) return K <= 8192;
    if (n_out <= 6656) return true;
    if (n_out <= 8192) return K <= 2048 || (tokens <= 4 && K <= 8192);
    if (n_out < 16384) return K > 1024 && K <= 5120;
    if (n_out <= 65536) return K >= 1024 && K <= 8192;
    return K >= 1024 && K < 8192 && (K <= 2048 || K >= 5120);
  };
  if (tokens > 16 || !faster()) return HB_ERR_UNSUPPORTED;
  if (tokens > 8)
    return K >= 4096 ? launch_skinny<2, 4, 512>(x, x_ld, w, bias, out, f, tokens, n_out, K, stream)
                     : launch_skinny<2, 2, 512>(x, x_ld, w, bias, out, f, tokens, n_out, K, stream);
  if (narrow && K >= 4096) return launch_skinny<1, 4, 512>(x, x_ld, w, bias, out, f, tokens, n_out, K, stream);
  if (n_out <= 296 * 16) return launch_skinny<1, 2, 512>(x, x_ld, w, bias, out, f, tokens, n_out, K, stream);
  if (n_out <= 6656) return launch_skinny<1, 4, 256>(x, x_ld, w, bias, out, f, tokens, n_out, K, stream);
  return launch_skinny<1, 8, 128>(x, x_ld, w, bias, out, f, tokens, n_out, K, stream);
}
