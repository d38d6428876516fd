// The matrix memories' recurrences sixteen tokens at a time, for portions of prompts:
//   S <- diag(g_t) S + k_t u_t^T,   o_t = S^T q_t,   u_t = v_t (plain) or beta_t (v_t - (diag(g_t) S)^T k_t) (delta rule)
// With P_t = g_1 ... g_t (elementwise, from the chunk's start), R_s = g_(s+1) ... g_16 and S the chunk's first state:
//   u = T (v - (P k) S),     T = (I + diag(beta) A)^-1 diag(beta),  A_ts = sum_d k_t (g_(s+1) ... g_t) k_s,  s < t
//   o_t = (P_t q_t) S + sum_(s <= t) B_ts u_s,                      B_ts = sum_d q_t (g_(s+1) ... g_t) k_s
//   S <- diag(P_16) S + sum_s (R_s k_s) u_s^T
// Every factor is a product of decays, never a quotient: strong decays underflow to the zero they stand for.
//
// T meets what does not need the state ahead of it: u = T v - (T P k) S, so that one product and one sum over the rows of S
// lie between a chunk's state and its u.
//
//   chunk_prepare_kernel    everything that needs no state, of all chunks and heads side by side, once a head: T and B, and the
//     rows T P k, P q, R k as three bfloat16 pieces a float (see hb::split3) in the order in which the tensor cores read them.
//   chunk_recurrence_kernel per (request, head, 16 or 32 columns of S): chunk after chunk. NW warps own 16 rows of S each,
//     in registers as accumulator tiles; the sums over all rows are brought together in shared memory in a fixed order.
//     Two groups of four more warps take turns: they copy the prepared chunks in (bulk copies, three or four chunks ahead),
//     make T v, and add up and write the outputs, which nothing waits for.
// The prepared chunks (7.5 to 39.5 KB a head, by key size and rule) go through a scratch of bounded size: see slices_of.
//
// Measured (B200, one request of 2,048 tokens, 16 heads of 128 x 128; token after token / sixteen at a time with the rows
// prepared by every block for itself / now): delta rule 576 / 224 / 182 us (45 of them the preparation); mLSTM with 1,101 and
// 467 tokens beside single ones 328 / 133 / 107; 1,100 tokens of the rule without correction, 16 heads of 128 x 128 307 / 85 / 74,
// of 64 x 128 263 / 66 / 52. Over 900 steps of all three rules (4 to 40 heads of 16 x 16 to 128 x 128, 1 to 73 requests) 0.80 of
// the second. The preparation costs the same whatever the columns are, so steps of many requests and few columns pay for it: delta
// rule, 40 heads of 96 x 64, 16 requests of 100 tokens 222 -> 227; 20 heads of 128 x 16, 19 uneven ones of 8,084 in all 262 -> 351
// (ops._chunked_recurrence gives most of them to the other form). Error against 64 bits (2-norm) of the first: 7.0e-8 before and now.
// What bounds it: the chain from chunk to chunk, 1.1 us; 4,200 warp instructions of 16 warps that wait for one another (an empty
// chunk with its barriers takes 0.44 us; no part of it more than 0.1). Tried: twice the helpers (8 % slower: they share the
// issue slots), half as many at keys of 64 and less (1.1 to 1.4 times as long); P q S by two helper warps from pieces of S kept
// in shared memory (1.25 us a chunk); mbarriers in place of the named barriers (1.4); T v from memory a chunk ahead (1.4: the
// loads arrive too late); the products as float32 fma; two tf32 pieces a factor (error 1.1e-7).
//
// What is not finite in a token's inputs reaches that token's and later outputs of the request, never an earlier one (an
// infinite value or state comes out of the products as NaN, where token after token the sum could stay infinite).
#include <algorithm>

#include "api.h"
#include "common.cuh"
#include "mma.cuh"
#include "tc.cuh"

namespace {

constexpr int C = 16;       // tokens of a chunk
constexpr int SMS = 148;

__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int n) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory"); }

// x(at) + ... + x(at + N - 1), neighbours first
template <int N, typename F>
__device__ __forceinline__ float tree_sum(F x, int at = 0) {
  if constexpr (N == 1) return x(at);
  else return tree_sum<N - N / 2>(x, at) + tree_sum<N / 2>(x, at + N - N / 2);
}

// a + b; what its rounding loses is added to `lost` (Knuth's two-sum)
__device__ __forceinline__ float two_sum(float a, float b, float& lost) {
  const float s = a + b, bb = s - a;
  lost += (a - (s - bb)) + (b - bb);
  return s;
}

// A running product of decays with the rest that its roundings leave: a decay that all rows share would carry the same
// rounding error into all of them, and a sum over the rows would not average it away.
struct Product {
  float hi = 1.f, lo = 0.f;
  __device__ __forceinline__ void times(float g) {
    const float h = hi * g;
    lo = fmaf(lo, g, fmaf(hi, g, -h));
    hi = h;
  }
  __device__ __forceinline__ float of(float x) const { return fmaf(hi, x, lo * x); }
  // the product with x, and in `rest` what its rounding leaves
  __device__ __forceinline__ float of(float x, float& rest) const {
    const float y = hi * x;
    rest = fmaf(lo, x, fmaf(hi, x, -y));
    return y;
  }
};

struct ChunkArgs {
  const void* q;             // element (token, d) of key head h at q[token * q_ld + h * dim + d]; k the same
  const void* k;
  const void* v;             // v[token * v_ld + head * vdim + c]
  long long q_ld, v_ld;
  const float* decay;        // [N, heads * dim], or [N, heads]: one decay for all rows
  const float* take;         // [N, heads] or null: factor of v; with it column vdim of S has the value 1 * take
  const float* beta;         // [N, heads]
  float o_scale;             // factor of the outputs
  float* state;
  long long state_stride, head_floats;
  int row_step, col_step;    // strides of S in the state
  const int* cu_seqlens;
  const int* slots;
  unsigned char* images;     // [units of the launch, heads]: ChunkImage
  float* out;                // [N, heads * vdim]
  float* nq;                 // [N, heads] (with take): outputs of column vdim
  int* status;
  int n_seqs, heads, kvh, dim, vdim, cols;
  int share, shares;         // which share of every request's chunks, and how many there are
  int unit0, units;          // the launch's first unit of the share and how many
};

// A request's chunks in a launch: the first of them, how many, and the first one's place among the launch's units.
struct Span {
  int chunk, count, unit;
};

// Share i of a request of c chunks is the i-th run of ceil(c / shares) of them. A unit is a chunk of the share; those of request s
// start at cu[s] / (C shares) + s, which leaves every request room for ceil(its tokens / (C shares)).
__host__ __device__ inline Span span_of(const int* cu, int s, int share, int shares, int unit0, int units) {
  const int begin = cu[s], chunks = (cu[s + 1] - begin + C - 1) / C;
  int at = begin / C + s - unit0, chunk = 0, to = chunks;
  if (shares > 1) {                  // (the divisions and what hangs on them are 0.2 us of a short step)
    const int run = (chunks + shares - 1) / shares;
    at = begin / (C * shares) + s - unit0;
    chunk = share * run;
    to = run < chunks - chunk ? run : chunks - chunk;
  }
  const int from = at < 0 ? -at : 0;
  if (to > units - at) to = units - at;
  return {chunk + from, to - from, at + from};
}

// hb::split3 with the rests of the two floats in the last pieces
__device__ __forceinline__ void split_more(float2 v, float2 rest, uint32_t (&p)[3]) {
  p[0] = hb::pack_bf16_sat(v.x, v.y);
  v.x -= __uint_as_float(p[0] << 16);
  v.y -= __uint_as_float(p[0] & 0xffff0000u);
  p[1] = hb::pack_bf16(v.x, v.y);
  v.x -= __uint_as_float(p[1] << 16);
  v.y -= __uint_as_float(p[1] & 0xffff0000u);
  p[2] = hb::pack_bf16(v.x + rest.x, v.y + rest.y);
}

// What the recurrence reads of a chunk, as two blocks of memory that are copied into shared memory as they lie. The factors
// that meet the tensor cores are there as three bfloat16 pieces (see hb::split3) in the order of the mma.sync fragments: lane l
// of warp w has its 12 registers of 16 rows of S, [8-wide tile][piece][half], as three 16-byte words at [w][0 .. 2][l].
template <int NW, bool PLAIN>
struct ChunkImage {
  struct Factors {
    uint4 w[PLAIN ? 0 : NW][3][32];   // T P k (not with the plain rule)
    uint4 pq[NW][3][32];              // P q
    uint4 rk[NW][3][32];              // R k
    float2 full[16 * NW];             // the whole chunk's decay and the rest of its rounding
  } f;
  struct Matrices {
    float t[PLAIN ? 0 : C][20];       // T
    float b[C][20];                   // B, zero above the diagonal
  } m;
};

// grid (units, heads), 128 threads: warp w takes s = w, w + 4, w + 8, w + 12; a running row w_s = k_s g_(s+1) ... g_t
// meets k_t and q_t, eight sums a token, brought together by a halving butterfly. Then a thread per row d of S: the products
// of its decays with k and q, and its column of T P k.
template <typename T, int NW, bool SCALAR, bool PLAIN>
__global__ void __launch_bounds__(128) chunk_prepare_kernel(const ChunkArgs a) {
  using Image = ChunkImage<NW, PLAIN>;
  // row lengths that put a fragment's rows into different banks
  constexpr int DP = 16 * NW, DL = (DP + 31) / 32, W = DL * 32, LD = W + 8;
  __shared__ __align__(16) float ks[C][LD], qs[C][LD];
  __shared__ __align__(16) float gr[SCALAR ? W * 20 : (C * LD > W * 20 ? C * LD : W * 20)];    // [token][row] decays, then [row][token] R k
  __shared__ __align__(16) float A[C][C + 1], B[C][20], Ts[C][20], bet[C], g1[C];
  // what the roundings of T P k, P q and R k leave: with the delta rule it goes into their third pieces
  __shared__ __align__(4) __nv_bfloat16 kl[PLAIN ? 1 : C][LD], ql[PLAIN ? 1 : C][LD], rl[PLAIN ? 1 : W][C + 2];     // (read in pairs)
  __shared__ int where[2];
  const int unit = blockIdx.x, head = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) where[0] = -1;
  __syncthreads();
  for (int s = tid; s < a.n_seqs; s += 128) {
    const Span span = span_of(a.cu_seqlens, s, a.share, a.shares, a.unit0, a.units);
    const int c = unit - span.unit;
    if (c >= 0 && c < span.count) { where[0] = a.cu_seqlens[s] + (span.chunk + c) * C; where[1] = a.cu_seqlens[s + 1]; }
  }
  __syncthreads();
  const int t0 = where[0];
  if (t0 < 0) return;
  const int count = min(C, where[1] - t0);
  const int kvhead = head / (a.heads / a.kvh);
  Image& img = reinterpret_cast<Image*>(a.images)[(size_t)unit * a.heads + head];
  {
    // a column of the chunk a thread (or every STEP-th token of one)
    constexpr int STEP = 128 / W > 0 ? 128 / W : 1;
    const int d = tid % W, from = tid / W;
    const T* q = reinterpret_cast<const T*>(a.q) + (size_t)(t0 + from) * a.q_ld + (size_t)kvhead * a.dim + d;
    const T* k = reinterpret_cast<const T*>(a.k) + (size_t)(t0 + from) * a.q_ld + (size_t)kvhead * a.dim + d;
    const float* g = a.decay + (size_t)(t0 + from) * a.heads * a.dim + (size_t)head * a.dim + d;
    if (from < STEP) {
#pragma unroll
      for (int t = from; t < C; t += STEP, q += STEP * a.q_ld, k += STEP * a.q_ld, g += STEP * (size_t)a.heads * a.dim) {
        const bool in = t < count && d < a.dim;
        ks[t][d] = in ? hb::to_f32(*k) : 0.f;
        qs[t][d] = in ? hb::to_f32(*q) : 0.f;
        if (!SCALAR) gr[t * LD + d] = in ? *g : 1.f;
      }
    }
  }
  if (tid < C) {
    if (SCALAR) g1[tid] = tid < count ? a.decay[(size_t)(t0 + tid) * a.heads + head] : 1.f;
    bet[tid] = (!PLAIN && tid < count) ? a.beta[(size_t)(t0 + tid) * a.heads + head] : 0.f;
  }
  __syncthreads();
  // lane: rows lane * DL ..; the warp's running rows start one by one, s = warp + 4 j in the tokens 4 j .. 4 j + 3
  float w[4][DL], rest[4][DL];
#pragma unroll
  for (int tb = 0; tb < 4; ++tb) {
#pragma unroll
    for (int tt = 0; tt < 4; ++tt) {
      const int t = 4 * tb + tt;
      if (tb == 0 && tt < warp) continue;
      float kt[DL], qt[DL], gt[DL];
#pragma unroll
      for (int i = 0; i < DL; ++i) {
        kt[i] = ks[t][lane * DL + i];
        qt[i] = qs[t][lane * DL + i];
        gt[i] = SCALAR ? g1[t] : gr[SCALAR ? 0 : t * LD + lane * DL + i];
      }
      float v[8];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        v[j] = v[4 + j] = 0.f;
        if (j > tb) continue;
        if (j == tb && tt < warp) continue;
        if (j == tb && tt == warp) {
#pragma unroll
          for (int i = 0; i < DL; ++i) { w[j][i] = kt[i]; rest[j][i] = 0.f; v[j] = fmaf(kt[i], qt[i], v[j]); }
        } else {
#pragma unroll
          for (int i = 0; i < DL; ++i) {
            const float h = w[j][i] * gt[i];                      // with the rest of its roundings, as Product
            rest[j][i] = fmaf(rest[j][i], gt[i], fmaf(w[j][i], gt[i], -h));
            w[j][i] = h;
            const float x = h + rest[j][i];
            if (!PLAIN) v[4 + j] = fmaf(x, kt[i], v[4 + j]);
            v[j] = fmaf(x, qt[i], v[j]);
          }
        }
      }
      constexpr int LIVE = PLAIN ? 4 : 8;
      // halve the values a lane holds while the lanes that share them double
      int mine = 0;
#pragma unroll
      for (int half = LIVE / 2, off = 16; half >= 1; half >>= 1, off >>= 1) {
        const bool up = lane & off;
#pragma unroll
        for (int i = 0; i < half; ++i) {
          const float give = up ? v[i] : v[i + half], keep = up ? v[i + half] : v[i];
          v[i] = keep + __shfl_xor_sync(0xffffffffu, give, off);
        }
        mine += up ? half : 0;
      }
#pragma unroll
      for (int off = 16 / LIVE; off >= 1; off >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
      if ((lane & (32 / LIVE - 1)) == 0) {
        const int s = warp + 4 * (mine & 3);
        if (mine < 4) B[t][s] = v[0];
        else A[t][s] = v[0];
      }
    }
  }
  const int d = tid;
  float gt[C], pk[C], pl[C];
  if (d < W) {
#pragma unroll
    for (int t = 0; t < C; ++t) gt[t] = SCALAR ? g1[t] : gr[SCALAR ? 0 : t * LD + d];
  }
  __syncthreads();
  for (int e = tid; e < C * C; e += 128) img.m.b[e / C][e % C] = (e % C) <= e / C ? B[e / C][e % C] : 0.f;
  if (!PLAIN && tid < C) {
    // column tid of T by forward substitution
    float x[C];
#pragma unroll
    for (int t = 0; t < C; ++t) {
      float s0 = t == tid ? 1.f : 0.f, s1 = 0.f;
#pragma unroll
      for (int s = 0; s < t; ++s) {
        if (s & 1) s1 = fmaf(-A[t][s], x[s], s1);
        else s0 = fmaf(-A[t][s], x[s], s0);
      }
      x[t] = t < tid ? 0.f : bet[t] * (s0 + s1);
      Ts[t][tid] = x[t];
      img.m.t[t][tid] = x[t];
    }
  }
  if (d < W) {
    Product p;
#pragma unroll
    for (int t = 0; t < C; ++t) {
      p.times(gt[t]);
      if constexpr (PLAIN) {
        qs[t][d] = p.of(qs[t][d]);
      } else {
        float rest;
        pk[t] = p.of(ks[t][d], pl[t]);
        qs[t][d] = p.of(qs[t][d], rest);
        ql[t][d] = __float2bfloat16_rn(rest);
      }
    }
    if (d < DP) img.f.full[d] = make_float2(p.hi, p.lo);
    Product r;
#pragma unroll
    for (int t = C - 4; t >= 0; t -= 4) {
      float x[4];
#pragma unroll
      for (int i = 3; i >= 0; --i) {
        if constexpr (PLAIN) {
          x[i] = r.of(ks[t + i][d]);
        } else {
          float rest;
          x[i] = r.of(ks[t + i][d], rest);
          rl[d][t + i] = __float2bfloat16_rn(rest);
        }
        r.times(gt[t + i]);
      }
      *reinterpret_cast<float4*>(&gr[d * 20 + t]) = make_float4(x[0], x[1], x[2], x[3]);
    }
  }
  __syncthreads();
  if (!PLAIN) {
    if (d < W) {
#pragma unroll
      for (int t = 0; t < C; ++t) {
        float tr[C], w0 = 0.f, w1 = 0.f;
#pragma unroll
        for (int s = 0; s <= t; s += 4) *reinterpret_cast<float4*>(&tr[s]) = *reinterpret_cast<const float4*>(&Ts[t][s]);
        // a later token's rows never reach an earlier one, whatever they hold
#pragma unroll
        for (int s = 0; s < t; ++s) {
          if (s & 1) w1 = fmaf(tr[s], pk[s], w1);
          else w0 = fmaf(tr[s], pk[s], w0);
        }
        // the token's own row, the largest term, comes last
        const float big = tr[t] * pk[t];
        float rest = fmaf(tr[t], pl[t], fmaf(tr[t], pk[t], -big));
        ks[t][d] = two_sum(big, w0 + w1, rest);
        kl[t][d] = __float2bfloat16_rn(rest);
      }
    }
    __syncthreads();
  }
  // the fragments: the mma's k is the row of S for T P k and P q (n the token), the token for R k (n the row)
  for (int f = tid; f < NW * 32; f += 128) {
    const int fw = f >> 5, g = (f & 31) >> 2, q4 = f & 3;
    auto put = [&](uint4 (&to)[3][32], auto of, auto rest) {
      uint32_t r[12];
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float2 v = *reinterpret_cast<const float2*>(of(n, h));
          uint32_t p[3];
          if constexpr (PLAIN) hb::split3(v.x, v.y, p);
          else split_more(v, __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(rest(n, h))), p);
#pragma unroll
          for (int x = 0; x < 3; ++x) r[n * 6 + x * 2 + h] = p[x];
        }
#pragma unroll
      for (int j = 0; j < 3; ++j) to[j][f & 31] = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
    };
    auto token_row = [&](auto* rows) { return [=](int n, int h) { return &rows[8 * n + g][fw * 16 + 8 * h + 2 * q4]; }; };
    auto row_token = [&](auto* rows, int ld) { return [=](int n, int h) { return &rows[(fw * 16 + 8 * n + g) * ld + 8 * h + 2 * q4]; }; };
    if constexpr (!PLAIN) put(img.f.w[fw], token_row(ks), token_row(kl));
    put(img.f.pq[fw], token_row(qs), token_row(ql));
    put(img.f.rk[fw], row_token(gr, 20), row_token(&rl[0][0], C + 2));
  }
}

// the pieces of hb::split3, of one float
__device__ __forceinline__ void put_pieces(__nv_bfloat16* at, int step, float x) {
  unsigned short first;
  asm("cvt.rn.satfinite.bf16.f32 %0, %1;" : "=h"(first) : "f"(x));
  __nv_bfloat16 h = __ushort_as_bfloat16(first);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    at[i * step] = h;
    x -= __bfloat162float(h);
    h = __float2bfloat16_rn(x);
  }
}
__device__ __forceinline__ void mma16(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
__device__ __forceinline__ void mma8(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(b));
}
// Two products [16, 16] times [16, 8], side by side: the small ones among themselves, the large one in two halves by
// itself, then their sum: the tensor core cuts a sum where it does not fit, and is so kept from cutting more than a
// product's last bits.
__device__ __forceinline__ void mma3(float (&out)[2][4], const uint32_t (&a)[3][4], const uint32_t (&b)[2][3][2]) {
  constexpr int from[5][2] = {{2, 0}, {0, 2}, {1, 1}, {1, 0}, {0, 1}};
  float lo[2][4], half[2][4];
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) lo[n][e] = half[n][e] = out[n][e] = 0.f;
#pragma unroll
  for (int n = 0; n < 2; ++n) mma8(out[n], a[0][0], a[0][1], b[n][0][0]);
#pragma unroll
  for (int n = 0; n < 2; ++n) mma8(half[n], a[0][2], a[0][3], b[n][0][1]);
#pragma unroll
  for (int p = 0; p < 5; ++p)
#pragma unroll
    for (int n = 0; n < 2; ++n) mma16(lo[n], a[from[p][0]], b[n][from[p][1]]);
#pragma unroll
  for (int n = 0; n < 2; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) out[n][e] = (out[n][e] + half[n][e]) + lo[n][e];
}

// the 12 registers of a fragment of 16 rows of S (ChunkImage)
__device__ __forceinline__ void load_fragment(uint32_t (&r)[2][3][2], const uint4 (&from)[3][32], int lane) {
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const uint4 v = from[j][lane];
    const uint32_t x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) r[(4 * j + i) / 6][(4 * j + i) % 6 / 2][i & 1] = x[i];
  }
}

template <int NW, int CT, bool PLAIN>
struct ChunkSmem {
  // row lengths that put a fragment's rows into different banks
  static constexpr int CG = 16 * CT, STAGES = CT == 1 ? 4 : 3, RING = 4, HELP = 128;
  struct All {
    typename ChunkImage<NW, PLAIN>::Factors factors[STAGES];
    typename ChunkImage<NW, PLAIN>::Matrices matrices[RING];
    float part_w[PLAIN ? 0 : NW][CG][24];      // [column][token]: a warp's share of (T P k S)^T
    float part_q[2][NW][C][CG + 4];            // [token][column]: a warp's share of P q S
    float2 u0[PLAIN ? 0 : RING][CG][20];       // [column][token]: T v and the rest of its rounding
    float v[PLAIN ? 0 : 2][CG][20];            // [column][token]
    float u[PLAIN ? RING : 2][CG][20];         // [column][token]
    __nv_bfloat16 up[PLAIN ? RING : 1][3][CG][24];    // the pieces of u
    uint64_t full[STAGES], full_m[RING];
    int gave_up;                               // a wait for a copy
  };
};

template <typename T, int NW, int CT, bool PLAIN>
__global__ void __launch_bounds__(32 * NW + 2 * ChunkSmem<NW, CT, PLAIN>::HELP) chunk_recurrence_kernel(const ChunkArgs a) {
  using Smem = ChunkSmem<NW, CT, PLAIN>;
  using Image = ChunkImage<NW, PLAIN>;
  constexpr int CG = Smem::CG, COMP = 32 * NW, HELP = Smem::HELP, STAGES = Smem::STAGES, RING = Smem::RING;
  // barriers: (+ chunk & 3) T v or the pieces of v there; (+ chunk & 1) u and the shares of P q S there, the factors read;
  // the outputs written; among a helper group; among the COMP threads
  constexpr int FULL = 1, DONE = 5, FREED = 7, GROUP = 9, PEER = 11;
  extern __shared__ __align__(128) unsigned char raw[];
  typename Smem::All& sm = *reinterpret_cast<typename Smem::All*>(raw);
  const int head = blockIdx.y, seq = blockIdx.z, col0 = blockIdx.x * CG;
  // (Blocks of 32 columns read it from shared memory: worked out by every thread it cost the delta rule 1 to 3 % there, 96.6 us where
  // these are 93.9 for 527 tokens of 32 heads of 128 x 128; blocks of 16 columns are the faster ones without, 181.9 and 186.7 for 2,048 of 16.)
  Span span;
  if constexpr (CT == 2) {
    __shared__ Span once;
    if (threadIdx.x == 0) once = span_of(a.cu_seqlens, seq, a.share, a.shares, a.unit0, a.units);
    __syncthreads();
    span = once;
  } else {
    span = span_of(a.cu_seqlens, seq, a.share, a.shares, a.unit0, a.units);
  }
  const int first = a.cu_seqlens[seq] + span.chunk * C, last = a.cu_seqlens[seq + 1], chunks = span.count;
  if (chunks <= 0) return;
  const int tid = threadIdx.x;
  if (tid == 0) {
#pragma unroll
    for (int i = 0; i < STAGES; ++i) tc::mbar_init(&sm.full[i], 1);
#pragma unroll
    for (int i = 0; i < RING; ++i) tc::mbar_init(&sm.full_m[i], 1);
    sm.gave_up = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  const Image* images = reinterpret_cast<const Image*>(a.images) + (size_t)span.unit * a.heads + head;
  bool ok = true;
  auto there = [&](uint64_t* full, int use) {          // a copy has arrived
    if (ok && !tc::mbar_wait(full, use & 1)) {
      atomicExch(a.status, 41);
      sm.gave_up = 1;
      tc::mbar_wait(full, use & 1);                   // once more, so that the copy does not outlive the block
      ok = false;                                     // go on without waiting: every barrier of the block is still met
    }
  };

  if (tid < COMP) {
    const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, q4 = lane & 3;
    // S^T as accumulator tiles [16 columns][8 rows]: s[m][n][0, 1] = column 16 m + g, rows 8 n + 2 q4 and the next;
    // [2, 3] = column 16 m + g + 8
    float* S = a.state + (size_t)a.slots[seq] * a.state_stride + (size_t)head * a.head_floats;
    float s[CT][2][4];
    auto at = [&](int m, int n, int e, bool& in) {
      const int d = warp * 16 + n * 8 + 2 * q4 + (e & 1), col = col0 + 16 * m + g + (e >> 1) * 8;
      in = d < a.dim && col < a.cols;
      return (size_t)d * a.row_step + (size_t)col * a.col_step;
    };
#pragma unroll
    for (int m = 0; m < CT; ++m)
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          bool in;
          const size_t i = at(m, n, e, in);
          s[m][n][e] = in ? S[i] : 0.f;
        }
    // sums over all warps: token lane & 15 of one of two columns two apart (different banks)
    constexpr int EN = (CG / 2 + NW - 1) / NW;
    const int t = lane & 15;
    auto pair_column = [&](int p) { return (p & 1) + 2 * (lane >> 4) + (p >> 1) * 4; };
    for (int i = 0; i < chunks; ++i) {
      const int b = i & 1, ring = i & 3;
      // the tiles of S^T are the A operand as they lie in the accumulators
      uint32_t sp[CT][3][4];
#pragma unroll
      for (int m = 0; m < CT; ++m)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          uint32_t p[3];
          hb::split3(s[m][e >> 1][2 * (e & 1)], s[m][e >> 1][2 * (e & 1) + 1], p);
#pragma unroll
          for (int x = 0; x < 3; ++x) sp[m][x][e] = p[x];
        }
      there(&sm.full[i % STAGES], i / STAGES);
      const auto& img = sm.factors[i % STAGES];
      uint32_t fr[2][3][2], qf[2][3][2];
      if constexpr (!PLAIN) {
        load_fragment(fr, img.w[warp], lane);
#pragma unroll
        for (int m = 0; m < CT; ++m) {
          float z[2][4];
          mma3(z, sp[m], fr);
#pragma unroll
          for (int n = 0; n < 2; ++n) {
            *reinterpret_cast<float2*>(&sm.part_w[warp][16 * m + g][8 * n + 2 * q4]) = make_float2(z[n][0], z[n][1]);
            *reinterpret_cast<float2*>(&sm.part_w[warp][16 * m + g + 8][8 * n + 2 * q4]) = make_float2(z[n][2], z[n][3]);
          }
        }
      }
      load_fragment(qf, img.pq[warp], lane);
      bar_sync(FULL + ring, COMP + HELP);
      if (i >= 2) bar_sync(FREED + b, COMP + HELP);
      auto outputs = [&]() {                     // the warp's share of P q S
#pragma unroll
        for (int m = 0; m < CT; ++m) {
          float z[2][4];
          mma3(z, sp[m], qf);
#pragma unroll
          for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) sm.part_q[b][warp][8 * n + 2 * q4 + (e & 1)][16 * m + g + (e >> 1) * 8] = z[n][e];
        }
      };
      if constexpr (!PLAIN) {
        const int count = min(C, last - first - i * C);
        bar_sync(PEER, COMP);
        float z[EN];
        float2 u0[EN];
#pragma unroll
        for (int j = 0; j < EN; ++j) {
          const int p = warp + j * NW, c = pair_column(p);
          if (p >= CG / 2) break;
          z[j] = tree_sum<NW>([&](int w) { return sm.part_w[w][c][t]; });
          u0[j] = sm.u0[ring][c][t];
        }
        outputs();               // nothing waits for them, they fill the time
#pragma unroll
        for (int j = 0; j < EN; ++j) {
          const int p = warp + j * NW, c = pair_column(p);
          if (p >= CG / 2) break;
          const float u = t < count ? (u0[j].x - z[j]) + u0[j].y : 0.f;
          sm.u[b][c][t] = u;
          put_pieces(&sm.up[0][0][c][t], CG * 24, u);
        }
        bar_sync(PEER, COMP);
      } else {
        outputs();
      }
      load_fragment(fr, img.rk[warp], lane);
      float4 full[2];
#pragma unroll
      for (int n = 0; n < 2; ++n) full[n] = *reinterpret_cast<const float4*>(&img.full[warp * 16 + 8 * n + 2 * q4]);
      uint32_t up[CT][3][4];
#pragma unroll
      for (int m = 0; m < CT; ++m)
#pragma unroll
        for (int x = 0; x < 3; ++x)
          hb::ldmatrix_x4(up[m][x], &sm.up[PLAIN ? ring : 0][x][16 * m + (lane & 15)][(lane >> 4) * 8]);
      bar_arrive(DONE + b, COMP + HELP);
#pragma unroll
      for (int m = 0; m < CT; ++m) {
        float z[2][4];
        mma3(z, up[m], fr);
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            s[m][n][e] = fmaf(s[m][n][e], (e & 1) ? full[n].z : full[n].x,
                              fmaf(s[m][n][e], (e & 1) ? full[n].w : full[n].y, z[n][e]));
      }
    }
    // Where a wait was given up, no copy is under way when the block ends: the last ones into each place are waited for, again with
    // the limit. (Behind the helpers' loop, or behind the states below, the same lines cost the delta rule 2 to 4 %.)
    if (*reinterpret_cast<volatile int*>(&sm.gave_up))
      for (int i = max(0, chunks - RING); i < chunks; ++i) {
        if (i >= chunks - STAGES) tc::mbar_wait(&sm.full[i % STAGES], (i / STAGES) & 1);
        tc::mbar_wait(&sm.full_m[i % RING], (i / RING) & 1);
      }
#pragma unroll
    for (int m = 0; m < CT; ++m)
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          bool in;
          const size_t i = at(m, n, e, in);
          if (in) S[i] = s[m][n][e];
        }
    return;
  }

  // ---- two groups of helpers that take turns: group b brings the images of the chunks of parity b in, makes T v of the
  // next one while the other threads are at this one, and writes this one's outputs
  const int b = (tid - COMP) / HELP, h = (tid - COMP) % HELP, hw = h >> 5, lane = h & 31;
  const T* v = reinterpret_cast<const T*>(a.v) + (size_t)head * a.vdim;
  constexpr int VN = (C * CG + HELP - 1) / HELP;
  T vr[VN];
  float fr[VN];
  auto copy = [&](void* dst, const void* src, uint32_t bytes, uint64_t* full) {      // one thread
    tc::mbar_expect_tx(full, bytes);
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(tc::smem_u32(dst)), "l"(src), "r"(bytes), "r"(tc::smem_u32(full)) : "memory");
  };
  auto bring_factors = [&](int i) {
    copy(&sm.factors[i % STAGES], &images[(size_t)i * a.heads].f, sizeof(sm.factors[0]), &sm.full[i % STAGES]);
  };
  auto bring_matrices = [&](int i) {
    copy(&sm.matrices[i % RING], &images[(size_t)i * a.heads].m, sizeof(sm.matrices[0]), &sm.full_m[i % RING]);
  };
  auto load = [&](int i) {               // nothing is computed from the values here, so nothing waits for them
    const int t0 = first + i * C, count = min(C, last - t0);
#pragma unroll
    for (int j = 0; j < VN; ++j) {
      const int e = h + j * HELP, t = e / CG, col = col0 + e % CG;
      const bool in = t < count && col < a.cols;
      vr[j] = in && col < a.vdim ? v[(size_t)(t0 + t) * a.v_ld + col] : hb::from_f32<T>(in ? 1.f : 0.f);
      fr[j] = in && a.take ? a.take[(size_t)(t0 + t) * a.heads + head] : 1.f;
    }
  };
  auto values = [&](int i) {             // of chunk i, from the registers
    const int ring = i & 3;
#pragma unroll
    for (int j = 0; j < VN; ++j) {
      const int e = h + j * HELP;
      if (e >= C * CG) break;
      const float x = hb::to_f32(vr[j]) * fr[j];
      if (PLAIN) {
        sm.u[ring][e % CG][e / CG] = x;
        put_pieces(&sm.up[ring][0][e % CG][e / CG], CG * 24, x);
      } else {
        sm.v[b][e % CG][e / CG] = x;
      }
    }
    if constexpr (!PLAIN) {
      there(&sm.full_m[ring], i / RING);
      const auto& img = sm.matrices[ring];
      bar_sync(GROUP + b, HELP);
      const int t = lane & 15;
      float4 tr[C / 4];
#pragma unroll
      for (int r = 0; r < C / 4; ++r) tr[r] = *reinterpret_cast<const float4*>(&img.t[t][4 * r]);
      const float own = img.t[t][t];
#pragma unroll
      for (int j = 0; j < VN; ++j) {
        const int p = hw + j * (HELP / 32), c = (p & 1) + 2 * (lane >> 4) + (p >> 1) * 4;
        if (p >= CG / 2) break;
        float u0 = 0.f, u1 = 0.f;
#pragma unroll
        for (int r = 0; r < C; r += 4) {
          const float4 x = *reinterpret_cast<const float4*>(&sm.v[b][c][r]);
          // a later token's rows never reach an earlier one, whatever they hold
          if (r < t) u0 = fmaf(tr[r / 4].x, x.x, u0);
          if (r + 1 < t) u1 = fmaf(tr[r / 4].y, x.y, u1);
          if (r + 2 < t) u0 = fmaf(tr[r / 4].z, x.z, u0);
          if (r + 3 < t) u1 = fmaf(tr[r / 4].w, x.w, u1);
        }
        // the token's own row, the largest term, comes last, and what is rounded off is kept: u rounds once
        const float vt = sm.v[b][c][t], big = own * vt;
        float lost = fmaf(own, vt, -big);
        const float sum = two_sum(big, u0 + u1, lost);
        sm.u0[ring][c][t] = make_float2(sum, lost);
      }
    }
    bar_arrive(FULL + ring, COMP + HELP);
  };
  if (h == 0) {
    for (int i = b; i < min(chunks, RING); i += 2) {
      bring_matrices(i);
      if (i < STAGES) bring_factors(i);
    }
  }
  if (b < chunks) { load(b); values(b); }
  bar_sync(GROUP + b, HELP);
  if (b + 2 < chunks) load(b + 2);
  for (int i = b; i < chunks; i += 2) {
    const int t0 = first + i * C, count = min(C, last - t0), ring = i & 3;
    if (i + 2 < chunks) values(i + 2);
    if (i + 4 < chunks) load(i + 4);
    bar_sync(DONE + b, COMP + HELP);
    if (PLAIN) there(&sm.full_m[ring], i / RING);
    const auto& img = sm.matrices[ring];
#pragma unroll
    for (int j = 0; j < VN; ++j) {
      const int e = h + j * HELP, t = e / CG, c = e % CG, col = col0 + c;
      if (e >= C * CG) break;
      float y0 = 0.f, y1 = 0.f;
#pragma unroll
      for (int x = 0; x < C; x += 4) {
        const float4 br = *reinterpret_cast<const float4*>(&img.b[t][x]);
        const float4 u = *reinterpret_cast<const float4*>(&sm.u[PLAIN ? ring : b][c][x]);
        if (x <= t) y0 = fmaf(br.x, u.x, y0);
        if (x + 1 <= t) y1 = fmaf(br.y, u.y, y1);
        if (x + 2 <= t) y0 = fmaf(br.z, u.z, y0);
        if (x + 3 <= t) y1 = fmaf(br.w, u.w, y1);
      }
      // the last three sums with what they round off, so that the output rounds once
      auto z = [&](int w) { return sm.part_q[b][w][t][c]; };
      float lost = 0.f;
      const float y = two_sum(y0, y1, lost);
      const float o = (two_sum(two_sum(tree_sum<NW - NW / 2>(z), tree_sum<NW / 2>(z, NW - NW / 2), lost), y, lost) + lost) * a.o_scale;
      if (t < count && col < a.vdim) a.out[(size_t)(t0 + t) * a.heads * a.vdim + (size_t)head * a.vdim + col] = o;
      else if (t < count && col < a.cols) a.nq[(size_t)(t0 + t) * a.heads + head] = o;
    }
    bar_sync(GROUP + b, HELP);                        // the group has read the matrices and the values
    if (h == 0) {
      if (i + STAGES < chunks) bring_factors(i + STAGES);
      if (i + RING < chunks) bring_matrices(i + RING);
    }
    if (i + 2 < chunks) bar_arrive(FREED + b, COMP + HELP);
  }
}

template <typename T, int NW, int CT, bool PLAIN>
int launch_columns(const ChunkArgs& a, cudaStream_t stream) {
  const size_t smem = sizeof(typename ChunkSmem<NW, CT, PLAIN>::All);
  cudaError_t e = cudaFuncSetAttribute(chunk_recurrence_kernel<T, NW, CT, PLAIN>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  chunk_recurrence_kernel<T, NW, CT, PLAIN>
      <<<dim3((a.cols + 16 * CT - 1) / (16 * CT), a.heads, a.n_seqs), 32 * NW + 2 * ChunkSmem<NW, CT, PLAIN>::HELP, smem, stream>>>(a);
  HB_LAUNCH_CHECK();
  return HB_OK;
}

// How a step's chunks go through `most_bytes` of scratch: every request's in `shares` runs, and the units of a share `units` at a
// time, launch after launch (the states go through memory).
// Shares keep the requests side by side, so the chain is the longest request's however many launches there are. Slices of
// 128 MB that took the chunks in order ran the requests one after another: two of 4,096 tokens (delta rule, 16 heads of
// 128 x 128) 1,037 us, 660 by shares; four of 2,048, 8 heads, 524 and 335. A launch more costs about 25 us, so the scratch is not
// small (those in 256 / 64 / 32 MB: 654 / 687 / 761 and 327 / 343 / 362).
// In order is the better way where a slice's blocks keep the SMs busy four times as long as the longest chain (64 requests of 100
// tokens, 64 heads: 2,550 us, by shares of 128 MB 2,896; with "once as long" instead of four times, four requests of 2,048 and
// 16 heads are 841 instead of 659), and where the requests' room for a partial chunk each would fill most of the scratch.
struct Slices {
  int shares, units;
};
inline Slices slices_of(int n_tokens, int n_seqs, int longest, int heads, int cols, size_t image_bytes, long long most_bytes) {
  const long long images = most_bytes / (long long)image_bytes;
  const int all = n_tokens / C + n_seqs, fit = (int)std::min<long long>(std::max(images / heads, 1LL), all), room = fit - n_seqs;
  if (all == fit) return {1, all};
  if (longest <= 0 || longest > n_tokens) longest = n_tokens;
  const bool full = 4LL * ((longest + C - 1) / C) * SMS <= images * ((cols + 31) / 32);
  if (full || 4 * (long long)room < fit) return {1, fit};
  const int shares = (n_tokens / C + room - 1) / room;
  return {shares, n_tokens / (C * shares) + n_seqs};
}

// Whether blocks of 32 columns take less time than blocks of 16: a chunk of theirs takes 1.6 times as long (with 1.4 or 1.9 in its
// place 300 steps took 1.006 or 1.001 of the time, single ones up to 1.1 or 1.3). A step's time is that of all blocks' chunks over
// all SMs or, if that is more, the rounds of the long requests' blocks, each a chain of the longest; a block's start and end count
// as four chunks. (mLSTM, 16 heads, two requests of 4,096 tokens: 129 columns are 160 blocks of 32 and two rounds, 723 us, or 288
// of 16 and two rounds, 498; 40 heads without correction, one of 304 tokens and 70 of one: 500 us in blocks of 16, 362 of 32.)
inline bool wide_blocks(int n_tokens, int n_seqs, int longest, int heads, int cols) {
  if (longest <= 0 || longest > n_tokens) longest = (n_tokens + n_seqs - 1) / n_seqs;
  const long long chain = (longest + C - 1) / C + 4, work = n_tokens / C + 5LL * n_seqs;
  const int requests = std::min(n_seqs, (2 * n_tokens + longest) / (2 * longest));
  auto steps = [&](int width) {
    const long long blocks = (long long)heads * ((cols + width - 1) / width);
    return std::max(work * blocks / SMS, (requests * blocks + SMS - 1) / SMS * chain);
  };
  return 10 * steps(16) > 16 * steps(32);
}

template <typename T, int NW, bool SCALAR, bool PLAIN>
int launch_chunked(ChunkArgs a, int n_tokens, int longest, long long most_bytes, cudaStream_t stream) {
  const Slices slices = slices_of(n_tokens, a.n_seqs, longest, a.heads, a.cols, sizeof(ChunkImage<NW, PLAIN>), most_bytes);
  a.shares = slices.shares;
  const bool wide = wide_blocks(n_tokens, a.n_seqs, longest, a.heads, a.cols);
  const int units = n_tokens / (C * a.shares) + a.n_seqs;
  for (a.share = 0; a.share < a.shares; ++a.share)
    for (a.unit0 = 0; a.unit0 < units; a.unit0 += slices.units) {
      a.units = units - a.unit0 < slices.units ? units - a.unit0 : slices.units;
      chunk_prepare_kernel<T, NW, SCALAR, PLAIN><<<dim3(a.units, a.heads), 128, 0, stream>>>(a);
      HB_LAUNCH_CHECK();
      const int rc = wide ? launch_columns<T, NW, 2, PLAIN>(a, stream) : launch_columns<T, NW, 1, PLAIN>(a, stream);
      if (rc != HB_OK) return rc;
    }
  return HB_OK;
}

size_t image_bytes(int dim, bool plain) {
  if (dim <= 32) return plain ? sizeof(ChunkImage<2, true>) : sizeof(ChunkImage<2, false>);
  if (dim <= 64) return plain ? sizeof(ChunkImage<4, true>) : sizeof(ChunkImage<4, false>);
  if (dim <= 96) return plain ? sizeof(ChunkImage<6, true>) : sizeof(ChunkImage<6, false>);
  return plain ? sizeof(ChunkImage<8, true>) : sizeof(ChunkImage<8, false>);
}

template <typename T, bool SCALAR, bool PLAIN>
int launch_by_dim(const ChunkArgs& a, int n_tokens, int longest, long long most_bytes, cudaStream_t stream) {
  if (a.dim <= 32) return launch_chunked<T, 2, SCALAR, PLAIN>(a, n_tokens, longest, most_bytes, stream);
  if (a.dim <= 64) return launch_chunked<T, 4, SCALAR, PLAIN>(a, n_tokens, longest, most_bytes, stream);
  if (a.dim <= 96) return launch_chunked<T, 6, SCALAR, PLAIN>(a, n_tokens, longest, most_bytes, stream);
  return launch_chunked<T, 8, SCALAR, PLAIN>(a, n_tokens, longest, most_bytes, stream);
}

}  // namespace

// Floats of scratch that the chunked recurrences need for `n_tokens` tokens of `n_seqs` requests, `cols` columns a head (vdim; the
// mLSTM vdim + 1), where `most_bytes` are to be enough or a single chunk of all heads needs more; `longest`: the longest portion,
// 0 where it is not known. The recurrence is called with the same numbers.
extern "C" long long hb_recurrence_chunked_scratch_floats(int n_tokens, int n_seqs, int longest, int heads, int dim, int cols, int plain,
                                                          long long most_bytes) {
  const size_t bytes = image_bytes(dim, plain != 0);
  return (long long)(slices_of(n_tokens, n_seqs, longest, heads, cols, bytes, most_bytes).units * (heads * bytes) / 4);
}

// What the launches of such a step take, for a look without a GPU: `out` = shares, units a launch; with `cu_seqlens` (of the host)
// also request `seq`'s first chunk, number of chunks (<= 0: none) and first unit in the launch of `share` that starts at `unit0`.
extern "C" void hb_recurrence_chunked_slices(int n_tokens, int n_seqs, int longest, int heads, int dim, int cols, int plain,
                                             long long most_bytes, const int* cu_seqlens, int seq, int share, int unit0, int* out) {
  const Slices slices = slices_of(n_tokens, n_seqs, longest, heads, cols, image_bytes(dim, plain != 0), most_bytes);
  out[0] = slices.shares;
  out[1] = slices.units;
  if (!cu_seqlens) return;
  const Span span = span_of(cu_seqlens, seq, share, slices.shares, unit0, slices.units);
  out[2] = span.chunk; out[3] = span.count; out[4] = span.unit;
}

extern "C" int hb_delta_recurrence_chunked(const float* q, const float* k, const float* v, const float* beta,
                                           const float* decay, float* state, long long state_stride,
                                           const int* cu_seqlens, const int* slots, float* scratch, float* out,
                                           int n_tokens, int n_seqs, int longest, int heads, int kvh, int dim,
                                           int vdim, int plain, long long most_bytes, int* status, cudaStream_t stream) {
  if (!q || !k || !v || (!beta && !plain) || !decay || !state || !cu_seqlens || !slots || !scratch || !out || !status) return HB_ERR_BAD_ARG;
  if (heads <= 0 || kvh <= 0 || heads % kvh || dim <= 0 || vdim <= 0 || n_seqs < 0 || n_tokens < 0) return HB_ERR_BAD_ARG;
  if (dim > 128 || heads > 65535 || n_seqs > 65535 || (reinterpret_cast<uintptr_t>(scratch) & 15)) return HB_ERR_UNSUPPORTED;
  if (n_seqs == 0 || n_tokens == 0) return HB_OK;
  ChunkArgs a = {};
  a.q = q; a.k = k; a.v = v; a.q_ld = (long long)kvh * dim; a.v_ld = (long long)heads * vdim; a.decay = decay; a.beta = beta;
  a.o_scale = 1.f; a.state = state; a.state_stride = state_stride; a.head_floats = (long long)dim * vdim;
  a.row_step = vdim; a.col_step = 1; a.cu_seqlens = cu_seqlens; a.slots = slots; a.images = reinterpret_cast<unsigned char*>(scratch); a.out = out; a.status = status;
  a.n_seqs = n_seqs; a.heads = heads; a.kvh = kvh; a.dim = dim; a.vdim = vdim; a.cols = vdim;
  return plain ? launch_by_dim<float, false, true>(a, n_tokens, longest, most_bytes, stream) : launch_by_dim<float, false, false>(a, n_tokens, longest, most_bytes, stream);
}

extern "C" int hb_mlstm_recurrence_chunked(const void* proj, int proj_dtype, long long ld, int q_off, int k_off, int v_off,
                                           float q_scale, const float* keep, const float* take, float* state,
                                           long long state_stride, const int* cu_seqlens, const int* slots, float* scratch,
                                           float* o, float* nq, int n_tokens, int n_seqs, int longest, int heads, int dim, int vdim,
                                           long long most_bytes, int* status, cudaStream_t stream) {
  if (!proj || !keep || !take || !state || !cu_seqlens || !slots || !scratch || !o || !nq || !status || n_seqs < 0 || n_tokens < 0 ||
      heads <= 0 || dim <= 0 || vdim <= 0)
    return HB_ERR_BAD_ARG;
  if (proj_dtype != HB_DTYPE_F32 && proj_dtype != HB_DTYPE_BF16) return HB_ERR_BAD_ARG;
  if (dim > 128 || heads > 65535 || n_seqs > 65535 || (reinterpret_cast<uintptr_t>(scratch) & 15)) return HB_ERR_UNSUPPORTED;
  if (n_seqs == 0 || n_tokens == 0) return HB_OK;
  ChunkArgs a = {};
  const size_t el = proj_dtype == HB_DTYPE_F32 ? 4 : 2;
  const char* base = reinterpret_cast<const char*>(proj);
  a.q = base + q_off * el; a.k = base + k_off * el; a.v = base + v_off * el; a.q_ld = ld; a.v_ld = ld; a.decay = keep;
  a.take = take; a.o_scale = q_scale; a.state = state; a.state_stride = state_stride;
  a.head_floats = (long long)(vdim + 1) * dim; a.row_step = 1; a.col_step = dim; a.cu_seqlens = cu_seqlens; a.slots = slots;
  a.images = reinterpret_cast<unsigned char*>(scratch); a.out = o; a.status = status; a.nq = nq; a.n_seqs = n_seqs; a.heads = heads; a.kvh = heads; a.dim = dim; a.vdim = vdim;
  a.cols = vdim + 1;
  return proj_dtype == HB_DTYPE_F32 ? launch_by_dim<float, true, true>(a, n_tokens, longest, most_bytes, stream)
                                    : launch_by_dim<__nv_bfloat16, true, true>(a, n_tokens, longest, most_bytes, stream);
}
