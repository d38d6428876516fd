// The matrix memories' recurrences sixteen tokens at a time, for portions of prompts:
//   S <- diag(g_t) S + k_t u_t^T,   o_t = S^T q_t,   u_t = v_t (plain) or beta_t (v_t - (diag(g_t) S)^T k_t) (delta rule)
// With P_t = g_1 ... g_t (elementwise, from the chunk's start), R_s = g_(s+1) ... g_16 and S the chunk's first state:
//   u = T (v - (P k) S),     T = (I + diag(beta) A)^-1 diag(beta),  A_ts = sum_d k_t (g_(s+1) ... g_t) k_s,  s < t
//   o_t = (P_t q_t) S + sum_(s <= t) B_ts u_s,                      B_ts = sum_d q_t (g_(s+1) ... g_t) k_s
//   S <- diag(P_16) S + sum_s (R_s k_s) u_s^T
// Every factor is a product of decays, never a quotient: strong decays underflow to the zero they stand for.
//
//   chunk_matrices_kernel   T and B of all chunks and heads, side by side (they need no state)
//   chunk_recurrence_kernel per (request, head, 16 or 32 columns of S): chunk after chunk. NW warps own 16 rows of S each,
//     in registers as accumulator tiles; their products run on the tensor cores with every float32 factor as three
//     bfloat16 pieces (see hb::split3), and the sums over all rows are brought together in shared memory in a fixed order.
//     NW more warps, in two groups that take turns, prepare the next chunk's rows (decay products) and write the chunk's
//     outputs, which nothing waits for.
//
// Measured (B200, one request of 2,048 tokens, 16 heads of 128 x 128; before: token after token, a chain of 2,048 steps):
// delta rule 582 -> 224 us (24 of them the matrices), the rule without correction 573 -> 155, mLSTM 437 -> 158; 32 heads of
// Mamba-2 709 -> 249. Error against 64 bits (2-norm, outputs / states): delta rule 9.1e-8 / 1.3e-7 -> 7.1e-8 / 7.0e-8, without
// correction 1.4e-7 / 1.1e-7 -> 8.7e-8 / 5.4e-8. A chunk is 1.6 us of a block: 6,000 warp instructions, of which the
// preparation of its rows is 40 %, between three barriers. Tried: the products as float32 fma (the shared-memory reads of 4 x 4
// tiles bound it: 293 us); two tf32 pieces a factor (error 1.1e-7, states of Mamba-2 1.9 times as far off: taken back).
//
// What is not finite in a token's inputs reaches that token's and later outputs of the request, never an earlier one (an
// infinite value or state comes out of the products as NaN, where token after token the sum could stay infinite).
#include "api.h"
#include "common.cuh"
#include "mma.cuh"

namespace {

constexpr int C = 16;       // tokens of a chunk

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
  float* matrices;           // [units, heads, 2, C, C]: T (not used by the plain rule), B
  float* out;                // [N, heads * vdim]
  float* nq;                 // [N, heads] (with take): outputs of column vdim
  int n_seqs, heads, kvh, dim, vdim, cols;
};

// unit = a request's chunk: those of request s start at cu[s] / C + s (there is room for a partial one each)
__device__ __forceinline__ int first_unit(const int* cu, int s) { return cu[s] / C + s; }

// grid (units, heads), 128 threads: warp w takes s = w, w + 4, w + 8, w + 12; a running row w_s = k_s g_(s+1) ... g_t
// meets k_t and q_t, eight sums a token, brought together by a halving butterfly.
template <typename T, int NW, bool SCALAR, bool PLAIN>
__global__ void __launch_bounds__(128) chunk_matrices_kernel(const ChunkArgs a) {
  constexpr int DP = 16 * NW, DL = (DP + 31) / 32;
  __shared__ __align__(16) float ks[C][DL * 32], qs[C][DL * 32], gs[SCALAR ? 1 : C][SCALAR ? C : DL * 32];
  __shared__ float A[C][C + 1], B[C][C], bet[C];
  __shared__ int where[2];
  const int unit = blockIdx.x, head = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) where[0] = -1;
  __syncthreads();
  for (int s = tid; s < a.n_seqs; s += 128) {
    const int c = unit - first_unit(a.cu_seqlens, s), n = a.cu_seqlens[s + 1] - a.cu_seqlens[s];
    if (c >= 0 && c * C < n) { where[0] = a.cu_seqlens[s] + c * C; where[1] = a.cu_seqlens[s + 1]; }
  }
  __syncthreads();
  const int t0 = where[0];
  if (t0 < 0) return;
  const int count = min(C, where[1] - t0);
  const int kvhead = head / (a.heads / a.kvh);
  {
    // a column of the chunk a thread (or every STEP-th token of one)
    constexpr int W = DL * 32, STEP = 128 / W > 0 ? 128 / W : 1;
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
        if (!SCALAR) gs[t][d] = in ? *g : 1.f;
      }
    }
  }
  if (tid < C) {
    if (SCALAR) gs[0][tid] = tid < count ? a.decay[(size_t)(t0 + tid) * a.heads + head] : 1.f;
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
        gt[i] = SCALAR ? gs[0][t] : gs[SCALAR ? 0 : t][lane * DL + i];
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
  __syncthreads();
  float* dst = a.matrices + ((size_t)unit * a.heads + head) * (2 * C * C);
  for (int e = tid; e < C * C; e += 128) dst[C * C + e] = (e % C) <= e / C ? B[e / C][e % C] : 0.f;
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
      dst[t * C + tid] = x[t];
    }
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

template <int NW, int CT, bool PLAIN>
struct ChunkSmem {
  // row lengths that put a fragment's rows into different banks
  static constexpr int DP = 16 * NW, LD = DP + 8, ROWS = PLAIN ? C : 2 * C, LZ = ROWS + 8, CG = 16 * CT;
  struct Stage {
    float p[ROWS][LD];       // P k (not with the plain rule), then P q
    float rk[DP][24];        // R k, [row][token]
    float2 full[DP];         // the whole chunk's decay and the rest of its rounding
    float t[C][20];          // T
    float b[C][C];           // B
    float v[C][CG + 4];      // values (0 past the end)
  };
  struct All {
    Stage stage[2];
    float part[2][NW][CG][LZ];         // [column][token]: a warp's share of (P S)^T
    float x[CG][20];                   // [column][token]
    float u[2][CG][20];                // [column][token]
    __nv_bfloat16 up[2][3][CG][24];    // the pieces of u
  };
};

template <typename T, int NW, int CT, bool SCALAR, bool PLAIN>
__global__ void __launch_bounds__(64 * NW) chunk_recurrence_kernel(const ChunkArgs a) {
  using Smem = ChunkSmem<NW, CT, PLAIN>;
  constexpr int CG = Smem::CG, COMP = 32 * NW, HELP = 16 * NW;
  // barriers (+ the buffer's parity): chunk prepared; u and the shares of P S there; chunk used up; among the COMP threads
  constexpr int FULL = 1, DONE = 3, EMPTY = 5, PEER = 7;
  extern __shared__ __align__(16) unsigned char raw[];
  typename Smem::All& sm = *reinterpret_cast<typename Smem::All*>(raw);
  const int head = blockIdx.y, seq = blockIdx.z, col0 = blockIdx.x * CG;
  const int first = a.cu_seqlens[seq], last = a.cu_seqlens[seq + 1];
  if (first >= last) return;
  const int chunks = (last - first + C - 1) / C;
  const int tid = threadIdx.x;

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
    for (int i = 0; i < chunks; ++i) {
      const int b = i & 1;
      auto& st = sm.stage[b];
      bar_sync(FULL + b, COMP + HELP);
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
      // the warp's share of (P S)^T for sixteen rows of P
      auto share = [&](int row) {
        uint32_t pp[2][3][2];
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float2 v = *reinterpret_cast<const float2*>(&st.p[row + 8 * n + g][warp * 16 + 8 * h + 2 * q4]);
            uint32_t p[3];
            hb::split3(v.x, v.y, p);
#pragma unroll
            for (int x = 0; x < 3; ++x) pp[n][x][h] = p[x];
          }
#pragma unroll
        for (int m = 0; m < CT; ++m) {
          float z[2][4];
          mma3(z, sp[m], pp);
#pragma unroll
          for (int n = 0; n < 2; ++n) {
            *reinterpret_cast<float2*>(&sm.part[b][warp][16 * m + g][row + 8 * n + 2 * q4]) = make_float2(z[n][0], z[n][1]);
            *reinterpret_cast<float2*>(&sm.part[b][warp][16 * m + g + 8][row + 8 * n + 2 * q4]) = make_float2(z[n][2], z[n][3]);
          }
        }
      };
      share(0);
      if constexpr (!PLAIN) {
        const int count = min(C, last - first - i * C);
        constexpr int EN = (C * CG + COMP - 1) / COMP;
        const int t = tid % C;
        float4 tr[C / 4];
        float vv[EN], xx[EN];
#pragma unroll
        for (int r = 0; r < C / 4; ++r) tr[r] = *reinterpret_cast<const float4*>(&st.t[t][4 * r]);
        const float own = st.t[t][t];
#pragma unroll
        for (int j = 0; j < EN; ++j) vv[j] = tid + j * COMP < C * CG ? st.v[t][(tid + j * COMP) / C] : 0.f;
        bar_sync(PEER, COMP);
#pragma unroll
        for (int j = 0; j < EN; ++j) {
          const int c = (tid + j * COMP) / C;
          if (tid + j * COMP >= C * CG) break;
          xx[j] = vv[j] - tree_sum<NW>([&](int w) { return sm.part[b][w][c][t]; });
          sm.x[c][t] = xx[j];
        }
        share(C);                // (P q) S: nothing waits for it, it fills the time
        __syncwarp();            // a warp reads back its own columns only
#pragma unroll
        for (int j = 0; j < EN; ++j) {
          const int c = (tid + j * COMP) / C;
          if (tid + j * COMP >= C * CG) break;
          float u0 = 0.f, u1 = 0.f;
#pragma unroll
          for (int r = 0; r < C; r += 4) {
            const float4 xr = *reinterpret_cast<const float4*>(&sm.x[c][r]);
            // a later token's rows never reach an earlier one, whatever they hold
            if (r < t) u0 = fmaf(tr[r / 4].x, xr.x, u0);
            if (r + 1 < t) u1 = fmaf(tr[r / 4].y, xr.y, u1);
            if (r + 2 < t) u0 = fmaf(tr[r / 4].z, xr.z, u0);
            if (r + 3 < t) u1 = fmaf(tr[r / 4].w, xr.w, u1);
          }
          // the token's own row, the largest term, comes last
          const float u = t < count ? fmaf(own, xx[j], u0 + u1) : 0.f;
          sm.u[b][c][t] = u;
          put_pieces(&sm.up[b][0][c][t], CG * 24, u);
        }
        bar_sync(PEER, COMP);
      }
      bar_arrive(DONE + b, COMP + HELP);
      uint32_t rp[2][3][2];
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float2 v = *reinterpret_cast<const float2*>(&st.rk[warp * 16 + 8 * n + g][8 * h + 2 * q4]);
          uint32_t p[3];
          hb::split3(v.x, v.y, p);
#pragma unroll
          for (int x = 0; x < 3; ++x) rp[n][x][h] = p[x];
        }
      float4 full[2];
#pragma unroll
      for (int n = 0; n < 2; ++n) full[n] = *reinterpret_cast<const float4*>(&st.full[warp * 16 + 8 * n + 2 * q4]);
#pragma unroll
      for (int m = 0; m < CT; ++m) {
        uint32_t up[3][4];
#pragma unroll
        for (int x = 0; x < 3; ++x)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            up[x][e] = *reinterpret_cast<const uint32_t*>(&sm.up[b][x][16 * m + g + (e & 1) * 8][2 * q4 + (e >> 1) * 8]);
        float z[2][4];
        mma3(z, up, rp);
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            s[m][n][e] = fmaf(s[m][n][e], (e & 1) ? full[n].z : full[n].x,
                              fmaf(s[m][n][e], (e & 1) ? full[n].w : full[n].y, z[n][e]));
      }
      if (i + 2 < chunks) bar_arrive(EMPTY + b, COMP + HELP);
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

  // ---- two groups of helpers, a thread per row of S: group b prepares the chunks of parity b and writes their outputs,
  // so the inputs of its next chunk, asked for as soon as the registers are free, have two chunks' time to arrive
  const int b = (tid - COMP) / HELP, d = (tid - COMP) % HELP;
  auto& st = sm.stage[b];
  const int kvhead = head / (a.heads / a.kvh);
  const T* q = reinterpret_cast<const T*>(a.q) + (size_t)kvhead * a.dim + d;
  const T* k = reinterpret_cast<const T*>(a.k) + (size_t)kvhead * a.dim + d;
  const T* v = reinterpret_cast<const T*>(a.v) + (size_t)head * a.vdim;
  const float* decay = a.decay + (SCALAR ? (size_t)head : (size_t)head * a.dim + d);
  const size_t decay_ld = SCALAR ? a.heads : (size_t)a.heads * a.dim;
  constexpr int TB4 = (PLAIN ? 1 : 2) * C * C / 4, TBN = (TB4 + HELP - 1) / HELP, VN = (C * CG + HELP - 1) / HELP;
  T kr[C], qr[C], vr[VN];
  float gr[C], fr[VN];
  float4 tbr[TBN];
  const int unit0 = first_unit(a.cu_seqlens, seq);
  auto load = [&](int i) {               // nothing is computed from the values here, so nothing waits for them
    const int t0 = first + i * C, count = min(C, last - t0);
    const T* kp = k + (size_t)t0 * a.q_ld;
    const T* qp = q + (size_t)t0 * a.q_ld;
    const float* gp = decay + (size_t)t0 * decay_ld;
    // (one decay a head: most chunks have nothing to ask about; 10 us of the mLSTM's 173 on ragged portions. With a decay a
    // row the same made the delta rule slower, by 9 us of 235.)
    if (SCALAR && count == C && d < a.dim && a.q_ld < (1 << 26)) {
      const int ql = (int)a.q_ld, gl = (int)decay_ld;
#pragma unroll
      for (int t = 0; t < C; ++t) {
        kr[t] = kp[t * ql];
        qr[t] = qp[t * ql];
        gr[t] = gp[t * gl];
      }
    } else {
#pragma unroll
      for (int t = 0; t < C; ++t, kp += a.q_ld, qp += a.q_ld, gp += decay_ld) {
        const bool in = t < count && d < a.dim;
        kr[t] = in ? *kp : hb::from_f32<T>(0.f);
        qr[t] = in ? *qp : hb::from_f32<T>(0.f);
        gr[t] = in ? *gp : 1.f;
      }
    }
    const float4* m = reinterpret_cast<const float4*>(a.matrices + ((size_t)(unit0 + i) * a.heads + head) * (2 * C * C) + (PLAIN ? C * C : 0));
#pragma unroll
    for (int j = 0; j < TBN; ++j)
      if (d + j * HELP < TB4) tbr[j] = m[d + j * HELP];
#pragma unroll
    for (int j = 0; j < VN; ++j) {
      const int e = d + j * HELP, t = e / CG, col = col0 + e % CG;
      const bool in = t < count && col < a.cols;
      vr[j] = in && col < a.vdim ? v[(size_t)(t0 + t) * a.v_ld + col] : hb::from_f32<T>(in ? 1.f : 0.f);
      fr[j] = in && a.take ? a.take[(size_t)(t0 + t) * a.heads + head] : 1.f;
    }
  };
  if (b < chunks) load(b);
  for (int i = b; i < chunks; i += 2) {
    const int t0 = first + i * C, count = min(C, last - t0);
    if (i >= 2) bar_sync(EMPTY + b, COMP + HELP);
    Product p;
#pragma unroll
    for (int t = 0; t < C; ++t) {
      p.times(gr[t]);
      if constexpr (!PLAIN) st.p[t][d] = p.of(hb::to_f32(kr[t]));
      st.p[(PLAIN ? 0 : C) + t][d] = p.of(hb::to_f32(qr[t]));
    }
    st.full[d] = make_float2(p.hi, p.lo);
    Product r;
#pragma unroll
    for (int t = C - 4; t >= 0; t -= 4) {
      float4 w;
      w.w = r.of(hb::to_f32(kr[t + 3])); r.times(gr[t + 3]);
      w.z = r.of(hb::to_f32(kr[t + 2])); r.times(gr[t + 2]);
      w.y = r.of(hb::to_f32(kr[t + 1])); r.times(gr[t + 1]);
      w.x = r.of(hb::to_f32(kr[t])); r.times(gr[t]);
      *reinterpret_cast<float4*>(&st.rk[d][t]) = w;
    }
#pragma unroll
    for (int j = 0; j < TBN; ++j) {
      const int e = d + j * HELP;
      if (e >= TB4) break;
      if (!PLAIN && e < C * C / 4) *reinterpret_cast<float4*>(&st.t[e / (C / 4)][e % (C / 4) * 4]) = tbr[j];
      else reinterpret_cast<float4*>(&st.b[0][0])[PLAIN ? e : e - C * C / 4] = tbr[j];
    }
#pragma unroll
    for (int j = 0; j < VN; ++j) {
      const int e = d + j * HELP;
      if (e >= C * CG) break;
      const float x = hb::to_f32(vr[j]) * fr[j];
      if (PLAIN) {
        sm.u[b][e % CG][e / CG] = x;
        put_pieces(&sm.up[b][0][e % CG][e / CG], CG * 24, x);
      } else {
        st.v[e / CG][e % CG] = x;
      }
    }
    bar_arrive(FULL + b, COMP + HELP);
    if (i + 2 < chunks) load(i + 2);
    bar_sync(DONE + b, COMP + HELP);
#pragma unroll
    for (int j = 0; j < VN; ++j) {
      const int e = d + j * HELP, t = e / CG, c = e % CG, col = col0 + c;
      if (e >= C * CG) break;
      float y0 = 0.f, y1 = 0.f;
#pragma unroll
      for (int x = 0; x < C; x += 4) {
        const float4 br = *reinterpret_cast<const float4*>(&st.b[t][x]);
        const float4 u = *reinterpret_cast<const float4*>(&sm.u[b][c][x]);
        if (x <= t) y0 = fmaf(br.x, u.x, y0);
        if (x + 1 <= t) y1 = fmaf(br.y, u.y, y1);
        if (x + 2 <= t) y0 = fmaf(br.z, u.z, y0);
        if (x + 3 <= t) y1 = fmaf(br.w, u.w, y1);
      }
      // the last three sums with what they round off, so that the output rounds once
      auto z = [&](int w) { return sm.part[b][w][c][(PLAIN ? 0 : C) + t]; };
      float lost = 0.f;
      const float y = two_sum(y0, y1, lost);
      const float o = (two_sum(two_sum(tree_sum<NW - NW / 2>(z), tree_sum<NW / 2>(z, NW - NW / 2), lost), y, lost) + lost) * a.o_scale;
      if (t < count && col < a.vdim) a.out[(size_t)(t0 + t) * a.heads * a.vdim + (size_t)head * a.vdim + col] = o;
      else if (t < count && col < a.cols) a.nq[(size_t)(t0 + t) * a.heads + head] = o;
    }
  }
}

template <typename T, int NW, int CT, bool SCALAR, bool PLAIN>
int launch_columns(const ChunkArgs& a, cudaStream_t stream) {
  const size_t smem = sizeof(typename ChunkSmem<NW, CT, PLAIN>::All);
  cudaError_t e = cudaFuncSetAttribute(chunk_recurrence_kernel<T, NW, CT, SCALAR, PLAIN>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  chunk_recurrence_kernel<T, NW, CT, SCALAR, PLAIN>
      <<<dim3((a.cols + 16 * CT - 1) / (16 * CT), a.heads, a.n_seqs), 64 * NW, smem, stream>>>(a);
  HB_LAUNCH_CHECK();
  return HB_OK;
}

template <typename T, int NW, bool SCALAR, bool PLAIN>
int launch_chunked(const ChunkArgs& a, int units, cudaStream_t stream) {
  chunk_matrices_kernel<T, NW, SCALAR, PLAIN><<<dim3(units, a.heads), 128, 0, stream>>>(a);
  HB_LAUNCH_CHECK();
  // 32 columns a block share the preparation of a chunk's rows, once 16 a block are more than a block per SM
  const long long blocks = (long long)((a.cols + 15) / 16) * a.heads * a.n_seqs;
  return blocks > 148 && a.cols > 16 ? launch_columns<T, NW, 2, SCALAR, PLAIN>(a, stream)
                                     : launch_columns<T, NW, 1, SCALAR, PLAIN>(a, stream);
}

template <typename T, bool SCALAR, bool PLAIN>
int launch_by_dim(const ChunkArgs& a, int units, cudaStream_t stream) {
  if (a.dim <= 32) return launch_chunked<T, 2, SCALAR, PLAIN>(a, units, stream);
  if (a.dim <= 64) return launch_chunked<T, 4, SCALAR, PLAIN>(a, units, stream);
  if (a.dim <= 96) return launch_chunked<T, 6, SCALAR, PLAIN>(a, units, stream);
  return launch_chunked<T, 8, SCALAR, PLAIN>(a, units, stream);
}

}  // namespace

// Floats of scratch that the chunked recurrences need for `n_tokens` tokens of `n_seqs` requests.
extern "C" long long hb_recurrence_chunked_scratch_floats(int n_tokens, int n_seqs, int heads) {
  return ((long long)n_tokens / C + n_seqs) * heads * (2 * C * C);
}

extern "C" int hb_delta_recurrence_chunked(const float* q, const float* k, const float* v, const float* beta,
                                           const float* decay, float* state, long long state_stride,
                                           const int* cu_seqlens, const int* slots, float* scratch, float* out,
                                           int n_tokens, int n_seqs, int heads, int kvh, int dim, int vdim, int plain,
                                           cudaStream_t stream) {
  if (!q || !k || !v || (!beta && !plain) || !decay || !state || !cu_seqlens || !slots || !scratch || !out) return HB_ERR_BAD_ARG;
  if (heads <= 0 || kvh <= 0 || heads % kvh || dim <= 0 || vdim <= 0 || n_seqs < 0 || n_tokens < 0) return HB_ERR_BAD_ARG;
  if (dim > 128 || heads > 65535 || n_seqs > 65535 || (reinterpret_cast<uintptr_t>(scratch) & 15)) return HB_ERR_UNSUPPORTED;
  if (n_seqs == 0 || n_tokens == 0) return HB_OK;
  ChunkArgs a = {};
  a.q = q; a.k = k; a.v = v; a.q_ld = (long long)kvh * dim; a.v_ld = (long long)heads * vdim; a.decay = decay; a.beta = beta;
  a.o_scale = 1.f; a.state = state; a.state_stride = state_stride; a.head_floats = (long long)dim * vdim;
  a.row_step = vdim; a.col_step = 1; a.cu_seqlens = cu_seqlens; a.slots = slots; a.matrices = scratch; a.out = out;
  a.n_seqs = n_seqs; a.heads = heads; a.kvh = kvh; a.dim = dim; a.vdim = vdim; a.cols = vdim;
  const int units = n_tokens / C + n_seqs;
  return plain ? launch_by_dim<float, false, true>(a, units, stream) : launch_by_dim<float, false, false>(a, units, stream);
}

extern "C" int hb_mlstm_recurrence_chunked(const void* proj, int proj_dtype, long long ld, int q_off, int k_off, int v_off,
                                           float q_scale, const float* keep, const float* take, float* state,
                                           long long state_stride, const int* cu_seqlens, const int* slots, float* scratch,
                                           float* o, float* nq, int n_tokens, int n_seqs, int heads, int dim, int vdim,
                                           cudaStream_t stream) {
  if (!proj || !keep || !take || !state || !cu_seqlens || !slots || !scratch || !o || !nq || n_seqs < 0 || n_tokens < 0 ||
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
  a.matrices = scratch; a.out = o; a.nq = nq; a.n_seqs = n_seqs; a.heads = heads; a.kvh = heads; a.dim = dim; a.vdim = vdim;
  a.cols = vdim + 1;
  const int units = n_tokens / C + n_seqs;
  return proj_dtype == HB_DTYPE_F32 ? launch_by_dim<float, true, true>(a, units, stream)
                                    : launch_by_dim<__nv_bfloat16, true, true>(a, units, stream);
}
