// Attention of portions of prompts over the paged cache in true 32 bits, on the tensor cores.
//
// A row is a (new token, query head) pair of one kv head: a block takes 64 rows of a request, 16 a warp, so the heads of a
// group read a key tile together. Keys come 32 at a time; queries, keys, values and softmax weights are taken apart into
// three bfloat16 pieces each that sum to them exactly (8 + 8 + 8 bits), and the six products of pieces down to 2^-24 of the
// whole are summed in float32: the large one by itself and added with float32's own rounding, since a tensor core cuts a sum
// where it does not fit. Maximum, exponentials and sums are float32 as in the general kernel, and so are the rules of what a
// token may read (see attention.cu). A value that is not finite reaches only the rows that may read it; a score that comes
// out not finite (an infinite key may weigh nothing) is worked out again as the general kernel does.
//
// What bounds it: mma.sync, at 2 cycles of an SM for [16, 16] x [16, 8], six of them a product (0.4 of the time), and the
// chains between them: a block of four warps splits, multiplies and takes exponentials in turn, two blocks per SM (104 KB of
// pieces each). The general kernel (a warp per row, uncoalesced rows of keys, every key read once per row) took 1,622 us for
// 600 tokens behind 301, 16 heads / 4 kv heads of 128, and 18.1 ms for 2,048 tokens, 40 / 8 heads; this one 112 us and
// 1.19 ms. Steps (beside a merge of shares that took 27 us longer): keys and values loaded where they are needed, two key tiles
// of products side by side 187 us; four side by side (the five small terms are a chain) 174; a tile's rows loaded into registers
// under the products before them 150; the shares of a row tile's keys chosen by fractional rounds 139; the merge a warp a row 112.
// Error against 64 bits 4.8e-7 -> 1.9e-7.
#include "api.h"
#include "common.cuh"
#include "mma.cuh"

namespace {

constexpr int ROWS = 64, KEYS = 32, WARPS = 4;

struct PortionArgs {
  const float* q;               // [N, nh, hd]
  const float* k_pages;         // [pages, nkv, page_size, hd]
  const float* v_pages;
  const int* block_table;
  int table_stride;
  const int* cu_seqlens;
  const int* positions;
  float* out;                   // [N, nh, hd]
  int nh, nkv, page_size, chunk, window, keep;
  float scale;
  int sink;
  float softcap;
  const float* slopes;
  const float* sink_values;
  int splits;                   // > 1: blocks that share a row tile's key tiles; their rows go to the parts
  float* part_acc;              // [N * nh, splits, hd]
  float* part_ml;               // [N * nh, splits, 2]
};

__device__ __forceinline__ void mma16(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ bool finite(float x) { return fabsf(x) <= 3.402823466e38f; }

// four floats into the three pieces' rows
template <int PIECE>
__device__ __forceinline__ void put4(__nv_bfloat16* at, float4 v) {
  uint32_t a[3], b[3];
  hb::split3(v.x, v.y, a);
  hb::split3(v.z, v.w, b);
#pragma unroll
  for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2*>(at + i * PIECE) = make_uint2(a[i], b[i]);
}

template <int NT>               // head_dim = 16 NT
__global__ void __launch_bounds__(32 * WARPS, NT <= 8 ? 2 : 1) portion_attention_kernel(const PortionArgs a) {
  constexpr int HD = 16 * NT, LD = HD + 8;          // rows of LD bfloat16 start in different banks (an odd number of 16 bytes)
  constexpr int QP = ROWS * LD, KP = KEYS * LD, PER = HD / 4;
  extern __shared__ __align__(16) unsigned char raw[];
  __nv_bfloat16* qs = reinterpret_cast<__nv_bfloat16*>(raw);      // [3][ROWS][LD]
  __nv_bfloat16* ks = qs + 3 * QP;                                // [3][KEYS][LD]
  __nv_bfloat16* vs = ks + 3 * KP;
  __shared__ long long offs[2][KEYS];                             // of a key's row in the pools, -1: no row may read it
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q4 = lane & 3;
  const int seq = blockIdx.z / a.splits, split = blockIdx.z % a.splits, kvh = blockIdx.y;
  const int group = a.nh / a.nkv;
  const int begin = a.cu_seqlens[seq], rows = (a.cu_seqlens[seq + 1] - begin) * group;
  const int r0 = (gridDim.x - 1 - blockIdx.x) * ROWS;             // the longest key ranges first
  if (r0 >= rows) return;
  const int* table = a.block_table + (size_t)seq * a.table_stride;
  auto first_key = [&](int pos) {
    int lo = a.chunk > 0 ? pos / a.chunk * a.chunk : 0;
    return a.window > 0 ? max(lo, pos - a.window + 1) : lo;
  };
  // the tile's keys: those kept from the sequence's start, then from the first row's first to the last row's own
  const int pos_last = a.positions[begin + min(rows - 1, r0 + ROWS - 1) / group];
  const int lo_first = first_key(a.positions[begin + r0 / group]), kept_most = min(a.keep, first_key(pos_last));
  const int main0 = lo_first / KEYS, head_tiles = min((kept_most + KEYS - 1) / KEYS, main0);
  const int tiles = head_tiles + pos_last / KEYS - main0 + 1, per = (tiles + a.splits - 1) / a.splits;
  const int tile0 = split * per, tile1 = min(tiles, tile0 + per);
  // this thread's two rows of scores and outputs
  int pos[2], lo[2], kept[2];
  size_t th[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r = r0 + warp * 16 + g + 8 * i;
    pos[i] = -1; lo[i] = 0; kept[i] = 0; th[i] = 0;
    if (r < rows) {
      pos[i] = a.positions[begin + r / group];
      lo[i] = first_key(pos[i]);
      kept[i] = min(a.keep, lo[i]);
      th[i] = (size_t)(begin + r / group) * a.nh + kvh * group + r % group;
    }
  }
  if (tile0 >= tile1) {
    if (a.splits > 1 && q4 == 0)
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (pos[i] >= 0) *reinterpret_cast<float2*>(a.part_ml + (th[i] * a.splits + split) * 2) = make_float2(-INFINITY, 0.f);
    return;
  }
  auto key0_of = [&](int tile) { return (tile < head_tiles ? tile : main0 + tile - head_tiles) * KEYS; };
  auto find = [&](int tile) {
    if (tid < KEYS) {
      const int key = key0_of(tile) + tid;
      long long off = -1;
      if (key <= pos_last && (key >= lo_first || key < kept_most)) {
        const int page = table[key / a.page_size];
        if (page >= 0) off = (((long long)page * a.nkv + kvh) * a.page_size + key % a.page_size) * HD;
      }
      offs[tile & 1][tid] = off;
    }
  };
  find(tile0);
  for (int e = tid; e < ROWS * PER; e += 32 * WARPS) {
    const int r = e / PER, c = (e % PER) * 4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r0 + r < rows)
      v = *reinterpret_cast<const float4*>(a.q + ((size_t)(begin + (r0 + r) / group) * a.nh + kvh * group + (r0 + r) % group) * HD + c);
    put4<QP>(qs + r * LD + c, v);
  }
  __syncthreads();

  float o[2 * NT][4], m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
#pragma unroll
  for (int n = 0; n < 2 * NT; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[n][e] = 0.f;
  const float inv_cap = a.softcap > 0.f ? 1.f / a.softcap : 0.f;
  float slope[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) slope[i] = a.slopes ? a.slopes[th[i] % a.nh] : 0.f;
  const __nv_bfloat16* q_at = qs + (warp * 16 + (lane & 15)) * LD + (lane >> 4) * 8;
  const __nv_bfloat16* k_at = ks + ((lane & 7) + (lane >> 4) * 8) * LD + ((lane >> 3) & 1) * 8;
  const __nv_bfloat16* v_at = vs + (lane & 15) * LD + (lane >> 4) * 8;

  // A tile's rows come as registers while the warps multiply something else: its values under its own scores, the next
  // tile's keys under its weights times values.
  constexpr int LOADS = KEYS * PER / (32 * WARPS);
  float4 in[LOADS];
  auto load = [&](const float* pages, const long long* off_of) {
#pragma unroll
    for (int i = 0; i < LOADS; ++i) {
      const int e = tid + i * 32 * WARPS;
      const long long off = off_of[e / PER];
      in[i] = off >= 0 ? *reinterpret_cast<const float4*>(pages + off + (e % PER) * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  auto store = [&](__nv_bfloat16* to) {
#pragma unroll
    for (int i = 0; i < LOADS; ++i) {
      const int e = tid + i * 32 * WARPS;
      put4<KP>(to + (e / PER) * LD + (e % PER) * 4, in[i]);
    }
  };
  load(a.k_pages, offs[tile0 & 1]);
  store(ks);
  __syncthreads();
  for (int tile = tile0; tile < tile1; ++tile) {
    const int key0 = key0_of(tile);
    const long long* off_of = offs[tile & 1];
    load(a.v_pages, off_of);
    if (tile + 1 < tile1) find(tile + 1);

    // scores
    float s[4][4], lo_s[4][4];
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) s[n][e] = lo_s[n][e] = 0.f;
#pragma unroll 1
    for (int kk = 0; kk < NT; ++kk) {
      unsigned qa[3][4];
#pragma unroll
      for (int p = 0; p < 3; ++p) hb::ldmatrix_x4(qa[p], q_at + p * QP + kk * 16);
      // four key tiles side by side: a product's five small terms are a chain
      unsigned kb[2][3][4];
#pragma unroll
      for (int np = 0; np < 2; ++np)
#pragma unroll
        for (int p = 0; p < 3; ++p) hb::ldmatrix_x4(kb[np][p], k_at + p * KP + np * 16 * LD + kk * 16);
      float hi[4][4];
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) hi[n][e] = 0.f;
      constexpr int from[6][2] = {{0, 0}, {2, 0}, {0, 2}, {1, 1}, {1, 0}, {0, 1}};
#pragma unroll
      for (int x = 0; x < 6; ++x)
#pragma unroll
        for (int n = 0; n < 4; ++n) {
          const unsigned(&kx)[4] = kb[n / 2][from[x][1]];
          mma16(x == 0 ? hi[n] : lo_s[n], qa[from[x][0]], kx[2 * (n % 2)], kx[2 * (n % 2) + 1]);
        }
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) s[n][e] += hi[n][e];
    }
    bool odd = false;                       // a value that is not finite
#pragma unroll
    for (int i = 0; i < LOADS; ++i) {
      float4& v = in[i];
      if (!(finite(v.x) && finite(v.y) && finite(v.z) && finite(v.w))) {
        odd = true;
        v.x = finite(v.x) ? v.x : 0.f; v.y = finite(v.y) ? v.y : 0.f;
        v.z = finite(v.z) ? v.z : 0.f; v.w = finite(v.w) ? v.w : 0.f;
      }
    }
    store(vs);                              // read last before the end of the tile before this one
    const int any_odd = __syncthreads_or(odd);          // ... and all warps are through with the keys
    if (tile + 1 < tile1) load(a.k_pages, offs[(tile + 1) & 1]);
    auto seen = [&](int i, int at) {
      const int key = key0 + at;
      return key <= pos[i] && (key >= lo[i] || key < kept[i]) && off_of[at] >= 0;
    };
    bool again = false;                     // a score that is not finite
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        s[n][e] = (s[n][e] + lo_s[n][e]) * a.scale;
        again |= !finite(s[n][e]);
      }
    if (again)
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int i = e >> 1, at = n * 8 + 2 * q4 + (e & 1);
          if (finite(s[n][e]) || !seen(i, at)) continue;
          const float *qr = a.q + th[i] * HD, *kr = a.k_pages + off_of[at];
          float dot = 0.f;
#pragma unroll 1
          for (int d = 0; d < HD; ++d) dot += (qr[d] * a.scale) * kr[d];
          s[n][e] = dot;
        }
    float most[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = e >> 1, at = n * 8 + 2 * q4 + (e & 1);
        float x = s[n][e];
        if (a.softcap > 0.f) x = a.softcap * tanhf(x * inv_cap);
        x -= slope[i] * (float)(pos[i] - key0 - at);
        s[n][e] = seen(i, at) ? x : -INFINITY;
        most[i] = fmaxf(most[i], s[n][e]);
      }
    float corr[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float x = most[i];
      x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 1));
      x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 2));
      x = fmaxf(x, m[i]);
      corr[i] = m[i] == -INFINITY ? 0.f : expf(m[i] - x);
      m[i] = x;
      l[i] *= corr[i];
    }
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float p = s[n][e] == -INFINITY ? 0.f : expf(s[n][e] - m[e >> 1]);
        s[n][e] = p;
        l[e >> 1] += p;
      }
    // weights times values
    unsigned pa[2][3][4];
#pragma unroll
    for (int kk = 0; kk < 2; ++kk)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        uint32_t p[3];
        hb::split3(s[2 * kk + (e >> 1)][2 * (e & 1)], s[2 * kk + (e >> 1)][2 * (e & 1) + 1], p);
#pragma unroll
        for (int x = 0; x < 3; ++x) pa[kk][x][e] = p[x];
      }
#pragma unroll
    for (int n0 = 0; n0 < 2 * NT; n0 += 4) {
      constexpr int TILES = 4;
      const int live = n0 + TILES <= 2 * NT ? TILES : 2;          // 2 NT is even
      float hi[TILES][4], lo_o[TILES][4];
#pragma unroll
      for (int n = 0; n < TILES; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) hi[n][e] = lo_o[n][e] = 0.f;
#pragma unroll
      for (int kk = 0; kk < 2; ++kk) {
        unsigned vb[2][3][4];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int p = 0; p < 3; ++p)
            if (2 * h < live) hb::ldmatrix_x4_trans(vb[h][p], v_at + p * KP + kk * 16 * LD + n0 * 8 + h * 16);
        constexpr int from[6][2] = {{0, 0}, {2, 0}, {0, 2}, {1, 1}, {1, 0}, {0, 1}};
#pragma unroll
        for (int x = 0; x < 6; ++x)
#pragma unroll
          for (int n = 0; n < TILES; ++n)
            if (n < live) {
              const unsigned(&vx)[4] = vb[n / 2][from[x][1]];
              mma16(x == 0 ? hi[n] : lo_o[n], pa[kk][from[x][0]], vx[2 * (n % 2)], vx[2 * (n % 2) + 1]);
            }
      }
#pragma unroll
      for (int n = 0; n < TILES; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (n < live) o[n0 + n][e] = fmaf(o[n0 + n][e], corr[e >> 1], hi[n][e] + lo_o[n][e]);
    }
    if (any_odd)
      for (int j = 0; j < KEYS; ++j) {
        const long long off = off_of[j];
        if (off < 0) continue;
#pragma unroll
        for (int n = 0; n < 2 * NT; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int i = e >> 1, key = key0 + j;
            const float v = *const_cast<const volatile float*>(a.v_pages + off + n * 8 + 2 * q4 + (e & 1));
            if (!finite(v) && key <= pos[i] && (key >= lo[i] || key < kept[i])) o[n][e] += v;
          }
      }
    if (tile + 1 < tile1) store(ks);
    __syncthreads();                        // the tile is read, the next one's keys are there
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 1);
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 2);
    if (pos[i] < 0) continue;
    float* dst;
    float mul = 1.f;
    if (a.splits > 1) {
      dst = a.part_acc + (th[i] * a.splits + split) * HD;
      if (q4 == 0) *reinterpret_cast<float2*>(a.part_ml + (th[i] * a.splits + split) * 2) = make_float2(m[i], l[i]);
    } else {
      dst = a.out + th[i] * HD;
      if (a.sink && l[i] > 0.f) l[i] += expf((a.sink_values ? a.sink_values[th[i] % a.nh] : 0.f) - m[i]);
      mul = l[i] > 0.f ? 1.f / l[i] : 0.f;
    }
#pragma unroll
    for (int n = 0; n < 2 * NT; ++n)
      *reinterpret_cast<float2*>(dst + n * 8 + 2 * q4) = make_float2(o[n][2 * i] * mul, o[n][2 * i + 1] * mul);
  }
}

template <int NT>
int launch_portions(const PortionArgs& a, int max_new, int n_seqs, cudaStream_t stream) {
  const size_t smem = (size_t)3 * (ROWS + 2 * KEYS) * (16 * NT + 8) * sizeof(__nv_bfloat16);
  cudaError_t e = cudaFuncSetAttribute(portion_attention_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  const long long row_tiles = ((long long)max_new * (a.nh / a.nkv) + ROWS - 1) / ROWS;
  portion_attention_kernel<NT><<<dim3((unsigned)row_tiles, a.nkv, n_seqs * a.splits), 32 * WARPS, smem, stream>>>(a);
  HB_LAUNCH_CHECK();
  return HB_OK;
}

}  // namespace

// Float32 attention of portions: request s owns rows cu_seqlens[s] .. of q, at consecutive positions. `splits` > 1: partial
// rows in part_acc / part_ml, to be merged by hb_attention_merge.
extern "C" int hb_attention_portions(const float* q, const float* k_pages, const float* v_pages, const int* block_table,
                                     int table_stride, const int* cu_seqlens, const int* positions, float* out, int n_seqs,
                                     int max_new, int nh, int nkv, int hd, int page_size, int chunk, int window, int keep,
                                     float scale, int sink, float softcap, const float* slopes, const float* sink_values,
                                     int splits, float* part_acc, float* part_ml, cudaStream_t stream) {
  if (!q || !k_pages || !v_pages || !block_table || !cu_seqlens || !positions || !out || splits < 1 ||
      (splits > 1 && (!part_acc || !part_ml)))
    return HB_ERR_BAD_ARG;
  if (n_seqs < 0 || max_new < 0 || nh <= 0 || nkv <= 0 || nh % nkv || page_size <= 0 || table_stride <= 0 || chunk < 0 ||
      window < 0 || keep < 0)
    return HB_ERR_BAD_ARG;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k_pages) | reinterpret_cast<uintptr_t>(v_pages) |
       reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(part_acc) | reinterpret_cast<uintptr_t>(part_ml)) & 15)
    return HB_ERR_UNSUPPORTED;
  if (nkv > 65535 || (long long)n_seqs * splits > 65535) return HB_ERR_UNSUPPORTED;
  if (n_seqs == 0 || max_new == 0) return HB_OK;
  const PortionArgs a = {q, k_pages, v_pages, block_table, table_stride, cu_seqlens, positions, out, nh, nkv, page_size, chunk,
                         window, keep, scale, sink, softcap, slopes, sink_values, splits, part_acc, part_ml};
  switch (hd) {
    case 16: return launch_portions<1>(a, max_new, n_seqs, stream);
    case 32: return launch_portions<2>(a, max_new, n_seqs, stream);
    case 48: return launch_portions<3>(a, max_new, n_seqs, stream);
    case 64: return launch_portions<4>(a, max_new, n_seqs, stream);
    case 80: return launch_portions<5>(a, max_new, n_seqs, stream);
    case 96: return launch_portions<6>(a, max_new, n_seqs, stream);
    case 112: return launch_portions<7>(a, max_new, n_seqs, stream);
    case 128: return launch_portions<8>(a, max_new, n_seqs, stream);
    case 192: return launch_portions<12>(a, max_new, n_seqs, stream);
    default: return HB_ERR_UNSUPPORTED;
  }
}
