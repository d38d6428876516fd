// Prefill attention on the 5th-generation tensor cores (tcgen05), bfloat16, two query tiles a block. An item is 128 consecutive new
// tokens of a request and one query head; the items of a key head are taken in the order (tile, head), two neighbours a block: most
// pairs are two heads of the same tokens, which read the same keys, and share every K and V tile in shared memory.
//   warps 0..3, 4..7  softmax of item 0 and item 1: thread = row = tensor-memory lane. A row of 128 scores is read at once, masked by
//                     absolute position (causal, chunk, sliding window), its maximum and sum kept in float32; P goes back as
//                     bfloat16 over the first half of its own S, and the P V product takes it from there.
//   warp 8            TMA loads: both Q tiles, then K and V tiles of 128 keys in turn through one ring, a box per page.
//   warp 9            issues the products, tile after tile: O0 += P0 V, S0 = Q0 K^T of the next tile, then the same of item 1. While
//                     one item's softmax runs, the tensor cores have the other's two products.
// S and O of both items take all of tensor memory, so one block lives on an SM; when a work's loads are under way, the block takes the
// next one that has not started (cluster launch control), and its Q and first K arrive while the last tiles of this one are worked at.
//
// Measured (B200, one tile a block and two blocks an SM / this, us): 2,048 tokens of 40 heads of 128 on 8 69.3 / 44.7, 4,096 205 / 141,
// 1,024 behind 16,384 424 / 336, 600 beside 700 behind 300 and 400 behind 100 49 / 35, 2,048 behind 8,192 in a window of 1,024 92 / 61,
// 24 heads on 24 49 / 37. Short launches whose last 128 keys are half empty are a block's latency and stay one tile a block
// (ops.prefill_one_tile).
// What bounds it: a pair of 128-key tiles takes 3,000 cycles where its products take 2,048 and its exponentials, 16 a cycle, as many:
// a chain of softmax (1,550), the last 32 keys' P V and Q K^T (640) and the hand-overs between them (about 350 from the last
// product to the softmax's first load, 200 back). What mattered on the way there, in us for 256 tokens behind 16,384: one lane that
// walked the products' loop alone 285, the warp together 231; waits that vote over each lane's own loop 235, over one try 230; P V
// begun before the last 32 keys of P are there 215 (64 keys: the same). Two warps that issue the products, one an item, 284: both
// items then wait for their products at the same time. Rows stored by the lane that holds them, 32 lines an instruction: 2.5 us a
// pair, by fours of lanes 1.4.
// Keys are multiplied in steps of 16, those that any row of an item reads: what the pool holds on pages given back reaches no row, rows
// behind the request's end are cleared, and a value that is not finite reaches rows of its request that come before it where a step of
// theirs ends behind it (with one tile a block: where their tile did).
// Every mbarrier wait is bounded; on a time-out a code goes to `status` and the block leaves through the common exit.
#include <cuda.h>
#include <cuda_bf16.h>
#include <stdint.h>

#include "api.h"
#include "attention_prefill_pair.h"
#include "common.cuh"
#include "tc.cuh"

namespace {

constexpr int BQ = 128;          // query rows of an item (UMMA M)
constexpr int BK = 128;          // key positions of a tile
constexpr int EARLY = 96;        // of them that the P V product starts with, before the rest of P is there
constexpr int THREADS = 384;     // three warpgroups: of 208, 208 and 88 registers a thread

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// The largest of a row's scores, in four chains of pairs (a maximum takes three operands).
__device__ __forceinline__ float row_max(const float (&v)[BK]) {
  float top[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
  for (int i = 0; i < BK; i += 8)
#pragma unroll
    for (int c = 0; c < 4; ++c) top[c] = fmaxf(fmaxf(top[c], v[i + 2 * c]), v[i + 2 * c + 1]);
  return fmaxf(fmaxf(top[0], top[1]), fmaxf(top[2], top[3]));
}

// An item: its first token, how many there are, the head, the first and last position, the first key that any row reads, its key tiles
// [begin, end).
struct Item {
  int tok0, n_valid, head, p_first, p_last, first, begin, end;
};

// What a block works at: two items (the second may have no tokens), their key tiles in one run, the last position.
struct Work {
  Item x[2];
  int there, begin, end, p_end, seq, kvh, piece;
};

template <int HD>
struct Layout {
  static constexpr int DBLK = HD / 64;                         // 64-element blocks of a row
  static constexpr int QBYTES = BQ * HD * 2, KBYTES = BK * HD * 2, BLOCK = BK * 128;
  static constexpr int STAGES = HD == 128 ? 5 : 8;
  static constexpr int OTHER = 512;                            // barriers and works
  static constexpr size_t SMEM = 2 * (size_t)QBYTES + STAGES * (size_t)KBYTES + OTHER;
};

__device__ __forceinline__ int first_visible(const PrefillPairArgs& a, int pos) {
  int lo = 0;
  if (a.chunk > 0) lo = (pos / a.chunk) * a.chunk;
  if (a.window > 0 && pos - a.window + 1 > lo) lo = pos - a.window + 1;
  return lo;
}

// The work of block (bx, by, bz) of the grid; false if there is none. A row that a share of the keys leaves out weighs nothing in
// the merge: such an item has tokens and no tiles.
__device__ __forceinline__ bool work_of(const PrefillPairArgs& a, int bx, int by, int bz, Work& w) {
  const int group = a.nh / a.nkv, seq_begin = a.cu_seqlens[by], n_new = a.cu_seqlens[by + 1] - seq_begin;
  const int items = (n_new + BQ - 1) / BQ * group, first = 2 * ((items + 1) / 2 - 1 - bz);   // a request's last tokens first
  if (n_new <= 0 || first < 0) return false;
  const bool left_out = a.skip_single && n_new == 1;
  if (left_out && a.key_splits == 1) return false;
  w.there = 1;
  w.seq = by;
  w.kvh = bx % a.nkv;
  w.piece = bx / a.nkv;
  const int p0 = a.positions[seq_begin];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    Item& x = w.x[k];
    const bool in = first + k < items;
    const int t = in ? (first + k) / group : 0;
    x.head = w.kvh * group + (first + k) % group;
    x.tok0 = seq_begin + t * BQ;
    x.n_valid = in ? min(BQ, n_new - t * BQ) : 0;
    x.p_first = p0 + t * BQ;
    x.p_last = x.p_first + x.n_valid - 1;
    x.first = first_visible(a, x.p_first);
    x.begin = x.first / BK;
    x.end = in ? x.p_last / BK + 1 : x.begin;
  }
  // neighbours in tokens, so what they read is one run
  w.begin = w.x[0].begin;
  w.end = left_out ? w.begin : max(w.x[0].end, w.x[1].end);
  w.p_end = max(w.x[0].p_last, w.x[1].p_last);
  if (a.key_splits > 1) {                                      // this block's share of it
    const int share = (w.end - w.begin + a.key_splits - 1) / a.key_splits;
    w.begin += w.piece * share;
    w.end = max(min(w.end, w.begin + share), w.begin);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      w.x[k].begin = max(w.x[k].begin, w.begin);
      w.x[k].end = max(min(w.x[k].end, w.end), w.x[k].begin);
    }
  }
  return true;
}

template <int HD>
__global__ void __launch_bounds__(THREADS, 1)
attn_prefill_pair_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                         const __grid_constant__ CUtensorMap map_v, const PrefillPairArgs a) {
  using L = Layout<HD>;
  constexpr int STAGES = L::STAGES, DBLK = L::DBLK;
  extern __shared__ __align__(1024) uint8_t smem[];
  if ((tc::smem_u32(smem) & 1023u) != 0) {
    if (threadIdx.x == 0) atomicExch(a.status, 51);
    return;
  }
  uint8_t* q_s = smem;                                         // two tiles
  uint8_t* ring = q_s + 2 * L::QBYTES;                         // K V K V ...
  uint8_t* other = ring + STAGES * L::KBYTES;
  uint4* answer = reinterpret_cast<uint4*>(other);
  Work* works = reinterpret_cast<Work*>(other + 16);           // 2
  uint64_t* bars = reinterpret_cast<uint64_t*>(other + 16 + 2 * sizeof(Work));
  uint64_t* full = bars;                                       // STAGES
  uint64_t* empty = full + STAGES;                             // STAGES
  uint64_t* q_full = empty + STAGES;                           // 1: both Q tiles
  uint64_t* q_empty = q_full + 1;                              // 1: a work's last S = Q K^T through
  uint64_t* s_full = q_empty + 1;                              // 2: S there, and every product before it through
  uint64_t* p_ready = s_full + 2;                              // 2: 96 keys of P there, S read, O rescaled, the O of the work before read
  uint64_t* p_rest = p_ready + 2;                              // 2: all of P there
  uint64_t* o_done = p_rest + 2;                               // 2: a work's last P V through
  uint64_t* tail = o_done + 2;                                 // 1: a work's last V tile, before its rows past the end are cleared
  uint64_t* work_full = tail + 1;                              // 2
  uint64_t* work_read = work_full + 2;                         // 2
  uint64_t* answered = work_read + 2;                          // 1
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(answered + 1);
  static_assert(sizeof(Work) % 4 == 0 && 16 + 2 * sizeof(Work) + (2 * STAGES + 16) * 8 + 4 <= L::OTHER, "barriers and works fit");

  const int warp = tc::uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  // What a block does first hangs together in a chain of memory latencies: the barriers, the tensor memory, the maps and the first
  // work's numbers are fetched side by side.
  if (warp == 11) {
    const int barriers = reinterpret_cast<uint64_t*>(tmem_slot) - bars;
    for (int i = lane; i < barriers; i += 32) {
      uint64_t* bar = bars + i;
      tc::mbar_init(bar, bar == p_ready || bar == p_ready + 1 || bar == p_rest || bar == p_rest + 1 ? 4
                         : bar == work_read || bar == work_read + 1                                  ? 9
                                                                                                     : 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  } else if (warp == 10 && lane < 3) {
    tc::prefetch_map(lane == 0 ? &map_q : lane == 1 ? &map_k : &map_v);
  }
  Work job = {};                                               // of the loads' warp
  bool some = true;
  int page = -1;                                               // this lane's of the tile that is loaded next
  // a lane a box of K or V: 64 elements of a page's rows (or of 64 of them)
  const int box = lane / DBLK, box_col = lane % DBLK * 64;
  const bool boxes = box < BK / a.box_rows;
  auto page_of = [&](int j) {
    const int key0 = j * BK + box * a.box_rows;
    return boxes && key0 <= job.p_end ? a.block_table[(size_t)job.seq * a.table_stride + key0 / a.page_size] : -1;
  };
  if (warp == 8) {
    if (!work_of(a, blockIdx.x, blockIdx.y, blockIdx.z, job)) job.there = 0;
    else if (job.begin < job.end) page = page_of(job.begin);
  }
  if (warp == 9) tc::alloc(tmem_slot, 512);
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t tmem_s[2] = {tmem, tmem + BK}, tmem_o[2] = {tmem + 2 * BK, tmem + 2 * BK + HD};
  if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
    if (warp == 8) {                            // ---- which work, and the TMA loads
      bool ok = true;
      int n = 0, queries = 0, bx = 0, by = 0, bz = 0, asked = 0, tails = 0;
      // When a work's loads are under way, the next block of the grid that has not started becomes this block's next work.
      auto bid = [&]() {
        if (lane == 0) {
          tc::mbar_expect_tx(answered, 16);
          asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];"
                       ::"r"(tc::smem_u32(answer)), "r"(tc::smem_u32(answered)) : "memory");
        }
        __syncwarp();
        if (!tc::mbar_wait_warp(answered, asked & 1)) {
          if (lane == 0) atomicExch(a.status, 67);
          ok = false;
          return;
        }
        ++asked;
        uint32_t got;
        asm volatile(
            "{\n.reg .b128 h;\n.reg .pred p;\n"
            "ld.shared.b128 h, [%4];\n"
            "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\n"
            "selp.u32 %3, 1, 0, p;\n"
            "mov.u32 %0, 0;\nmov.u32 %1, 0;\nmov.u32 %2, 0;\n"
            "@p clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {%0, %1, %2, _}, h;\n}"
            : "=r"(bx), "=r"(by), "=r"(bz), "=r"(got) : "r"(tc::smem_u32(answer)) : "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        some = got != 0;
        if (!some || !work_of(a, bx, by, bz, job)) job.there = 0;
        else if (job.begin < job.end) page = page_of(job.begin);
      };
      for (int w = 0; ok; ) {
        if (!job.there && some) {               // nothing in this block of the grid
          bid();
          continue;
        }
        const bool loads = job.there && job.begin < job.end;
        // (every work's Q phase is waited for, also of those without keys: the barrier is never two phases on)
        if ((w >= 2 && !tc::mbar_wait_warp(&work_read[w & 1], ((w >> 1) - 1) & 1)) ||
            (w >= 1 && !tc::mbar_wait_warp(q_empty, (w - 1) & 1))) {
          if (lane == 0) atomicExch(a.status, 65);
          ok = false;
          break;
        }
        if (lane == 0 && loads) {
          const bool two = job.x[1].n_valid > 0;
          tc::mbar_expect_tx(q_full, (two ? 2 : 1) * L::QBYTES);
          for (int d = 0; d < DBLK; ++d) {
            tc::tma_load_2d(q_s + d * L::BLOCK, &map_q, job.x[0].head * HD + d * 64, job.x[0].tok0, q_full);
            if (two) tc::tma_load_2d(q_s + L::QBYTES + d * L::BLOCK, &map_q, job.x[1].head * HD + d * 64, job.x[1].tok0, q_full);
          }
        }
        queries += loads;
        auto publish = [&]() {                  // to the products' and the softmax's warps
          if (lane == 0) {
            works[w & 1] = job;
            tc::mbar_arrive(&work_full[w & 1]);
          }
          ++w;
        };
        if (!loads) publish();
        if (!some) break;
        if (loads) {
          // Rows of V past the last position meet weights of zero in their step of 16 keys, and may hold anything: they are cleared.
          const int clear = (job.p_end + 1) % 16 != 0 && job.p_end / BK == job.end - 1 ? job.p_end % BK + 1 : 0;
          for (int j = job.begin; j < job.end && ok; ++j) {
            const int next = j + 1 < job.end ? page_of(j + 1) : -1;
            // keys past the last position, or on pages given back, are read by no row: any row will do
            const int row = page >= 0 ? (page * a.nkv + job.kvh) * a.page_size + (j * BK + box * a.box_rows) % a.page_size : 0;
            for (int v = 0; v < 2 && ok; ++v, ++n) {
              const int s = n % STAGES, use = n / STAGES;
              uint8_t* dst = ring + s * L::KBYTES;
              if (use >= 1 && !tc::mbar_wait_warp(&empty[s], (use - 1) & 1)) {
                if (lane == 0) atomicExch(a.status, 52);
                ok = false;
                break;
              }
              const bool last = v && j + 1 == job.end && clear;
              uint64_t* bar = last ? tail : &full[s];
              if (lane == 0) tc::mbar_expect_tx(bar, L::KBYTES);
              __syncwarp();
              if (boxes) tc::tma_load_2d(dst + box_col / 64 * L::BLOCK + box * a.box_rows * 128, v ? &map_v : &map_k, box_col, row, bar);
              if (v == 0 && j == job.begin) publish();       // the first K is under way
              if (last) {
                if (!tc::mbar_wait_warp(tail, tails & 1)) {
                  if (lane == 0) atomicExch(a.status, 53);
                  ok = false;
                }
                ++tails;
                const int to = (clear + 15) / 16 * 16;
                for (int e = lane; e < (to - clear) * DBLK * 8; e += 32) {
                  const int r = clear + e / (DBLK * 8), at = e % (DBLK * 8);
                  *reinterpret_cast<uint4*>(dst + at / 8 * L::BLOCK + r * 128 + at % 8 * 16) = make_uint4(0, 0, 0, 0);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&full[s]);
              }
            }
            page = next;
          }
        }
        if (ok) bid();
      }
      // nothing reaches for the block's memory when it ends: the commits on the last stages have arrived, which come behind their copies;
      // where a wait ran out they may never come, and the copies on their way are waited for
      if (!ok && queries > 0) tc::mbar_wait_warp(q_full, (queries - 1) & 1);
      for (int i = max(0, n - STAGES); i < n; ++i) tc::mbar_wait_warp(ok ? &empty[i % STAGES] : &full[i % STAGES], (i / STAGES) & 1);
    } else if (warp == 9) {                     // ---- the products: the whole warp walks, one lane issues
      constexpr uint32_t idesc_qk = tc::idesc_bf16(BQ, BK, false);
      constexpr uint32_t idesc_pv = tc::idesc_bf16(BQ, HD, true);
      const uint32_t q_addr = tc::smem_u32(q_s), ring_addr = tc::smem_u32(ring);
      bool ok = true;
      int stage = 0, turn = 0, loads = 0, phase[2] = {0, 0};    // the ring's; Q tiles taken; P tiles taken of either item
      auto wait = [&](uint64_t* bar, int parity, int code) {
        if (!tc::mbar_wait_warp(bar, parity)) {
          if (lane == 0) atomicExch(a.status, code);
          ok = false;
        }
      };
      auto advance = [&]() {
        if (++stage == STAGES) { stage = 0; turn ^= 1; }
      };
      for (int w = 0; ok; ++w) {
        wait(&work_full[w & 1], (w >> 1) & 1, 68);
        if (!ok) break;
        const Work& job = works[w & 1];
        const int there = tc::uniform(job.there), begin = tc::uniform(job.begin), end = tc::uniform(job.end);
        int x_begin[2], x_end[2], x_first[2], x_last[2];        // first key read; last position
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          x_begin[i] = tc::uniform(job.x[i].begin);
          x_end[i] = tc::uniform(job.x[i].end);
          x_first[i] = tc::uniform(job.x[i].first);
          x_last[i] = tc::uniform(job.x[i].p_last);
        }
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&work_read[w & 1]);
        if (!there) break;
        if (begin == end) {
          if (lane == 0) tc::mbar_arrive(q_empty);
          continue;
        }
        wait(q_full, loads++ & 1, 54);
        if (!ok) break;
        // S_i = Q_i K^T; the K tile is in the ring's stage
        auto scores = [&](uint32_t mine, int i) {
          const uint64_t q = tc::desc_kmajor(q_addr + i * L::QBYTES), k = tc::desc_kmajor(ring_addr + stage * L::KBYTES);
#pragma unroll
          for (int t = 0; t < HD / 16; ++t) {
            const uint32_t at = ((t / 4) * L::BLOCK + (t % 4) * 32) >> 4;
            tc::mma_if(mine, tmem_s[i], q + at, k + at, idesc_qk, t != 0);
          }
          tc::commit_if(mine, &s_full[i]);
        };
        const uint32_t mine = tc::elect_one();
        for (int j = begin - 1; j < end; ++j) {
          const int v_stage = stage;
          if (j >= begin) {
            wait(&full[stage], turn, 56);       // V of this tile
            advance();
          }
          if (j + 1 < end) wait(&full[stage], turn, 57);        // K of the next
          if (!ok) break;
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            if (x_begin[i] <= j && j < x_end[i]) {
              // steps of 16 keys that any row of the item reads
              const int from = max(0, x_first[i] - j * BK) / 16, to = min(BK - 1, x_last[i] - j * BK) / 16;
              const uint64_t v = tc::desc_mnmajor(ring_addr + v_stage * L::KBYTES, L::BLOCK);
              const uint32_t more = j > x_begin[i];
              const bool whole = from == 0 && to == BK / 16 - 1;
              wait(&p_ready[i], phase[i] & 1, 58 + i);
              if (!ok) break;
              tc::fence_after();
              if (whole) {
#pragma unroll
                for (int t = 0; t < EARLY / 16; ++t)
                  tc::mma_a_tmem_if(mine, tmem_o[i], tmem_s[i] + t * 8, v + t * (2048 >> 4), idesc_pv, t == 0 ? more : 1u);
              }
              wait(&p_rest[i], phase[i] & 1, 70 + i);
              if (!ok) break;
              tc::fence_after();
              if (whole) {
#pragma unroll
                for (int t = EARLY / 16; t < BK / 16; ++t)
                  tc::mma_a_tmem_if(mine, tmem_o[i], tmem_s[i] + t * 8, v + t * (2048 >> 4), idesc_pv, 1u);
              } else {
#pragma unroll 1
                for (int t = from; t <= to; ++t)
                  tc::mma_a_tmem_if(mine, tmem_o[i], tmem_s[i] + t * 8, v + t * (2048 >> 4), idesc_pv, more || t > from);
              }
              if (j + 1 == x_end[i]) tc::commit_if(mine, &o_done[i]);
              ++phase[i];
            }
            if (i == 1 && j >= begin) tc::commit_if(mine, &empty[v_stage]);
            if (x_begin[i] <= j + 1 && j + 1 < x_end[i]) scores(mine, i);
          }
          if (!ok) break;
          if (j + 1 < end) {
            tc::commit_if(mine, &empty[stage]);
            if (j + 2 == end) tc::commit_if(mine, q_empty);
            advance();
          }
        }
      }
    }
  } else {                                      // ---- softmax
    asm volatile("setmaxnreg.inc.sync.aligned.u32 208;");
    const int i = warp >> 2;
    const int r = (warp & 3) * 32 + lane;
    const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t s_addr = (i ? tmem_s[1] : tmem_s[0]) + lane_addr, o_addr = (i ? tmem_o[1] : tmem_o[0]) + lane_addr;
    bool ok = true;
    int phase = 0, done = 0;                    // tiles and works of this item so far
    for (int w = 0; ok; ++w) {
      if (!tc::mbar_wait_warp(&work_full[w & 1], (w >> 1) & 1)) {
        if (lane == 0) atomicExch(a.status, 64);
        break;
      }
      const Work& job = works[w & 1];
      const bool there = job.there;
      const Item x = job.x[i];
      const int piece = job.piece;
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&work_read[w & 1]);
      if (!there) break;
      const bool row_ok = r < x.n_valid;
      const int pos = x.p_first + r, warp_first = x.p_first + (warp & 3) * 32;
      const int lo = first_visible(a, pos), warp_lo = first_visible(a, warp_first + 31);
      // rows without a token start above every score, so they never move the maximum
      float m = row_ok ? -INFINITY : INFINITY, l = 0.f;
      for (int j = x.begin; j < x.end; ++j, ++phase) {
        if (!tc::mbar_wait_warp(&s_full[i], phase & 1)) {
          if (lane == 0) atomicExch(a.status, 60 + i);
          ok = false;
          break;
        }
        tc::fence_after();
        const int key_base = j * BK;
        float sv[BK];
        {
          uint32_t raw[4][32];
#pragma unroll
          for (int c = 0; c < 4; ++c) tc::ld32_nowait(s_addr + 32 * c, raw[c]);
          tc::wait_ld();
#pragma unroll
          for (int c = 0; c < BK; ++c) sv[c] = __uint_as_float(raw[c / 32][c % 32]);
        }
        // a tile that every row of this warp sees whole needs no masks (rows past the portion's end are not written)
        if (key_base + BK - 1 > warp_first) {
          const int most = row_ok ? pos - key_base : -1;
#pragma unroll
          for (int c = 0; c < BK; ++c) sv[c] = c <= most ? sv[c] : -INFINITY;
        }
        if (key_base < warp_lo) {
          const int least = lo - key_base;
#pragma unroll
          for (int c = 0; c < BK; ++c) sv[c] = c >= least ? sv[c] : -INFINITY;
        }
        const float mx = fmaxf(m, row_max(sv) * a.scale_log2);           // the scale is positive
        // The exponentials are taken against `m`, which follows the maximum only when a row of the warp has grown by more than 2^8:
        // P stays below 256 and most tiles leave O as it is. A row that has seen nothing yet has nothing to move to.
        const bool move = __any_sync(0xffffffffu, mx > m + 8.f);
        float corr = 1.f;
        if (move) {
          corr = m == -INFINITY ? 0.f : fast_exp2(m - mx);
          m = mx;
          if (j > x.begin) {                      // S came after the product of the tile before: O stands still
#pragma unroll 1
            for (int c = 0; c < HD; c += 32) {
              float o[32];
              tc::ld32(o_addr + c, o);
#pragma unroll
              for (int e = 0; e < 32; ++e) o[e] *= corr;
              tc::st32(o_addr + c, o);
            }
          }
        }
        const float base = m == -INFINITY ? 0.f : -m;                    // of a row that has seen nothing: 2^-inf = 0 all the same
        const float2 scale2 = make_float2(a.scale_log2, a.scale_log2), base2 = make_float2(base, base);
        float2 part[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          uint32_t packed[16];
#pragma unroll
          for (int c = 0; c < 16; ++c) {
            const int at = 32 * h + 2 * c;
            const float2 y = __ffma2_rn(make_float2(sv[at], sv[at + 1]), scale2, base2);
            const float2 p = make_float2(fast_exp2(y.x), fast_exp2(y.y));
            part[c & 1] = __fadd2_rn(part[c & 1], p);
            __nv_bfloat162 hh = __floats2bfloat162_rn(p.x, p.y);
            packed[c] = *reinterpret_cast<uint32_t*>(&hh);
          }
          tc::st16_nowait(s_addr + 16 * h, packed);
          if (32 * (h + 1) == EARLY || 32 * (h + 1) == BK) {
            tc::wait_st();
            tc::fence_before();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(32 * (h + 1) == BK ? &p_rest[i] : &p_ready[i]);
          }
        }
        const float2 both = __fadd2_rn(part[0], part[1]);
        l = l * corr + (both.x + both.y);
      }
      if (!ok) break;
      if (x.begin == x.end) {
        if (row_ok && a.key_splits > 1) {
          float* ml = a.part_ml + (((size_t)(x.tok0 + r) * a.nh + x.head) * a.key_splits + piece) * 2;
          ml[0] = -INFINITY;
          ml[1] = 0.f;
        }
        continue;
      }
      if (!tc::mbar_wait_warp(&o_done[i], done++ & 1)) {
        if (lane == 0) atomicExch(a.status, 62 + i);
        break;
      }
      tc::fence_after();
      if (a.key_splits > 1) {
        // this share of the keys only: the row as it is, with its maximum and sum, for the merge
        const size_t at = ((size_t)(x.tok0 + r) * a.nh + x.head) * a.key_splits + piece;
        if (row_ok) {
          a.part_ml[at * 2] = m == -INFINITY ? -INFINITY : m * 0.6931471805599453f;
          a.part_ml[at * 2 + 1] = l;
        }
#pragma unroll 1
        for (int c = 0; c < HD; c += 32) {
          uint32_t o[32];
          tc::ld32_nowait(o_addr + c, o);
          tc::wait_ld();
#pragma unroll
          for (int h = 0; h < 32; h += 16) {
            uint4 v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = make_uint4(o[h + 4 * e], o[h + 4 * e + 1], o[h + 4 * e + 2], o[h + 4 * e + 3]);
            tc::trade_rows(v, lane);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int to = (r & ~3) + e;
              if (to < x.n_valid)
                *reinterpret_cast<uint4*>(a.part_acc + (((size_t)(x.tok0 + to) * a.nh + x.head) * a.key_splits + piece) * HD + c + h +
                                          4 * (lane & 3)) = v[e];
            }
          }
        }
      } else {
        if (a.sink && l > 0.f) l += exp2f((a.sink_values ? a.sink_values[x.head] * 1.4426950408889634f : 0.f) - m);
        const float inv = l > 0.f ? 1.f / l : 0.f;
#pragma unroll 1
        for (int c = 0; c < HD; c += 32) {
          uint32_t o[32];
          tc::ld32_nowait(o_addr + c, o);
          tc::wait_ld();
          uint4 v[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            uint32_t u[4];
#pragma unroll
            for (int f = 0; f < 4; ++f) {
              __nv_bfloat162 hh = __floats2bfloat162_rn(__uint_as_float(o[8 * e + 2 * f]) * inv, __uint_as_float(o[8 * e + 2 * f + 1]) * inv);
              u[f] = *reinterpret_cast<uint32_t*>(&hh);
            }
            v[e] = make_uint4(u[0], u[1], u[2], u[3]);
          }
          tc::trade_rows(v, lane);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int to = (r & ~3) + e;
            if (to < x.n_valid)
              *reinterpret_cast<uint4*>(a.out + ((size_t)(x.tok0 + to) * a.nh + x.head) * HD + c + 8 * (lane & 3)) = v[e];
          }
        }
      }
    }
  }
  tc::fence_before();
  __syncthreads();
  if (warp == 9) {
    tc::fence_after();
    tc::dealloc(tmem, 512);
  }
}

template <int HD>
int launch(const void* q, const void* k_pages, const void* v_pages, const PrefillPairArgs& a, int n_tokens, long long pool_rows,
           int n_seqs, int max_new, cudaStream_t stream) {
  CUtensorMap mq, mk, mv;
  if (!tc::make_map_bf16(&mq, q, (uint64_t)n_tokens, (uint64_t)a.nh * HD, BQ) ||
      !tc::make_map_bf16(&mk, k_pages, (uint64_t)pool_rows, HD, a.box_rows) ||
      !tc::make_map_bf16(&mv, v_pages, (uint64_t)pool_rows, HD, a.box_rows))
    return HB_ERR_UNSUPPORTED;
  const size_t smem = Layout<HD>::SMEM;
  cudaError_t e = cudaFuncSetAttribute(attn_prefill_pair_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  const long long pairs = ((long long)((max_new + BQ - 1) / BQ) * (a.nh / a.nkv) + 1) / 2;
  if (pairs > 65535 || n_seqs > 65535 || (long long)a.nkv * a.key_splits > 0x7fffffffLL) return HB_ERR_UNSUPPORTED;
  attn_prefill_pair_kernel<HD><<<dim3(a.nkv * a.key_splits, n_seqs, (unsigned)pairs), THREADS, smem, stream>>>(mq, mk, mv, a);
  HB_LAUNCH_CHECK();
  return HB_OK;
}

}  // namespace

int hb_prefill_pair_launch(const void* q, const void* k_pages, const void* v_pages, const PrefillPairArgs& a, int n_tokens,
                           long long pool_rows, int n_seqs, int max_new, int hd, cudaStream_t stream) {
  if (hd == 128) return launch<128>(q, k_pages, v_pages, a, n_tokens, pool_rows, n_seqs, max_new, stream);
  if (hd == 64) return launch<64>(q, k_pages, v_pages, a, n_tokens, pool_rows, n_seqs, max_new, stream);
  return HB_ERR_UNSUPPORTED;
}
