// The tcgen05 prefill attention of plain softmax rows, two query tiles a block (attention_prefill_pair.cu).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

struct PrefillPairArgs {
  const int* block_table;
  const int* cu_seqlens;
  const int* positions;
  __nv_bfloat16* out;
  int* status;
  int table_stride, nh, nkv, page_size, chunk, window, skip_single, box_rows;
  float scale_log2;          // softmax scale * log2(e)
  // With key_splits > 1 that many blocks share the key tiles of every pair of items; a block leaves its rows unnormalised in
  // part_acc [row][split][head_dim] with (maximum, sum) in part_ml [row][split][2], and hb_attention_merge combines them.
  int key_splits;
  float* part_acc;
  float* part_ml;
  int sink;                  // 1: the denominator has one more term, e^0, or e^sink_values[head]
  const float* sink_values;
};

// head_dim 64 or 128; HB_ERR_UNSUPPORTED for others
int hb_prefill_pair_launch(const void* q, const void* k_pages, const void* v_pages, const PrefillPairArgs& a, int n_tokens,
                           long long pool_rows, int n_seqs, int max_new, int hd, cudaStream_t stream);
