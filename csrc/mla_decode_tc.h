// Absorbed latent attention on tcgen05 (mla_decode_tc.cu), called by pg_latent_attention.
#pragma once
#include "common.cuh"

struct MlaDecodeTc {
  const bf16 *q_abs, *q_pe, *latent;  // queries and outputs by strides in elements; cache [pages, page_size, 512 + r]
  bf16* out;
  long long q_tok, q_head, pe_tok, pe_head, o_tok, o_head;
  const float *cos, *sin;  // turn the q_pe columns (null: they come rotated)
  int max_pos, window;
  const int *q_indptr, *kv_lens, *table, *unit_seq;
  int table_stride, first_row, tokens, heads, page_size, splits;
  float scale_log2;
  float *part_o, *part_lse;
  const float* sink;
  const bf16* gate;
  long long ld_gate;
  uint32_t* status;
};

int mla_decode_tc(const MlaDecodeTc& p, int r, long long pages, cudaStream_t stream);
