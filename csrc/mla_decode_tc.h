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
  int table_stride, first_row, tokens, heads, page_size;
  int splits;  // blocks that the caller would like to share a row's keys: how small the groups of heads may get
  int shared;  // the blocks share all rows' keys evenly, rows cut where need be (0: a block walks one row's keys)
  float scale_log2;
  float *part_o, *part_lse;  // of cut rows: two slots a block, [heads of a group, 512] and [heads of a group]
  int* cuts;                 // a block's last row, where that ends in other blocks' shares: (unit or -1, pieces)
  const float* sink;
  const bf16* gate;
  long long ld_gate;
  uint32_t* status;
};

// part: scratch for cut rows; too little, and no row is cut
int mla_decode_tc(MlaDecodeTc p, int r, long long pages, void* part, long long part_bytes, cudaStream_t stream);
