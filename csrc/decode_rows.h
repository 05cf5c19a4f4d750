// Projections of one to four token rows as streams of weight rows (decode_rows.cu).
#pragma once
#include "common.cuh"

constexpr int DR_MAX_ROWS = 4;
constexpr int DR_MAX_PHASES = 4;
enum { DR_PLAIN = 0, DR_SWIGLU = 1, DR_RESID_NORM = 2, DR_QKV_ROPE = 3 };

struct DecodeRowsPhase {
  int M, K, epi;
  int rows, splits, per_row;  // weight rows per block, warps that share a row's k, pieces per warp and row (decode_rows_plan)
  const bf16 *x, *w;
  long long ldx, ldw, ld_out;
  bf16* out;
  int out_f32;                // PLAIN: f32 rows
  const bf16* norm_w;         // RESID_NORM
  int norm_offset;
  const float* in_ssp;        // the input rows owe their RMSNorm scale (null: none); behind the first phase they are the residual's
  int in_parts, in_ld, in_width;
  float in_eps;
  float* out_ssp;             // RESID_NORM: [T][out_ld], one sum per tile of 128 columns
  int out_ld;
  const bf16 *q_w, *k_w, *cos, *sin;  // QKV_ROPE (heads of 128)
  const int *positions, *slots;
  bf16* kv;
  int hq, hkv, rot, page_size, max_pos;
  long long num_slots;
  float qk_eps;
};

struct DecodeRows {
  DecodeRowsPhase ph[DR_MAX_PHASES];
  int nphase, barriers;  // barriers: blocks wait for one another (several phases, or a pass behind the last)
  bf16* residual;
  long long ld_res;
  float* scratch;        // QKV_ROPE: f32 [T, M]
  uint32_t *counters, *status;  // counters: DR_MAX_PHASES + 1 words, zero before and after
  int x_bytes, part_bytes, smem, grid;
};

// Fills in the plan; false: these phases are not for this kernel (row counts, sizes, alignment).
bool decode_rows_plan(DecodeRows& p, int T);
int decode_rows_run(const DecodeRows& p, int T, cudaStream_t stream);
