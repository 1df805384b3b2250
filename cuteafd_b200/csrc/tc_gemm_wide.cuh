// Entry of the wide tcgen05 GEMM (tc_gemm_wide.cu) for the two GEMM entry points that hand it their prompt-sized products.
#pragma once
#include "common.cuh"

struct WideArgs {
  const CUtensorMap* tmX;        // activations, box of 128 rows
  const CUtensorMap* tmW;        // [G] weights, box of 128 rows (the gate's in the two-weight form)
  const CUtensorMap* tmW2;       // [G] up weights (two-weight form)
  const uint8_t* const* sfw;     // [G] FP4 weight scales in the 128 x 4 atom layout
  const uint8_t* const* sfw2;
  const uint8_t* sfx;            // FP4 activation scales, row-major
  const float* sw;               // FP8: weight scales [ceil(N / 128), ceil(K / 128)], activation scales [rows, ceil(K / 128)]
  const float* sx;
  const float* alpha;            // [G] output scale or null
  const float* alpha2;
  const int4* tiles;             // grouped: {group, first row, rows, 0}; null = dense
  const int* n_tiles;
  void* Y;
  const bf16* R;
  int* status;
  uint8_t* q_out;                // FP4 copy of a two-weight product, scales, 1 / global scale of the consumer
  uint8_t* sf_out;
  const float* inv_gs_out;
  int ldsfx, ldsf_out, ldy, rows_total, N, K, epi, act;
  int parts;                     // K in this many parts, each a sum of its own, added in order (dense, no activation; 0 and 1: one sum)
};

// kind: 0 bf16, 1 NVFP4, 2 MXFP4, 3 FP8 with 128-wide fp32 scales.  `max_items`: most token tiles the launch can meet.
int ca_gemm_wide(int kind, bool swiglu, const WideArgs& a, long long max_items, cudaStream_t stream);
