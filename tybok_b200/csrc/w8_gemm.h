// What the two W8 GEMM kernels (w8_gemm.cu, w8_gemm_pair.cu) share: epilogue codes and the call description.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace tb {

// EPI_GEGLU_PACKED: one weight matrix whose 128-row tiles hold 64 gate rows followed by the 64
// up rows of the same channels; the tile yields 64 output channels gelu(gate) * up.
// EPI_QKV_ROPE: packed q/k/v projection whose 128-row tiles hold 64 head dimensions followed by
// their rotate-half partners (d, d + D/2); the tile is rotated and stored as q rows / cache rows.
enum : int { EPI_NONE = 0, EPI_GELU = 1, EPI_RESIDUAL = 2, EPI_GEGLU = 3, EPI_GEGLU_PACKED = 4, EPI_QKV_ROPE = 5 };

struct RopeEpi {
  const int* pos;              // [M] position of every token row
  const __nv_bfloat16* cos;    // [max_pos][D]
  const __nv_bfloat16* sin;
  __nv_bfloat16* q;            // [M][H*D]
  __nv_bfloat16* kcache;       // [B][G][Lcap][D]
  __nv_bfloat16* vcache;
  int L, H, G, D, Lcap, key_off;
};

// One GEMM call as the C entry points describe it (arguments already checked).
struct GemmCall {
  const uint8_t* planes;   // [np][M][K]
  int np;                  // 3 e5m2 planes (fixed exponent shift) or 2 e4m3 planes with row_scale
  const float* row_scale;  // [M], two-plane form
  const void* w0;          // [N][K] e4m3 (packed forms: the interleaved matrix)
  const void* w1;          // second matrix of EPI_GEGLU, else NULL
  const float* s0;
  const float* s1;
  const __nv_bfloat16* bias;
  __nv_bfloat16* y;
  long long ldy;
  uint8_t* y_planes;
  int M, N, K, n_out;
  int epi;
  const __nv_bfloat16* res;
  long long ldres;
  const void* gate;
  long long ldgate;
  int rows_per_gate, gate_bf16;
  float out_scale, plane_scale;
  const RopeEpi* rope;
  bool split;              // K over the pairs of a cluster (EPI_NONE, EPI_GELU, EPI_RESIDUAL)
  int* status;
  cudaStream_t stream;
};

// True when w8_gemm_pair.cu is the faster kernel for this shape (`nw` weight matrices of N rows).
bool gemm_pair_suits(int M, int N, int nw, int np);
// Estimated SM clocks of the split form (a cluster of pairs per tile) for one wave of clusters; negative: does not apply.
double gemm_pair_split_cost(int M, int N, int K, int np);
int launch_gemm_pair(const GemmCall& c);

}  // namespace tb
