// The weight-streaming W8A8 product (w8a8_stream.cu) and the output arithmetic it shares with the tiled GEMM.
#pragma once

#include "common.cuh"

namespace mp {

enum : int { STREAM_F16 = 0, STREAM_AFFINE = 1, STREAM_SWIGLU = 2 };

struct StreamParams {
  int M, N, K;                 // activation rows (ungrouped), output columns per expert, bytes of K
  int steps;                   // ceil(K / 128)
  int row_blocks;              // ceil(N / 128)
  int min_share;               // least steps a block is given
  int early_weights;           // 1: only the previous kernel of the stream may still run, and it writes neither the weights
                               //    nor the counts and segments
  const int* counts;           // grouped: rows of every expert ...
  const int* segments;         // ... and where they begin in the activation and output rows
  int experts;
  int rows_per_expert;         // weight rows of an expert
  int up_row_offset;           // SwiGLU: weight rows between a gate row and its up row
  const float* a_scale;
  const float* b_scale;        // indexed like the weight rows
  const __half* bias;
  void* out;                   // f16 [rows][N]
  float* row_absmax;           // SwiGLU: max |h| of every (row, 128 columns), [rows][row_blocks]
  const float* a_zero;
  const int* a_rowsum;
  const float* b_zero;
  const int* b_rowsum;
  uint32_t* tiles;             // workspace: [grid][parts][tokens][128], zero between calls
  int* error_word;
  int x_box;                   // activation rows a load brings: no more than there are (a copy that reaches beyond a small
                               // tensor is slow: 14 us instead of 8 for 24 rows of 4096 in a box of 128)
  const __half* x;             // rows to quantise in the kernel, or null; then ...
  int8_t* qx;                  // ... their codes and ...
  float* qx_scale;             // ... scales are left here
};

// Rows of a linear, rows per expert.  From 9 rows on the tiled kernel is as fast or faster (16 rows, us: 4096x4096 10.6 vs
// 10.0, 28672x4096 26.5 vs 25.4; at 64: 19.5 vs 10.2, 37.3 vs 26.5); at 8 this one is (9.3 vs 9.9, 4096x14336 15.7 vs 17).
constexpr int kStreamMaxRows = 8, kStreamMaxExpertRows = 64;

// Most rows a call (grouped: an expert of it) has; MP_ERR_UNSUPPORTED where the kernel does not apply.
int launch_w8a8_stream(int epi, const void* x_i8, int x_rows, const void* w_i8, int w_rows, StreamParams p, int max_rows,
                       void* workspace, size_t workspace_bytes, cudaStream_t st);

size_t w8a8_stream_workspace_bytes(int epi, int max_rows);

// The tiled asymmetric GEMM (w8a8_gemm.cu); scratch for split-K as for mp_w8a8_gemm_ex, or null.
int w8a8_affine_gemm(const void* qx_u8, const void* x_scale_f32, const void* x_zero_f32, const void* x_rowsum_i32,
                     const void* w_u8, const void* w_scale_f32, const void* w_zero_f32, const void* w_rowsum_i32,
                     const void* bias_f16, void* y_f16, int M, int N, int K, void* workspace, size_t workspace_bytes,
                     int* error_word, cudaStream_t st);

#ifdef __CUDACC__
// acc * s_token * s_channel (+ bias) with every fp32 operation rounded on its own (no contraction into
// an fma), so that every kernel that ends in it produces the same bits.
__device__ __forceinline__ float scaled_output(int acc, float s_token, float s_channel) {
  return __fmul_rn(__fmul_rn(static_cast<float>(acc), s_token), s_channel);
}

// sum (qx - zx)(qw - zw) = acc - zw * sum(qx) - zx * (sum(qw) - K * zw), exactly.  With both zero points in [0, 255] the
// result fits 32 bits (K * 255 * 255 < 2^31 is required), so arithmetic modulo 2^32 gives it whatever the products do;
// zero points beyond the codes (rows on one side of zero) take 64 bits, which cost the tiled GEMM 40 % of its time when
// every element did.
__device__ __forceinline__ float affine_output(int acc, int K, float zx, int sum_x, float zw, int sum_w, float sa, float sb) {
  float t;
  if (zx >= 0.0f && zx <= 255.0f && zw >= 0.0f && zw <= 255.0f) {
    const unsigned int x = static_cast<unsigned int>(zx), w = static_cast<unsigned int>(zw);
    t = static_cast<float>(static_cast<int>(static_cast<unsigned int>(acc) - w * static_cast<unsigned int>(sum_x) -
                                            x * (static_cast<unsigned int>(sum_w) - static_cast<unsigned int>(K) * w)));
  } else {
    const long long x = static_cast<long long>(zx), w = static_cast<long long>(zw);
    t = static_cast<float>(static_cast<long long>(acc) - w * sum_x - x * sum_w + static_cast<long long>(K) * x * w);
  }
  return __fmul_rn(__fmul_rn(t, sa), sb);
}

// the reference rounds gate/up (F.linear output), silu(gate) and the product to fp16; silu in fp32 with the hardware
// exp2 / reciprocal: the result is rounded to fp16 right away, which hides their ~2 ulp fp32 error
__device__ __forceinline__ __half swiglu_f16(int g, int u, float sa, float sg, float su) {
  const __half g16 = f2h(static_cast<float>(g) * sa * sg);
  const __half u16 = f2h(static_cast<float>(u) * sa * su);
  const float gf = h2f(g16);
  const __half s16 = f2h(__fdividef(gf, 1.0f + __expf(-gf)));
  return hmul_t(s16, u16);
}
#endif

}  // namespace mp
