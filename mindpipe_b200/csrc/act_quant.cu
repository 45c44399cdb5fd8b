// Per-row (token / output channel) symmetric int8 quantisation.
//
// Arithmetic of quantize_activation_per_token_absmax and
// quantize_weight_per_channel_absmax
// (algorithm/quantization/ptq/smoothquant/source/smoothquant/fake_quant.py:10-31)
// with the integer codes kept, which is what npu_dynamic_quant returns at
// acceleration/runtime_patches/vllm_ascend.patch:3950:
//   s    = f16( max(absmax, f16(1e-5)) / 127 )
//   code = rint( f16( x / s ) )         (division in fp32, rounded to fp16 first)
//   fake = f16( code * s )
// The row is read with 128-bit loads, reduced with warp shuffles and kept in
// registers for the rounding step (rows up to 16384 columns), so it is read once.
#include "common.cuh"

namespace mp {

// Quantise eight values held in one 128-bit register group and store the codes and / or the
// fake-quantised values f16(code * s).
__device__ __forceinline__ void emit_codes(const uint4& raw, const RowQuant& rq, int8_t* q8, __half* fake8) {
  if (fake8) {
    uint4 fk;
    const uint2 codes = quant8_pack_fake(raw, rq, fk);
    if (q8) *reinterpret_cast<uint2*>(q8) = codes;
    *reinterpret_cast<uint4*>(fake8) = fk;
  } else if (q8) {
    *reinterpret_cast<uint2*>(q8) = quant8_pack(raw, rq);
  }
}

// One warp per row (many rows of up to 32 * 8 * NV columns): the row is read once with NV independent
// 128-bit loads per lane, reduced with shuffles only, and quantised from registers -- no block-level
// synchronisation at all.
// CODES / FAKE select the outputs at compile time and the rare tiny-scale rows take a rolled loop that
// re-reads the row, so the unrolled body holds one route only (the kernel stays small enough for the
// instruction cache).
template <int NV, bool CODES, bool FAKE>
__global__ void __launch_bounds__(128)
act_quant_warp_kernel(const __half* __restrict__ x, int M, int K, int8_t* __restrict__ q,
                      float* __restrict__ scale, __half* __restrict__ fake) {
  chain_wait();              // programmatic dependent launch: the producer of x has finished
  chain_release();
  const int row = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (row >= M) return;
  const int lane = threadIdx.x & 31;
  const __half* xr = x + (size_t)row * K;
  const int chunks = K >> 3;
  uint4 held[NV];
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int c = lane + v * 32;
    held[v] = c < chunks ? *reinterpret_cast<const uint4*>(xr + c * 8) : make_uint4(0, 0, 0, 0);
  }
  __half2 m2 = __float2half2_rn(0.0f);
#pragma unroll
  for (int v = 0; v < NV; ++v) m2 = absmax8(m2, held[v]);
  const float amax = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(absmax_to_float(m2))));
  const float eps = h2f(f2h(1e-5f));                                   // clamp_(min=1e-5) on an fp16 tensor
  const float sf = h2f(f2h(__fdiv_rn(fmaxf(amax, eps), 127.0f)));      // div_(q_max), rounded to fp16
  RowQuant rq = make_row_quant(sf);
  if (lane == 0 && scale) scale[row] = sf;
  int8_t* qr = CODES ? q + (size_t)row * K : nullptr;
  __half* fr = FAKE ? fake + (size_t)row * K : nullptr;
  if (!rq.packed) {                                   // scale below 2^-14: fp32 route, rolled
#pragma unroll 1
    for (int c = lane; c < chunks; c += 32)
      emit_codes(*reinterpret_cast<const uint4*>(xr + c * 8), rq, CODES ? qr + c * 8 : nullptr,
                 FAKE ? fr + c * 8 : nullptr);
    return;
  }
  rq.packed = true;                                   // lets the compiler drop the other route below
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int c = lane + v * 32;
    if (c >= chunks) continue;
    emit_codes(held[v], rq, CODES ? qr + c * 8 : nullptr, FAKE ? fr + c * 8 : nullptr);
  }
}

template <int NV>
static int launch_act_quant_warp(const __half* x, int M, int K, int8_t* q, float* sc, __half* fk, cudaStream_t st) {
  const unsigned blocks = static_cast<unsigned>((M + 3) / 4);
  if (q && fk) {
    return launch_chained(act_quant_warp_kernel<NV, true, true>, dim3(blocks), dim3(128), 0, st, x, M, K, q, sc, fk);
  } else if (q) {
    return launch_chained(act_quant_warp_kernel<NV, true, false>, dim3(blocks), dim3(128), 0, st, x, M, K, q, sc, fk);
  } else {
    return launch_chained(act_quant_warp_kernel<NV, false, true>, dim3(blocks), dim3(128), 0, st, x, M, K, q, sc, fk);
  }
}

// NV = 128-bit vectors per thread.  NV > 0: the row (K <= THREADS * 8 * NV) is held in
// registers between the abs-max and the rounding step, so global memory is read once;
// NV == 0: any K, second pass re-reads the row (an L1/L2 hit).
template <int THREADS, int NV>
__global__ void __launch_bounds__(THREADS)
act_quant_kernel(const __half* __restrict__ x, int M, int K, int8_t* __restrict__ q,
                 float* __restrict__ scale, __half* __restrict__ fake) {
  chain_wait();
  chain_release();
  __shared__ uint32_t s_red[THREADS / 32];
  const int row = blockIdx.x;
  const __half* xr = x + (size_t)row * K;
  const int chunks = K >> 3;
  constexpr int NREG = NV > 0 ? NV : 1;
  uint4 held[NREG];
  __half2 m2 = __float2half2_rn(0.0f);
  auto absmax_of = [&](const uint4& raw) { m2 = absmax8(m2, raw); };
  if (NV > 0) {
#pragma unroll
    for (int v = 0; v < NREG; ++v) {
      const int c = threadIdx.x + v * THREADS;
      held[v] = c < chunks ? *reinterpret_cast<const uint4*>(xr + c * 8) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int v = 0; v < NREG; ++v) absmax_of(held[v]);
  } else {
    for (int c = threadIdx.x; c < chunks; c += THREADS) absmax_of(*reinterpret_cast<const uint4*>(xr + c * 8));
  }
  // (bit patterns of non-negative numbers order as the numbers do)
  uint32_t top = __reduce_max_sync(0xffffffffu, __float_as_uint(absmax_to_float(m2)));
  if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = top;
  __syncthreads();
  top = __reduce_max_sync(0xffffffffu, (threadIdx.x & 31) < THREADS / 32 ? s_red[threadIdx.x & 31] : 0u);
  const float eps = h2f(f2h(1e-5f));                                                  // clamp_(min=1e-5) on an fp16 tensor
  const float sf = h2f(f2h(__fdiv_rn(fmaxf(__uint_as_float(top), eps), 127.0f)));     // div_(q_max), rounded to fp16
  if (threadIdx.x == 0 && scale) scale[row] = sf;
  const RowQuant rq = make_row_quant(sf);
  auto emit = [&](int c, const uint4& raw) {
    emit_codes(raw, rq, q ? q + (size_t)row * K + c * 8 : nullptr,
               fake ? fake + (size_t)row * K + c * 8 : nullptr);
  };
  if (NV > 0) {
#pragma unroll
    for (int v = 0; v < NREG; ++v) {
      const int c = threadIdx.x + v * THREADS;
      if (c < chunks) emit(c, held[v]);
    }
  } else {
    for (int c = threadIdx.x; c < chunks; c += THREADS) emit(c, *reinterpret_cast<const uint4*>(xr + c * 8));
  }
}

// OmniQuant-style dynamic asymmetric quantisation of each row to unsigned 8-bit codes:
// UniformAffineQuantizer.per_token_dynamic_calibration + fake_quant
// (algorithm/quantization/ptq/omniquant/source/omniquant/quantizer.py:124-150, 89-111;
// symmetric=False, no group, no learned clipping), every op rounded to fp16 as torch does:
//   s  = clamp(f16(f16(max - min) / 255), 1e-5, 1e4)
//   zp = rint(clamp(f16(-min / s), -1e4, 1e4))
//   u  = clamp(f16(rint(f16(x / s)) + zp), 0, 255);   fake = f16(f16(u - zp) * s)
// Also emits the row sum of the codes, which the integer GEMM's zero-point correction needs.
// A row (K <= THREADS * 8 * NV) is read once and stays in registers; NV == 0: any K, the second pass re-reads it.  The
// codes come from the packed f16x2 quotient (exact, see common.cuh): with a zero point in [0, 255] quotients stay within
// +-512, where adding 1536 rounds to an integer, and the code is the low byte.  Zero points beyond the codes (rows on one
// side of zero) and scales below 2^-14 take fp32 divisions.  333 rows of 4096 / 11008: 5.2 / 9.6 us with a division per
// value and two passes.
__device__ __forceinline__ uint32_t affine_code_pair(__half2 x, const RowQuant& rq, __half2 zp2) {
  const __half2 r = __hadd2_rn(quant_pair_packed(x, rq), zp2);
  return h2_bits(__hmin2(__hmax2(r, __float2half2_rn(1536.0f)), __float2half2_rn(1791.0f)));
}

template <int THREADS, int NV>
__global__ void __launch_bounds__(THREADS)
affine_quant_kernel(const __half* __restrict__ x, int K, uint8_t* __restrict__ q, float* __restrict__ scale,
                    float* __restrict__ zero, int* __restrict__ rowsum, __half* __restrict__ fake) {
  chain_wait();
  chain_release();
  __shared__ __half2 s_range[THREADS / 32];
  __shared__ int s_sum[THREADS / 32];
  const int row = blockIdx.x;
  const __half* xr = x + (size_t)row * K;
  const int chunks = K >> 3;
  constexpr int NREG = NV > 0 ? NV : 1;
  uint4 held[NREG];
  // (a thread without a piece of its own takes the first one)
  __half2 mx = *reinterpret_cast<const __half2*>(xr), mn = mx;
  auto range_of = [&](const uint4& raw) {
    const __half2* h = reinterpret_cast<const __half2*>(&raw);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      mx = __hmax2(mx, h[j]);
      mn = __hmin2(mn, h[j]);
    }
  };
  if (NV > 0) {
#pragma unroll
    for (int v = 0; v < NREG; ++v) {
      const int c = threadIdx.x + v * THREADS;
      held[v] = *reinterpret_cast<const uint4*>(xr + (c < chunks ? c : 0) * 8);
    }
#pragma unroll
    for (int v = 0; v < NREG; ++v) range_of(held[v]);
  } else {
    for (int c = threadIdx.x; c < chunks; c += THREADS) range_of(*reinterpret_cast<const uint4*>(xr + c * 8));
  }
  // (max, -min) through the reductions as one register
  __half2 m = max_and_neg_min(mx, mn);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = __hmax2(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) s_range[threadIdx.x >> 5] = m;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < THREADS / 32; ++i) m = __hmax2(m, s_range[i]);
  const __half hmax = __low2half(m), hmin = __hneg(__high2half(m));
  __half sh = hdiv_t(hsub_t(hmax, hmin), f2h(255.0f));
  const float lo = h2f(f2h(1e-5f)), hi = h2f(f2h(1e4f));
  sh = f2h(fminf(fmaxf(h2f(sh), lo), hi));
  const float zp = rintf(fminf(fmaxf(h2f(hdiv_t(__hneg(hmin), sh)), -hi), hi));
  const float sf = h2f(sh);
  if (threadIdx.x == 0) {
    scale[row] = sf;
    zero[row] = zp;
  }
  const RowQuant rq = make_row_quant(sf);
  const bool fast = rq.packed && zp >= 0.0f && zp <= 255.0f;
  const __half2 zp2 = __float2half2_rn(zp);
  int local_sum = 0;
  auto emit = [&](int c, const uint4& raw) {
    const __half2* h = reinterpret_cast<const __half2*>(&raw);
    uint2 codes;
    if (fast) {
      const uint32_t c0 = affine_code_pair(h[0], rq, zp2), c1 = affine_code_pair(h[1], rq, zp2);
      const uint32_t c2 = affine_code_pair(h[2], rq, zp2), c3 = affine_code_pair(h[3], rq, zp2);
      codes = make_uint2(__byte_perm(c0, c1, 0x6420), __byte_perm(c2, c3, 0x6420));
    } else {
      uint32_t w[2] = {0, 0};
      const __half* hs = reinterpret_cast<const __half*>(&raw);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float u = rintf(h2f(f2h(__fdiv_rn(h2f(hs[j]), sf))));
        u = h2f(f2h(u + zp));
        u = fminf(fmaxf(u, 0.0f), 255.0f);
        w[j >> 2] |= static_cast<uint32_t>(u) << (8 * (j & 3));
      }
      codes = make_uint2(w[0], w[1]);
    }
    local_sum = static_cast<int>(__dp4a(codes.y, 0x01010101u, __dp4a(codes.x, 0x01010101u, static_cast<unsigned>(local_sum))));
    if (q) *reinterpret_cast<uint2*>(q + (size_t)row * K + c * 8) = codes;
    if (fake) {
      __align__(16) __half out[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const uint32_t code = ((j < 4 ? codes.x : codes.y) >> (8 * (j & 3))) & 0xFFu;
        out[j] = hmul_t(f2h(static_cast<float>(code) - zp), sh);
      }
      *reinterpret_cast<uint4*>(fake + (size_t)row * K + c * 8) = *reinterpret_cast<uint4*>(out);
    }
  };
  if (NV > 0) {
#pragma unroll
    for (int v = 0; v < NREG; ++v) {
      const int c = threadIdx.x + v * THREADS;
      if (c < chunks) emit(c, held[v]);
    }
  } else {
    for (int c = threadIdx.x; c < chunks; c += THREADS) emit(c, *reinterpret_cast<const uint4*>(xr + c * 8));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) local_sum += __shfl_xor_sync(0xffffffffu, local_sum, o);
  if ((threadIdx.x & 31) == 0) s_sum[threadIdx.x >> 5] = local_sum;
  __syncthreads();
  if (threadIdx.x == 0 && rowsum) {
    int tot = 0;
    for (int i = 0; i < THREADS / 32; ++i) tot += s_sum[i];
    rowsum[row] = tot;
  }
}

// Residual add + RMSNorm + per-token int8 quant in one pass over the row: the
// torch_npu.npu_add_rms_norm_dynamic_quant call that feeds the (codes, scale) tuple to
// the W8A8 linear (acceleration/runtime_patches/vllm_ascend.patch:754-770).
//   r   = f16(x + residual)                      (written back as the new residual)
//   y   = f16( f16(r * rsqrt(mean(r^2) + eps)) * gamma )   (RMSNorm as HF Llama computes it)
//   q,s = per-token absmax int8 of y             (same arithmetic as act_quant_kernel)
template <int THREADS, int NV>
__global__ void __launch_bounds__(THREADS)
add_rmsnorm_quant_kernel(const __half* __restrict__ x, __half* __restrict__ residual,
                         const __half* __restrict__ gamma, float eps, int H, int8_t* __restrict__ q,
                         float* __restrict__ scale) {
  __shared__ float s_red[THREADS / 32];
  __shared__ float s_bcast;
  const int row = blockIdx.x;
  const int chunks = H >> 3;
  const __half* xr = x + (size_t)row * H;
  __half* rr = residual + (size_t)row * H;
  auto block_reduce = [&](float v, bool is_max) -> float {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float other = __shfl_xor_sync(0xffffffffu, v, o);
      v = is_max ? fmaxf(v, other) : v + other;
    }
    __syncthreads();                               // s_red may still be read from the previous reduction
    if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x < 32) {
      float w = threadIdx.x < THREADS / 32 ? s_red[threadIdx.x] : 0.0f;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float other = __shfl_xor_sync(0xffffffffu, w, o);
        w = is_max ? fmaxf(w, other) : w + other;
      }
      if (threadIdx.x == 0) s_bcast = w;
    }
    __syncthreads();
    return s_bcast;
  };
  uint4 held[NV];
  float sumsq = 0.0f;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int c = threadIdx.x + v * THREADS;
    held[v] = make_uint4(0, 0, 0, 0);
    if (c < chunks) {
      const uint4 a = *reinterpret_cast<const uint4*>(xr + c * 8);
      const uint4 b = *reinterpret_cast<const uint4*>(rr + c * 8);
      const __half* ha = reinterpret_cast<const __half*>(&a);
      const __half* hb = reinterpret_cast<const __half*>(&b);
      __align__(16) __half hs[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        hs[j] = hadd_t(ha[j], hb[j]);
        const float f = h2f(hs[j]);
        sumsq += f * f;
      }
      held[v] = *reinterpret_cast<uint4*>(hs);
      *reinterpret_cast<uint4*>(rr + c * 8) = held[v];           // new residual
    }
  }
  const float inv = rsqrtf(block_reduce(sumsq, false) / static_cast<float>(H) + eps);
  float amax = 0.0f;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int c = threadIdx.x + v * THREADS;
    if (c < chunks) {
      const uint4 gw = *reinterpret_cast<const uint4*>(gamma + c * 8);
      const __half* hg = reinterpret_cast<const __half*>(&gw);
      __half* hs = reinterpret_cast<__half*>(&held[v]);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        hs[j] = hmul_t(f2h(h2f(hs[j]) * inv), hg[j]);
        amax = fmaxf(amax, fabsf(h2f(hs[j])));
      }
    }
  }
  const float eps_q = h2f(f2h(1e-5f));
  const float sf = h2f(f2h(__fdiv_rn(fmaxf(block_reduce(amax, true), eps_q), 127.0f)));
  const RowQuant rq = make_row_quant(sf);
  if (threadIdx.x == 0) scale[row] = sf;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int c = threadIdx.x + v * THREADS;
    if (c < chunks) {
      *reinterpret_cast<uint2*>(q + (size_t)row * H + c * 8) = quant8_pack(held[v], rq);
    }
  }
}

}  // namespace mp

using namespace mp;

extern "C" int mp_add_rmsnorm_quant(const void* x_f16, void* residual_f16, const void* gamma_f16, float eps, int M,
                                    int H, void* q_i8, void* scale_f32, mp_stream_t stream) {
  if (!x_f16 || !residual_f16 || !gamma_f16 || !q_i8 || !scale_f32 || M <= 0 || H <= 0) return MP_ERR_INVALID_ARG;
  if (H % 8 != 0 || H > 16384) return MP_ERR_UNSUPPORTED;
  if (!aligned(x_f16, 16) || !aligned(residual_f16, 16) || !aligned(gamma_f16, 16) || !aligned(q_i8, 8)) return MP_ERR_ALIGNMENT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const __half* x = static_cast<const __half*>(x_f16);
  __half* r = static_cast<__half*>(residual_f16);
  const __half* g = static_cast<const __half*>(gamma_f16);
  int8_t* q = static_cast<int8_t*>(q_i8);
  float* sc = static_cast<float*>(scale_f32);
  if (H <= 2048) {
    add_rmsnorm_quant_kernel<256, 1><<<M, 256, 0, st>>>(x, r, g, eps, H, q, sc);
  } else if (H <= 4096) {
    add_rmsnorm_quant_kernel<256, 2><<<M, 256, 0, st>>>(x, r, g, eps, H, q, sc);
  } else if (H <= 8192) {
    add_rmsnorm_quant_kernel<512, 2><<<M, 512, 0, st>>>(x, r, g, eps, H, q, sc);
  } else {
    add_rmsnorm_quant_kernel<512, 4><<<M, 512, 0, st>>>(x, r, g, eps, H, q, sc);
  }
  MP_LAUNCH_CHECK();
  return MP_OK;
}

// A block of these kernels loads its row, reduces, then stores: an SM streams only while its blocks are in different phases.
// With many rows narrow blocks with more pieces per thread keep more rows in flight (4096 rows, us: 14336 values 40.8 with 512
// threads, 29.7 with 256; 8192 values 23.4 / 16.7 with 128; with zero points 35.9 / 32.0 and 26.3 / 17.9; a warp per row up to
// 4096 values).  While all rows fit on the SMs side by side the chain of load, reduction, division and rounding is the time,
// so a thread has one or two pieces of the row.  A Llama-8B layer's four products with their quantisations, 1 / 4 / 16 / 64 /
// 148 rows, us: a warp per row of 4096 and 512 threads for 14336 58.8 / 60.4 / 65.0 / 69.1 / 86.5, wide blocks 56.3 / 57.7 /
// 62.6 / 67.2 / 85.2 (two and four pieces a thread above 4096 56.7 / 58.2 / 62.7 / 67.7 / 85.8).
// Where the line is, by a quantisation and its product (4096 / 14336 output columns), us, wide blocks / narrow ones:
//   above 8192 values a block has 1024 threads with two pieces each, and two of them fill an SM: 296 rows (11008 values, 297
//     rows 25.1 / 24.6 and 60.6 / 60.2, 500 rows 29.5 / 26.7 and 68.5 / 65.3; 14336 values, 200 rows 26.1 / 25.9 and 53.0 /
//     54.2)
//   up to 8192, one piece a thread (and with zero points, whose blocks have 512 threads, up to 16384), four rows to an SM: 592
//     (8192 values, 333 rows 20.2 / 21.3 and 51.3 / 52.8, 500 rows 21.1 / 21.7 and 52.1 / 53.0, 740 rows 27.4 / 26.1 at 4096
//     columns; with zero points 333 and 2000 rows of a Llama-7B layer 110.4 / 114.4 and 326.9 / 323.5)
//   up to 4096 values narrow is a warp, eight rows to a block.  From 65 to 256 rows (200 with zero points, 160 above 3072
//     values) the product gains more from the SMs this leaves to its blocks, which set up meanwhile (it seems: the times are
//     what was measured), than from the shorter chain: 2048 values, 64 rows 7.3 / 7.3 and 10.4 / 10.3, 224 rows 9.2 / 8.7 and
//     14.8 / 14.4, 333 rows 10.6 / 10.0 and 19.5 / 21.5; 4096 values, 148 rows 11.7 / 11.2 and 19.5 / 19.3, 333 rows
//     13.3 / 14.0 and 27.0 / 29.9
constexpr int kNarrowFrom = 65;
static bool wide_blocks(int M, int narrow_to, int wide_to) { return M < kNarrowFrom || (M > narrow_to && M <= wide_to); }

extern "C" int mp_act_quant_per_token(const void* x_f16, int M, int K, void* q_i8, void* scale_f32,
                                      void* fake_f16, mp_stream_t stream) {
  if (!x_f16 || M <= 0 || K <= 0 || (!q_i8 && !fake_f16)) return MP_ERR_INVALID_ARG;
  if (K % 8 != 0) return MP_ERR_UNSUPPORTED;
  if (!aligned(x_f16, 16) || (q_i8 && !aligned(q_i8, 8)) || (fake_f16 && !aligned(fake_f16, 16))) return MP_ERR_ALIGNMENT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const __half* x = static_cast<const __half*>(x_f16);
  int8_t* q = static_cast<int8_t*>(q_i8);
  float* sc = static_cast<float*>(scale_f32);
  __half* fk = static_cast<__half*>(fake_f16);
  if (K <= 16384 && wide_blocks(M, K > 4096 ? 0 : K > 3072 ? 160 : 256, K > 8192 ? 2 * kSmCount : 4 * kSmCount)) {
    if (K <= 1024) return launch_chained(act_quant_kernel<128, 1>, dim3(M), dim3(128), 0, st, x, M, K, q, sc, fk);
    if (K <= 2048) return launch_chained(act_quant_kernel<256, 1>, dim3(M), dim3(256), 0, st, x, M, K, q, sc, fk);
    if (K <= 4096) return launch_chained(act_quant_kernel<512, 1>, dim3(M), dim3(512), 0, st, x, M, K, q, sc, fk);
    if (K <= 8192) return launch_chained(act_quant_kernel<1024, 1>, dim3(M), dim3(1024), 0, st, x, M, K, q, sc, fk);
    return launch_chained(act_quant_kernel<1024, 2>, dim3(M), dim3(1024), 0, st, x, M, K, q, sc, fk);
  }
  if (K <= 1024) {
    return launch_act_quant_warp<4>(x, M, K, q, sc, fk, st);
  } else if (K <= 2048) {
    return launch_act_quant_warp<8>(x, M, K, q, sc, fk, st);
  } else if (K <= 4096) {
    return launch_act_quant_warp<16>(x, M, K, q, sc, fk, st);
  } else if (K <= 8192) {
    return launch_chained(act_quant_kernel<128, 8>, dim3(M), dim3(128), 0, st, x, M, K, q, sc, fk);
  } else if (K <= 16384) {
    return launch_chained(act_quant_kernel<256, 8>, dim3(M), dim3(256), 0, st, x, M, K, q, sc, fk);
  } else {
    return launch_chained(act_quant_kernel<512, 0>, dim3(M), dim3(512), 0, st, x, M, K, q, sc, fk);
  }
}

extern "C" int mp_affine_quant_per_row(const void* x_f16, int M, int K, void* q_u8, void* scale_f32, void* zero_f32,
                                       void* rowsum_i32, void* fake_f16, mp_stream_t stream) {
  if (!x_f16 || !scale_f32 || !zero_f32 || M <= 0 || K <= 0 || (!q_u8 && !fake_f16)) return MP_ERR_INVALID_ARG;
  if (K % 8 != 0) return MP_ERR_UNSUPPORTED;
  if (!aligned(x_f16, 16) || (q_u8 && !aligned(q_u8, 8)) || (fake_f16 && !aligned(fake_f16, 16))) return MP_ERR_ALIGNMENT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const __half* x = static_cast<const __half*>(x_f16);
  uint8_t* q = static_cast<uint8_t*>(q_u8);
  float *sc = static_cast<float*>(scale_f32), *ze = static_cast<float*>(zero_f32);
  int* rs = static_cast<int*>(rowsum_i32);
  __half* fk = static_cast<__half*>(fake_f16);
  if (K > 2048 && K <= 16384 && !wide_blocks(M, K > 4096 ? 0 : K > 3072 ? 160 : 200, 4 * kSmCount)) {
    if (K <= 4096) return launch_chained(affine_quant_kernel<128, 4>, dim3(M), dim3(128), 0, st, x, K, q, sc, ze, rs, fk);
    if (K <= 8192) return launch_chained(affine_quant_kernel<128, 8>, dim3(M), dim3(128), 0, st, x, K, q, sc, ze, rs, fk);
    return launch_chained(affine_quant_kernel<256, 8>, dim3(M), dim3(256), 0, st, x, K, q, sc, ze, rs, fk);
  }
  if (K <= 2048) return launch_chained(affine_quant_kernel<128, 2>, dim3(M), dim3(128), 0, st, x, K, q, sc, ze, rs, fk);
  if (K <= 4096) return launch_chained(affine_quant_kernel<256, 2>, dim3(M), dim3(256), 0, st, x, K, q, sc, ze, rs, fk);
  if (K <= 8192) return launch_chained(affine_quant_kernel<512, 2>, dim3(M), dim3(512), 0, st, x, K, q, sc, ze, rs, fk);
  if (K <= 16384) return launch_chained(affine_quant_kernel<512, 4>, dim3(M), dim3(512), 0, st, x, K, q, sc, ze, rs, fk);
  return launch_chained(affine_quant_kernel<512, 0>, dim3(M), dim3(512), 0, st, x, K, q, sc, ze, rs, fk);
}
