// W4A16 weight-side kernels: asymmetric group quantise + pack, dequantise
// (the bit-exact check of the GEMMs' dequant stage) and the one-time
// re-layout of scales / zero points for the GEMM kernels.
#include "common.cuh"

namespace mp {

// Eight weights -> one packed word with an fp32 division each; sz = (scale, zero point).
__device__ __forceinline__ uint32_t w4_codes_fp32(const uint4& raw, __half2 sz) {
  const __half* h = reinterpret_cast<const __half*>(&raw);
  const __half s = __low2half(sz);
  const float zf = __high2float(sz);
  uint32_t word = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    float q = rintf(h2f(hdiv_t(h[j], s)));                  // round(w / scales), may be +-inf
    q = h2f(f2h(q + zf));                                   // + zeros, rounded to fp16
    q = fminf(fmaxf(q, 0.0f), 15.0f);                       // clamp(0, 15)
    word |= static_cast<uint32_t>(q) << (4 * j);
  }
  return word;
}

// Groups of 32, 64, 128 and 256 columns: L = group / 8 lanes of a warp hold one group, eight columns (16 bytes) each,
// and a warp takes the groups of V such vectors per lane: 32 groups of 32 or 64 columns, 16 of 128, 8 of 256.  The
// weights are read once and stay in registers.  HBM moves 2.5 bytes per weight, which leaves about 110 issue slots per
// 256 weights, so the instruction count decides (the former kernel -- a warp per group, an fp32 division per weight, a
// second pass over the weights -- took 600 us for 12288x4096 + 4096x4096 + 22016x4096 + 4096x11008 in groups of 128):
//  * max and -min travel through the shuffles as the two halves of one register, and the reduction scatters: at each
//    step a lane passes on half of its vectors, so V vectors cost V - 1 exchanges and every lane ends with one group;
//  * that lane computes the group's scale and zero point -- the two divisions and the constants of its quotients;
//  * codes come from the packed f16x2 quotient of common.cuh (exactly round(f16(w / s)), see there);
//  * weights are paired (k, k + 4), so the eight codes drop into their nibbles with three multiply-adds.

// two weights of a group whose zero point did not need clamping -> f16x2 holding 1536 + min(round(f16(w / s)), 15 - z).
// pr = (2^-e, f16(1 / s')), nb = (-s', 1536 + 15 - z) with s = s' 2^e, see make_row_quant.  (With z = -round(min / s)
// no quotient rounds below -z, so the lower clamp has nothing to do.)
__device__ __forceinline__ uint32_t w4_code_pair(uint32_t w, __half2 pr, __half2 nb) {
  const __half2 wp = __hmul2_rn(*reinterpret_cast<const __half2*>(&w), __low2half2(pr));
  const __half2 q = __hmul2_rn(wp, __high2half2(pr));
  const __half2 rem = __hfma2(q, __low2half2(nb), wp);
  const __half2 q2 = __hfma2(rem, __high2half2(pr), q);
  return h2_bits(__hmin2(__hadd2_rn(q2, __float2half2_rn(1536.0f)), __high2half2(nb)));
}

__host__ __device__ constexpr int quantize_vectors(int lanes_per_group) { return lanes_per_group == 4 ? 4 : 8; }

template <int L>
__global__ void __launch_bounds__(256)
w4_quantize_groups_kernel(const __half* __restrict__ w, int N, int K, int groups, uint32_t* __restrict__ packed,
                          __half* __restrict__ scale, uint32_t* __restrict__ zero_words) {
  constexpr int V = quantize_vectors(L);       // 16-byte loads per lane
  constexpr int S = V == 4 ? 2 : 3;            // log2(V)
  constexpr int GPV = 32 / L;                  // groups per load of the warp
  constexpr int G = V * GPV;                   // groups per warp
  const int lane = threadIdx.x & 31;
  const unsigned units_per_row = static_cast<unsigned>(groups + G - 1) / G;
  const unsigned unit = blockIdx.x * 8 + (threadIdx.x >> 5);
  const unsigned n = unit / units_per_row;
  if (n >= static_cast<unsigned>(N)) return;
  const int g0 = static_cast<int>(unit - n * units_per_row) * G;     // first group of this warp
  const int vecs = K >> 3, v0 = g0 * L + lane; // 16-byte vectors per row, first one of this lane
  const uint4* row = reinterpret_cast<const uint4*>(w + (size_t)n * K);
  uint4 raw[V];
#pragma unroll
  for (int v = 0; v < V; ++v) raw[v] = v0 + v * 32 < vecs ? __ldcs(row + v0 + v * 32) : make_uint4(0, 0, 0, 0);
  __half2 m[V];                                // (max, -min)
#pragma unroll
  for (int v = 0; v < V; ++v) {
    const __half2* h = reinterpret_cast<const __half2*>(&raw[v]);
    const __half2 mx = __hmax2(__hmax2(h[0], h[1]), __hmax2(h[2], h[3]));
    m[v] = max_and_neg_min(mx, __hmin2(__hmin2(h[0], h[1]), __hmin2(h[2], h[3])));
  }
#pragma unroll
  for (int st = 0; st < S; ++st) {
    const bool upper = lane & (1 << st);
    const int half = V >> (st + 1);
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const __half2 keep = upper ? m[i + half] : m[i], pass = upper ? m[i] : m[i + half];
      m[i] = __hmax2(keep, __shfl_xor_sync(0xffffffffu, pass, 1 << st));
    }
  }
#pragma unroll
  for (int o = V; o < L; o <<= 1) m[0] = __hmax2(m[0], __shfl_xor_sync(0xffffffffu, m[0], o));
  // this lane's group: the vector its low S bits (most significant first) chose
  int my_v = 0;
#pragma unroll
  for (int st = 0; st < S; ++st) my_v |= (lane & (1 << st)) ? V >> (st + 1) : 0;
  const int my_g = my_v * GPV + lane / L;
  const bool live = g0 + my_g < groups, first = L <= V || (lane & (L - 1)) < V;   // larger groups: several lanes agree
  // scale and zero point, every op rounded to fp16 as torch does
  const __half hmax = __low2half(m[0]), hmin = __hneg(__high2half(m[0]));
  __half span = hsub_t(hmax, hmin);
  const __half eps = f2h(1e-5f);
  if (h2f(span) < h2f(eps)) span = eps;                       // clamp(min=1e-5)
  const __half s = hdiv_t(span, f2h(15.0f));                  // / max_int
  const float z_raw = -rintf(h2f(hdiv_t(hmin, s)));           // -round(min / scales)
  const float zf = fminf(fmaxf(z_raw, 0.0f), 15.0f);          // clamp_(0, 15)
  const uint32_t z = static_cast<uint32_t>(zf);
#pragma unroll
  for (int wd = 0; wd < G / 8; ++wd) {
    const uint32_t zw = __reduce_or_sync(0xffffffffu, (my_g >> 3) == wd && live ? z << (4 * (my_g & 7)) : 0u);
    if (lane == 0 && g0 + wd * 8 < groups) zero_words[(size_t)n * ((groups + 7) >> 3) + (g0 >> 3) + wd] = zw;
  }
  if (live && first) scale[(size_t)n * groups + g0 + my_g] = s;
  const RowQuant rq = make_row_quant(h2f(s));
  // the packed route needs a scale of at least 2^-14 that is finite; a zero point that was clamped (all weights of the
  // group on one side of zero) leaves quotients the short form does not cover
  const bool fast = rq.packed && rq.s < 65536.0f && z_raw >= 0.0f && z_raw <= 15.0f;
  const uint32_t pr_mine = fast ? h2_bits(__halves2half2(__low2half(rq.pow2), __low2half(rq.rcp)))
                                : h2_bits(__halves2half2(f2h(0.0f), s));   // marks the fp32 route
  const uint32_t nb_mine = h2_bits(__halves2half2(__low2half(rq.neg_sp), f2h(1551.0f - zf)));
  uint32_t* out = packed + (size_t)n * vecs;
#pragma unroll
  for (int v = 0; v < V; ++v) {
    if (v0 - lane + v * 32 >= vecs) break;     // the row ends inside this warp's span
    int src = lane & ~(L - 1);                 // lane that made the constants of this lane's group in vector v
#pragma unroll
    for (int st = 0; st < S; ++st) src |= (v & (V >> (st + 1))) ? 1 << st : 0;
    const uint32_t prw = __shfl_sync(0xffffffffu, pr_mine, src);
    const uint32_t nbw = __shfl_sync(0xffffffffu, nb_mine, src);
    const uint32_t zv = __shfl_sync(0xffffffffu, z, src);
    const __half2 pr = *reinterpret_cast<const __half2*>(&prw), nb = *reinterpret_cast<const __half2*>(&nbw);
    uint32_t word;
    if ((prw & 0xffffu) != 0) {
      // pairs (k0,k4) (k1,k5) (k2,k6) (k3,k7): each result is 0x66006600 + code - z in both halves, so with the
      // constants taken out their sum over 16^j is the packed word
      const uint32_t r0 = w4_code_pair(prmt(raw[v].x, raw[v].z, 0x5410), pr, nb);
      const uint32_t r1 = w4_code_pair(prmt(raw[v].x, raw[v].z, 0x7632), pr, nb);
      const uint32_t r2 = w4_code_pair(prmt(raw[v].y, raw[v].w, 0x5410), pr, nb);
      const uint32_t r3 = w4_code_pair(prmt(raw[v].y, raw[v].w, 0x7632), pr, nb);
      const uint32_t bias = zv * 0x11111111u - 0x66006600u * 0x1111u;
      word = (r3 * 4096u + r2 * 256u) + (r1 * 16u + (r0 + bias));
    } else {
      word = w4_codes_fp32(raw[v], __halves2half2(__high2half(pr), f2h(static_cast<float>(zv))));
    }
    if (v0 + v * 32 < vecs) __stcs(out + v0 + v * 32, word);
  }
}

// Any other group (a multiple of eight columns).
// One warp per (row, group); a block of 8 warps covers 8 consecutive groups
// of one row so that it can also emit the packed zero-point word.
// Arithmetic follows pseudo_quantize_tensor(zero_point=True) in
// algorithm/quantization/ptq/awq/source/awq/quantize/quantizer.py:72-97,
// every op rounded to fp16 as torch does on fp16 tensors.
__global__ void __launch_bounds__(256)
w4_quantize_kernel(const __half* __restrict__ w, int N, int K, int group, int groups,
                   uint32_t* __restrict__ packed, __half* __restrict__ scale,
                   uint32_t* __restrict__ zero_words) {
  __shared__ uint32_t s_zero[8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n = blockIdx.y;
  const int g = blockIdx.x * 8 + warp;
  if (threadIdx.x < 8) s_zero[threadIdx.x] = 0;
  __syncthreads();
  if (g < groups) {
    const __half* row = w + (size_t)n * K + (size_t)g * group;
    const int chunks = group >> 3;  // 8 columns (16 bytes) per chunk
    float vmax = -INFINITY, vmin = INFINITY;
    for (int c = lane; c < chunks; c += 32) {
      uint4 raw = *reinterpret_cast<const uint4*>(row + c * 8);
      const __half* h = reinterpret_cast<const __half*>(&raw);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float f = h2f(h[j]);
        vmax = fmaxf(vmax, f);
        vmin = fminf(vmin, f);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
      vmin = fminf(vmin, __shfl_xor_sync(0xffffffffu, vmin, o));
    }
    const __half hmax = f2h(vmax), hmin = f2h(vmin);  // exact: both are fp16 values
    __half span = hsub_t(hmax, hmin);
    const __half eps = f2h(1e-5f);
    if (h2f(span) < h2f(eps)) span = eps;                       // clamp(min=1e-5)
    const __half s = hdiv_t(span, f2h(15.0f));                  // / max_int
    float zf = -rintf(h2f(hdiv_t(hmin, s)));                    // -round(min / scales)
    zf = fminf(fmaxf(zf, 0.0f), 15.0f);                         // clamp_(0, 15)
    for (int c = lane; c < chunks; c += 32) {
      packed[(size_t)n * (K >> 3) + (size_t)g * chunks + c] =
          w4_codes_fp32(*reinterpret_cast<const uint4*>(row + c * 8), __halves2half2(s, f2h(zf)));
    }
    if (lane == 0) {
      scale[(size_t)n * groups + g] = s;
      s_zero[warp] = static_cast<uint32_t>(zf);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t zw = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) zw |= (s_zero[j] & 0xFu) << (4 * j);
    zero_words[(size_t)n * ((groups + 7) >> 3) + blockIdx.x] = zw;
  }
}

__device__ __forceinline__ __half zero_point_of(const uint32_t* zero_words, int n, int groups, int g) {
  if (zero_words == nullptr) return __float2half_rn(8.0f);
  uint32_t zw = zero_words[(size_t)n * ((groups + 7) >> 3) + (g >> 3)];
  return __float2half_rn(static_cast<float>((zw >> (4 * (g & 7))) & 0xFu));
}

// A thread expands one packed word (8 codes -> 16 bytes) in each of four consecutive rows, through the same dequant8 the
// GEMM kernels use: loads of 128 and stores of 512 contiguous bytes per warp, and the group a word belongs to (a
// division) is found once for the four.  Bound by the stores; with a word per thread and 64-bit index arithmetic the
// kernel issued twice the instructions and ran at 3.7 TB/s.
constexpr int kDequantRows = 4;
__global__ void __launch_bounds__(256)
w4_dequant_kernel(const uint32_t* __restrict__ packed, const __half* __restrict__ scale,
                  const uint32_t* __restrict__ zero_words, int N, int words_per_row, int words_per_group, int groups,
                  __half* __restrict__ out) {
  const int c = blockIdx.x * 256 + threadIdx.x;
  if (c >= words_per_row) return;
  const int g = c / words_per_group, gw = g >> 3, gs = 4 * (g & 7);
  const int zero_pitch = (groups + 7) >> 3;
  for (int n0 = blockIdx.y * kDequantRows; n0 < N; n0 += gridDim.y * kDequantRows) {
    uint32_t q[kDequantRows], z[kDequantRows];
    __half s[kDequantRows];
#pragma unroll
    for (int i = 0; i < kDequantRows; ++i) {
      const int n = min(n0 + i, N - 1);
      q[i] = __ldcs(packed + (size_t)n * words_per_row + c);
      s[i] = scale[(size_t)n * groups + g];
      z[i] = zero_words ? (zero_words[(size_t)n * zero_pitch + gw] >> gs) & 0xFu : 8u;
    }
#pragma unroll
    for (int i = 0; i < kDequantRows; ++i) {
      if (n0 + i >= N) break;
      // 1024 + z and -(64 + z) as fp16 bit patterns
      const uint32_t zl = 0x64006400u + z[i] * 0x00010001u, zh = 0xD400D400u + z[i] * 0x00100010u;
      ScaleZero p;
      p.s2 = __half2half2(s[i]);
      p.z_lo = *reinterpret_cast<const __half2*>(&zl);
      p.z_hi = *reinterpret_cast<const __half2*>(&zh);
      __half2 v[4];
      dequant8(q[i], p, v);
      // v = (k0,k4) (k1,k5) (k2,k6) (k3,k7) -> natural order
      const uint32_t a = h2_as_u32(v[0]), b = h2_as_u32(v[1]), cc = h2_as_u32(v[2]), d = h2_as_u32(v[3]);
      __stcs(reinterpret_cast<uint4*>(out) + (size_t)(n0 + i) * words_per_row + c,
             make_uint4(prmt(a, b, 0x5410), prmt(cc, d, 0x5410), prmt(a, b, 0x7632), prmt(cc, d, 0x7632)));
    }
  }
}

// sz[g, n] = (scale[n, g], f16(zero[n, g]))
__global__ void __launch_bounds__(256)
w4_prepare_kernel(const __half* __restrict__ scale, const uint32_t* __restrict__ zero_words,
                  int N, int groups, __half2* __restrict__ sz) {
  const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (size_t)N * groups) return;
  const int g = static_cast<int>(idx / N);
  const int n = static_cast<int>(idx % N);
  sz[idx] = __halves2half2(scale[(size_t)n * groups + g], zero_point_of(zero_words, n, groups, g));
}

}  // namespace mp

using namespace mp;

extern "C" int mp_w4a16_quantize(const void* w_f16, int N, int K, int group, void* packed_i32,
                                 void* scale_f16, void* zero_i32, mp_stream_t stream) {
  if (!w_f16 || !packed_i32 || !scale_f16 || !zero_i32 || N <= 0 || K <= 0 || group <= 0) return MP_ERR_INVALID_ARG;
  if (K % 8 != 0 || group % 8 != 0 || K % group != 0) return MP_ERR_UNSUPPORTED;
  if (!aligned(w_f16, 16)) return MP_ERR_ALIGNMENT;
  const int groups = K / group;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const __half* w = static_cast<const __half*>(w_f16);
  uint32_t* packed = static_cast<uint32_t*>(packed_i32);
  __half* scale = static_cast<__half*>(scale_f16);
  uint32_t* zero = static_cast<uint32_t*>(zero_i32);
  // groups that a warp of the kernels for these sizes takes
  const bool own = group == 32 || group == 64 || group == 128 || group == 256;
  const int per_warp = own ? quantize_vectors(group / 8) * 256 / group : 1;
  const long long units = (long long)N * ((groups + per_warp - 1) / per_warp);
  if (own && units > 0x7fffffffLL) return MP_ERR_UNSUPPORTED;
  const unsigned blocks = static_cast<unsigned>((units + 7) / 8);
  switch (group) {
    case 32: w4_quantize_groups_kernel<4><<<blocks, 256, 0, st>>>(w, N, K, groups, packed, scale, zero); break;
    case 64: w4_quantize_groups_kernel<8><<<blocks, 256, 0, st>>>(w, N, K, groups, packed, scale, zero); break;
    case 128: w4_quantize_groups_kernel<16><<<blocks, 256, 0, st>>>(w, N, K, groups, packed, scale, zero); break;
    case 256: w4_quantize_groups_kernel<32><<<blocks, 256, 0, st>>>(w, N, K, groups, packed, scale, zero); break;
    default:
      w4_quantize_kernel<<<dim3((groups + 7) / 8, N), 256, 0, st>>>(w, N, K, group, groups, packed, scale, zero);
  }
  MP_LAUNCH_CHECK();
  return MP_OK;
}

extern "C" int mp_w4a16_dequant(const void* packed_i32, const void* scale_f16, const void* zero_i32,
                                int N, int K, int group, void* w_out_f16, mp_stream_t stream) {
  if (!packed_i32 || !scale_f16 || !w_out_f16 || N <= 0 || K <= 0 || group <= 0) return MP_ERR_INVALID_ARG;
  if (K % 8 != 0 || group % 8 != 0 || K % group != 0) return MP_ERR_UNSUPPORTED;
  if (!aligned(w_out_f16, 16)) return MP_ERR_ALIGNMENT;
  const int row_groups = (N + kDequantRows - 1) / kDequantRows;
  const dim3 grid((K / 8 + 255) / 256, row_groups < 65535 ? row_groups : 65535);
  w4_dequant_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint32_t*>(packed_i32), static_cast<const __half*>(scale_f16),
      static_cast<const uint32_t*>(zero_i32), N, K / 8, group / 8, K / group, static_cast<__half*>(w_out_f16));
  MP_LAUNCH_CHECK();
  return MP_OK;
}

extern "C" int mp_w4a16_prepare(const void* scale_f16, const void* zero_i32, int N, int K, int group,
                                void* sz_f16x2, mp_stream_t stream) {
  if (!scale_f16 || !sz_f16x2 || N <= 0 || K <= 0 || group <= 0) return MP_ERR_INVALID_ARG;
  if (K % group != 0) return MP_ERR_UNSUPPORTED;
  const int groups = K / group;
  const size_t total = (size_t)N * groups;
  const unsigned blocks = static_cast<unsigned>((total + 255) / 256);
  w4_prepare_kernel<<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __half*>(scale_f16), static_cast<const uint32_t*>(zero_i32), N, groups,
      static_cast<__half2*>(sz_f16x2));
  MP_LAUNCH_CHECK();
  return MP_OK;
}
