// W8A8 products with few activation rows (up to 8, or 64 to an expert): the weights are streamed once as the MMA's
// 128-row operand, the activation rows are its N.
//
//   D[128 weight rows][tokens] (int32, TMEM) += W[128 rows x 128 bytes] (shared memory) x X[tokens x 128 bytes]^T
//
// What bounds it: HBM.  A stage of 16 KB of weights takes the SM's share of HBM about 700 clocks; its four MMAs take 160
// (operands in shared memory, up to 64 tokens), the MMA thread's wait 170 and the producer about 320.  The former form --
// activations as a 128-row operand padded with zero rows, K cut into slices, partial sums written out and added by a
// second kernel -- took 10.2 + 2.8 us for 6144x4096 and 36.6 us for 28672x4096 at 4 rows.
//
// Work is divided as in w4a16_decode_umma.cu: the (expert, row block, 128-byte step of K) sequence is cut evenly over one
// block per SM, a block walks its range backwards, the part of a row block that continues in later blocks goes to the
// block's tile in the workspace, and the block that holds a row block's end adds the tiles of the earlier ones (integer
// sums: the cut changes no bit).  A tile word is stored with its sign bit flipped, so that zero -- "not there yet" -- would
// be the sum -2^31, which 8-bit products over K < 2^17 do not reach; the reader polls the words and puts the zeros back.
//
//   warps 0-7   epilogue: accumulator -> shared memory (lane = weight row) -> a warp per token, four weight rows per lane:
//               scales, bias or SwiGLU, stores of 256 contiguous bytes
//   warp 8      TMA producer: one copy of weights and one of activations per stage
//   warp 9      TMEM allocation and the MMA issuer
// Where its stream is short a block takes less than half an SM, so the next product of a chain starts beside the end of this
// one; its first weights are then already on the way (see early_weights).  A long stream has a longer ring (long_stream).
//
// With few activation values (quantise_in_stream) the kernel quantises the rows itself (QUANT): a launch less between two
// products of a chain, which was 1 to 2 us of its own chain of load, reduction and store.  The epilogue warps and four more
// look through all rows for their maxima, then
//   warps 10-13 quantise 128 columns of two rows each per stage, into the stage's activations as TMA would lay them out
#include "common.cuh"
#include "tc.cuh"
#include "moe_api.cuh"
#include "w8a8_stream.cuh"

namespace mp {

using namespace tc;

namespace ws {
constexpr int kRows = 128;
constexpr int kStepK = 128;
constexpr int kEpiWarps = 8, kLoadWarp = 8, kMmaWarp = 9;
constexpr int kQuantWarp0 = 10, kQuantWarps = 4; // with rows quantised here: two rows to a warp
constexpr int kMaxQuantRows = 2 * kQuantWarps;
constexpr int kWBytes = kRows * kStepK;
constexpr int kChunk = 16;                       // tokens that pass through shared memory at a time
constexpr int kPitch = kRows + 4;                // words between tokens there: 16-byte rows, lanes on different banks
constexpr int kMaxRing = 8;
// Blocks of at least long_stream() stages have kLongRing of them in flight, though they then take more than half an SM and the
// next product of a chain starts behind their end: with four (32 tokens) an SM has too little under way, with more than six
// the HBM rate falls again (the Mixtral-shaped experts at 32 tokens, us: 4 stages 284, 6 262, 7 263, 8 270; 28672x4096 at one
// row, 5 / 6 / 8 stages 24.0 / 23.4 / 23.6).  Rings of half an SM are four stages or less from 32 tokens on, so there, and
// where the start of the next product has less to hide because it quantises its rows first, half the length is enough
// (line at 40 / 20 stages: experts of 3072x3072 at 64 tokens 69.0 / 65.8, of 2048x2048 at 32 41.1 / 40.9, a layer with its
// rows quantised inside 52.0 / 51.6; but experts of 2048x4096 at 16 tokens 54.7 / 55.0, an asymmetric layer at 8 rows 91.8 /
// 92.8).
constexpr int kLongRing = 6;
constexpr int long_stream(int tokens, bool quantising) { return tokens > 16 || quantising ? 20 : 40; }
constexpr int kMaxExperts = 256;
constexpr int kMaxGroups = 512;

template <int TOK, int EPI, bool LONG, bool QUANT>
struct Cfg {
  static_assert(!QUANT || (TOK >= kMaxQuantRows && EPI == STREAM_F16), "rows quantised here");
  static constexpr int kThreads = 32 * (kMmaWarp + 1 + (QUANT ? kQuantWarps : 0));
  static constexpr int kParts = EPI == STREAM_SWIGLU ? 2 : 1;       // gate rows and up rows
  static constexpr int kStageBytes = kWBytes + TOK * kStepK;
  static constexpr int kSmemMax = 112 * 1024;
  static constexpr int kFixed = 1024 + 2 * kChunk * kPitch * 4 + (2 * kMaxRing + 4) * 8 + 64;
  static constexpr int kFit = (kSmemMax - kFixed) / kStageBytes;
  static constexpr int kRing = LONG ? kLongRing : kFit < kMaxRing ? kFit : kMaxRing;
  static constexpr int kSmem = kFixed + kRing * kStageBytes;
  static constexpr int kTmemUsed = 2 * kParts * TOK;                // two accumulator buffers
  static constexpr uint32_t kTmemCols = kTmemUsed <= 64 ? 64 : kTmemUsed <= 128 ? 128 : 256;
  static_assert(kRing >= 3 && kSmem <= 224 * 1024 && kTmemUsed <= 256, "shared or tensor memory");
};
}  // namespace ws

__device__ __forceinline__ void stream_tmem_ld_x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ uint4 stream_ld_v4(const uint32_t* p) {
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void stream_st_v4(uint32_t* p, const uint4& v) {
  asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// Position in the work sequence, walked backwards.
struct StreamAt {
  int group, rb, kb;
  __device__ __forceinline__ void set(int t, int row_blocks, int steps) {
    const int g = t / steps;
    kb = t - g * steps;
    group = g / row_blocks;
    rb = g - group * row_blocks;
  }
  __device__ __forceinline__ void back(int row_blocks, int steps) {
    if (--kb >= 0) return;
    kb = steps - 1;
    if (--rb >= 0) return;
    rb = row_blocks - 1;
    --group;
  }
};

template <int TOK, int EPI, bool LONG, bool QUANT>
__global__ void __launch_bounds__(ws::Cfg<TOK, EPI, LONG, QUANT>::kThreads, 2)
w8a8_stream_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                   const StreamParams p) {
  using C = ws::Cfg<TOK, EPI, LONG, QUANT>;
  constexpr int kRing = C::kRing, kParts = C::kParts;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint32_t* s_chunk = reinterpret_cast<uint32_t*>(base + kRing * C::kStageBytes);      // two of [kChunk][kPitch]
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_chunk + 2 * ws::kChunk * ws::kPitch);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * ws::kMaxRing + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  // grouped: the (expert, first row of up to TOK) pairs that have rows; more than kMaxGroups are not expected (see the
  // launcher) and would be dropped
  __shared__ int s_group[EPI == STREAM_AFFINE ? 1 : ws::kMaxGroups];
  __shared__ int s_active;
  __shared__ uint32_t s_top[QUANT ? ws::kMaxQuantRows : 1];     // the rows' largest magnitudes
  const uint32_t ring = smem_u32(base);
  const uint32_t full0 = smem_u32(bars), empty0 = full0 + 8 * ws::kMaxRing;
  const uint32_t dfull0 = empty0 + 8 * ws::kMaxRing, dempty0 = dfull0 + 16;

  const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
  const int blk = static_cast<int>(blockIdx.x), grid = static_cast<int>(gridDim.x);
  const bool grouped = p.counts != nullptr;
  if (warp == ws::kLoadWarp && elect_one()) {
    prefetch_tensormap(&tmap_w);
    prefetch_tensormap(&tmap_x);
    for (int s = 0; s < kRing; ++s) {
      mbar_init(full0 + 8 * s, QUANT ? 1 + (p.M + 1) / 2 : 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int d = 0; d < 2; ++d) {
      mbar_init(dfull0 + 8 * d, 1);
      mbar_init(dempty0 + 8 * d, ws::kEpiWarps);
    }
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == ws::kMmaWarp) {
    tmem_alloc(smem_u32(tmem_slot), C::kTmemCols);
    tmem_relinquish();
  }
  if (QUANT && tid < ws::kMaxQuantRows) s_top[tid] = 0;
  if (!QUANT && !p.early_weights) chain_wait();
  if (grouped && warp == 0) {
    // (the counts are complete: they are older than the previous kernel, or it was waited for)
    int n = 0;
    for (int e0 = 0; e0 < p.experts; e0 += 32) {
      const int tiles = e0 + lane < p.experts ? (p.counts[e0 + lane] + TOK - 1) / TOK : 0;
      int upto = tiles;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += v;
      }
      for (int i = 0; i < tiles; ++i) {
        const int at = n + upto - tiles + i;
        if (EPI != STREAM_AFFINE && at < ws::kMaxGroups) s_group[at] = (e0 + lane) | (i << 8);
      }
      n += __shfl_sync(0xffffffffu, upto, 31);
    }
    if (lane == 0) s_active = min(n, ws::kMaxGroups);
  }
  __syncwarp();
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  const int steps = p.steps, row_blocks = p.row_blocks;
  const int total = (grouped ? s_active : 1) * row_blocks * steps;
  // even ranges, the first `extra` blocks one longer; at least min_share steps each, so later blocks may have none
  int share = (total + grid - 1) / grid;
  if (share < p.min_share) share = p.min_share;
  const int blocks = (total + share - 1) / share;
  const int even = blocks ? total / blocks : 0, extra = total - even * blocks;
  const int t_lo = blk * even + min(blk, extra);
  const int t_hi = blk < blocks ? t_lo + even + (blk < extra ? 1 : 0) - 1 : t_lo - 1;
  const int n_steps = t_hi - t_lo + 1;

  if (warp == ws::kLoadWarp) {
    // ------------------------------------------------------------ TMA producer
    if (elect_one()) {
      StreamAt at;
      at.set(n_steps > 0 ? t_hi : 0, row_blocks, steps);
      auto load_w = [&](int s, const StreamAt& a, int part) {
        const int e = grouped ? s_group[a.group] & 0xFF : 0;
        mbar_arrive_expect_tx(full0 + 8 * s, ws::kWBytes + (QUANT ? 0 : p.x_box * ws::kStepK));
        tma_load_2d(ring + s * C::kStageBytes, &tmap_w, full0 + 8 * s, a.kb * ws::kStepK,
                    e * p.rows_per_expert + part * p.up_row_offset + a.rb * ws::kRows);
      };
      auto load_x = [&](int s, const StreamAt& a) {
        const int row = grouped ? p.segments[s_group[a.group] & 0xFF] + (s_group[a.group] >> 8) * TOK : 0;
        tma_load_2d(ring + s * C::kStageBytes + ws::kWBytes, &tmap_x, full0 + 8 * s, a.kb * ws::kStepK, row);
      };
      const int n_stages = n_steps * kParts;
      int ahead = 0;
      if constexpr (QUANT) {                       // the first weights as far as L2: a kernel before may write weights
        StreamAt a = at;
        for (int i = 0; i < kRing && i < n_stages; ++i, a.back(row_blocks, steps))
          tma_prefetch_2d(&tmap_w, a.kb * ws::kStepK, a.rb * ws::kRows);
        chain_wait();
      } else if (p.early_weights) {                // the ring's first weights, then what the previous kernel made
        StreamAt a = at;
        for (; ahead < kRing && ahead < n_stages; ++ahead) {
          load_w(ahead, a, ahead % kParts);
          if (ahead % kParts == kParts - 1) a.back(row_blocks, steps);
        }
        chain_wait();
      }
      int s = 0, part = 0;
      uint32_t phase = 1;
      for (int i = 0; i < n_stages; ++i) {
        if (i >= ahead) {
          if (!mbar_wait(empty0 + 8 * s, phase, abort_flag)) break;
          load_w(s, at, part);
        }
        if (!QUANT) load_x(s, at);
        if (++part == kParts) {
          part = 0;
          at.back(row_blocks, steps);
        }
        if (++s == kRing) { s = 0; phase ^= 1; }
      }
      chain_release();             // this block's loads are issued: the next kernel's blocks may start
    }
  } else if (warp == ws::kMmaWarp) {
    // ------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      constexpr uint32_t idesc =
          umma_idesc(kIdescDFormatS32 | (EPI == STREAM_AFFINE ? kIdescABFormatU8 : kIdescABFormatS8), ws::kRows, TOK);
      StreamAt at;
      at.set(n_steps > 0 ? t_hi : 0, row_blocks, steps);
      int s = 0, d = 0;
      uint32_t phase = 0, dphase = 1;
      bool fresh = true, ok = true;
      for (int i = 0; ok && i < n_steps; ++i) {
        if (fresh && !mbar_wait(dempty0 + 8 * d, dphase, abort_flag)) break;
#pragma unroll
        for (int part = 0; part < kParts; ++part) {
          if (!mbar_wait(full0 + 8 * s, phase, abort_flag)) { ok = false; break; }
          tcgen05_fence_after();
          const uint32_t stage = ring + s * C::kStageBytes;
          const uint64_t a_desc = umma_desc_k_sw128(stage), b_desc = umma_desc_k_sw128(stage + ws::kWBytes);
          const uint32_t d_tmem = tmem_base + (d * kParts + part) * TOK;
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) umma_i8(d_tmem, a_desc + 2 * kk, b_desc + 2 * kk, idesc, !(fresh && kk == 0));
          umma_commit(empty0 + 8 * s);
          if (++s == kRing) { s = 0; phase ^= 1; }
        }
        fresh = at.kb == 0;
        if (fresh || i == n_steps - 1) {
          umma_commit(dfull0 + 8 * d);
          if (++d == 2) { d = 0; dphase ^= 1; }
        }
        at.back(row_blocks, steps);
      }
    }
  } else {
    float sa_here = 0.0f;                          // QUANT: the scale of row `warp`
    if (QUANT || p.early_weights) chain_wait();    // before anything of the previous kernel is read or overwritten
    if constexpr (QUANT) {
      // a quantising warp has 128 columns of two rows per stage, eight values to a lane; the first stages' are on their way
      // while the rows are looked through
      const int r = 2 * (warp - ws::kQuantWarp0) + (lane >> 4), c = lane & 15;
      const bool mine = warp >= ws::kEpiWarps && r < p.M;
      auto load = [&](int kb) {
        return mine && kb * ws::kStepK + 8 * c < p.K
                   ? *reinterpret_cast<const uint4*>(p.x + (size_t)r * p.K + kb * ws::kStepK + 8 * c) : make_uint4(0, 0, 0, 0);
      };
      constexpr int kHeld = 4;                     // (3 is level, 6 is 2 us slower for four products)
      uint4 held[kHeld];
      StreamAt at, ahead;
      at.set(n_steps > 0 ? t_hi : 0, row_blocks, steps);
      ahead = at;
      const int n = warp >= ws::kEpiWarps && 2 * (warp - ws::kQuantWarp0) < p.M ? n_steps : 0;
#pragma unroll
      for (int u = 0; u < kHeld; ++u) {
        held[u] = u < n ? load(ahead.kb) : make_uint4(0, 0, 0, 0);
        ahead.back(row_blocks, steps);
      }
      // the largest magnitude of every row: the epilogue and quantising warps in equal parts over the rows (all warps over
      // all pieces, with a division and an atomic for each 32, took 0.8 us longer at four rows of 4096)
      constexpr int kLookWarps = ws::kEpiWarps + ws::kQuantWarps, kBatch = 6;
      const int me = warp < ws::kEpiWarps ? warp : warp - (ws::kQuantWarp0 - ws::kEpiWarps);
      const int per_row = kLookWarps / p.M, of = me / per_row, chunks = p.K >> 3;
      if (of < p.M) {
        const uint4* xr = reinterpret_cast<const uint4*>(p.x + (size_t)of * p.K);
        __half2 m2 = __float2half2_rn(0.0f);
        for (int i0 = (me - of * per_row) * 32 + lane; i0 < chunks; i0 += kBatch * per_row * 32) {
          uint4 look[kBatch];
#pragma unroll
          for (int j = 0; j < kBatch; ++j) {
            const int i = i0 + j * per_row * 32;
            look[j] = i < chunks ? xr[i] : make_uint4(0, 0, 0, 0);
          }
#pragma unroll
          for (int j = 0; j < kBatch; ++j) m2 = absmax8(m2, look[j]);
        }
        // (bit patterns of non-negative numbers order as the numbers do)
        __syncwarp();
        const uint32_t top = __reduce_max_sync(0xffffffffu, __float_as_uint(absmax_to_float(m2)));
        if (lane == 0) atomicMax(&s_top[of], top);
      }
      asm volatile("bar.sync 2, %0;" ::"n"(32 * kLookWarps) : "memory");
      // (as in act_quant.cu)
      auto scale_of = [&](int r) {
        const float eps = h2f(f2h(1e-5f));
        return h2f(f2h(__fdiv_rn(fmaxf(__uint_as_float(s_top[r]), eps), 127.0f)));
      };
      if (warp < ws::kEpiWarps) {
        sa_here = warp < p.M ? scale_of(warp) : 0.0f;
      } else {
        // ---------------------------------------------------------- quantising warps
        const float sf = mine ? scale_of(r) : 1.0f;
        const RowQuant rq = make_row_quant(sf);
        int8_t* qr = p.qx + (size_t)r * p.K + 8 * c;
        // row r of the stage's activations, 128 bytes, its 16-byte units swizzled as TMA would
        const uint32_t slot = ws::kWBytes + r * ws::kStepK + (((c >> 1) ^ (r & 7)) << 4) + ((c & 1) << 3);
        int s = 0;
        uint32_t phase = 1;
        bool ok = true;
        for (int i0 = 0; ok && i0 < n; i0 += kHeld) {
#pragma unroll
          for (int u = 0; u < kHeld; ++u) {
            if (i0 + u >= n) break;
            const uint2 codes = quant8_pack(held[u], rq);
            if (i0 + u + kHeld < n) held[u] = load(ahead.kb);
            ahead.back(row_blocks, steps);
            ok = __all_sync(0xffffffffu, mbar_wait(empty0 + 8 * s, phase, abort_flag));
            if (!ok) break;
            if (mine) *reinterpret_cast<uint2*>(base + s * C::kStageBytes + slot) = codes;
            fence_proxy_async_smem();
            mbar_arrive_warp(full0 + 8 * s, lane);
            if (++s == kRing) { s = 0; phase ^= 1; }
            if (at.rb == 0 && mine) {              // the caller's codes and scales, by the blocks of the first 128 rows
              if (at.kb * ws::kStepK + 8 * c < p.K) *reinterpret_cast<uint2*>(qr + at.kb * ws::kStepK) = codes;
              if (at.kb == 0 && c == 0) p.qx_scale[r] = sf;
            }
            at.back(row_blocks, steps);
          }
        }
      }
    }
    // ------------------------------------------------------------ epilogue
    const int quarter = warp & 3, half = warp >> 2;
    const uint32_t lane_field = static_cast<uint32_t>(quarter * 32) << 16;
    const int row = quarter * 32 + lane;
    StreamAt at;
    at.set(n_steps > 0 ? t_hi : 0, row_blocks, steps);
    int d = 0;
    uint32_t dphase = 0;
    for (int t = QUANT && warp >= ws::kEpiWarps ? t_lo - 1 : t_hi; t >= t_lo;) {
      const int seg_lo = max(t_lo, t - at.kb);                  // this segment: steps [seg_lo, t] of one row block
      const bool ends = at.kb == steps - 1, whole = ends && seg_lo == t - at.kb;
      // the first block of this row block (its tiles are added by the block that holds the end)
      const int first_t = t - at.kb;
      const int longer = extra * (even + 1);
      const int first_block = first_t < longer ? first_t / (even + 1) : extra + (first_t - longer) / max(even, 1);
      const int e = grouped ? s_group[at.group] & 0xFF : 0, first_row = grouped ? (s_group[at.group] >> 8) * TOK : 0;
      const int x_row0 = grouped ? p.segments[e] + first_row : 0;
      const int tokens = grouped ? min(p.counts[e] - first_row, TOK) : p.M;
      // (a wait that gave up skips the work but not the barriers: the other warps may have come through)
      const bool ok = __all_sync(0xffffffffu, mbar_wait(dfull0 + 8 * d, dphase, abort_flag));
      tcgen05_fence_after();
      // SwiGLU: 16 tokens of both accumulators per pass; else 32 tokens, 16 per half of the warps
      constexpr int kPass = kParts == 2 ? 16 : 32;
      const int n0 = at.rb * ws::kRows + 4 * lane;
      float sc[kParts][4];
#pragma unroll
      for (int q = 0; q < kParts; ++q)
#pragma unroll
        for (int i = 0; i < 4; ++i)
          sc[q][i] = n0 + i < p.N ? __ldg(p.b_scale + (size_t)e * p.rows_per_expert + q * p.up_row_offset + n0 + i) : 0.0f;
      bool gave_up = !ok;
      for (int m0 = 0; m0 < TOK && m0 < tokens; m0 += kPass) {
        const int mine = kParts == 2 ? m0 : m0 + half * 16;     // first token of this warp's 16 columns
        if (TOK > 16 || kParts == 2 || half == 0) {
          if (ok && mine < TOK) {
            uint32_t r[16];
            stream_tmem_ld_x16(tmem_base + lane_field + (d * kParts + (kParts == 2 ? half : 0)) * TOK + mine, r);
            tmem_ld_wait();
            uint32_t* dst = s_chunk + half * ws::kChunk * ws::kPitch + row;
#pragma unroll
            for (int m = 0; m < 16; ++m) dst[m * ws::kPitch] = r[m];
          }
        }
        asm volatile("bar.sync 1, 256;" ::: "memory");
        const int in_pass = min(min(kPass, TOK - m0), tokens - m0);
        for (int j = warp; j < in_pass && !gave_up; j += ws::kEpiWarps) {
          const int m = m0 + j;
          // words of token m: part 0 (and, SwiGLU, part 1)
          uint4 acc[kParts];
#pragma unroll
          for (int q = 0; q < kParts; ++q)
            acc[q] = *reinterpret_cast<const uint4*>(
                s_chunk + ((kParts == 2 ? q : j >> 4) * ws::kChunk + (j & 15)) * ws::kPitch + 4 * lane);
          if (!ends) {
#pragma unroll
            for (int q = 0; q < kParts; ++q)
              stream_st_v4(p.tiles + (((size_t)blk * kParts + q) * TOK + m) * ws::kRows + 4 * lane,
                           make_uint4(acc[q].x ^ 0x80000000u, acc[q].y ^ 0x80000000u, acc[q].z ^ 0x80000000u,
                                      acc[q].w ^ 0x80000000u));
            continue;
          }
          if (!whole) {
            for (int b2 = first_block; b2 < blk && !gave_up; b2 += 4) {
              uint4 w[4][kParts];
              uint64_t since = 0;
              for (uint32_t it = 1;; ++it) {
                bool there = true;
#pragma unroll
                for (int k = 0; k < 4; ++k)
#pragma unroll
                  for (int q = 0; q < kParts; ++q) {
                    w[k][q] = b2 + k < blk ? stream_ld_v4(p.tiles + (((size_t)(b2 + k) * kParts + q) * TOK + m) * ws::kRows + 4 * lane)
                                           : make_uint4(1u, 1u, 1u, 1u);
                    there = there && w[k][q].x != 0u && w[k][q].y != 0u && w[k][q].z != 0u && w[k][q].w != 0u;
                  }
                if (there) break;
                if ((it & 0x3F) == 0) {
                  const uint64_t now = globaltimer_ns();
                  if (since == 0) since = now;
                  if (now - since > kWaitLimitNs) *abort_flag = 1;
                  if (*abort_flag) { gave_up = true; break; }
                }
              }
#pragma unroll
              for (int k = 0; k < 4; ++k)
                if (b2 + k < blk && !gave_up) {
#pragma unroll
                  for (int q = 0; q < kParts; ++q) {
                    acc[q].x += w[k][q].x ^ 0x80000000u;
                    acc[q].y += w[k][q].y ^ 0x80000000u;
                    acc[q].z += w[k][q].z ^ 0x80000000u;
                    acc[q].w += w[k][q].w ^ 0x80000000u;
                    stream_st_v4(p.tiles + (((size_t)(b2 + k) * kParts + q) * TOK + m) * ws::kRows + 4 * lane,
                                 make_uint4(0u, 0u, 0u, 0u));                      // ready for the next call
                  }
                }
            }
            if (gave_up) break;
          }
          const size_t out_row = (size_t)(x_row0 + m);
          const float sa = QUANT ? sa_here : __ldg(p.a_scale + out_row);       // (QUANT: row j is warp j's)
          __half hv[4];
          if constexpr (EPI == STREAM_SWIGLU) {
            const int* g = reinterpret_cast<const int*>(&acc[0]);
            const int* u = reinterpret_cast<const int*>(&acc[kParts - 1]);
            float hmax = 0.0f;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              hv[i] = swiglu_f16(g[i], u[i], sa, sc[0][i], sc[kParts - 1][i]);
              if (n0 + i < p.N) hmax = fmaxf(hmax, fabsf(h2f(hv[i])));
            }
            const unsigned int top = __reduce_max_sync(0xffffffffu, __float_as_uint(hmax));    // non-negative: ordered as bits
            if (lane == 0) p.row_absmax[out_row * row_blocks + at.rb] = __uint_as_float(top);
          } else {
            const int* a = reinterpret_cast<const int*>(&acc[0]);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              float v;
              if constexpr (EPI == STREAM_AFFINE) {
                v = n0 + i < p.N ? affine_output(a[i], p.K, __ldg(p.a_zero + out_row), __ldg(p.a_rowsum + out_row),
                                                 __ldg(p.b_zero + n0 + i), __ldg(p.b_rowsum + n0 + i), sa, sc[0][i])
                                 : 0.0f;
              } else {
                v = scaled_output(a[i], sa, sc[0][i]);
              }
              if (p.bias && n0 + i < p.N) v = __fadd_rn(v, h2f(p.bias[n0 + i]));
              hv[i] = f2h(v);
            }
          }
          __half* out = static_cast<__half*>(p.out) + out_row * p.N + n0;
          if (n0 + 4 <= p.N && (p.N & 3) == 0) {
            *reinterpret_cast<uint2*>(out) = *reinterpret_cast<const uint2*>(hv);
          } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (n0 + i < p.N) out[i] = hv[i];
          }
        }
        asm volatile("bar.sync 1, 256;" ::: "memory");          // the chunk may be overwritten
      }
      tcgen05_fence_before();
      mbar_arrive_warp(dempty0 + 8 * d, lane);
      if (++d == 2) { d = 0; dphase ^= 1; }
      // on to the next row block
      at.kb = 0;
      at.back(row_blocks, steps);
      t = seg_lo - 1;
    }
  }

  __syncwarp();
  tcgen05_fence_before();
  __syncthreads();
  if (*abort_flag) {
    if (tid == 0 && p.error_word) atomicExch(p.error_word, 6);
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == ws::kMmaWarp) {
    tcgen05_fence_after();
    tmem_dealloc(tmem_base, C::kTmemCols);
  }
}

template <int TOK, int EPI, bool LONG, bool QUANT = false>
static int launch_stream(const CUtensorMap& tw, const CUtensorMap& tx, const StreamParams& p, int grid, cudaStream_t st) {
  using C = ws::Cfg<TOK, EPI, LONG, QUANT>;
  auto kern = w8a8_stream_kernel<TOK, EPI, LONG, QUANT>;
  static thread_local int configured_device = -1;
  int device = 0;
  MP_CUDA_TRY(cudaGetDevice(&device));
  if (configured_device != device) {
    MP_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmem));
    configured_device = device;
  }
  return launch_chained(kern, dim3(grid), dim3(C::kThreads), C::kSmem, st, tw, tx, p);
}

static int stream_tokens(int rows) { return rows <= 16 ? 16 : rows <= 32 ? 32 : 64; }

size_t w8a8_stream_workspace_bytes(int epi, int max_rows) {
  const int parts = epi == STREAM_SWIGLU ? 2 : 1;
  return kW4CounterBytes + (size_t)kSmCount * parts * stream_tokens(max_rows) * ws::kRows * sizeof(uint32_t);
}

int launch_w8a8_stream(int epi, const void* x_i8, int x_rows, const void* w_i8, int w_rows, StreamParams p, int max_rows,
                       void* workspace, size_t workspace_bytes, cudaStream_t st) {
  if (max_rows > kStreamMaxExpertRows || p.K % 16 != 0 || p.K >= (1 << 17) || p.experts > ws::kMaxExperts)
    return MP_ERR_UNSUPPORTED;
  if (!workspace || workspace_bytes < w8a8_stream_workspace_bytes(epi, max_rows) || !aligned(workspace, 16))
    return MP_ERR_UNSUPPORTED;
  if (!aligned(x_i8, 16) || !aligned(w_i8, 16) || !aligned(p.out, 8)) return MP_ERR_UNSUPPORTED;
  const int tok = stream_tokens(max_rows);
  CUtensorMap tw, tx;
  int rc = encode_tensor_map_2d(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, w_i8, (uint64_t)p.K, (uint64_t)w_rows, (uint64_t)p.K,
                                ws::kStepK, ws::kRows);
  if (rc != MP_OK) return rc;
  p.x_box = x_rows < tok ? x_rows : tok;
  rc = encode_tensor_map_2d(&tx, CU_TENSOR_MAP_DATA_TYPE_UINT8, x_i8, (uint64_t)p.K, (uint64_t)x_rows, (uint64_t)p.K,
                            ws::kStepK, p.x_box);
  if (rc != MP_OK) return rc;
  p.steps = (p.K + ws::kStepK - 1) / ws::kStepK;
  p.row_blocks = (p.N + ws::kRows - 1) / ws::kRows;
  // grouped: an expert is taken again for every `tok` rows it has beyond the first
  const int groups = p.counts ? min(p.experts + x_rows / tok, ws::kMaxGroups) : 1;
  const long long most = (long long)groups * p.row_blocks * p.steps;
  if (most > (1 << 24)) return MP_ERR_UNSUPPORTED;
  // as in w4a16_decode_umma.cu: at b steps per block a row block costs b steps and steps / b tiles; a tile costs about 0.4
  // (16 tokens) to 0.7 (64) steps
  const int tile_cost_x10 = tok == 16 ? 4 : tok == 32 ? 5 : 7;
  p.min_share = 2;
  while (p.min_share * p.min_share * 10 < p.steps * tile_cost_x10) ++p.min_share;
  p.tiles = reinterpret_cast<uint32_t*>(static_cast<unsigned char*>(workspace) + kW4CounterBytes);
  const long long want = (most + p.min_share - 1) / p.min_share;
  const int grid = want < kSmCount ? (int)want : kSmCount;
  // (with every expert taken once)
  const long long stages = (long long)(p.counts ? p.experts : 1) * p.row_blocks * p.steps * (epi == STREAM_SWIGLU ? 2 : 1);
  const bool is_long = stages >= (long long)ws::long_stream(tok, p.x != nullptr) * grid;
  if (p.x) {
    if (epi != STREAM_F16 || max_rows > ws::kMaxQuantRows || !aligned(p.x, 16)) return MP_ERR_UNSUPPORTED;
    return is_long ? launch_stream<16, STREAM_F16, true, true>(tw, tx, p, grid, st)
                       : launch_stream<16, STREAM_F16, false, true>(tw, tx, p, grid, st);
  }
#define MP_STREAM_EPI(TOK, EPI) \
  return is_long ? launch_stream<TOK, EPI, true>(tw, tx, p, grid, st) : launch_stream<TOK, EPI, false>(tw, tx, p, grid, st);
#define MP_STREAM(TOK)                                     \
  switch (epi) {                                           \
    case STREAM_F16: MP_STREAM_EPI(TOK, STREAM_F16)        \
    case STREAM_AFFINE: MP_STREAM_EPI(TOK, STREAM_AFFINE)  \
    default: MP_STREAM_EPI(TOK, STREAM_SWIGLU)             \
  }
  switch (tok) {
    case 16: MP_STREAM(16)
    case 32: MP_STREAM(32)
    default: MP_STREAM(64)
  }
#undef MP_STREAM_EPI
#undef MP_STREAM
}

// ---- the W8A8 linears: quantisation of the rows, then the product -------------------------------------------------
static size_t split_bytes(int M, int N, int K) { return mp_w8a8_gemm_workspace_bytes(M, N, K); }
constexpr size_t kSplitOffset = kW4CounterBytes + kW4TileBytes;
static bool stream_rows(int M, int K) { return M <= kStreamMaxRows && K % 16 == 0 && K < (1 << 17); }

// Rows quantised inside the product: every block reads all of x for the rows' maxima, at about 45 bytes a clock, which has to
// cost less than the kernel that it saves.  The four products of a Llama-8B layer, us, with the quantisation before / inside
// all of them: 1 row 56.9 / 50.0, 4 rows 58.2 / 52.3, 6 rows 58.9 / 54.6, 8 rows 59.2 / 56.6 (56.1 without the 8 x 14336 one);
// of a Llama-70B layer 1 row 157.1 / 146.1, 4 rows 159.8 / 151.8 (155.6 without 4 x 28672), 8 rows 162.9 / 161.5 (161.3).
// x may not share memory with what other blocks write meanwhile.
static bool overlap(const void* a, size_t a_bytes, const void* b, size_t b_bytes) {
  const char *p = static_cast<const char*>(a), *q = static_cast<const char*>(b);
  return p < q + b_bytes && q < p + a_bytes;
}
static bool quantise_in_stream(const void* x, const void* qx, const void* scale, const void* y, int M, int N, int K) {
  if (!x || M <= 0 || K <= 0 || !stream_rows(M, K) || (long long)M * K > (M <= 6 ? 131072 : 65536)) return false;
  const size_t values = (size_t)M * K;
  return !overlap(x, 2 * values, qx, values) && !overlap(x, 2 * values, scale, 4 * (size_t)M) &&
         !overlap(x, 2 * values, y, 2 * (size_t)M * N);
}

static size_t linear_workspace_bytes(int epi, int M, int N, int K) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (stream_rows(M, K)) return w8a8_stream_workspace_bytes(epi, M);
  const size_t split = split_bytes(M, N, K);
  return split ? kSplitOffset + split : 0;
}

}  // namespace mp

using namespace mp;

extern "C" size_t mp_w8a8_linear_workspace_bytes(int M, int N, int K) { return linear_workspace_bytes(STREAM_F16, M, N, K); }

extern "C" int mp_w8a8_linear(const void* x_f16, const void* w_i8, const void* w_scale_f32, const void* bias_f16, void* y_f16,
                              int M, int N, int K, void* qx_i8, void* x_scale_f32, void* workspace, size_t workspace_bytes,
                              int* error_word, mp_stream_t stream) {
  if (!w_i8 || !w_scale_f32 || !y_f16 || !qx_i8 || !x_scale_f32 || N <= 0) return MP_ERR_INVALID_ARG;
  StreamParams p{};
  p.M = M; p.N = N; p.K = K;
  p.b_scale = static_cast<const float*>(w_scale_f32);
  p.bias = static_cast<const __half*>(bias_f16);
  p.out = y_f16;
  p.error_word = error_word;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (quantise_in_stream(x_f16, qx_i8, x_scale_f32, y_f16, M, N, K)) {
    p.x = static_cast<const __half*>(x_f16);
    p.qx = static_cast<int8_t*>(qx_i8);
    p.qx_scale = static_cast<float*>(x_scale_f32);
    const int rc = launch_w8a8_stream(STREAM_F16, qx_i8, M, w_i8, N, p, M, workspace, workspace_bytes, st);
    if (rc != MP_ERR_UNSUPPORTED) return rc;
    p.x = nullptr;
  }
  int rc = mp_act_quant_per_token(x_f16, M, K, qx_i8, x_scale_f32, nullptr, stream);
  if (rc != MP_OK) return rc;
  if (stream_rows(M, K)) {
    p.early_weights = 1;                 // the kernel before is the quantisation, which waited for everything older
    p.a_scale = static_cast<const float*>(x_scale_f32);
    rc = launch_w8a8_stream(STREAM_F16, qx_i8, M, w_i8, N, p, M, workspace, workspace_bytes, st);
    if (rc != MP_ERR_UNSUPPORTED) return rc;
  }
  const bool scratch = workspace && workspace_bytes > kSplitOffset;
  return mp_w8a8_gemm_ex(qx_i8, x_scale_f32, w_i8, w_scale_f32, bias_f16, y_f16, M, N, K,
                         scratch ? static_cast<unsigned char*>(workspace) + kSplitOffset : nullptr,
                         scratch ? workspace_bytes - kSplitOffset : 0, error_word, stream);
}

extern "C" size_t mp_w8a8_affine_linear_workspace_bytes(int M, int N, int K) {
  return linear_workspace_bytes(STREAM_AFFINE, M, N, K);
}

extern "C" int mp_w8a8_affine_linear(const void* x_f16, const void* w_u8, const void* w_scale_f32, const void* w_zero_f32,
                                     const void* w_rowsum_i32, const void* bias_f16, void* y_f16, int M, int N, int K,
                                     void* qx_u8, void* x_scale_f32, void* x_zero_f32, void* x_rowsum_i32, void* workspace,
                                     size_t workspace_bytes, int* error_word, mp_stream_t stream) {
  if (!w_u8 || !w_scale_f32 || !w_zero_f32 || !w_rowsum_i32 || !y_f16 || !qx_u8 || !x_scale_f32 || !x_zero_f32 ||
      !x_rowsum_i32 || N <= 0)
    return MP_ERR_INVALID_ARG;
  if ((long long)K * 255 * 255 > 2147483647LL) return MP_ERR_UNSUPPORTED;   // the unsigned sums must fit int32
  int rc = mp_affine_quant_per_row(x_f16, M, K, qx_u8, x_scale_f32, x_zero_f32, x_rowsum_i32, nullptr, stream);
  if (rc != MP_OK) return rc;
  if (stream_rows(M, K)) {
    StreamParams p{};
    p.M = M; p.N = N; p.K = K;
    p.early_weights = 1;
    p.a_scale = static_cast<const float*>(x_scale_f32);
    p.b_scale = static_cast<const float*>(w_scale_f32);
    p.a_zero = static_cast<const float*>(x_zero_f32);
    p.a_rowsum = static_cast<const int*>(x_rowsum_i32);
    p.b_zero = static_cast<const float*>(w_zero_f32);
    p.b_rowsum = static_cast<const int*>(w_rowsum_i32);
    p.bias = static_cast<const __half*>(bias_f16);
    p.out = y_f16;
    p.error_word = error_word;
    rc = launch_w8a8_stream(STREAM_AFFINE, qx_u8, M, w_u8, N, p, M, workspace, workspace_bytes,
                            static_cast<cudaStream_t>(stream));
    if (rc != MP_ERR_UNSUPPORTED) return rc;
  }
  const bool scratch = workspace && workspace_bytes > kSplitOffset;
  return w8a8_affine_gemm(qx_u8, x_scale_f32, x_zero_f32, x_rowsum_i32, w_u8, w_scale_f32, w_zero_f32, w_rowsum_i32, bias_f16,
                          y_f16, M, N, K, scratch ? static_cast<unsigned char*>(workspace) + kSplitOffset : nullptr,
                          scratch ? workspace_bytes - kSplitOffset : 0, error_word, static_cast<cudaStream_t>(stream));
}
