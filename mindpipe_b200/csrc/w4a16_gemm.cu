// W4A16 product for many tokens: y[M,N] = x[M,K] @ dequant(W)[N,K]^T on the fp16 tensor cores, the int4 unpack and
// group dequantisation fused in as a producer stage.
//
// The weights are the A operand, in tensor memory: a pair of CTAs (a cluster of 2, cta_group::2) multiplies 256 weight
// rows -- 128 in each CTA -- with up to 256 tokens, whose activations are the B operand, half of them in each CTA's shared
// memory.  Why this way round:
//   * expanded weights never pass through shared memory.  Per 256 columns of K a CTA takes 16 KB of packed words and at
//     256 tokens 64 KB of activations into shared memory and reads them once, 1250 clocks at 128 B/clk, beside 2048 clocks
//     of MMA.  With the expanded tile as B in shared memory (512 tokens x 256 rows to a pair) it was 1800 of 2048, and a
//     batch of 129 rows was multiplied as 256, one of 300 as 512.
//   * the tokens are the MMA's N, any multiple of 32, so little is multiplied for padding.
//   * expanding 32768 weights takes the SM's ALUs 660 clocks of those 2048.
// A persistent pair per two SMs, roles by warp:
//   warps 0-11   expansion, three sets of four warps taking 128-column steps in turn: a lane holds a weight row, makes
//                exactly f16((u - z) * s) of its words and stores them to a tensor memory slot
//   warps 12-19  epilogue: accumulators -> fp16 (+ bias), transposed through shared memory -> y; or fp32 partial tiles
//   warp 20      TMA producer of the packed words (256 columns a stage)
//   warp 21      MMA issuer (the even CTA's)
//   warp 22      TMA producer of the activations (128 columns a step)
// Work is cut in one of three ways, whichever an estimate of clocks says is shortest (see w4_gemm_shape): whole tiles to a
// pair; a tile shared by a cluster of two or four pairs, each with its part of K, which exchange their sums through
// distributed shared memory; or, with scratch, an equal run of all tiles' steps to every pair, the tiles cut in between left
// as fp32 partial tiles that a second kernel adds in K order.  Whole tiles and clusters are the usual ones; equal runs win
// where K is long beside few tiles that do not fill the pairs (97 rows of 1024 x 28672, 300 rows of 8192 x 28672).
//
// Measured (us, groups of 128; in brackets the form it replaces, expanded weights as the B operand in shared memory):
// 12288 x 4096 at 129 / 333 / 512 / 2048 rows 22.0 / 35.8 / 42.1 / 155.8 [40.8 / 59.7 / 59.6 / 171.6], 4096 x 11008 at
// 129 / 2048 rows 23.5 / 142.4 [38.1 / 149.5].  With many rows the MMAs bound it (1050 clocks a step of 1024 at 256 tokens,
// 5000 of 38000 a tile in the epilogue); below 160 rows the expansion warps (about 800 a step).
//
// With the warp's number a uniform value (uniform_warp, tc.cuh) the single-thread roles issue faster: the four linears of a
// 7B layer at 100 / 200 / 333 rows 89.6 / 115.5 / 141.5 -> 87.2 / 112.9 / 139.8.
//
// Every mbarrier wait is bounded (tc.cuh); on a timeout the pair records an error word, lets its copies land, frees its
// tensor memory and returns.
#include <algorithm>

#include "common.cuh"
#include "tc.cuh"

namespace mp {

using namespace tc;

namespace w4 {
constexpr int kRows = 128;                 // weight rows of a CTA
constexpr int kStepK = 128, kStageK = 256;
constexpr int kSets = 3;
constexpr int kEpiWarp0 = 4 * kSets, kEpiWarps = 8, kWeightWarp = kEpiWarp0 + kEpiWarps, kMmaWarp = kWeightWarp + 1,
              kXWarp = kWeightWarp + 2;
constexpr int kThreads = 32 * (kXWarp + 1);
constexpr int kStageBytes = kRows * kStageK / 2;
constexpr int kMaxT = 256;
constexpr int kSlotCols = kStepK / 2;      // tensor memory columns of a step's expanded weights
constexpr int kMaxSlots = 6, kMaxRing = 8;
constexpr int kRingBytes = 192 * 1024;     // both rings
constexpr int kStagingBytes = kEpiWarps * 4096;           // two chunks of 32 tokens x 32 rows for each epilogue warp
constexpr int kTailBytes = 512;
constexpr size_t kSmem = 1024 + kRingBytes + kStagingBytes + kTailBytes;
constexpr int kTmemCols = 512;
constexpr int kPairs = kSmCount / 2;

__host__ __device__ constexpr int accumulators(int T) { return T <= 128 ? 2 : 1; }
__host__ __device__ constexpr int x_step_bytes(int T) { return T / 2 * kStepK * 2; }
// Slots of a step's operands: tensor memory for the expanded weights, shared memory for the activations.  There are four
// or more, and at least as many weight stages, see the waits of the expansion.
__host__ __device__ constexpr int slots(int T) {
  int n = (kTmemCols - accumulators(T) * T) / kSlotCols;
  if (n > kMaxSlots) n = kMaxSlots;
  while ((kRingBytes - n * x_step_bytes(T)) / kStageBytes < n) --n;
  return n;
}
__host__ __device__ constexpr int ring(int T) {
  const int n = (kRingBytes - slots(T) * x_step_bytes(T)) / kStageBytes;
  return n < kMaxRing ? n : kMaxRing;
}
static_assert(slots(256) == 4 && slots(128) == 4 && slots(160) == 5 && slots(192) == 4 && slots(224) == 4 && ring(256) == 4 && ring(160) == 5, "rings");
}  // namespace w4

struct W4GemmParams {
  const uint32_t* sz;       // [K/group, N] (scale, zero) f16 pairs
  const __half* bias;
  __half* y;
  int M, N, K, group;
  int T;                    // tokens of a tile, a multiple of 32
  int m_tiles, steps;       // tiles along the tokens; 128-column steps of a tile
  int unit_steps;           // 1, or `steps` when pairs take whole tiles
  int split;                // > 1: a cluster of this many pairs shares a tile, a pair takes steps / split of it
  int share, extra;         // units of a pair: share, one more for the first `extra` pairs
  float* partial;           // [pair][2][rank][T / 4][128][4 tokens]: the first segment of a pair that begins inside a tile, and the last
                            // one that ends inside a tile whose beginning it holds
  int* error_word;
};

__host__ __device__ inline int w4_range_start(int pair, int share, int extra) {
  return pair * share + (pair < extra ? pair : extra);
}
__device__ __forceinline__ int w4_pair_of(int unit, int share, int extra) {
  const int longer = extra * (share + 1);
  return unit < longer ? unit / (share + 1) : extra + (unit - longer) / share;
}

// A pair's walk over its units: one segment per tile.
struct W4Segment {
  int tile, s0, s1;         // steps [s0, s1) of the tile
};

// D[tmem] (+)= A[tmem] * B[smem] over a CTA pair: M = 256, 128 lanes of A and D in each CTA's tensor memory, B's rows
// split in halves between the two shared memories.
template <bool ACCUMULATE = true>
__device__ __forceinline__ void umma_f16_ts_pair(uint32_t tmem_d, uint32_t tmem_a, uint32_t desc_lo, uint32_t desc_hi,
                                                 uint32_t idesc, bool accumulate = true) {
  if (ACCUMULATE) {
    asm volatile(
        "{\n\t.reg .b64 b;\n\tmov.b64 b, {%2, %3};\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], b, %4, 1;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "r"(desc_lo), "r"(desc_hi), "r"(idesc) : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .b64 b;\n\t.reg .pred p;\n\tmov.b64 b, {%2, %3};\n\tsetp.ne.b32 p, %5, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], b, %4, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "r"(desc_lo), "r"(desc_hi), "r"(idesc), "r"(static_cast<uint32_t>(accumulate))
        : "memory");
  }
}

__device__ __forceinline__ uint4 w4_lds_v4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}

// One packed word -> f16((u - z) * s) of its eight columns in order.
__device__ __forceinline__ void expand_word(uint32_t word, const ScaleZero& sp, uint32_t* out) {
  __half2 v[4];
  dequant8(word, sp, v);
  const uint32_t a = h2_as_u32(v[0]), b = h2_as_u32(v[1]), c = h2_as_u32(v[2]), d = h2_as_u32(v[3]);
  out[0] = prmt(a, b, 0x5410);
  out[1] = prmt(c, d, 0x5410);
  out[2] = prmt(a, b, 0x7632);
  out[3] = prmt(c, d, 0x7632);
}

// Rows n and n + 1 of up to four tokens from `m` on.
__device__ __forceinline__ void store_quad(const W4GemmParams& p, int m, int tokens, int n, const float (&a)[4],
                                           const float (&b)[4]) {
  const float bias0 = p.bias ? h2f(p.bias[n]) : -0.0f, bias1 = p.bias && n + 1 < p.N ? h2f(p.bias[n + 1]) : -0.0f;
  __half* y = p.y + (size_t)m * p.N + n;
#pragma unroll
  for (int j = 0; j < 4; ++j, y += p.N) {
    if (j >= tokens) break;
    const __half2 h = __floats2half2_rn(a[j] + bias0, b[j] + bias1);
    if (p.N % 2 == 0) {
      *reinterpret_cast<__half2*>(y) = h;
    } else {
      y[0] = __low2half(h);
      if (n + 1 < p.N) y[1] = __high2half(h);
    }
  }
}

__global__ void __launch_bounds__(w4::kThreads, 1)
w4a16_gemm_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w,
                  const W4GemmParams p) {
  using namespace w4;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int T = p.T, n_slots = slots(T), n_w = ring(T), n_acc = accumulators(T);
  const int x_bytes = x_step_bytes(T), x_half = x_bytes / 2;
  unsigned char* tail = smem + kRingBytes + kStagingBytes;
  const uint32_t xring = smem_u32(smem), wring = xring + n_slots * x_bytes, staging = xring + kRingBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(tail);
  const uint32_t wfull0 = smem_u32(bars);                  // packed words landed
  const uint32_t wempty0 = wfull0 + 8 * kMaxRing;          // ... and were read
  const uint32_t ready0 = wempty0 + 8 * kMaxRing;          // leader: both CTAs' halves of a slot's operands are in place
  const uint32_t done0 = ready0 + 8 * kMaxSlots;           // ... and were multiplied
  const uint32_t tfull0 = done0 + 8 * kMaxSlots;           // a segment's accumulator is complete
  const uint32_t tempty0 = tfull0 + 16;                    // leader: both CTAs have read it
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tail + 8 * (2 * kMaxRing + 2 * kMaxSlots + 4));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const uint32_t cta = cluster_ctarank(), rank = cta & 1u, leader_cta = cta & ~1u;
  const bool leader = rank == 0;
  const int pair = static_cast<int>(blockIdx.x) >> 1, steps = p.steps, split = p.split;
  // this pair's steps
  int u0, u1;
  if (split > 1) {
    const int tile = pair / split, i = pair - tile * split;
    u0 = tile * steps + steps * i / split;
    u1 = tile * steps + steps * (i + 1) / split;
  } else {
    u0 = w4_range_start(pair, p.share, p.extra) * p.unit_steps;
    u1 = w4_range_start(pair + 1, p.share, p.extra) * p.unit_steps;
  }
  // the segment that begins at unit u
  auto segment_at = [&](int u, W4Segment& g) {
    g.tile = u / steps;
    g.s0 = u - g.tile * steps;
    g.s1 = min(steps, g.s0 + u1 - u);
  };
  auto first_row = [&](int tile) { return (tile / p.m_tiles) * (2 * kRows) + static_cast<int>(rank) * kRows; };

  // weight producer: where its walk stands, and a stage's load
  W4Segment wg{0, 0, 0};
  int w_end = u0, w_st = 0, w_row = 0;
  auto next_stage = [&]() {                    // false: none left
    if (w_st > (wg.s1 - 1) >> 1 || w_end == u0) {
      if (w_end >= u1) return false;
      segment_at(w_end, wg);
      w_end += wg.s1 - wg.s0;
      w_st = wg.s0 >> 1;
      w_row = first_row(wg.tile);
    }
    return true;
  };
  auto load_stage = [&](int s) {
    mbar_arrive_expect_tx(wfull0 + 8 * s, kStageBytes);
    tma_load_2d(wring + s * kStageBytes, &tmap_w, wfull0 + 8 * s, w_st++ * (kStageK / 2), w_row);
  };
  bool w_more = false;

  // the barriers of the first weights, which come while the rest is set up, are this CTA's own
  if (warp == kWeightWarp) {
    if (elect_one()) {
      for (int s = 0; s < n_w; ++s) {
        mbar_init(wfull0 + 8 * s, 1);
        mbar_init(wempty0 + 8 * s, 8);                     // four warps for each of the stage's two steps
      }
      fence_mbar_init();
    }
  } else if (warp == kXWarp) {
    if (elect_one()) {
      prefetch_tensormap(&tmap_x);
      for (int q = 0; q < n_slots; ++q) {
        mbar_init(ready0 + 8 * q, 9);                      // four warps of each CTA, the leader's TMA producer
        mbar_init(done0 + 8 * q, 1);
      }
      for (int b = 0; b < 2; ++b) {
        mbar_init(tfull0 + 8 * b, 1);
        mbar_init(tempty0 + 8 * b, 2 * kEpiWarps);
      }
      *abort_flag = 0;
      fence_mbar_init();
    }
  } else if (warp == kMmaWarp) {
    tmem_alloc_pair(smem_u32(tmem_slot), kTmemCols);
    tmem_relinquish_pair();
  }
  __syncwarp();
  tcgen05_fence_before();
  cluster_arrive();              // the peer's barriers exist before anything signals them
  chain_wait();
  chain_release();
  if (warp == kWeightWarp && elect_one()) {      // (tensor memory and the cluster's barrier take about 1.1 us)
    for (int s = 0; s < n_w; ++s) {
      w_more = next_stage();
      if (!w_more) break;
      load_stage(s);
    }
  }
  __syncwarp();
  cluster_wait();                // (and this CTA's: every thread of the cluster takes part)
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == kWeightWarp) {
    if (w_more) {                              // the thread that issued the first loads
      int s = 0;
      uint32_t phase = 0;
      while (next_stage()) {
        if (!mbar_wait(wempty0 + 8 * s, phase, abort_flag)) break;
        load_stage(s);
        if (++s == n_w) { s = 0; phase ^= 1; }
      }
    }
  } else if (warp == kXWarp) {
    if (elect_one()) {
      const uint32_t ready_leader0 = map_to_cta(ready0, leader_cta);
      int s = 0;
      uint32_t phase = 1;
      bool ok = true;
      W4Segment g;
      for (int u = u0; ok && u < u1; u += g.s1 - g.s0) {
        segment_at(u, g);
        const int m0 = (g.tile % p.m_tiles) * T + static_cast<int>(rank) * (T / 2);
        for (int st = g.s0; st < g.s1; ++st) {
          if (!mbar_wait(done0 + 8 * s, phase, abort_flag)) { ok = false; break; }
          const int k0 = st * kStepK;
          const bool both = k0 + 64 < p.K;
          if (leader) mbar_arrive_expect_tx(ready0 + 8 * s, both ? 2 * x_bytes : x_bytes);     // of both CTAs
          tma_load_2d_pair(xring + s * x_bytes, &tmap_x, ready_leader0 + 8 * s, k0, m0);
          if (both) tma_load_2d_pair(xring + s * x_bytes + x_half, &tmap_x, ready_leader0 + 8 * s, k0 + 64, m0);
          if (++s == n_slots) { s = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == kMmaWarp) {
    if (leader && elect_one()) {
      const uint32_t idesc = umma_idesc(kIdescDFormatF32 | kIdescABFormatF16, 2 * kRows, T);
      const unsigned short pair_mask = static_cast<unsigned short>(3u << leader_cta);
      // This thread's instructions wait their turn among those of the expansion: at 160 tokens and fewer they set the pace, so
      // a step has as few as possible.
      const uint64_t b_desc0 = umma_desc_k_sw128(xring);
      const uint32_t desc_hi = static_cast<uint32_t>(b_desc0 >> 32), desc_lo0 = static_cast<uint32_t>(b_desc0);
      const uint32_t a0 = tmem_base + n_acc * T, slot_step = x_bytes >> 4, half_step = x_half >> 4;
      uint32_t desc = desc_lo0, a_tmem = a0;
      int q = 0, d = 0;
      uint32_t phase = 0, dphase = 1;
      bool ok = true;
      W4Segment g;
      for (int u = u0; ok && u < u1; u += g.s1 - g.s0) {
        segment_at(u, g);
        if (!mbar_wait(tempty0 + 8 * d, dphase, abort_flag)) break;
        const uint32_t d_tmem = tmem_base + d * T;
        for (int st = g.s0; st < g.s1; ++st) {
          if (!mbar_wait(ready0 + 8 * q, phase, abort_flag)) { ok = false; break; }
          tcgen05_fence_after();
          // 16 K per instruction: 8 columns of A, 32 bytes of B's rows
          umma_f16_ts_pair<false>(d_tmem, a_tmem, desc, desc_hi, idesc, st != g.s0);
#pragma unroll
          for (int kk = 1; kk < 4; ++kk) umma_f16_ts_pair(d_tmem, a_tmem + kk * 8, desc + 2 * kk, desc_hi, idesc);
          if (st * kStepK + 64 < p.K) {
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              umma_f16_ts_pair(d_tmem, a_tmem + 32 + kk * 8, desc + half_step + 2 * kk, desc_hi, idesc);
          }
          umma_commit_both(done0 + 8 * q, pair_mask);
          desc += slot_step;
          a_tmem += kSlotCols;
          if (++q == n_slots) { q = 0; phase ^= 1; desc = desc_lo0; a_tmem = a0; }
        }
        if (!ok) break;
        umma_commit_both(tfull0 + 8 * d, pair_mask);
        if (++d == n_acc) { d = 0; dphase ^= 1; }
      }
    }
  } else if (warp < kEpiWarp0) {
    // ---- expansion: this warp's 32 rows of every third step
    const int quarter = warp & 3, set = warp >> 2;
    const int row = quarter * 32 + lane, sw = row & 7;
    const uint32_t a_tmem0 = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + n_acc * T;
    const uint32_t ready_leader0 = map_to_cta(ready0, leader_cta);
    const int sub_blocks = p.K / 64, g64 = p.group / 64;
    // x / d for the small quotients here is the high word of x * ceil(2^32 / d), d > 1
    const uint32_t by_slots = 0xffffffffu / n_slots + 1, by_ring = 0xffffffffu / n_w + 1, by_group = 0xffffffffu / g64 + 1;
    W4Segment g{0, 0, 0};
    int n = 0, end = u0;                       // the segment's row, and the unit after it
    int stage0 = 0, stages = 0;                // its first weight stage's number in this pair's run, and how many it has
    auto seek = [&](int u) {
      while (u >= end) {
        stage0 += stages;
        segment_at(end, g);
        stages = ((g.s1 - 1) >> 1) - (g.s0 >> 1) + 1;
        end += g.s1 - g.s0;
        n = min(first_row(g.tile) + row, p.N - 1);
      }
      return g.s1 - (end - u);
    };
    // (scale, zero) of this row for the step's two blocks of 64 columns.  Two loads, the same word twice or not: a copy of
    // one would wait for it here.  Rows and columns that do not exist take another's; nothing of theirs is kept.
    auto load_sz = [&](int st, uint32_t (&z)[2]) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int b = min(2 * st + i, sub_blocks - 1);
        const int grp = g64 == 1 ? b : static_cast<int>(__umulhi(static_cast<uint32_t>(b), by_group));
        z[i] = __ldg(p.sz + (size_t)grp * p.N + n);
      }
    };
    int u = u0 + set, st = 0;
    uint32_t sz_next[2];
    if (u < u1) {
      st = seek(u);
      load_sz(st, sz_next);
    }
    while (u < u1) {
      const int use = static_cast<int>(__umulhi(static_cast<uint32_t>(u - u0), by_slots)), q = u - u0 - use * n_slots;
      const int stage = stage0 + (st >> 1) - (g.s0 >> 1);
      const int lap = static_cast<int>(__umulhi(static_cast<uint32_t>(stage), by_ring)), s = stage - lap * n_w;
      const int reads = (st ^ 1) < g.s0 || (st ^ 1) >= g.s1 ? 2 : 1;    // the stage's other step may not be this pair's
      const int h = st & 1;
      const bool both = 2 * st + 1 < sub_blocks;                         // K may end in the middle of the step
      const uint32_t sz_now[2] = {sz_next[0], sz_next[1]};
      u += kSets;
      if (u < u1) {                            // the next step's scales arrive while this one is expanded
        st = seek(u);
        load_sz(st, sz_next);
      }
      // The slot first: the unit three before this one waited for the unit n_slots before it, which is no earlier than the
      // slot's use before its last one, so the barrier's parity is not ambiguous; and when the unit n_slots before this one
      // is done, every stage n_w >= n_slots before this one has been filled and read, so the stage's is not either.
      if (!__all_sync(0xffffffffu, mbar_wait(done0 + 8 * q, (use & 1) ^ 1, abort_flag) &&
                                       mbar_wait(wfull0 + 8 * s, lap & 1, abort_flag))) break;
      tcgen05_fence_after();
      const uint32_t src = wring + s * kStageBytes + row * 128;
      uint4 w[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) w[j] = w4_lds_v4(src + (((h * 4 + j) ^ sw) << 4));
      const uint32_t a_tmem = a_tmem0 + q * kSlotCols;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (j == 2 && !both) break;
        const __half2 szh = *reinterpret_cast<const __half2*>(&sz_now[j >> 1]);
        const ScaleZero sp = make_scale_zero(__low2half(szh), __high2half(szh));
        uint32_t r[16];
        expand_word(w[j].x, sp, r);
        expand_word(w[j].y, sp, r + 4);
        expand_word(w[j].z, sp, r + 8);
        expand_word(w[j].w, sp, r + 12);
        tmem_st_32x32_x16(a_tmem + j * 16, r);
      }
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(wempty0 + 8 * s);
        if (reads == 2) mbar_arrive(wempty0 + 8 * s);
      }
      tmem_st_wait();
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_tmem(ready_leader0 + 8 * q);
    }
  } else {
    // ---- epilogue: lane = weight row, column = token; two warps to a quarter of the rows take 32 tokens in turn
    const int quarter = warp & 3, half = (warp - kEpiWarp0) >> 2;
    const int row = quarter * 32 + lane;
    const uint32_t tempty_leader0 = map_to_cta(tempty0, leader_cta);
    const uint32_t stage = staging + (warp - kEpiWarp0) * 4096;
    const bool vec = p.N % 8 == 0;
    int d = 0;
    uint32_t dphase = 0;
    W4Segment g;
    for (int u = u0; u < u1; u += g.s1 - g.s0) {
      segment_at(u, g);
      const int n0 = first_row(g.tile) + quarter * 32, n = n0 + lane, m0 = (g.tile % p.m_tiles) * T;
      const bool whole = g.s0 == 0 && g.s1 == steps;
      const float bias = p.bias && n < p.N ? h2f(p.bias[n]) : 0.0f;
      if (!__all_sync(0xffffffffu, mbar_wait(tfull0 + 8 * d, dphase, abort_flag))) break;
      if (split > 1) break;                    // its one segment; exchanged below
      tcgen05_fence_after();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + d * T;
      const int last = min(T, p.M - m0);                     // tokens that exist
      const int chunks = (last - 32 * half + 63) >> 6;       // of 32 tokens; this warp's are c, c + 2, ...: four at most
      uint32_t r[32], h[16];
      auto load = [&](int i) { tmem_ld_32x32(taddr + 32 * half + 64 * i, r); };
      auto pack = [&](uint32_t (&h)[16]) {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          float v0 = __uint_as_float(r[2 * j]), v1 = __uint_as_float(r[2 * j + 1]);
          if (p.bias) { v0 += bias; v1 += bias; }
          h[j] = h2_as_u32(__floats2half2_rn(v0, v1));
        }
      };
      // a chunk through shared memory: 16 token pairs x 32 rows of words; the 16-byte pieces of odd pairs trade places,
      // against bank conflicts
      auto stage_chunk = [&](const uint32_t (&h)[16], int buf) {
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 16; ++j)
          asm volatile("st.shared.u32 [%0], %1;" ::"r"(stage + buf * 2048 + j * 128 + (((lane >> 2) ^ (j & 1)) << 4) + (lane & 3) * 4), "r"(h[j]) : "memory");
        __syncwarp();
      };
      auto flush = [&](int buf, int i) {
        const int c0 = 32 * half + 64 * i;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int j = k * 8 + (lane >> 2), piece = (lane & 3) * 2, t = c0 + 2 * j;      // pair of tokens, eight rows
          const uint32_t src = stage + buf * 2048 + j * 128;
          const uint4 a = w4_lds_v4(src + ((piece ^ (j & 1)) << 4)), b = w4_lds_v4(src + (((piece + 1) ^ (j & 1)) << 4));
          __half* dst = p.y + (size_t)(m0 + t) * p.N + n0 + (lane & 3) * 8;
          if (t < last)
            *reinterpret_cast<uint4*>(dst) = make_uint4(prmt(a.x, a.y, 0x5410), prmt(a.z, a.w, 0x5410), prmt(b.x, b.y, 0x5410), prmt(b.z, b.w, 0x5410));
          if (t + 1 < last)
            *reinterpret_cast<uint4*>(dst + p.N) = make_uint4(prmt(a.x, a.y, 0x7632), prmt(a.z, a.w, 0x7632), prmt(b.x, b.y, 0x7632), prmt(b.z, b.w, 0x7632));
        }
      };
      auto release = [&]() {
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_tmem(tempty_leader0 + 8 * d);
      };
      if (!whole) {
        float* dst = p.partial + (((size_t)pair * 2 + (g.s0 == 0)) * 2 + rank) * ((size_t)T * kRows) + row * 4;
#pragma unroll 1
        for (int i = 0; i < chunks; ++i) {
          load(i);
          tmem_ld_wait();
          uint4* to = reinterpret_cast<uint4*>(dst + (32 * half + 64 * i) * kRows);
#pragma unroll
          for (int j = 0; j < 8; ++j) to[j * kRows] = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
        }
        release();
      } else if (vec && n0 + 32 <= p.N) {
        // The accumulator is given back as soon as its last columns are in registers: nothing is stored to memory before
        // (with the chunks stored one after another the MMAs waited 5800 clocks a tile for 256 tokens).
        if (chunks > 0) load(0);
        tmem_ld_wait();
        if (chunks <= 1) release();
        if (chunks > 0) pack(h);
        if (chunks > 1) load(1);
        if (chunks > 0) stage_chunk(h, 0);
        if (chunks > 1) {
          tmem_ld_wait();
          if (chunks == 2) release();
          pack(h);
          if (chunks > 2) load(2);
          stage_chunk(h, 1);
        }
        if (chunks > 2) {
          tmem_ld_wait();
          if (chunks == 3) release();
          pack(h);
        }
        if (chunks > 3) {
          load(3);
          tmem_ld_wait();
          release();
        }
        if (chunks > 0) flush(0, 0);
        if (chunks > 2) stage_chunk(h, 0);
        if (chunks > 1) flush(1, 1);
        if (chunks > 3) {
          pack(h);
          stage_chunk(h, 1);
        }
        if (chunks > 2) flush(0, 2);
        if (chunks > 3) flush(1, 3);
      } else {
#pragma unroll 1
        for (int i = 0; i < chunks; ++i) {
          load(i);
          tmem_ld_wait();
          pack(h);
          const int c0 = 32 * half + 64 * i;
          __half* y = p.y + (size_t)(m0 + c0) * p.N + n;
          if (n < p.N) {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (c0 + j < last)
                y[(size_t)j * p.N] = __ushort_as_half(static_cast<unsigned short>((j & 1) ? h[j >> 1] >> 16 : h[j >> 1]));
          }
        }
        release();
      }
      if (++d == n_acc) { d = 0; dphase ^= 1; }
    }
  }

  // a CTA that gave up tells its peer (whose waits poll the flag) before both meet at the cluster barrier; the peer
  // cannot have left yet, so its shared memory is still there
  __syncwarp();
  if (*abort_flag && lane == 0) st_cluster_u32(map_to_cta(smem_u32(const_cast<int*>(abort_flag)), cta ^ 1u), 1u);
  __syncwarp();
  cluster_arrive();       // the leader's MMAs read the peer's shared memory: nobody leaves early
  cluster_wait();
  if (split > 1) {
    // Every CTA of the cluster has finished its products and its rings are free.  CTA (i, rank) gets, from the CTAs of its
    // rank, their sums of the i-th part of the tile's tokens, adds them in K order and stores that part.  Through global
    // memory the partial tiles took 2.1 us to write and about 4 to read again (12 MB each way at 160 tokens).
    const int tile = pair / split, i = pair - tile * split;
    const int m0 = (tile % p.m_tiles) * T, last = min(T, p.M - m0);
    const int quads = T / (4 * split);                       // of tokens, a CTA's part
    if (warp >= kEpiWarp0 && warp < kEpiWarp0 + kEpiWarps) {
      const int quarter = warp & 3, half = (warp - kEpiWarp0) >> 2;
      const uint32_t own = xring + static_cast<uint32_t>(i * quads * kRows + quarter * 32 + lane) * 16;
      tcgen05_fence_after();
      for (int c0 = 32 * half; c0 < last; c0 += 64) {
        uint32_t r[32];
        tmem_ld_32x32(tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + c0, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int quad = c0 / 4 + j, to = quad / quads;
          const uint32_t dst = map_to_cta(own + static_cast<uint32_t>(quad - to * quads) * kRows * 16, 2 * to + rank);
          asm volatile("st.shared::cluster.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(dst), "r"(r[4 * j]), "r"(r[4 * j + 1]),
                       "r"(r[4 * j + 2]), "r"(r[4 * j + 3]) : "memory");
        }
      }
      tcgen05_fence_before();
    }
    __syncwarp();
    cluster_arrive();
    cluster_wait();
    const int n0 = first_row(tile);
    for (int e = threadIdx.x; e < quads * (kRows / 2); e += kThreads) {
      const int quad = e / (kRows / 2), row = (e % (kRows / 2)) * 2, t = (i * quads + quad) * 4, n = n0 + row;
      if (t >= last || n >= p.N) continue;
      float v[2][4] = {};
      for (int from = 0; from < split; ++from) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const uint4 w = w4_lds_v4(xring + static_cast<uint32_t>((from * quads + quad) * kRows + row + k) * 16);
          v[k][0] += __uint_as_float(w.x); v[k][1] += __uint_as_float(w.y);
          v[k][2] += __uint_as_float(w.z); v[k][3] += __uint_as_float(w.w);
        }
      }
      store_quad(p, m0 + t, min(4, last - t), n, v[0], v[1]);
    }
    __syncthreads();
  }
  if (*abort_flag) {
    if (threadIdx.x == 0 && p.error_word) atomicExch(p.error_word, 2);
    const uint64_t t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == kMmaWarp) {
    tcgen05_fence_after();
    tmem_dealloc_pair(tmem_base, kTmemCols);
  }
}

// The tiles that more than one pair worked on: y = f16(sum of their partial tiles in K order (+ bias)).  Block (b, z): the
// tile in which pair b + 1 begins, slice z of its tokens.
__global__ void __launch_bounds__(256)
w4a16_gemm_reduce_kernel(const W4GemmParams p) {
  chain_wait();
  chain_release();
  const int start = w4_range_start(static_cast<int>(blockIdx.x) + 1, p.share, p.extra);
  const int tile = start / p.steps;
  if (start == tile * p.steps) return;                       // the pair begins with the tile
  const int first = w4_pair_of(tile * p.steps, p.share, p.extra);
  if (first != static_cast<int>(blockIdx.x)) return;         // an earlier boundary in the same tile does it
  const int last = w4_pair_of((tile + 1) * p.steps - 1, p.share, p.extra);
  const int m0 = (tile % p.m_tiles) * p.T, n0 = (tile / p.m_tiles) * (2 * w4::kRows);
  const int tokens = min(p.T, p.M - m0);
  const size_t tile_words = (size_t)p.T * w4::kRows;
  // two rows of four tokens to a thread
  const int i = blockIdx.y * 256 + threadIdx.x, t = (i / w4::kRows) * 4, r = (i % w4::kRows) * 2;
  if (t >= tokens) return;
  const int rank = r / w4::kRows;
  const float4* src = reinterpret_cast<const float4*>(p.partial + rank * tile_words + (size_t)t * w4::kRows) + (r - rank * w4::kRows);
  const size_t pair_step = tile_words;                         // four tiles of four words
  float4 a = src[first * pair_step + tile_words / 2], b = src[first * pair_step + tile_words / 2 + 1];
  for (int q = first + 1; q <= last; q += 4) {                 // four requests at a time
    float4 va[4], vb[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (q + j <= last) {
        va[j] = src[(q + j) * pair_step];
        vb[j] = src[(q + j) * pair_step + 1];
      }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (q + j <= last) {
        a.x += va[j].x; a.y += va[j].y; a.z += va[j].z; a.w += va[j].w;
        b.x += vb[j].x; b.y += vb[j].y; b.z += vb[j].z; b.w += vb[j].w;
      }
  }
  const int n = n0 + r;
  if (n >= p.N) return;
  const float va[4] = {a.x, a.y, a.z, a.w}, vb[4] = {b.x, b.y, b.z, b.w};
  store_quad(p, m0 + t, min(4, tokens - t), n, va, vb);
}

static void w4_launch_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* cluster, int pairs, int split) {
  cfg.gridDim = dim3(2 * pairs, 1, 1);
  cfg.blockDim = dim3(w4::kThreads, 1, 1);
  cfg.dynamicSmemBytes = w4::kSmem;
  cluster->id = cudaLaunchAttributeClusterDimension;
  cluster->val.clusterDim.x = 2 * split;
  cluster->val.clusterDim.y = 1;
  cluster->val.clusterDim.z = 1;
  cfg.attrs = cluster;
  cfg.numAttrs = 1;
}

// How a product is cut, by the shortest estimate in SM clocks: the tokens of a tile, and then
//   * whole tiles to a pair, in as many waves as it takes;
//   * a tile to a cluster of two or four pairs, which exchange their sums through their shared memories;
//   * with scratch, an equal run of all tiles' steps to every pair, the cut tiles added by a second kernel.
// A step is 4 T clocks of MMA but no less than the 600 of its expansion, and 110 for its barriers; the last tile's
// epilogue 16 T.  The exchange in a cluster takes about 4000 and 16 T, the second kernel 4000 and, with the partial tiles'
// way to L2 and back, 100 T.  With these the choice was the fastest of all cuts, or within 4 % of it, over 65..1024 rows of
// seven shapes from 2688 x 2944 to 22016 x 4096.
struct W4Shape {
  int T;
  int split;                // pairs to a tile
  bool runs;                // equal runs
  int pairs;
};
struct W4Device {
  int id = -1;
  int clusters[3];          // clusters of 1, 2, 4 pairs that fit the device at once
};
static int w4_device(const W4Device** out) {
  static thread_local W4Device d;
  *out = &d;
  int device = 0;
  MP_CUDA_TRY(cudaGetDevice(&device));
  if (d.id == device) return MP_OK;
  MP_CUDA_TRY(cudaFuncSetAttribute(w4a16_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)w4::kSmem));
  for (int i = 0; i < 3; ++i) {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr;
    w4_launch_config(cfg, &attr, w4::kPairs / 4 * 4, 1 << i);
    MP_CUDA_TRY(cudaOccupancyMaxActiveClusters(&d.clusters[i], w4a16_gemm_kernel, &cfg));
  }
  d.id = device;
  return MP_OK;
}

static W4Shape w4_gemm_shape(int M, int N, int K, bool scratch, const int (&clusters)[3]) {
  const long long n_tiles = (N + 2 * w4::kRows - 1) / (2 * w4::kRows), steps = (K + w4::kStepK - 1) / w4::kStepK;
  W4Shape best{};
  long long best_cost = -1;
  auto offer = [&](long long cost, const W4Shape& shape) {
    if (best_cost >= 0 && cost >= best_cost) return;
    best_cost = cost;
    best = shape;
  };
  for (int T = w4::kMaxT; T >= 32; T -= 32) {
    const long long tiles = n_tiles * ((M + T - 1) / T), units = tiles * steps;
    const long long step = std::max(4 * T, 600) + 110, waves = (tiles + w4::kPairs - 1) / w4::kPairs;
    offer(waves * steps * step + 16 * T, W4Shape{T, 1, false, (int)std::min<long long>(tiles, w4::kPairs)});
    for (int i = 1; i <= 2; ++i) {
      const int split = 1 << i;
      if (tiles > clusters[i] || steps < 2 * split) continue;
      offer((steps + split - 1) / split * step + 4000 + (16 + 16 / split) * T, W4Shape{T, split, false, (int)tiles * split});
    }
    const long long pairs = std::min<long long>(w4::kPairs, units / 4);
    if (!scratch || pairs < 2 || (units % pairs == 0 && units / pairs % steps == 0)) continue;
    offer((units + pairs - 1) / pairs * step + 4000 + 116 * T, W4Shape{T, 1, true, (int)pairs});
  }
  return best;
}

static size_t w4_partial_bytes(int pairs, int T) { return (size_t)pairs * 4 * T * w4::kRows * sizeof(float); }

static W4Shape w4_gemm_shape_here(int M, int N, int K) {
  const W4Device* d;
  const int none[3] = {0, 0, 0};
  return w4_gemm_shape(M, N, K, true, w4_device(&d) == MP_OK ? d->clusters : none);
}

// What the chosen cut writes: partial tiles for equal runs, nothing for whole tiles and clusters.
size_t w4a16_gemm_partial_bytes(int M, int N, int K) {
  if (M <= 0 || N <= 0 || K <= 0 || K % 64 != 0) return 0;
  const W4Shape s = w4_gemm_shape_here(M, N, K);
  return s.runs ? w4_partial_bytes(s.pairs, s.T) : 0;
}

}  // namespace mp

using namespace mp;

// What the entry with scratch insists on: the same, and for fewer pairs than the device has also where the cut writes none of
// it (a smaller buffer has always been refused there).
extern "C" size_t mp_w4a16_prefill_workspace_bytes(int M, int N, int K) {
  if (M <= 0 || N <= 0 || K <= 0 || K % 64 != 0) return 0;
  const W4Shape s = w4_gemm_shape_here(M, N, K);
  return s.runs || s.pairs < w4::kPairs ? w4_partial_bytes(s.pairs, s.T) : 0;
}

extern "C" int mp_w4a16_linear_prefill(const void* x_f16, const void* packed_i32, const void* sz_f16x2,
                                       const void* bias_f16, void* y_f16, int M, int N, int K, int group,
                                       int* error_word, mp_stream_t stream) {
  return mp_w4a16_linear_prefill_ex(x_f16, packed_i32, sz_f16x2, bias_f16, y_f16, M, N, K, group, nullptr, 0,
                                    error_word, stream);
}

extern "C" int mp_w4a16_linear_prefill_ex(const void* x_f16, const void* packed_i32, const void* sz_f16x2,
                                          const void* bias_f16, void* y_f16, int M, int N, int K, int group,
                                          void* workspace, size_t workspace_bytes, int* error_word,
                                          mp_stream_t stream) {
  if (!x_f16 || !packed_i32 || !sz_f16x2 || !y_f16 || M <= 0 || N <= 0 || K <= 0 || group <= 0) return MP_ERR_INVALID_ARG;
  if (K % 64 != 0 || group % 64 != 0 || K % group != 0) return MP_ERR_UNSUPPORTED;
  if (!aligned(x_f16, 16) || !aligned(packed_i32, 16) || !aligned(sz_f16x2, 4) || !aligned(y_f16, 16)) return MP_ERR_ALIGNMENT;
  const W4Device* d;
  int rc = w4_device(&d);
  if (rc != MP_OK) return rc;
  const W4Shape shape = w4_gemm_shape(M, N, K, workspace != nullptr, d->clusters);
  if (workspace) {
    if (workspace_bytes < mp_w4a16_prefill_workspace_bytes(M, N, K)) return MP_ERR_WORKSPACE;
    if (!aligned(workspace, 16)) return MP_ERR_ALIGNMENT;
  }
  CUtensorMap tx, tw;
  rc = encode_tensor_map_2d(&tx, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, x_f16, (uint64_t)K, (uint64_t)M, (uint64_t)K * 2, 64,
                                shape.T / 2);
  if (rc != MP_OK) return rc;
  rc = encode_tensor_map_2d(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, packed_i32, (uint64_t)K / 2, (uint64_t)N, (uint64_t)K / 2,
                            w4::kStageK / 2, w4::kRows);
  if (rc != MP_OK) return rc;
  W4GemmParams p{};
  p.sz = static_cast<const uint32_t*>(sz_f16x2);
  p.bias = static_cast<const __half*>(bias_f16);
  p.y = static_cast<__half*>(y_f16);
  p.M = M; p.N = N; p.K = K; p.group = group;
  p.T = shape.T;
  p.m_tiles = (M + shape.T - 1) / shape.T;
  p.steps = (K + w4::kStepK - 1) / w4::kStepK;
  p.error_word = error_word;
  const long long tiles = (long long)p.m_tiles * ((N + 2 * w4::kRows - 1) / (2 * w4::kRows)), units = tiles * p.steps;
  if (units > 2000000000LL) return MP_ERR_UNSUPPORTED;
  p.split = shape.split;
  const long long parts = shape.runs ? units : tiles;       // shared out evenly (split > 1: by the cluster's place)
  p.share = (int)(parts / shape.pairs);
  p.extra = (int)(parts % shape.pairs);
  p.unit_steps = shape.runs ? 1 : p.steps;
  p.partial = static_cast<float*>(workspace);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr[2];
  w4_launch_config(cfg, attr, shape.pairs, shape.split);
  cfg.stream = st;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.numAttrs = 2;
  MP_CUDA_TRY(cudaLaunchKernelEx(&cfg, w4a16_gemm_kernel, tx, tw, p));
  if (!shape.runs) return MP_OK;
  return launch_chained(w4a16_gemm_reduce_kernel, dim3(shape.pairs - 1, (shape.T / 4 * w4::kRows + 255) / 256), dim3(256), 0, st, p);
}
