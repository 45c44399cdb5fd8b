// W4A16 linear for up to 128 rows (above 96 the linear's dispatch sends small weights to the GEMM) on the tcgen05 tensor core
// with the weights as the TENSOR-MEMORY operand: y = x @ dequant(W)^T, the packed weights streamed once.
//
// A thread owns ONE weight row: it reads its row of a stage from the shared-memory ring, expands it and stores the packed
// registers straight into tensor memory (tcgen05.st, lane = row, column = pair of K).  One elected
// thread then issues tcgen05.mma kind::f16 with A = those TMEM columns (128 rows x 16 K per instruction), B = the
// activation tile in shared memory (token rows, K-major, 128-byte swizzle) and the fp32 accumulator [128 rows x tokens]
// in TMEM.  No dequantised weight touches shared or global memory, and no dequant warp issues an MMA, shuffles a fragment
// or touches an activation.
//
// What bounds it (clocks per 16 KB stage of weights and SM; HBM delivers one in about 700):
//   expansion   alone, twelve warps: exact f16((u - z) * s) in order 750 (17 instructions per eight weights, nine of them half
//               rate); FOLD, the exact integers u - z with the group's scale applied to its dot product, 460, of which the
//               stores to tensor memory are 230.  Four warps, one on each scheduler, take 540, eight 480.
//   MMA         16 instructions of N / 2 clocks (operand A in tensor memory): 154 at 16 tokens, 768 at 96
//   producer    one thread per stream, weights and activations, with no division in their loops (with both streams in one
//               thread this was what held the kernel at 0.45 of HBM)
// every role has its own warps and its own barriers, and none waits for another that is not its input.
//
// FOLD (up to 16 rows, groups of a multiple of 128 columns): the accumulator of every 128-column unit is read back by
// the epilogue warps, which add scale * dot to fp32 registers: more accurate than the fp16-rounded f16((u - z) * s) and
// three instructions per eight weights cheaper.  Otherwise (more rows, shorter groups) the exact form accumulates in TMEM.
//
// Work is cut stream-K style: the (row block, 256-column stage) pairs form one sequence divided evenly over a persistent
// grid of one block per SM.  A block walks its range BACKWARDS.  Of the row blocks in its range only the first it meets
// can continue in later blocks: that part's fp32 tile goes to the block's slot in the workspace.  Any other row block ends
// inside the range, and the block that holds a row block's end adds the tiles of the earlier blocks and writes y.  So a
// block waits only for blocks of lower number, which wrote their tile at the beginning of their range, and adds in block
// order (results are identical from run to run).  A tile word is stored inverted and zero means "not there yet": the
// reader polls the words themselves (bounded) and puts the zeros back, with no fence, counter or second round trip.
//
// Warps, by role and in this order (Cfg has the numbers):
//   16 (or 12)   expansion: two sets of eight take stages in turn, a warp does 32 rows of half a stage; three sets of four and
//                whole stages for the exact form up to 16 rows (see Cfg::kParts).  At the end they fetch the tiles of the row
//                block that this block closes
//   4            epilogue
//   1            TMA producer of weights and (scale, zero) pairs
//   1            TMEM allocation and the MMA issuer
//   1            TMA producer of activations
//   1            side warp: copies from host memory, in a launch that brings some; tiles to L2 from 17 to 64 rows.  Up to 16
//                rows only a launch that brings copies has it
// Expansion emits the columns of a packed word in the order (k0,k4,k1,k5,k2,k6,k3,k7).  Up to 16 rows the expansion warps
// apply the same permutation in place to the 16-byte chunks of the stage's activation tile (a chunk is one token's eight
// columns of one word, so the swizzle does not matter); with more rows they put the words back in order, see Cfg.  (Warps
// of their own for the permutation were starved by the expansion warps: 2100 clocks per stage with one; in the epilogue warps it
// took a 7B layer at 16 rows from 42 to 49 us.)
// One block fills an SM: its ring is what hides HBM's latency.  Smaller blocks, two of them to an SM so that the next linear
// of a chain starts beside the end of this one, took 38 us where this takes 28 (28672x8192, 16 rows).
// What a launch costs beyond the stream: 1.3 us from the end of the kernel before to the first MMA, 1.3 from the last MMA to the
// last block's end.  The first was 2.1 to 2.9 with the whole ring requested before the activations, which then queued behind
// it, and the (scale, zero) pairs not brought to L2 with the weights; the second 2 to 2.6, and 5 at 77 rows, with the tiles
// read, an element at a time, after the last MMA.  Measured without early weights (us; in brackets that form): 12288x4096 at 16
// rows 9.4 [11.5], 10240x8192 at 8 12.0 [14.4], 28672x8192 at 8 25.6 [28.5], 12288x4096 at 77 13.6 [16.2].  Streaming the
// same bytes with nothing done to them takes 5.0, 8.0, 19.0 and 5.0.
// Every wait is bounded.
#include "common.cuh"
#include "tc.cuh"

namespace mp {

using namespace tc;

namespace du {
constexpr int kRows = 128;
constexpr int kStageK = 256;
constexpr int kSlots = 3;                             // stages between expansion and MMA: stage i is in slot i % 3
constexpr int kWBytes = kRows * (kStageK / 2);        // 16384
constexpr int kMaxRing = 8, kMaxXRing = 8;          // (eight weight stages; ten 1 to 5 % slower: 40960x8192 at 8 rows 36.3 us, 34.7 with eight)
// Weight stages requested before the activations, which queue behind them: with early weights the time up to the wait for
// the kernel before is theirs (12288x4096 at 16 rows in a chain, us: 4 or 5 stages 9.2, 6 9.5, the whole ring 10.1).
constexpr int kFirstEarly = 5, kFirst = 1;
// Stages brought to L2 while the kernel before ends.  A prefetch and the load after it cost L2 more than the load alone (us
// without early weights, 3 / 4 / 6 / 10 stages: 4096x4096 at 1 row 5.20 / 5.38 / 5.36 / 5.31, 12288x4096 at 16 9.22 / 9.13 /
// 9.40 / 9.92 and at 77 13.20 / 13.03 / 13.06 / 13.43, 8192x28672 at 8 24.95 / 24.85 / 24.74 / 25.29, 28672x8192 at 8 24.46 /
// 24.44 / 24.67 / 25.20; groups of 64: 12288x4096 at 16 10.14 / 10.10 / 10.34 / 10.93, 8192x28672 at 8 28.69 / 27.83 / 28.44 /
// 29.37).
constexpr int kPrefetch = 4;
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kASlotCols = kStageK / 2;          // two columns of K per 32-bit register
constexpr size_t kSmemMax = 224 * 1024;

template <int N>
struct Int { static constexpr int value = N; };

// TOK: token rows of the MMA (its N); XROWS: token rows of the activation tile in shared memory (8 where no more exist:
// the MMA then reads whatever follows for the other eight, whose results are not used)
// CARRY: a warp more, for copies from host memory
template <int TOK, int XROWS, bool FOLD, bool CARRY>
struct Cfg {
  // the columns of an expanded word come out as (k0,k4) (k1,k5) ..: the activations are put into that order, in shared
  // memory, or (PERM false) the words back into theirs.  Permuting the activations of 64 tokens per block and stage cost the
  // expansion warps a third of their time, permuting them in a kernel of its own 2 us a call.
  static constexpr int kTokens = XROWS;               // that can exist
  static constexpr bool PERM = TOK <= 16;
  // Warps that share 32 rows of a stage.  Two, in two sets, have a stage expanded soonest; where a stage costs both the exact
  // products and the permutation, one to a stage in three sets spends less on barriers (us without early weights, halves /
  // whole stages: 28672x8192 at 8 rows 25.6 / 28.1, 10240x8192 12.0 / 13.8, 4096x4096 at 48 8.5 / 9.5; groups of 64:
  // 8192x28672 at 9 rows 40.1 / 34.9).
  static constexpr int kParts = PERM && !FOLD ? 1 : 2;
  static constexpr int kSets = kParts == 1 ? 3 : 2;       // expansion sets, a stage each in turn
  static constexpr int kPieces = 8 / kParts;              // 16-byte pieces of a row that a warp does
  static constexpr int kEpiWarp0 = 4 * kParts * kSets;
  static constexpr int kWeightWarp = kEpiWarp0 + 4, kMmaWarp = kWeightWarp + 1, kXWarp = kMmaWarp + 1;
  static constexpr int kSideWarp = kXWarp + 1;
  static constexpr int kThreads = 32 * (kSideWarp + (CARRY ? 1 : 0));
  static constexpr int kXSub = XROWS * 128;           // [XROWS x 64 columns] fp16
  static constexpr int kXBytes = (PERM ? 4 : 2) * kXSub;        // a tile of the ring: a stage, or half of one
  // activation tiles in flight: enough to hide the latency of their loads behind the stages before (with one per slot the
  // expansion warps waited half their time); with PERM at most six, see the wait for a slot
  static constexpr int kXRing = TOK <= 64 ? 6 : 4;
  // accumulators: FOLD two per slot (one for each 128 columns), else one per segment in turn
  static constexpr int kAccs = FOLD ? 2 * kSlots : TOK > 64 ? 1 : 2;
  static constexpr uint32_t kASlot0 = kAccs * TOK;
  static_assert(kASlot0 + kSlots * kASlotCols <= kTmemCols, "tensor memory");
};
__host__ __device__ constexpr int sz_bytes(int groups_per_stage) { return (groups_per_stage * kRows * 4 + 1023) & ~1023; }
constexpr int kBars = 2 * kMaxRing + 2 * kMaxXRing + 2 * kSlots + 4;
constexpr int kScaleWords = kSlots * 2 * 2 * kRows;   // [slot][use parity][half][row]
constexpr int kTailBytes = kBars * 8 + kScaleWords * 4 + 64;
constexpr int kMaxGrid = kSmCount;
// The least stages a block is given.  More blocks per row block shorten the stream but lengthen the closing step, which
// reads a tile per block: at b stages per block a row block of ST stages takes about b stages + ST / b tiles, so b is the
// root of ST times the cost of a tile in stages (0.4 at 16 tokens to 1 at 128; 1024x8192 at 16 tokens: 7.0 us with b = 2,
// 6.3 with 4).
inline int min_share(int stages_per_row, int tok) {
  const int tile_cost_x10 = tok == 16 ? 4 : tok <= 32 ? 5 : tok <= 64 ? 7 : tok <= 96 ? 9 : 10;
  int b = 2;
  while (b * b * 10 < stages_per_row * tile_cost_x10) ++b;
  return b;
}
__host__ __device__ constexpr int tokens_for(int M) { return M <= 16 ? 16 : (M + 15) / 16 * 16; }
// workspace: the other kernels' arrival counters | one tile per block
constexpr size_t kTileOffset = kW4CounterBytes;
static_assert(kW4TileBytes >= (size_t)kMaxGrid * 128 * kRows * sizeof(uint32_t), "tiles");
// (tiles of 16 tokens: at 77 rows 80 are multiplied where tiles of 32 took 96, 12288x4096 13.6 -> 13.0 us, 28672x8192 at 48
// rows 36.5 -> 34.5)
inline size_t workspace_bytes(int M) { return kTileOffset + (size_t)kMaxGrid * tokens_for(M) * kRows * sizeof(uint32_t); }
}  // namespace du

struct DecodeUmmaParams {
  const __half* bias;
  __half* y;
  int M, N, K, group;
  int stages_per_row;      // ST = ceil(K / 256)
  int share, extra;        // stages per block: share, one more for the first `extra` blocks
  int groups_per_stage;    // rows of the (scale, zero) box
  int gshift;              // log2(group) for groups of up to 128 columns
  int ring;                // weight stages in the ring
  int first;               // weight stages requested before the activations, at most `ring`
  int early_weights;       // 1: fetch weights before the previous kernel of the stream has finished
  int early_tiles;         // 1: tiles to L2 before the first stage (up to 16 rows)
  uint32_t* tiles;         // workspace: [grid][TOK][128] inverted fp32 words, zero between calls
  int* error_word;
};

// The list of copies is in the arguments, and the warp that copies in the block, of the launches that bring copies alone: in
// all of them they cost four captured linears of a 7B layer at 16 rows 0.15 us (41.15 -> 41.00), a 70B layer at 8 rows 0.5
// (106.4 -> 105.8), and the exact form up to 16 rows a spilled register.  Beyond 16 rows nothing is carried, but the forms keep
// list and warp: the compiler's code without them is slower (us: 1024x8192 at 48 rows 10.5 -> 10.8, 12288x4096 at 64 12.3 ->
// 12.6, 8192x8192 at 96 16.8 -> 17.2).
template <bool CARRY>
struct DecodeUmmaArgs : DecodeUmmaParams {};
template <>
struct DecodeUmmaArgs<true> : DecodeUmmaParams {
  HostCopies copies;       // from host memory, every block its share; count 0: none
};

// The stage range of block b is [range_start(b), range_start(b + 1)): p.share stages each, one more for the first p.extra.
__device__ __forceinline__ int range_start(int b, const DecodeUmmaParams& p) { return b * p.share + min(b, p.extra); }
// the block whose range holds stage t
__device__ __forceinline__ int block_of(int t, const DecodeUmmaParams& p) {
  const int longer = p.extra * (p.share + 1);
  return t < longer ? t / (p.share + 1) : p.extra + (t - longer) / p.share;
}


__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}

// D[tmem] (+)= A[tmem] * B[smem]: the A operand is read from tensor memory (lane = row, one 32-bit
// column = two consecutive K elements), 16 K per instruction.
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint32_t desc_lo, uint32_t desc_hi,
                                            uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .b64 b;\n\t.reg .pred p;\n\tmov.b64 b, {%2, %3};\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %4, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "r"(desc_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Shared-memory accesses by 32-bit shared-window address (the 1 KB-aligned ring pointer hides the address space from the
// compiler; plain dereferences of it are generic loads and stores).
__device__ __forceinline__ uint4 du_lds_v4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint32_t du_lds_u32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ void du_sts_v4(uint32_t addr, const uint4& v) {
  asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w));
}
__device__ __forceinline__ void du_sts_u32(uint32_t addr, uint32_t v) {
  asm volatile("st.shared.u32 [%0], %1;" ::"r"(addr), "r"(v));
}
__device__ __forceinline__ uint4 ld_relaxed_gpu_v4(const uint32_t* p) {
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void prefetch_l2(const uint32_t* p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}
__device__ __forceinline__ void st_relaxed_gpu_v4_zero(uint32_t* p) {
  asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1,%1,%1,%1};" ::"l"(p), "r"(0u) : "memory");
}
__device__ __forceinline__ void st_relaxed_gpu(uint32_t* p, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// eight fp16 values (k0..k7) -> (k0,k4,k1,k5,k2,k6,k3,k7), the column order of an expanded word
__device__ __forceinline__ uint4 pair_permute_u4(const uint4 in) {
  uint4 v;
  v.x = prmt(in.x, in.z, 0x5410);
  v.y = prmt(in.x, in.z, 0x7632);
  v.z = prmt(in.y, in.w, 0x5410);
  v.w = prmt(in.y, in.w, 0x7632);
  return v;
}

// (k0,k4) (k1,k5) (k2,k6) (k3,k7) -> (k0,k1) .. (k6,k7)
__device__ __forceinline__ void in_order(uint32_t* v) {
  const uint32_t a = prmt(v[0], v[1], 0x5410), b = prmt(v[2], v[3], 0x5410);
  const uint32_t c = prmt(v[0], v[1], 0x7632), d = prmt(v[2], v[3], 0x7632);
  v[0] = a; v[1] = b; v[2] = c; v[3] = d;
}

// One packed word -> the exact fp16 integers u - z of its eight columns, in dequant8's order.  zl = 1024 + z and
// zh = 64 + z: the even nibbles are planted in the mantissa of 1024 (step 1), the odd ones, left in place, in that of
// 64 (step 1/16), so both differences are exact.
__device__ __forceinline__ void expand8(uint32_t q, __half2 zl, __half2 zh, uint32_t* v) {
  const uint32_t q8 = q >> 8;
  const uint32_t a = lop3_and_or(q, 0x000f000fu, 0x64006400u), b = lop3_and_or(q, 0x00f000f0u, 0x54005400u);
  const uint32_t c = lop3_and_or(q8, 0x000f000fu, 0x64006400u), d = lop3_and_or(q8, 0x00f000f0u, 0x54005400u);
  v[0] = h2_as_u32(__hsub2(*reinterpret_cast<const __half2*>(&a), zl));
  v[1] = h2_as_u32(__hsub2(*reinterpret_cast<const __half2*>(&b), zh));
  v[2] = h2_as_u32(__hsub2(*reinterpret_cast<const __half2*>(&c), zl));
  v[3] = h2_as_u32(__hsub2(*reinterpret_cast<const __half2*>(&d), zh));
}

template <int TOK, int XROWS, bool FOLD, bool CARRY>
__global__ void __launch_bounds__(du::Cfg<TOK, XROWS, FOLD, CARRY>::kThreads, 1)
w4a16_decode_umma_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                         const __grid_constant__ CUtensorMap tmap_sz, const DecodeUmmaArgs<CARRY> p) {
  using C = du::Cfg<TOK, XROWS, FOLD, CARRY>;
  constexpr int kXSub = C::kXSub, kXBytes = C::kXBytes, kXRing = C::kXRing;
  constexpr bool PERM = C::PERM;
  extern __shared__ unsigned char smem_raw[];
  // activation ring | weight ring | barriers, scales, flags
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int stage_bytes = du::kWBytes + du::sz_bytes(p.groups_per_stage);
  unsigned char* tail = base + kXRing * kXBytes + p.ring * stage_bytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(tail);
  uint32_t* s_scale = reinterpret_cast<uint32_t*>(bars + du::kBars);
  uint32_t* tmem_slot = s_scale + du::kScaleWords;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const uint32_t xring = smem_u32(base), wring = xring + kXRing * kXBytes;
  const uint32_t full0 = smem_u32(bars);                      // a stage's weights landed
  const uint32_t empty0 = full0 + 8 * du::kMaxRing;           // its weights have been read
  const uint32_t xempty0 = empty0 + 8 * du::kMaxRing;         // activation tile has been read
  const uint32_t xfull0 = xempty0 + 8 * du::kMaxXRing;        // activation tile landed
  const uint32_t ready0 = xfull0 + 8 * du::kMaxXRing;         // slot holds an expanded stage (FOLD: and its accumulators are free)
  const uint32_t done0 = ready0 + 8 * du::kSlots;             // its MMAs are complete
  const uint32_t dfull0 = done0 + 8 * du::kSlots;             // not FOLD: a segment's accumulator is complete
  const uint32_t dempty0 = dfull0 + 16;                       // ... and has been read

  const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;
  const int blk = static_cast<int>(blockIdx.x);
  const int ST = p.stages_per_row;
  const int t_lo = range_start(blk, p), t_hi = range_start(blk + 1, p) - 1;   // walked from t_hi down
  const int n_stages = t_hi - t_lo + 1;

  // whether the block's last segment ends a row block that earlier blocks began, whose tiles it then adds (see the expansion)
  const int rb_lo = t_lo / ST;
  const bool closes = t_lo > rb_lo * ST && t_hi >= rb_lo * ST + ST - 1;
  constexpr int kExpThreads = 32 * C::kEpiWarp0;
  constexpr int kMine = (C::kTokens * (du::kRows / 4) + kExpThreads - 1) / kExpThreads;     // elements of an expansion thread
  float others[kMine][4];

  // weight producer: the stage it is at (its first loads are issued before the block is set up)
  int w_row = 0, w_st = 0;
  auto group_of = [&](int st) { return p.group <= du::kStageK ? st * p.groups_per_stage : (st * du::kStageK) / p.group; };
  auto load_weights = [&](int s) {
    const uint32_t full = full0 + 8 * s, dst = wring + s * stage_bytes;
    mbar_arrive_expect_tx(full, du::kWBytes + p.groups_per_stage * du::kRows * 4);
    tma_load_2d(dst, &tmap_w, full, w_st * (du::kStageK / 2), w_row);
    tma_load_2d(dst + du::kWBytes, &tmap_sz, full, w_row, group_of(w_st));
    if (--w_st < 0) { w_st = ST - 1; w_row -= du::kRows; }
  };
  if (warp == C::kWeightWarp) {
    if (elect_one()) {
      for (int s = 0; s < p.ring; ++s) {
        mbar_init(full0 + 8 * s, 1);
        mbar_init(empty0 + 8 * s, 4 * C::kParts);
      }
      fence_mbar_init();
      w_row = (t_hi / ST) * du::kRows;
      w_st = t_hi % ST;
      if (!p.early_weights) {
        for (int s = 0, row = w_row, st = w_st; s < du::kPrefetch && s < n_stages; ++s) {     // to L2 while the kernel before ends
          tma_prefetch_2d(&tmap_sz, row, group_of(st));
          tma_prefetch_2d(&tmap_w, st * (du::kStageK / 2), row);
          if (--st < 0) { st = ST - 1; row -= du::kRows; }
        }
        chain_wait();
      }
      for (int s = 0; s < p.first && s < n_stages; ++s) load_weights(s);
    }
  } else if (warp == C::kXWarp) {
    if (elect_one()) {
      prefetch_tensormap(&tmap_x);
      for (int s = 0; s < kXRing; ++s) {
        mbar_init(xempty0 + 8 * s, 1);
        mbar_init(xfull0 + 8 * s, 1);
      }
      for (int q = 0; q < du::kSlots; ++q) {
        mbar_init(ready0 + 8 * q, 4 * C::kParts + (FOLD ? 4 : 0));
        mbar_init(done0 + 8 * q, 1);
      }
      for (int d = 0; d < 2; ++d) {
        mbar_init(dfull0 + 8 * d, 1);
        mbar_init(dempty0 + 8 * d, 4);
      }
      *abort_flag = 0;
      fence_mbar_init();
      // The first activations on their way to L2, where they are already unless the kernel before did not write them (a 7B
      // layer at 16 rows 43.3 -> 42.1 us; with more than 16 rows nothing).
      if (PERM) {
        for (int i = 0, st = t_hi % ST; i < 2 && i < n_stages; ++i) {
          tma_prefetch_3d(&tmap_x, 0, 0, st * (du::kStageK / 64));
          if (--st < 0) st = ST - 1;
        }
      }
    }
  } else if (warp == C::kMmaWarp) {
    tmem_alloc(smem_u32(tmem_slot), du::kTmemCols);
    tmem_relinquish();
  }
  __syncwarp();
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == C::kWeightWarp) {
    // ------------------------------------------------------------ TMA producer: weights
    if (elect_one()) {
      chain_wait();                // (early weights: the activations come before the rest of the ring)
      int s = p.first;
      uint32_t phase = 1;
      if (s == p.ring) { s = 0; phase = 0; }
      for (int i = p.first; i < n_stages; ++i) {
        if (!mbar_wait(empty0 + 8 * s, phase, abort_flag)) break;
        load_weights(s);
        if (++s == p.ring) { s = 0; phase ^= 1; }
      }
      chain_release();             // all of this block's loads are issued: the next kernel's blocks may start
    }
  } else if (warp == C::kXWarp) {
    // ------------------------------------------------------------ TMA producer: activations
    if (elect_one()) {
      chain_wait();
      int st = t_hi % ST, xs = 0;
      uint32_t phase = 1;
      bool ok = true;
      for (int i = 0; ok && i < n_stages; ++i) {
#pragma unroll
        for (int h = 0; h < (PERM ? 1 : 2); ++h) {
          if (!mbar_wait(xempty0 + 8 * xs, phase, abort_flag)) { ok = false; break; }
          mbar_arrive_expect_tx(xfull0 + 8 * xs, kXBytes);
          tma_load_3d(xring + xs * kXBytes, &tmap_x, xfull0 + 8 * xs, 0, 0, st * (du::kStageK / 64) + h * 2);
          if (++xs == kXRing) { xs = 0; phase ^= 1; }
        }
        if (--st < 0) st = ST - 1;
      }
    }
  } else if (warp == C::kMmaWarp) {
    // ------------------------------------------------------------ MMA issuer: one wait, 16 MMAs, one commit per stage
    if (elect_one()) {
      constexpr uint32_t idesc = umma_idesc(kIdescDFormatF32 | kIdescABFormatF16, du::kRows, TOK);
      bool fresh = true;                                       // the next MMA starts a segment
      int st = t_hi % ST, q = 0, xs = 0, d = 0;
      uint32_t phase = 0, xphase = 0, dphase = 1;
      bool ok = true;
      const uint64_t b_desc0 = umma_desc_k_sw128(xring);
      const uint32_t desc_hi = static_cast<uint32_t>(b_desc0 >> 32), desc_lo0 = static_cast<uint32_t>(b_desc0);
      for (int i = 0; i < n_stages; ++i) {
        if (!FOLD && fresh && !mbar_wait(dempty0 + 8 * d, dphase, abort_flag)) break;
        if (!mbar_wait(ready0 + 8 * q, phase, abort_flag)) break;
        tcgen05_fence_after();
        const uint32_t a_tmem = tmem_base + C::kASlot0 + q * du::kASlotCols;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (!PERM && !mbar_wait(xfull0 + 8 * xs, xphase, abort_flag)) { ok = false; break; }
          const uint32_t d_tmem = tmem_base + (FOLD ? 2 * q + h : d) * TOK;
          const uint32_t desc = desc_lo0 + ((xs * kXBytes + (PERM ? h * 2 * kXSub : 0)) >> 4);
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)       // 16 K per instruction: 8 TMEM columns of A, 32 bytes of B's rows
            umma_f16_ts(d_tmem, a_tmem + (h * 8 + kk) * 8, desc + ((kk >> 2) * kXSub >> 4) + 2 * (kk & 3), desc_hi, idesc,
                        FOLD ? kk != 0 : !(fresh && h == 0 && kk == 0));
          if (!PERM || h == 1) {
            umma_commit(xempty0 + 8 * xs);
            if (++xs == kXRing) { xs = 0; xphase ^= 1; }
          }
        }
        if (!ok) break;
        umma_commit(done0 + 8 * q);
        fresh = st == 0;
        if (!FOLD && (fresh || i == n_stages - 1)) {
          umma_commit(dfull0 + 8 * d);
          if (++d == C::kAccs) { d = 0; dphase ^= 1; }
        }
        if (--st < 0) st = ST - 1;
        if (++q == du::kSlots) { q = 0; phase ^= 1; }
      }
    }
  } else if (warp < C::kEpiWarp0) {
    // ------------------------------------------------------------ expansion: a warp does 32 rows of a stage, or half of it
    constexpr int kPieces = C::kPieces;
    const int quarter = warp & 3, part = C::kParts == 1 ? 0 : (warp >> 2) & 1, set = warp / (4 * C::kParts);
    const int row = quarter * 32 + lane;
    const uint32_t a_tmem0 = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + C::kASlot0 + part * kPieces * 16;
    const uint32_t lane_w = row * 128 + ((row & 7) << 4);      // a swizzled row's 16-byte pieces are at lane_w ^ (piece << 4)
    const uint32_t scale0 = smem_u32(s_scale + row);
    const uint32_t sz_lane = du::kWBytes + row * 4;
    int s = set, xs = set, q = set;
    uint32_t phase = 0, xphase = 0, use = 0;
    // The tiles that this block will add on their way to L2, from which the weights of other linears push those of a graph that
    // is not replayed all the time (three graphs of a 7B layer at 16 rows in turn, us: without 41.7, here 41.0, by the side warp
    // after the wait for the kernel before 41.1, from the loop below 43.0; not beside host copies, 65.7 -> 66.3).  With more rows
    // the idle side warp does it, a line at a time (that layer at 35 / 64 rows 51.3 / 58.8 -> 50.9 / 57.2; here, eagerly, 77
    // rows took 65.0 -> 67.2), up to 64: at 77 rows the tiles are there already in an eager call, 55.7 -> 56.1.
    if (PERM && closes && p.early_tiles) {
      const int first_block = block_of(rb_lo * ST, p);
      for (int b2 = first_block; b2 < blk; ++b2)
#pragma unroll
        for (int k = 0; k < kMine; ++k)
          if (tid + k * kExpThreads < p.M * (du::kRows / 4))
            prefetch_l2(p.tiles + (size_t)b2 * TOK * du::kRows + (tid + k * kExpThreads) * 4);
    }
    for (int i = set; i < n_stages; i += C::kSets) {
      // FOLD: one look at all three barriers and one vote, where nothing is to be waited for: a wait that is over and its vote
      // cost 38 clocks a stage (the four linears of a 70B layer at 8 rows 95.1 -> 91.7 us; the exact form, whose arithmetic is
      // longer, gains nothing)
      const bool wait = !FOLD || !__all_sync(0xffffffffu, mbar_test(full0 + 8 * s, phase) & mbar_test(done0 + 8 * q, use ^ 1) &
                                                              mbar_test(xfull0 + 8 * xs, xphase));
      if (wait && !__all_sync(0xffffffffu, mbar_wait(full0 + 8 * s, phase, abort_flag))) break;
      const uint32_t stage = wring + s * stage_bytes, src = (stage + lane_w) ^ (part * kPieces * 16), sz = stage + sz_lane;
      uint4 q4[kPieces];
#pragma unroll
      for (int j = 0; j < kPieces; ++j) q4[j] = du_lds_v4(src ^ (j << 4));
      constexpr int kScales = FOLD ? kPieces / 4 : kPieces;    // one for 128 columns or one for 32
      uint32_t szw[kScales];
#pragma unroll
      for (int j = 0; j < kScales; ++j)
        szw[j] = du_lds_u32(sz + (p.groups_per_stage > 1 ? ((part * 128 + j * (FOLD ? 128 : 32)) >> p.gshift) * (du::kRows * 4) : 0));
      // (the slot's use before its last one is over: this warp has waited for the MMAs of a stage at most six before this
      // one, and they complete in order, so the parity is not ambiguous)
      if (wait && !__all_sync(0xffffffffu, mbar_wait(done0 + 8 * q, use ^ 1, abort_flag))) break;
      mbar_arrive_warp(empty0 + 8 * s, lane);
      tcgen05_fence_after();
      const uint32_t a_tmem = a_tmem0 + q * du::kASlotCols;
      if constexpr (FOLD) {
#pragma unroll
        for (int h = 0; h < kScales; ++h) {
          du_sts_u32(scale0 + ((q * 2 + use) * 2 + part + h) * (du::kRows * 4), szw[h]);
          const __half2 z2 = __high2half2(*reinterpret_cast<const __half2*>(&szw[h]));
          const __half2 zl = __hadd2(z2, __float2half2_rn(1024.0f)), zh = __hadd2(z2, __float2half2_rn(64.0f));
#pragma unroll
          for (int j = 4 * h; j < 4 * h + 4; ++j) {
            uint32_t r[16];
            expand8(q4[j].x, zl, zh, r);
            expand8(q4[j].y, zl, zh, r + 4);
            expand8(q4[j].z, zl, zh, r + 8);
            expand8(q4[j].w, zl, zh, r + 12);
            tmem_st_32x32_x16(a_tmem + j * 16, r);
          }
        }
      } else {
#pragma unroll
        for (int j = 0; j < kPieces; ++j) {
          const __half2 szh = *reinterpret_cast<const __half2*>(&szw[j]);
          const ScaleZero sp = make_scale_zero(__low2half(szh), __high2half(szh));
          uint32_t r[16];
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const uint32_t word = c == 0 ? q4[j].x : c == 1 ? q4[j].y : c == 2 ? q4[j].z : q4[j].w;
            __half2 v[4];
            dequant8(word, sp, v);
#pragma unroll
            for (int e = 0; e < 4; ++e) r[4 * c + e] = h2_as_u32(v[e]);
            if constexpr (!PERM) in_order(&r[4 * c]);
          }
          tmem_st_32x32_x16(a_tmem + j * 16, r);
        }
      }
      if constexpr (PERM) {
        // this warp's share of the stage's activations: chunks of XROWS tokens x 256 columns
        if (wait && !__all_sync(0xffffffffu, mbar_wait(xfull0 + 8 * xs, xphase, abort_flag))) break;
        constexpr int kChunks = kXBytes / 2048 / C::kParts;
        const uint32_t xt = xring + xs * kXBytes + part * (kXBytes / C::kParts) + row * 16;
        uint4 v[kChunks];
#pragma unroll
        for (int j = 0; j < kChunks; ++j) v[j] = du_lds_v4(xt + j * 2048);
#pragma unroll
        for (int j = 0; j < kChunks; ++j) du_sts_v4(xt + j * 2048, pair_permute_u4(v[j]));
        fence_proxy_async_smem();                                  // generic-proxy stores -> visible to the MMA's reads
      }
      tmem_st_wait();
      tcgen05_fence_before();
      mbar_arrive_warp(ready0 + 8 * q, lane);
      s += C::kSets;
      if (s >= p.ring) { s -= p.ring; phase ^= 1; }
      if (PERM && (xs += C::kSets) >= kXRing) { xs -= kXRing; xphase ^= 1; }
      q += C::kSets;
      if (q >= du::kSlots) { q -= du::kSlots; use ^= 1; }
    }
    // The sums of the tiles that this block closes, fetched while the last MMAs and the epilogue run: four rows of a token to
    // an element, ELEMENTS elements of TILES tiles requested together.
    auto fetch = [&](auto elements, auto tiles) {
      constexpr int ELEMENTS = decltype(elements)::value, TILES = decltype(tiles)::value;
      const int first_block = block_of(rb_lo * ST, p);
      uint32_t* tile0 = p.tiles + (size_t)first_block * TOK * du::kRows + tid * 4;
      for (int b2 = first_block; b2 < blk && !*abort_flag; b2 += TILES, tile0 += (size_t)TILES * TOK * du::kRows) {
        uint4 w[ELEMENTS][TILES];
        uint64_t since = 0;
        for (uint32_t it = 1;; ++it) {
          bool there = true;
#pragma unroll
          for (int k = 0; k < ELEMENTS; ++k)
#pragma unroll
            for (int j = 0; j < TILES; ++j)
              w[k][j] = b2 + j < blk && tid + k * kExpThreads < p.M * (du::kRows / 4)
                            ? ld_relaxed_gpu_v4(tile0 + (size_t)j * TOK * du::kRows + k * kExpThreads * 4)
                            : make_uint4(1u, 1u, 1u, 1u);
#pragma unroll
          for (int k = 0; k < ELEMENTS; ++k)
#pragma unroll
            for (int j = 0; j < TILES; ++j)
              there = there && w[k][j].x != 0u && w[k][j].y != 0u && w[k][j].z != 0u && w[k][j].w != 0u;
          if (there) break;
          if ((it & 0x3F) == 0) {
            const uint64_t now = globaltimer_ns();
            if (since == 0) since = now;
            if (now - since > kWaitLimitNs) *abort_flag = 1;
            if (*abort_flag) break;
          }
        }
#pragma unroll
        for (int k = 0; k < ELEMENTS; ++k)
#pragma unroll
          for (int j = 0; j < TILES; ++j)
            if (b2 + j < blk && tid + k * kExpThreads < p.M * (du::kRows / 4)) {
              others[k][0] += __uint_as_float(~w[k][j].x);
              others[k][1] += __uint_as_float(~w[k][j].y);
              others[k][2] += __uint_as_float(~w[k][j].z);
              others[k][3] += __uint_as_float(~w[k][j].w);
              st_relaxed_gpu_v4_zero(tile0 + (size_t)j * TOK * du::kRows + k * kExpThreads * 4);       // ready for the next call
            }
      }
    };
    if (closes) {
      chain_wait();       // (with more than 16 rows nothing that this warp waited for came after it) the tiles are this call's
#pragma unroll
      for (int k = 0; k < kMine; ++k)
#pragma unroll
        for (int i = 0; i < 4; ++i) others[k][i] = 0.0f;
      // as many requests as registers hold
      const int mine = (p.M * (du::kRows / 4) + kExpThreads - 1) / kExpThreads;
      if (kMine <= 3 || mine <= 3) {
        fetch(du::Int<kMine < 3 ? kMine : 3>{}, du::Int<4>{});
      } else if (mine <= 4) {
        fetch(du::Int<kMine < 4 ? kMine : 4>{}, du::Int<2>{});
      } else {
        fetch(du::Int<kMine>{}, du::Int<1>{});
      }
    }
  } else if (warp == C::kSideWarp) {
    // ------------------------------------------------------------ copies: beside the product, which ends when they have ended
    if (TOK > 16 && TOK <= 64 && closes) {       // tiles to L2, as the expansion warps do up to 16 rows
      const int first_block = block_of(rb_lo * ST, p);
      for (int b2 = first_block; b2 < blk; ++b2)
        for (int e = lane; e < p.M * (du::kRows / 32); e += 32)
          prefetch_l2(p.tiles + (size_t)b2 * TOK * du::kRows + e * 32);
    }
    if constexpr (CARRY) {
      if (p.copies.count > 0) {
        chain_wait();
        copy_pieces(p.copies, blk * 32 + lane, static_cast<int>(gridDim.x) * 32, true);
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue: lane = weight row, column = token
    constexpr int CH = FOLD ? XROWS : 16;                      // tokens held at a time
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;
    const uint32_t d_tmem = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    chain_wait();                                              // before anything of the previous kernel is overwritten
    // v = a segment's sums for tokens [m0, m0 + CH): to y, to this block's tile, or to shared memory for the closing step
    auto finish = [&](const float (&v)[CH], int m0, int rb, bool ends_row_block, bool whole) {
      if (whole) {
        const int n = rb * du::kRows + row;
        if (n < p.N) {
          const float bias = p.bias ? h2f(p.bias[n]) : 0.0f;
#pragma unroll
          for (int m = 0; m < CH; ++m)
            if (m0 + m < p.M) p.y[(size_t)(m0 + m) * p.N + n] = f2h(v[m] + bias);
        }
      } else if (!ends_row_block) {
        uint32_t* tile = p.tiles + ((size_t)blk * TOK + m0) * du::kRows + row;
#pragma unroll
        for (int m = 0; m < CH; ++m)
          if (m0 + m < p.M) {
            const uint32_t b = ~__float_as_uint(v[m]);
            st_relaxed_gpu(tile + m * du::kRows, b == 0u ? 0x80000000u : b);     // (one NaN pattern becomes another)
          }
      } else {
        // the block's last segment: every weight stage has been read, so the ring is free
        const uint32_t own = wring + (m0 * du::kRows + row) * 4;
#pragma unroll
        for (int m = 0; m < CH; ++m)
          if (m0 + m < p.M) du_sts_u32(own + m * du::kRows * 4, __float_as_uint(v[m]));
      }
    };
    bool ok = true;
    int q = 0;
    uint32_t phase = 0;
    if constexpr (FOLD) {
      for (int i = 0; i < du::kSlots; ++i) mbar_arrive_warp(ready0 + 8 * i, lane);       // all accumulators are free
    }
    int rb = t_hi / ST, d = 0;
    for (int t = t_hi; ok && t >= t_lo; --rb) {
      const int row_first = rb * ST, lo = max(t_lo, row_first);
      const bool ends = t == row_first + ST - 1, whole = ends && lo == row_first;
      if constexpr (FOLD) {
        float acc[CH];
#pragma unroll
        for (int m = 0; m < CH; ++m) acc[m] = 0.0f;
        for (; t >= lo; --t) {
          if (!__all_sync(0xffffffffu, mbar_wait(done0 + 8 * q, phase & 1, abort_flag))) { ok = false; break; }
          tcgen05_fence_after();
          uint32_t r0[CH], r1[CH];
          tmem_ld_cols(d_tmem + 2 * q * TOK, r0);
          tmem_ld_cols(d_tmem + (2 * q + 1) * TOK, r1);
          const uint32_t sa = smem_u32(s_scale + ((q * 2 + (phase & 1)) * 2) * du::kRows + row);
          const uint32_t sz0 = du_lds_u32(sa), sz1 = du_lds_u32(sa + du::kRows * 4);
          tmem_ld_wait();
          tcgen05_fence_before();
          mbar_arrive_warp(ready0 + 8 * q, lane);
          const float s0 = __low2float(*reinterpret_cast<const __half2*>(&sz0));
          const float s1 = __low2float(*reinterpret_cast<const __half2*>(&sz1));
#pragma unroll
          for (int m = 0; m < CH; ++m)
            acc[m] = fmaf(s1, __uint_as_float(r1[m]), fmaf(s0, __uint_as_float(r0[m]), acc[m]));
          if (++q == du::kSlots) { q = 0; phase ^= 1; }
        }
        if (!ok) break;
        finish(acc, 0, rb, ends, whole);
      } else {
        if (!__all_sync(0xffffffffu, mbar_wait(dfull0 + 8 * d, phase & 1, abort_flag))) break;
        tcgen05_fence_after();
#pragma unroll 1
        for (int m0 = 0; m0 < TOK && m0 < p.M; m0 += 16) {
          uint32_t r[CH];
          tmem_ld_cols(d_tmem + d * TOK + m0, r);
          tmem_ld_wait();
          float v[CH];
#pragma unroll
          for (int m = 0; m < CH; ++m) v[m] = __uint_as_float(r[m]);
          finish(v, m0, rb, ends, whole);
          __syncwarp();
        }
        tcgen05_fence_before();
        mbar_arrive_warp(dempty0 + 8 * d, lane);
        if (++d == C::kAccs) { d = 0; phase ^= 1; }
      }
      t = lo - 1;
    }
  }

  tcgen05_fence_before();
  __syncthreads();
  // The closing step: when the block's last segment ends a row block that earlier blocks began, their sums and this block's.
  if (closes && warp < C::kEpiWarp0 && !*abort_flag) {
#pragma unroll
    for (int k = 0; k < kMine; ++k) {
      const int e = tid + k * kExpThreads, m = e / (du::kRows / 4), r4 = (e % (du::kRows / 4)) * 4, n = rb_lo * du::kRows + r4;
      if (m >= p.M || n >= p.N) continue;                      // N is a multiple of four
      const uint4 own = du_lds_v4(wring + (m * du::kRows + r4) * 4);
      float v[4] = {__uint_as_float(own.x) + others[k][0], __uint_as_float(own.y) + others[k][1],
                    __uint_as_float(own.z) + others[k][2], __uint_as_float(own.w) + others[k][3]};
      if (p.bias) {
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] += h2f(p.bias[n + i]);
      }
      __half* y = p.y + (size_t)m * p.N + n;
      *reinterpret_cast<__half2*>(y) = __floats2half2_rn(v[0], v[1]);
      *reinterpret_cast<__half2*>(y + 2) = __floats2half2_rn(v[2], v[3]);
    }
  }
  if (*abort_flag) {
    if (tid == 0 && p.error_word) atomicExch(p.error_word, 4);
    const uint64_t t_start = globaltimer_ns();
    while (globaltimer_ns() - t_start < 200000ull) __nanosleep(1000);  // let copies and MMAs in flight land
    __syncthreads();
  }
  if (warp == C::kMmaWarp) {
    tcgen05_fence_after();
    tmem_dealloc(tmem_base, du::kTmemCols);
  }
}

int* decode_error_word_ptr(int* out_rc);   // w4a16_decode_tma.cu: device address of the decode error word

size_t decode_umma_workspace_bytes(int M, int K) { return du::workspace_bytes(M); }

bool decode_umma_shape_ok(int M, int N, int K, int group) {
  if (M > 128 || K % 64 != 0 || N % 4 != 0) return false;
  return group == 32 || group == 64 || group == 128 || group == du::kStageK || group % du::kStageK == 0;
}

template <int TOK, int XROWS, bool FOLD, bool CARRY = false>
static int launch_umma(const CUtensorMap& tw, const CUtensorMap& tx, const CUtensorMap& tsz, const DecodeUmmaParams& params,
                       int grid, cudaStream_t st, const HostCopies* copies = nullptr) {
  using C = du::Cfg<TOK, XROWS, FOLD, CARRY>;
  auto kern = w4a16_decode_umma_kernel<TOK, XROWS, FOLD, CARRY>;
  DecodeUmmaArgs<CARRY> p;
  static_cast<DecodeUmmaParams&>(p) = params;
  if constexpr (CARRY) p.copies = copies ? *copies : HostCopies{};
  static thread_local int configured_device = -1;
  int device = 0;
  MP_CUDA_TRY(cudaGetDevice(&device));
  if (configured_device != device) {
    MP_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)du::kSmemMax));
    configured_device = device;
  }
  // as many weight stages as fit
  const int stage = du::kWBytes + du::sz_bytes(p.groups_per_stage);
  const size_t fixed = 1024 + (size_t)C::kXRing * C::kXBytes + du::kTailBytes;
  p.ring = (int)((du::kSmemMax - fixed) / stage);
  if (p.ring > du::kMaxRing) p.ring = du::kMaxRing;
  p.first = p.early_weights ? du::kFirstEarly : du::kFirst;
  if (p.first > p.ring) p.first = p.ring;
  return launch_chained(kern, dim3(grid), dim3(C::kThreads), fixed + (size_t)p.ring * stage, st, tw, tx, tsz, p);
}

// The tensor maps of weights and (scale, zero) pairs.  A map is made of an address and sizes and of nothing in memory, and a
// program calls with the same weights again and again, so those made last are kept, per thread, in the place that the weights'
// address gives.  Encoding all three in every call took what the stream kernel gains on a shape that the host bounds (one
// 4096x4096 linear at one row, eager, us: the ring kernel, which keeps its maps, 6.05, this 6.25; kept 5.64 where that took
// 5.84, and 6.14 where the ring kernel takes 6.14).  The activations' map is made in every call: their address is another one more often than not.
static int weight_maps(const void* packed, const void* sz, int N, int K, int group, int gps, const CUtensorMap** tw,
                       const CUtensorMap** tsz) {
  struct Entry {
    CUtensorMap tw, tsz;
    const void *packed, *sz;
    int N, K, group;
  };
  constexpr int kLog2Entries = 7;
  static thread_local Entry entries[1 << kLog2Entries];
  Entry& e = entries[(reinterpret_cast<uintptr_t>(packed) >> 4) * 0x9E3779B97F4A7C15ull >> (64 - kLog2Entries)];
  if (e.packed != packed || e.sz != sz || e.N != N || e.K != K || e.group != group) {
    e.packed = nullptr;
    int rc = encode_tensor_map_2d(&e.tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, packed, (uint64_t)K / 2, (uint64_t)N,
                                  (uint64_t)K / 2, 128, du::kRows, true);
    if (rc != MP_OK) return rc;
    rc = encode_tensor_map_2d(&e.tsz, CU_TENSOR_MAP_DATA_TYPE_UINT32, sz, (uint64_t)N, (uint64_t)(K / group),
                              (uint64_t)N * 4, du::kRows, gps, false);
    if (rc != MP_OK) return rc;
    e.packed = packed;
    e.sz = sz;
    e.N = N;
    e.K = K;
    e.group = group;
  }
  *tw = &e.tw;
  *tsz = &e.tsz;
  return MP_OK;
}

// Returns MP_ERR_UNSUPPORTED for shapes this kernel does not take (M > 128, K % 64 != 0, N % 4 != 0, groups
// other than 32, 64, 128, 256 or a multiple of 256) and when the workspace is missing or too small; the
// caller then uses another kernel.  The workspace starts zeroed and is left ready for the next call;
// calls that share it must not overlap on the GPU.
int launch_decode_umma(const void* x, const void* packed, const void* sz, const void* bias, void* y, int M, int N, int K,
                       int group, void* workspace, size_t workspace_bytes, cudaStream_t st, bool early_weights,
                       bool early_tiles, const HostCopies* copies) {
  if (!decode_umma_shape_ok(M, N, K, group)) return MP_ERR_UNSUPPORTED;
  const int tok = du::tokens_for(M);
  if (!workspace || workspace_bytes < du::workspace_bytes(M) || !aligned(workspace, 16)) return MP_ERR_UNSUPPORTED;
  if (!aligned(x, 16) || !aligned(packed, 16) || !aligned(sz, 16) || !aligned(y, 4)) return MP_ERR_UNSUPPORTED;
  const int row_blocks = (N + du::kRows - 1) / du::kRows;
  const int gps = group < du::kStageK ? du::kStageK / group : 1;
  const CUtensorMap *tw_at = nullptr, *tsz_at = nullptr;
  int rc = weight_maps(packed, sz, N, K, group, gps, &tw_at, &tsz_at);
  if (rc != MP_OK) return rc;
  const CUtensorMap &tw = *tw_at, &tsz = *tsz_at;
  // [64 columns][token][chunk of 64 columns]: one copy brings the sub-tiles of a stage or half of one
  CUtensorMap tx;
  const uint64_t x_dims[3] = {64, (uint64_t)M, (uint64_t)K / 64}, x_strides[2] = {(uint64_t)K * 2, 128};
  const uint32_t x_box[3] = {64, (uint32_t)(M <= 8 ? 8 : tok), tok <= 16 ? 4u : 2u};
  rc = encode_tensor_map_3d(&tx, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, x, x_dims, x_strides, x_box);
  if (rc != MP_OK) return rc;
  DecodeUmmaParams p{};
  p.bias = static_cast<const __half*>(bias);
  p.y = static_cast<__half*>(y);
  p.M = M; p.N = N; p.K = K; p.group = group;
  p.stages_per_row = (K + du::kStageK - 1) / du::kStageK;
  const long long total = (long long)row_blocks * p.stages_per_row;
  if (total > (1 << 24)) return MP_ERR_UNSUPPORTED;
  // as few blocks as finish as early as a block on every SM would
  int per_block = ((int)total + du::kMaxGrid - 1) / du::kMaxGrid;
  if (per_block < du::min_share(p.stages_per_row, tok)) per_block = du::min_share(p.stages_per_row, tok);
  const int grid = ((int)total + per_block - 1) / per_block;
  p.share = (int)total / grid;
  p.extra = (int)total % grid;
  p.groups_per_stage = gps;
  p.gshift = group == 32 ? 5 : group == 64 ? 6 : 7;
  p.early_weights = early_weights ? 1 : 0;
  p.early_tiles = early_tiles ? 1 : 0;
  p.tiles = reinterpret_cast<uint32_t*>(static_cast<unsigned char*>(workspace) + du::kTileOffset);
  int rc_err = MP_OK;
  p.error_word = decode_error_word_ptr(&rc_err);
  if (rc_err != MP_OK) return rc_err;
  const bool fold = group % 128 == 0;
  if (copies) {
    if (tok > 16) return MP_ERR_INVALID_ARG;
    if (M <= 8)
      return fold ? launch_umma<16, 8, true, true>(tw, tx, tsz, p, grid, st, copies)
                  : launch_umma<16, 8, false, true>(tw, tx, tsz, p, grid, st, copies);
    return fold ? launch_umma<16, 16, true, true>(tw, tx, tsz, p, grid, st, copies)
                : launch_umma<16, 16, false, true>(tw, tx, tsz, p, grid, st, copies);
  }
  if (M <= 8) return fold ? launch_umma<16, 8, true>(tw, tx, tsz, p, grid, st) : launch_umma<16, 8, false>(tw, tx, tsz, p, grid, st);
  if (tok == 16) return fold ? launch_umma<16, 16, true>(tw, tx, tsz, p, grid, st) : launch_umma<16, 16, false>(tw, tx, tsz, p, grid, st);
  switch (tok) {
    case 32: return launch_umma<32, 32, false, true>(tw, tx, tsz, p, grid, st);
    case 48: return launch_umma<48, 48, false, true>(tw, tx, tsz, p, grid, st);
    case 64: return launch_umma<64, 64, false, true>(tw, tx, tsz, p, grid, st);
    case 80: return launch_umma<80, 80, false, true>(tw, tx, tsz, p, grid, st);
    case 96: return launch_umma<96, 96, false, true>(tw, tx, tsz, p, grid, st);
    case 112: return launch_umma<112, 112, false, true>(tw, tx, tsz, p, grid, st);
    default: return launch_umma<128, 128, false, true>(tw, tx, tsz, p, grid, st);
  }
}

}  // namespace mp
