// W4A16 GEMM (M > 16: serving batches and prompts) on 5th-generation tensor cores: tcgen05.mma with the
// accumulators AND the dequantised weight operand in tensor memory.
//
//   out[m, n] = sum_k x[m, k] * (nib(n, k) - 8) * scales[n, k / 32]      (float32 accumulate)
//
// Orientation ("swap A/B"): the MMA's M dimension is the weight row n, its N dimension the
// activation row m.  A team -- one CTA (CG = 1) or the two CTAs of a cluster (CG = 2) -- owns
// D[128 * CG n x bm m], CTA r its rows 128 r .. 128 r + 127:
//   * Packed int4 tiles [128 n x 256 k] (+ their fp16 scales) arrive by TMA in each CTA; sixteen
//     dequant warps turn them into fp16 (exactly RN((q - 8) * s); K % 256 != 0: and the rest, a second term)
//     and write them with tcgen05.st into a ring of TMEM slots that the MMA reads as its A operand.  The packed weights cross shared
//     memory once (0.5 B/weight) and never as 2-byte values.
//   * X tiles [bm x 256 k] fp16 are the shared-memory B operand; in a pair each CTA holds half of their
//     rows, which both SMs' tensor cores read (cta_group::2).
//   * One warp of the team issues the MMAs; tcgen05.commit releases X stages and TMEM slots (in both
//     CTAs) and hands a finished accumulator to four epilogue warps (tcgen05.ld -> global).
// TMEM (512 columns): up to two accumulators of bm columns, so that the epilogue of one tile runs under
// the MMAs of the next; the A slots (128 columns each: 256 k as packed fp16 pairs) at the end.
//
// What bounds it.  In one call by itself at bm >= 192 the tensor cores (an MMA with its A operand in TMEM takes N / 2 clocks from
// N = 32 on); below, the dequant warps' instructions and HBM, and what is left of the issue of the MMAs beside them (see
// umma_steps).  The hand-over between the dequant warps, the MMA warp and back is a chain of barrier round trips -- hence whole 256-k
// stages per barrier (with 64-k steps every step took ~750 clocks whatever bm), two sets of dequant warps that take the
// stages in turn, and MMAs issued by an elected lane of a uniform warp.  Call after call, everything from M = 32 on large
// weights upwards runs at the GPU's 1000 W: then a call takes as long as its energy lasts.
// M = 64 on 8192 -> 28672, back to back in bursts / sustained: 47.5 / 56.9 us with an election per MMA, now 41.9 / 50.7.
//
// Split of the work: whole tiles in turn while they fill all teams.  The rest goes in pieces of fewer rows, or, on
// single SMs, is cut along K into equal shares (stream-K): a tile produced by several CTAs is combined through
// scratch, every contributor publishes its float32 partial and bumps a counter, the last one sums all in a
// fixed order and writes the output.  Nobody waits for another CTA.  With fewer tiles than SMs a cluster of 2 to 6
// single CTAs shares the K of each tile and adds up the partials over distributed shared memory.  Pairs are not cut
// along K: with all warps settling the shares, out of line, whole tiles took 58.9 -> 62.7 us at M = 512, 4096 -> 14336.
//
// Weight tiles are fp16 because bf16's 8-bit significand cannot hold (q-8)*s within the 1e-2 output
// tolerance; bf16 activations are converted to fp16 by a small pre-pass into the caller's workspace.
// Every mbarrier wait is bounded; on expiry the kernel records a status code and unwinds.
#pragma once
#include "common.cuh"

namespace lcq {
namespace gemm_tc {

constexpr int BN = 128;                 // weight rows per CTA
constexpr int BK = 64;                  // k per step (one 128-byte swizzle row of fp16): four MMAs
constexpr int WK = 256;                 // k per stage: of packed weights, of X and of TMEM
constexpr int W_STAGE = BN * (WK / 2);  // 16384
constexpr int S_STAGE = BN * (WK / 32) * 2;   // 2048
constexpr int WS_STAGE = W_STAGE + S_STAGE;
constexpr int MAX_XS = 6, MAX_WS = 9, MAX_AS = 3;    // ring depths: X stages, weight stages, TMEM A slots
constexpr int A_STEP_COLS = BK / 2;     // TMEM columns of 64 k as packed fp16 pairs
constexpr int A_SLOT_COLS = WK / 2;     // an A slot holds a whole weight stage
constexpr int TMEM_COLS = 512;
constexpr int N_DQ_WARPS = 16;          // two sets of two warpgroups
constexpr int WARP_EPI0 = N_DQ_WARPS, WARP_W = WARP_EPI0 + 4, WARP_X = WARP_W + 1, WARP_MMA = WARP_X + 1;
constexpr int NTHREADS = (WARP_MMA + 1) * 32;
// fp16 numbers that make up a weight: one where K is whole weight stages, else two (see RAGGED below)
__host__ __device__ constexpr int terms(bool ragged) { return ragged ? 2 : 1; }
constexpr int BAR_EPI = 1;              // named barrier of the epilogue warps

// ---------------------------------------------------------------- tcgen05 / cluster wrappers
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// CG = 1: the CTA alone; CG = 2: the pair of CTAs of a cluster (the two forms of every instruction below).
template <int CG> __device__ __forceinline__ void tmem_alloc(uint32_t* smem_slot, uint32_t cols) {
  if (CG == 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_slot)), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  } else {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_slot)), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
}
template <int CG> __device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
  if (CG == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
  else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem descriptor] for 64 k: four MMAs.  Called by a whole warp, issued by one elected
// lane: with every operand uniform over the warp the compiler keeps them in uniform registers, where the
// instruction wants them.  `b`: the low word of the descriptor (its start address); `first`: 0 overwrites D.
#define LCQ_MMA(CG, A, B, P) \
  "mov.b64 bd, {" B ", %5};\n\ttcgen05.mma.cta_group::" #CG ".kind::f16 [%0], [" A "], bd, %3, " P ";\n\t"
#define LCQ_MMA_STEP(CG, K, P0) \
  "add.u32 a1, a" #K ", 8;\n\tadd.u32 a2, a" #K ", 16;\n\tadd.u32 a3, a" #K ", 24;\n\t" \
  "add.u32 b1, b" #K ", 2;\n\tadd.u32 b2, b" #K ", 4;\n\tadd.u32 b3, b" #K ", 6;\n\t" \
  LCQ_MMA(CG, "a" #K, "b" #K, P0) LCQ_MMA(CG, "a1", "b1", "q") LCQ_MMA(CG, "a2", "b2", "q") LCQ_MMA(CG, "a3", "b3", "q")
#define LCQ_MMA_BEGIN \
  "{\n\t.reg .pred p, q, e;\n\t.reg .b64 bd;\n\t.reg .b32 a0, a1, a2, a3, a4, a8, a12, b0, b1, b2, b3, b4, b8, b12;\n\t" \
  "elect.sync _|e, 0xffffffff;\n\t@!e bra ISSUED;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.eq.b32 q, 0, 0;\n\t" \
  "mov.b32 a0, %1;\n\tmov.b32 b0, %2;\n\t"
#define LCQ_MMA_END "ISSUED:\n\t}"
// High word of the descriptor: 1024 bytes between 8-row groups, descriptor version (sm_100), 128-byte swizzle.
constexpr uint32_t B_DESC_HI = (1024u >> 4) | (1u << 14) | (2u << 29);
template <int CG> __device__ __forceinline__ void umma_step(uint32_t d_tmem, uint32_t a_tmem, uint32_t b, uint32_t idesc, uint32_t first) {
  if (CG == 2)
    asm volatile(LCQ_MMA_BEGIN LCQ_MMA_STEP(2, 0, "p") LCQ_MMA_END ::"r"(d_tmem), "r"(a_tmem), "r"(b), "r"(idesc), "r"(first), "n"(B_DESC_HI) : "memory");
  else
    asm volatile(LCQ_MMA_BEGIN LCQ_MMA_STEP(1, 0, "p") LCQ_MMA_END ::"r"(d_tmem), "r"(a_tmem), "r"(b), "r"(idesc), "r"(first), "n"(B_DESC_HI) : "memory");
}
// The same for a whole stage of 256 k (STEPS = 4) or half of one (2); `step`: descriptor units between 64-k steps.  One election and
// one branch for all: the issuing warp shares its scheduler with four dequant warps, and what it can issue bounds tiles of
// few rows.  Clocks per MMA beside four busy warps on the scheduler, N <= 64: an election per MMA in a loop over
// the steps 168, all sixteen unrolled 61, one election for four 63, one for all with predicated MMAs 52, with a branch 45.
template <int CG, int STEPS> __device__ __forceinline__ void umma_steps(uint32_t d_tmem, uint32_t a_tmem, uint32_t b, uint32_t step, uint32_t idesc, uint32_t first) {
#define LCQ_MMA_TWO_STEPS(G)                                                                                                 \
  LCQ_MMA_BEGIN "add.u32 a4, %1, 32;\n\tadd.u32 b4, %2, %6;\n\t" LCQ_MMA_STEP(G, 0, "p") LCQ_MMA_STEP(G, 4, "q")
#define LCQ_MMA_FOUR_STEPS(G)                                                                                                \
  LCQ_MMA_BEGIN                                                                                                              \
  "add.u32 a4, %1, 32;\n\tadd.u32 a8, %1, 64;\n\tadd.u32 a12, %1, 96;\n\t"                                                   \
  "add.u32 b4, %2, %6;\n\tadd.u32 b8, b4, %6;\n\tadd.u32 b12, b8, %6;\n\t"                                                   \
  LCQ_MMA_STEP(G, 0, "p") LCQ_MMA_STEP(G, 4, "q") LCQ_MMA_STEP(G, 8, "q") LCQ_MMA_STEP(G, 12, "q")
  static_assert(STEPS == 4 || (STEPS == 2 && CG == 1), "the forms that are used");
  if constexpr (CG == 2)
    asm volatile(LCQ_MMA_FOUR_STEPS(2) LCQ_MMA_END ::"r"(d_tmem), "r"(a_tmem), "r"(b), "r"(idesc), "r"(first), "n"(B_DESC_HI), "r"(step) : "memory");
  else if constexpr (STEPS == 4)
    asm volatile(LCQ_MMA_FOUR_STEPS(1) LCQ_MMA_END ::"r"(d_tmem), "r"(a_tmem), "r"(b), "r"(idesc), "r"(first), "n"(B_DESC_HI), "r"(step) : "memory");
  else
    asm volatile(LCQ_MMA_TWO_STEPS(1) LCQ_MMA_END ::"r"(d_tmem), "r"(a_tmem), "r"(b), "r"(idesc), "r"(first), "n"(B_DESC_HI), "r"(step) : "memory");
#undef LCQ_MMA_TWO_STEPS
#undef LCQ_MMA_FOUR_STEPS
}
#undef LCQ_MMA
#undef LCQ_MMA_STEP
#undef LCQ_MMA_BEGIN
#undef LCQ_MMA_END
// Arrives on this barrier (CG = 2: and on its counterpart in the other CTA) once the MMAs issued so far
// have completed.  Whole warp, like the MMAs: the same lane is elected.
template <int CG> __device__ __forceinline__ void umma_commit(uint64_t* bar) {
  if (CG == 2)
    asm volatile("{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
                 "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}"
                 ::"r"(smem_u32(bar)), "h"(static_cast<uint16_t>(3)) : "memory");
  else
    asm volatile("{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
                 "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_u32(bar)) : "memory");
}
// TMA load into this CTA's shared memory whose bytes are counted by a barrier of either CTA of the pair.
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const void* tmap, uint32_t bar_cluster_addr, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(dst)), "l"(tmap), "r"(bar_cluster_addr), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
        "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]),
        "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]),
        "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31]) : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
        "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
        "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr) : "memory");
}

// Low word of the shared-memory matrix descriptor of a K-major tile of 128-byte rows, 128-byte swizzle, 1024 bytes
// between 8-row groups: the start address, and a leading byte offset that is not used for swizzled K-major tiles.
__device__ __forceinline__ uint32_t make_b_desc(uint32_t smem_addr) { return ((smem_addr & 0x3FFFFu) >> 4) | (1u << 16); }
// The N of a kind::f16 MMA is a multiple of this.  For the pair form (M = 256) it is 32 that is specified; 48, 80 and 112 gave the
// right results, and are not used.
__host__ __device__ constexpr int mma_n_step(int cg) { return 16 * cg; }
// kind::f16 instruction descriptor: D=f32, A=B=f16, both K-major, M=128*CG, N=bm.
__host__ __device__ inline uint32_t make_idesc(int bm, int cg) {
  return (1u << 4) | (static_cast<uint32_t>(bm >> 3) << 17) | (static_cast<uint32_t>((BN * cg) >> 4) << 24);
}

// ---------------------------------------------------------------- work schedule
struct Params {
  void* out;            // [M, N]
  const void* scales;   // [N, K/32] fp16 (read directly when K % 256 != 0)
  float* partials;      // CG = 1: [2 * teams][bm][BN]
  int* counters;        // [sk_tiles], zero on entry, zero on exit
  int M, N, K;
  int bm;               // activation rows per tile (MMA N): multiple of 32, <= 256
  int n_tiles_n, n_tiles;
  int nst;              // 256-k weight stages per tile
  int teams;            // CTAs (CG = 1) or pairs (CG = 2) launched
  int sk_tiles;         // tiles 0 .. sk_tiles-1 (CG = 2: none) are cut along K, the others go whole to team (tile - sk_tiles) % teams
  int full, tail;       // tiles full .. are cut into `tail` pieces of bm / tail rows of x (a last wave that would be mostly empty)
  int split;            // > 1: a cluster of `split` teams per tile, each with its share of K (no whole tiles, no scratch)
  int nxs, nws;         // ring depths: X stages, weight stages
  int nas;              // TMEM A slots
  int nd;               // accumulators (1 or 2)
};

// First unit (a tile's weight stage, tile-major) of team p's share of the tiles that are cut along K.
__host__ __device__ inline unsigned share_begin(const Params& p, int team) {
  const unsigned units = static_cast<unsigned>(p.sk_tiles) * static_cast<unsigned>(p.nst);
  return static_cast<unsigned>(static_cast<unsigned long long>(units) * static_cast<unsigned>(team) / static_cast<unsigned>(p.teams));
}
__host__ __device__ inline int share_owner(const Params& p, unsigned unit) {
  const unsigned units = static_cast<unsigned>(p.sk_tiles) * static_cast<unsigned>(p.nst);
  return static_cast<int>((static_cast<unsigned long long>(unit + 1u) * static_cast<unsigned>(p.teams) - 1u) / units);
}

// The segments of one team: (tile, stages st0 .. st1-1).  Every role walks them in the same order.
struct Walk {
  unsigned u, u1;       // what is left of the team's share of the cut tiles
  int next_item;        // then the whole tiles and the pieces of the last ones
  int tile, st0, st1;
  int m0, bm;           // first row of x and their number
  __host__ __device__ Walk(const Params& p, int team) {
    if (p.split > 1) {
      const int t = team / p.split, r = team - t * p.split;
      u = static_cast<unsigned>(t * p.nst + p.nst * r / p.split);
      u1 = static_cast<unsigned>(t * p.nst + p.nst * (r + 1) / p.split);
      next_item = p.n_tiles;
      return;
    }
    u = share_begin(p, team);
    u1 = share_begin(p, team + 1);
    next_item = p.sk_tiles + team;
  }
  __host__ __device__ bool next(const Params& p) {
    if (u < u1) {
      tile = static_cast<int>(u / static_cast<unsigned>(p.nst));
      st0 = static_cast<int>(u - static_cast<unsigned>(tile) * static_cast<unsigned>(p.nst));
      const unsigned left = u1 - u, in_tile = static_cast<unsigned>(p.nst - st0);
      const unsigned take = left < in_tile ? left : in_tile;
      st1 = st0 + static_cast<int>(take);
      u += take;
      m0 = (tile / p.n_tiles_n) * p.bm;
      bm = p.bm;
      return true;
    }
    st0 = 0;
    st1 = p.nst;
    for (;;) {
      tile = next_item;
      bm = p.bm;
      int piece = 0;
      if (tile >= p.full) {
        const int i = tile - p.full;
        tile = p.full + i / p.tail;
        piece = i - (tile - p.full) * p.tail;
        bm = p.bm / p.tail;
      }
      if (tile >= p.n_tiles) return false;
      next_item += p.teams;
      m0 = (tile / p.n_tiles_n) * p.bm + piece * bm;
      if (m0 < p.M) return true;              // (a piece below the last row of x is no work)
    }
  }
};

enum { FLAG_ABORT, FLAG_SHARED, ISSUED_W, ISSUED_X0, ISSUED_X1, N_FLAGS = 6 };
struct Smem {           // offsets from the 1024-byte aligned dynamic shared memory base
  int w;                // nws stages of WS_STAGE
  int bars;
  int tmem_slot;
  int flags;            // abort flag, epilogue broadcast, stages issued: weights, X (in the pair's first CTA: of both CTAs)
  int total;
};
__host__ __device__ inline int x_step_bytes(int bm, int cg) { return (bm / cg) * 128; }   // this CTA's share of a tile's rows, 64 k
__host__ __device__ inline int x_stage_bytes(int bm, int cg) { return (WK / BK) * x_step_bytes(bm, cg); }
__host__ __device__ inline Smem smem_map(int bm, int cg, int nxs, int nws) {
  Smem s;
  s.w = nxs * x_stage_bytes(bm, cg);    // X stages first: steps are multiples of 1024 bytes, the swizzle's period
  s.bars = s.w + nws * WS_STAGE;
  // full_x, empty_x [MAX_XS]; full_w, empty_w [MAX_WS]; full_a, empty_a [MAX_AS]; full_d, empty_d [2]; drained
  s.tmem_slot = s.bars + (2 * MAX_XS + 2 * MAX_WS + 2 * MAX_AS + 5) * 8;
  s.flags = s.tmem_slot + 8;
  s.total = s.flags + 4 * N_FLAGS;
  return s;
}

// ---------------------------------------------------------------- dequantisation
__device__ __forceinline__ uint32_t lop_and_or(uint32_t a, uint32_t mask, uint32_t magic) {   // (a & mask) | magic
  uint32_t r;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(a), "r"(mask), "r"(magic));
  return r;
}
__device__ __forceinline__ uint32_t sub_mul(uint32_t v, uint32_t offset, __half2 s2) {        // (v - offset) * s, halves alike
  const __half2 d = __hsub2(*reinterpret_cast<const __half2*>(&v), *reinterpret_cast<const __half2*>(&offset));
  const __half2 r = __hmul2(d, s2);
  return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t sub_mul_rest(uint32_t v, uint32_t offset, __half2 s2) {   // what sub_mul rounds off, exactly
  const __half2 d = __hsub2(*reinterpret_cast<const __half2*>(&v), *reinterpret_cast<const __half2*>(&offset));
  const __half2 r = __hfma2(d, s2, __hneg2(__hmul2(d, s2)));
  return *reinterpret_cast<const uint32_t*>(&r);
}
// RN((q - 8) * s) for the 8 nibbles of a word, as 4 half2; REST: (q - 8) * s less that.  A nibble in bits 0-3 of a 16-bit lane under
// 0x6400 is the fp16 number 1024 + q, one in bits 4-7 under 0x5400 is 64 + q; the subtraction is exact.
// PERM = true leaves the pairs as the masks deliver them -- (e0,e4) (e1,e5) (e2,e6) (e3,e7) -- for
// activations whose k order was permuted the same way by the pre-pass (13 instructions a word); else
// each byte is copied to both halves first, so that its two nibbles come out as a natural pair (16).
template <bool PERM, bool REST>
__device__ __forceinline__ void dequant_word(uint32_t w, __half2 s2, uint32_t* o) {
  const auto scaled = [&](uint32_t v, uint32_t offset) { return REST ? sub_mul_rest(v, offset, s2) : sub_mul(v, offset, s2); };
  if (PERM) {
    const uint32_t w8 = w >> 8;
    o[0] = scaled(lop_and_or(w, 0x000F000Fu, 0x64006400u), 0x64086408u);
    o[1] = scaled(lop_and_or(w, 0x00F000F0u, 0x54005400u), 0x54805480u);
    o[2] = scaled(lop_and_or(w8, 0x000F000Fu, 0x64006400u), 0x64086408u);
    o[3] = scaled(lop_and_or(w8, 0x00F000F0u, 0x54005400u), 0x54805480u);
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      o[j] = scaled(lop_and_or(__byte_perm(w, 0u, 0x4040 + 0x0101 * j), 0x00F0000Fu, 0x54006400u), 0x54806408u);
  }
}
// The 64 weights of a row in two groups of 32, with a scale each.
template <bool PERM, bool REST>
__device__ __forceinline__ void dequant_step(const uint4* pk, __half2 s0, __half2 s1, uint32_t (&v)[32]) {
  dequant_word<PERM, REST>(pk[0].x, s0, v);
  dequant_word<PERM, REST>(pk[0].y, s0, v + 4);
  dequant_word<PERM, REST>(pk[0].z, s0, v + 8);
  dequant_word<PERM, REST>(pk[0].w, s0, v + 12);
  dequant_word<PERM, REST>(pk[1].x, s1, v + 16);
  dequant_word<PERM, REST>(pk[1].y, s1, v + 20);
  dequant_word<PERM, REST>(pk[1].z, s1, v + 24);
  dequant_word<PERM, REST>(pk[1].w, s1, v + 28);
}

__device__ __forceinline__ uint32_t peer_addr(uint32_t local_addr, uint32_t rank) {   // same offset in the CTA of that rank
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local_addr), "r"(rank));
  return a;
}
__device__ __forceinline__ void store_remote(uint32_t cluster_addr, int v) {
  asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(cluster_addr), "r"(v) : "memory");
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// Barriers of the MMA issuer's CTA, as the CTAs of the team address them.  What these arrivals hand over
// lives in tensor memory and is ordered by the tcgen05 fences around them.
template <int CG> __device__ __forceinline__ uint32_t leader_addr(uint64_t* bar) {
  return CG == 2 ? peer_addr(smem_u32(bar), 0) : smem_u32(bar);
}
template <int CG> __device__ __forceinline__ void arrive_leader(uint32_t addr) {
  if (CG == 2) asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
  else asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(addr) : "memory");
}
// Bounded wait; gives up when the CTA's abort flag is set or the library's wait limit has passed.  The
// clock is read only after many polls: waits of the ordinary kind end before that.
__device__ __noinline__ bool wait_slow(volatile int* flag_abort, uint64_t* bar, uint32_t parity) {
#pragma unroll 1
  for (int i = 0; i < 1024; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
  }
  const uint64_t t0 = global_timer_ns();
  const uint64_t limit = wait_limit_ns();
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 64; ++i) {
      if (mbar_try_wait(bar, parity)) return true;
    }
    if (*flag_abort != 0 || global_timer_ns() - t0 > limit) return false;
  }
}
__device__ __forceinline__ bool wait_bar(volatile int* flag_abort, uint64_t* bar, uint32_t parity) {
  if (mbar_try_wait(bar, parity)) return true;
  return wait_slow(flag_abort, bar, parity);
}
// The same with one verdict for the whole warp, so that warp-aligned instructions after it never run
// with a partial warp.
__device__ __forceinline__ bool warp_wait(volatile int* flag_abort, uint64_t* bar, uint32_t parity) {
  return __all_sync(0xffffffffu, wait_bar(flag_abort, bar, parity));
}
__device__ __forceinline__ int load_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ bool all_epilogue_warps(bool ok) {
  uint32_t all;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\t"
      "bar.red.and.pred q, %2, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(all) : "r"(ok ? 1u : 0u), "n"(BAR_EPI) : "memory");
  return all != 0;
}

// A position in a ring of n slots and the parity of its current lap.
struct Ring {
  uint32_t i, phase;
  __device__ __forceinline__ void step(uint32_t n) { if (++i == n) { i = 0; phase ^= 1u; } }
};

// Adds up the partials of a tile that was cut along K and writes its row r of the outputs: `count`
// contributors in team order, bit for bit the same whoever finishes; contributor `mine` (this CTA) is still
// in tensor memory.  16 columns at a time: a round trip to L2 under the stream of weights takes 2-3 us.
// With one other contributor (nearly always) its next columns are fetched while the current ones are added.
// Out of line: its registers would otherwise cost the dequant warps some of theirs.
template <typename OT>
__device__ __noinline__ void finish_tile(uint32_t d_t, OT* out, int rows_out, int rows, int N, const float* first, const float* second,
                                         long long stride, int count, int mine) {
  const bool two = count == 2;
  const float* other = mine == 0 ? second : first;
  float next[16];
  if (two) {
#pragma unroll
    for (int i = 0; i < 16; ++i) next[i] = __ldcg(other + i * BN);
  }
#pragma unroll 1
  for (int c0 = 0; c0 < rows; c0 += 16) {
    uint32_t v[16];
    tmem_ld16(d_t + c0, v);
    tmem_wait_ld();
    if (two) {
      other += 16 * BN;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        v[i] = __float_as_uint(__uint_as_float(v[i]) + next[i]);
        if (c0 + 16 < rows) next[i] = __ldcg(other + i * BN);
      }
    } else {
      float sum[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) sum[i] = 0.0f;
#pragma unroll 1
      for (int q = 0; q < count; ++q) {
        const float* src = (q == 0 ? first : second + (q - 1) * stride) + c0 * BN;
#pragma unroll
        for (int i = 0; i < 16; ++i) next[i] = q == mine ? __uint_as_float(v[i]) : __ldcg(src + i * BN);
#pragma unroll
        for (int i = 0; i < 16; ++i) sum[i] += next[i];
      }
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = __float_as_uint(sum[i]);
    }
    OT* o = out + static_cast<long long>(c0) * N;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      if (c0 + i < rows_out) *o = from_f32<OT>(__uint_as_float(v[i]));
      o += N;
    }
  }
}

// After a wait ran out in the CTA or its partner: waits for what they still have under way -- the MMAs, and the copies
// into the last stages, which nobody waits for any more -- so that nothing lands in shared memory or reads it after
// they have left.  A CTA of a pair may have loaded its half of an X stage whose other half was never issued: the
// barrier is then given the missing half, or armed for the one that comes.  Called by all threads; in a pair between
// two cluster barriers.
template <int CG, bool RAGGED>
__device__ __noinline__ void drain(const Params& p, uint8_t* smem, int team, uint32_t crank) {
  const Smem L = smem_map(p.bm, CG, p.nxs, p.nws);
  uint64_t* full_x = reinterpret_cast<uint64_t*>(smem + L.bars);
  uint64_t* full_w = full_x + 2 * MAX_XS;
  uint64_t* drained = full_w + 2 * MAX_WS + 2 * MAX_AS + 4;
  const volatile int* flags = reinterpret_cast<const volatile int*>(smem + L.flags);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (warp == WARP_MMA) {
    if (crank == 0) umma_commit<CG>(drained);            // (arrives in both CTAs, after all that was committed before)
    __syncwarp();
    mbar_wait_landed(drained, 0);
  } else if (warp == WARP_W && lane == 0) {
    const int n = flags[ISSUED_W];
    for (int i = n > p.nws ? n - p.nws : 0; i < n; ++i) mbar_wait_landed(full_w + i % p.nws, (i / p.nws) & 1);
  } else if (warp == WARP_X && lane == 0 && crank == 0) {
    const int mine = flags[ISSUED_X0], other = CG == 2 ? flags[ISSUED_X1] : mine, n = mine > other ? mine : other;
    const int nk = p.K / BK;
    int i = 0;
    for (Walk w(p, team); i < n && w.next(p);) {
      for (int st = w.st0; st < w.st1 && i < n; ++st, ++i) {
        if (i < n - p.nxs) continue;
        const int steps = RAGGED && nk - st * 4 < 4 ? nk - st * 4 : 4, bytes = steps * x_step_bytes(w.bm, CG);
        uint64_t* bar = full_x + i % p.nxs;
        if (i >= mine) mbar_expect_tx(bar, bytes);
        else if (i >= other) asm volatile("mbarrier.complete_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
        mbar_wait_landed(bar, (i / p.nxs) & 1);
      }
    }
  }
  __syncthreads();
}

// RAGGED: K % 256 != 0 -- the last weight stage of a tile is partial, and the scale rows are no 16-byte
// multiples, so no tensor map can describe them: the dequant warps load their scales from global
// memory, a stage ahead.  Such calls have exact products (TERMS = 2), as the decode kernel has that they ran on
// before this one took them: a weight is the sum of two fp16 numbers, RN((q - 8) * s) and what that rounds off
// ((q - 8) * s and its rounding are multiples of 2^-24, so the rest is an fp16 number), in two A slots that meet the
// same X stage.  The first set of dequant warps writes the one, the second set the other.
//
// HALVES: the sixteen MMAs of a stage under two elections, for tiles of more than 64 rows on one SM.  An MMA takes 48 clocks and up there, which hides
// the second election, while with all in one block the instance spills 60 bytes instead of 24, and calls of few stages pay for that: 116 x 1024 -> 9850
// 9.2 us with an election per MMA, 9.6 with one, 9.2 with two; 277 x 1280 -> 4077 10.0 / 10.2 / 9.9; 486 x 768 -> 3174 7.8 / 8.05 / 7.7; 128 x 2048 ->
// 16000 13.0 / 12.9 / 12.7.  Up to 64 rows one is faster on long K: 17 x 12032 -> 26539 60.4 / 45.2 / 46.0, 32 x 8192 -> 28672 46.1 / 35.2 / 35.7 (64 x 1280 ->
// 16000 9.1 / 8.5 / 8.4).  Pairs and RAGGED calls spill the same either way.
template <int CG, typename OT, bool PERM, bool RAGGED, bool HALVES>
__global__ void __launch_bounds__(NTHREADS, 1)
w4a16_gemm_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_piece,
                  const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_s,
                  const __grid_constant__ Params p) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const Smem L = smem_map(p.bm, CG, p.nxs, p.nws);
  uint64_t* full_x = reinterpret_cast<uint64_t*>(smem + L.bars);
  uint64_t* empty_x = full_x + MAX_XS;
  uint64_t* full_w = empty_x + MAX_XS;
  uint64_t* empty_w = full_w + MAX_WS;
  uint64_t* full_a = empty_w + MAX_WS;
  uint64_t* empty_a = full_a + MAX_AS;
  uint64_t* full_d = empty_a + MAX_AS;
  uint64_t* empty_d = full_d + 2;
  uint64_t* drained = empty_d + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L.tmem_slot);
  volatile int* flag_abort = reinterpret_cast<volatile int*>(smem + L.flags);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // (uniform over the warp)
  const uint32_t crank = CG == 2 ? blockIdx.x & 1 : 0;    // rank in the pair: clusters are consecutive blocks
  const int team = blockIdx.x / CG;
  const int nk = p.K / BK;                    // 64-k steps of a tile
  constexpr int TERMS = terms(RAGGED);        // A slots per weight stage

  if (threadIdx.x == 0) {
    // full_x, full_a and empty_d are used in the pair's first CTA only; commits arrive in both CTAs
    for (int i = 0; i < MAX_XS; ++i) { mbar_init(&full_x[i], 1); mbar_init(&empty_x[i], 1); }
    for (int i = 0; i < MAX_WS; ++i) { mbar_init(&full_w[i], 1); mbar_init(&empty_w[i], TERMS * N_DQ_WARPS / 2); }
    for (int i = 0; i < MAX_AS; ++i) { mbar_init(&full_a[i], CG * N_DQ_WARPS / 2); mbar_init(&empty_a[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&full_d[i], 1); mbar_init(&empty_d[i], 4 * CG); }
    mbar_init(drained, 1);
    *flag_abort = 0;
    fence_barrier_init();
    griddep_launch_dependents();
  }
  if (warp == WARP_MMA) tmem_alloc<CG>(tmem_slot, TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (CG == 2) cluster_barrier();             // the other CTA's barriers exist
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t a_base = tmem_base + TMEM_COLS - p.nas * A_SLOT_COLS;

  // (a pair gives up together: see drain)
#define LCQ_GIVE_UP(code)                                                                                                  \
  do {                                                                                                                     \
    *flag_abort = 1;                                                                                                       \
    if (CG == 2) store_remote(peer_addr(smem_u32(smem + L.flags + 4 * FLAG_ABORT), crank ^ 1u), 1);                        \
    atomicExch(&g_device_status, (code));                                                                                  \
  } while (0)

  if (warp == WARP_W) {
    // ------------------------------------------------------------ weights and scales (constants: no dependency wait)
    if (lane == 0) {
      tma_prefetch_desc(&tmap_w);
      if (!RAGGED) tma_prefetch_desc(&tmap_s);
      Ring r = {0, 0};
      bool ok = true;
      int issued = 0;
      for (Walk w(p, team); ok && w.next(p);) {
        const int n0 = (w.tile % p.n_tiles_n) * (CG * BN) + static_cast<int>(crank) * BN;
        for (int st = w.st0; st < w.st1; ++st, r.step(p.nws)) {
          if (!wait_bar(flag_abort, &empty_w[r.i], r.phase ^ 1u)) { LCQ_GIVE_UP(10); ok = false; break; }
          uint8_t* dst = smem + L.w + r.i * WS_STAGE;
          mbar_expect_tx(&full_w[r.i], RAGGED ? W_STAGE : WS_STAGE);
          tma_load_2d(dst, &tmap_w, &full_w[r.i], st * (WK / 2), n0);
          if (!RAGGED) tma_load_2d(dst + W_STAGE, &tmap_s, &full_w[r.i], st * (WK / 32), n0);
          ++issued;
        }
      }
      flag_abort[ISSUED_W] = issued;
    }
  } else if (warp == WARP_X) {
    // ------------------------------------------------------------ activations: this CTA's share of the rows of each tile
    if (lane == 0) {
      tma_prefetch_desc(&tmap_x);
      griddep_wait();                    // x is the preceding kernel's output
      const int stage_bytes = x_stage_bytes(p.bm, CG);
      Ring r = {0, 0};
      bool ok = true;
      int issued = 0;
      for (Walk w(p, team); ok && w.next(p);) {
        const int rows = w.bm / CG, bytes = x_step_bytes(w.bm, CG);
        const int m0 = w.m0 + static_cast<int>(crank) * rows;
        const CUtensorMap* tmap = w.bm == p.bm ? &tmap_x : &tmap_piece;
        for (int st = w.st0; st < w.st1; ++st, r.step(p.nxs)) {
          const int steps = RAGGED && nk - st * 4 < 4 ? nk - st * 4 : 4;
          if (!wait_bar(flag_abort, &empty_x[r.i], r.phase ^ 1u)) { LCQ_GIVE_UP(11); ok = false; break; }
          if (crank == 0) mbar_expect_tx(&full_x[r.i], CG * steps * bytes);
          const uint32_t bar = leader_addr<CG>(full_x + r.i);
          uint8_t* dst = smem + r.i * stage_bytes;
          for (int j = 0; j < steps; ++j) {
            if (CG == 2) tma_load_2d_pair(dst + j * bytes, tmap, bar, (st * 4 + j) * BK, m0);
            else tma_load_2d(dst + j * bytes, tmap, full_x + r.i, (st * 4 + j) * BK, m0);
          }
          ++issued;
        }
      }
      if (CG == 2) store_remote(peer_addr(smem_u32(smem + L.flags + 4 * (ISSUED_X0 + crank)), 0), issued);
      else flag_abort[ISSUED_X0] = issued;
    }
  } else if (warp == WARP_MMA) {
    // ------------------------------------------------------------ MMA issuer: one warp for the team
    if (crank == 0) {
      const uint32_t desc0 = make_b_desc(smem_u32(smem));                                 // descriptors count 16-byte units
      const uint32_t desc_stage = static_cast<uint32_t>(x_stage_bytes(p.bm, CG) >> 4);
      Ring rx = {0, 0}, ra = {0, 0}, rd = {0, 0};
      bool ok = true;
      for (Walk w(p, team); ok && w.next(p); rd.step(p.nd)) {
        if (!warp_wait(flag_abort, &empty_d[rd.i], rd.phase ^ 1u)) { if (lane == 0) LCQ_GIVE_UP(12); ok = false; break; }
        tc_fence_after();
        const uint32_t idesc = make_idesc(w.bm, CG);
        const uint32_t desc_step = static_cast<uint32_t>(x_step_bytes(w.bm, CG) >> 4);
        const uint32_t d_t = tmem_base + rd.i * p.bm;
        uint32_t acc = 0;
        for (int i = TERMS * w.st0; i < TERMS * w.st1; ++i, ra.step(p.nas)) {
          const int st = i / TERMS;
          const int steps = RAGGED && nk - st * 4 < 4 ? nk - st * 4 : 4;
          if (!warp_wait(flag_abort, &full_x[rx.i], rx.phase) || !warp_wait(flag_abort, &full_a[ra.i], ra.phase)) {
            if (lane == 0) LCQ_GIVE_UP(14);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t bdesc = desc0 + rx.i * desc_stage, a_t = a_base + ra.i * A_SLOT_COLS;
          if constexpr (HALVES) {
            umma_steps<1, 2>(d_t, a_t, bdesc, desc_step, idesc, acc);
            umma_steps<1, 2>(d_t, a_t + 2 * A_STEP_COLS, bdesc + 2 * desc_step, desc_step, idesc, 1u);
          } else if (!RAGGED || steps == WK / BK) {
            umma_steps<CG, 4>(d_t, a_t, bdesc, desc_step, idesc, acc);
          } else {
            for (int k = 0; k < steps; ++k) umma_step<CG>(d_t, a_t + k * A_STEP_COLS, bdesc + k * desc_step, idesc, k == 0 ? acc : 1u);
          }
          acc = 1;
          if (TERMS == 1 || (i & 1)) {
            umma_commit<CG>(&empty_x[rx.i]);
            rx.step(p.nxs);
          }
          umma_commit<CG>(&empty_a[ra.i]);
        }
        if (ok) umma_commit<CG>(&full_d[rd.i]);
      }
    }
  } else if (warp < N_DQ_WARPS) {
    // ------------------------------------------------------------ dequant warps: smem int4 -> TMEM fp16
    // Two sets of two warpgroups take the stages (TERMS = 2: the two terms of each stage) in turn, so that one set
    // computes while the other loads, stores or waits.  Thread = weight row = TMEM lane; warpgroup g of a set takes the 64-k steps 2g and
    // 2g + 1 of its stages (four scale groups).
    const int set = warp >> 3, g = (warp >> 2) & 1;
    const int r = (warp & 3) * 32 + lane;
    const uint32_t lane_taddr = a_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + 2 * g * A_STEP_COLS;
    const uint32_t full_a0 = leader_addr<CG>(full_a);
    const uint8_t* wrow = smem + L.w + r * 128;
    const uint8_t* srow = smem + L.w + W_STAGE + r * 16 + g * 8;
    const int swz = (4 * g) ^ (r & 7);         // 16-byte chunk 4g + j of the row sits at chunk (4g + j) ^ (r & 7): 128-byte swizzle
    Ring rw = {0, 0}, ra = {0, 0};
    int turn = 0;                              // whose A slot it is
    bool ok = true;
    for (Walk w(p, team); ok && w.next(p);) {
      const uint32_t* gs = nullptr;            // RAGGED: this row's scales in global memory, two groups a word
      uint2 s_next = make_uint2(0u, 0u);
      const auto fetch = [&](int st) {
        const int k = st * 4 + 2 * g;
        s_next.x = __ldg(gs + (k < nk ? k : nk - 1));
        s_next.y = __ldg(gs + (k + 1 < nk ? k + 1 : nk - 1));
      };
      if (RAGGED) {
        const int n = (w.tile % p.n_tiles_n) * (CG * BN) + static_cast<int>(crank) * BN + r;
        gs = reinterpret_cast<const uint32_t*>(p.scales) + static_cast<long long>(n < p.N ? n : p.N - 1) * nk;
        fetch(w.st0);
      }
      for (int i = TERMS * w.st0; i < TERMS * w.st1; ++i, turn ^= 1, ra.step(p.nas)) {
        const int st = i / TERMS;
        if (turn != set) {
          if (TERMS == 1) rw.step(p.nws);
          continue;
        }
        uint2 sc = s_next;
        if (RAGGED) fetch(st + 1);
        if (!warp_wait(flag_abort, &full_w[rw.i], rw.phase)) { if (lane == 0) LCQ_GIVE_UP(15); ok = false; break; }
        const uint8_t* src = wrow + rw.i * WS_STAGE;
        uint4 pk[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) pk[j] = *reinterpret_cast<const uint4*>(src + ((swz ^ j) << 4));
        if (!RAGGED) sc = *reinterpret_cast<const uint2*>(srow + rw.i * WS_STAGE);
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty_w[rw.i]);
        const uint32_t dst = lane_taddr + ra.i * A_SLOT_COLS;
#pragma unroll
        for (int h = 0; h < 2; ++h) {          // RAGGED: steps past K are stored too, and not multiplied
          const __half2 s01 = *reinterpret_cast<const __half2*>(h == 0 ? &sc.x : &sc.y);
          const __half2 s0 = __low2half2(s01), s1 = __high2half2(s01);
          uint32_t v[32];
          if (TERMS == 2 && set == 1) dequant_step<PERM, true>(pk + 2 * h, s0, s1, v);
          else dequant_step<PERM, false>(pk + 2 * h, s0, s1, v);
          if (h == 0) {
            if (!warp_wait(flag_abort, &empty_a[ra.i], ra.phase ^ 1u)) { if (lane == 0) LCQ_GIVE_UP(16); ok = false; break; }
            tc_fence_after();
          }
          tmem_st32(dst + h * A_STEP_COLS, v);
        }
        if (!ok) break;
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) arrive_leader<CG>(full_a0 + ra.i * 8);
        rw.step(p.nws);
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue warps: TMEM -> global
    // The accumulator is n-major (lane = n, column = m) while out is [M, N]: a warp writes 32
    // consecutive n of one m per store (64 or 128 contiguous bytes: whole sectors).
    griddep_wait();                            // out and the scratch may still be in the preceding kernel's use
    const int q4 = warp - WARP_EPI0;
    const int r = q4 * 32 + lane;
    const uint32_t lane_taddr = tmem_base + (static_cast<uint32_t>(q4 * 32) << 16);
    const uint32_t empty_d0 = leader_addr<CG>(empty_d);
    volatile int* shared_int = flag_abort + FLAG_SHARED;
    const long long part_elems = static_cast<long long>(p.bm) * BN;
    Ring rd = {0, 0};
    for (Walk w(p, team); w.next(p); rd.step(p.nd)) {
      const int n = (w.tile % p.n_tiles_n) * (CG * BN) + static_cast<int>(crank) * BN + r;
      const uint32_t d_t = lane_taddr + rd.i * p.bm;
      int rows = p.M - w.m0;                   // rows of out in this tile
      if (rows > w.bm) rows = w.bm;
      OT* out = static_cast<OT*>(p.out) + static_cast<long long>(w.m0) * p.N + n;
      // one verdict for the four warps: they meet at named barriers below
      if (!all_epilogue_warps(wait_bar(flag_abort, &full_d[rd.i], rd.phase))) { if (lane == 0) LCQ_GIVE_UP(17); break; }
      tc_fence_after();
      if (CG == 1 && p.split > 1) break;       // the cluster adds up its shares below
      // who else contributes to this tile: teams p0 .. p1
      int p0 = team, p1 = team, slot1 = 0;
      if (CG == 1 && w.tile < p.sk_tiles) {
        const unsigned t0 = static_cast<unsigned>(w.tile) * static_cast<unsigned>(p.nst);
        p0 = share_owner(p, t0);
        p1 = share_owner(p, t0 + static_cast<unsigned>(p.nst) - 1u);
        slot1 = share_begin(p, p0) < t0;       // p0 came from the tile before (slot 0); the others' shares begin here
      }
      const auto part = [&](int q) {
        return p.partials + static_cast<long long>(2 * q + (q == p0 ? slot1 : 0)) * part_elems + r;
      };
      if (CG == 2 || p1 == p0) {
        for (int c0 = 0; c0 < rows; c0 += 32) {
          uint32_t v[32];
          tmem_ld32(d_t + c0, v);
          tmem_wait_ld();
          if (n < p.N) {
            OT* o = out + static_cast<long long>(c0) * p.N;
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              if (c0 + i < rows) *o = from_f32<OT>(__uint_as_float(v[i]));
              o += p.N;
            }
          }
        }
      } else {
        int* counter = p.counters + w.tile;
        // published already by all the others?  Then this CTA finishes the tile without publishing.
        if (threadIdx.x == WARP_EPI0 * 32) *shared_int = load_acquire(counter);
        named_bar_sync(BAR_EPI, 128);
        bool finish = *shared_int == p1 - p0;
        named_bar_sync(BAR_EPI, 128);
        if (!finish) {
          float* mine = part(team);
          for (int c0 = 0; c0 < rows; c0 += 32) {
            uint32_t v[32];
            tmem_ld32(d_t + c0, v);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 32; ++i) __stcg(mine + (c0 + i) * BN, __uint_as_float(v[i]));
          }
          __threadfence();
          named_bar_sync(BAR_EPI, 128);
          if (threadIdx.x == WARP_EPI0 * 32) *shared_int = atomicAdd(counter, 1);
          named_bar_sync(BAR_EPI, 128);
          finish = *shared_int == p1 - p0;
          named_bar_sync(BAR_EPI, 128);
        }
        __threadfence();
        if (finish) {
          finish_tile<OT>(d_t, out, n < p.N ? rows : 0, rows, p.N, part(p0), part(p0) + (2 - slot1) * part_elems,
                          2 * part_elems, p1 - p0 + 1, team - p0);
          if (threadIdx.x == WARP_EPI0 * 32) *counter = 0;
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) arrive_leader<CG>(empty_d0 + rd.i * 8);
    }
  }
#undef LCQ_GIVE_UP

  tc_fence_before();
  __syncthreads();
  if (CG == 2) cluster_barrier();    // neither CTA leaves while the other may still arrive on its barriers or the pair's MMAs read its memory
  if (*flag_abort) {
    drain<CG, RAGGED>(p, smem, team, crank);
    if (CG == 2) cluster_barrier();
  }
  if (CG == 1 && p.split > 1) {
    // One tile per cluster, its K shared out: CTA d settles columns d * cw .. of the tile.  Every CTA sends
    // each of the others its part of their columns (distributed shared memory, into the rings, which
    // nobody uses any more), and adds up what it got in rank order.
    // The twenty dequant and epilogue warps each take 16 columns at a time.
    const int me = team % p.split, tile = team / p.split, cw = (p.bm + p.split - 1) / p.split;
    const int m0 = (tile / p.n_tiles_n) * p.bm;
    const int rows = p.M - m0 < p.bm ? p.M - m0 : p.bm;
    const int r = (warp & 3) * 32 + lane;
    cluster_barrier();
    if (warp < WARP_W) {
      tc_fence_after();
      const uint32_t mine = smem_u32(smem) + (me * cw * BN + r) * 4;
      for (int c0 = (warp >> 2) * 16; c0 < rows; c0 += (WARP_W / 4) * 16) {
        uint32_t v[16];
        tmem_ld16(tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + c0, v);
        tmem_wait_ld();
        int d = c0 / cw, j = c0 - d * cw;
        uint32_t dst = peer_addr(mine + j * (BN * 4), d);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          if (c0 + i < rows) store_remote(dst, static_cast<int>(v[i]));
          dst += BN * 4;
          if (++j == cw && d + 1 < p.split) { j = 0; ++d; dst = peer_addr(mine, d); }
        }
      }
      tc_fence_before();
    }
    cluster_barrier();
    const int n = (tile % p.n_tiles_n) * BN + r;
    if (warp < WARP_W && n < p.N) {
      const float* got = reinterpret_cast<const float*>(smem) + r;
      OT* out = static_cast<OT*>(p.out) + static_cast<long long>(m0 + me * cw) * p.N + n;
#pragma unroll 2
      for (int j = warp >> 2; j < cw && me * cw + j < rows; j += WARP_W / 4) {
        float sum = 0.0f;
        for (int q = 0; q < p.split; ++q) sum += got[(q * cw + j) * BN];
        out[static_cast<long long>(j) * p.N] = from_f32<OT>(sum);
      }
    }
  }
  if (warp == WARP_MMA) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc<CG>(tmem_base, TMEM_COLS);
  }
}

// bf16 -> fp16 copy of the activations (exact for |x| in fp16's normal range) with the 8 values
// of every 16-byte piece reordered to (0,4,1,5,2,6,3,7): the order in which the nibble masks
// deliver the weights, so the dequant warps need no re-pairing.
__global__ void __launch_bounds__(256) bf16_to_f16_perm_kernel(const uint4* __restrict__ in, uint4* __restrict__ out, long long n16) {
  griddep_launch_dependents();
  griddep_wait();
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n16; i += stride) {
    const uint4 a = __ldg(in + i);
    const uint32_t w[4] = {a.x, a.y, a.z, a.w};
    float f[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) { f[2 * j] = __uint_as_float(w[j] << 16); f[2 * j + 1] = __uint_as_float(w[j] & 0xFFFF0000u); }
    const __half2 h0 = __floats2half2_rn(f[0], f[4]), h1 = __floats2half2_rn(f[1], f[5]);
    const __half2 h2 = __floats2half2_rn(f[2], f[6]), h3 = __floats2half2_rn(f[3], f[7]);
    out[i] = make_uint4(*reinterpret_cast<const uint32_t*>(&h0), *reinterpret_cast<const uint32_t*>(&h1),
                        *reinterpret_cast<const uint32_t*>(&h2), *reinterpret_cast<const uint32_t*>(&h3));
  }
}

// ---------------------------------------------------------------------------- host side
struct Tiling { int cg, bm, n_tiles_n, n_tiles, teams, sk_tiles, full, tail, split, nd, nas, nxs, nws; };

// Microseconds of a 64-k step of a tile, measured at K = 8192 when every MMA had an election of its own: with few teams at work the hand-over
// of the weights through TMEM and the MMAs bound it; with all SMs busy (`used` = 1) L2 and power add to that.  Since the MMAs of a stage are
// issued in one block, steps of up to 64 rows take less than this says (64 x 8192 -> 28672: 0.22 us by the formula, 0.19 by the call's 42 us; 32 rows 46 ->
// 36 us a call), so low tiles, pieces and shares of K are priced too high against high tiles.  The constants have not been fitted again: forms are chosen as they
// were, and calls have become faster in them.  Two terms per weight are taken to cost twice as much, which has not been measured by itself.
inline double step_us(int cg, int bm, double used) {
  const double alone = 0.145 + 0.0005 * bm;
  const double busy = cg == 1 ? 0.145 + 0.00117 * bm : bm <= 128 ? 0.152 + 0.00088 * bm : 0.150 + 0.00100 * bm;
  const double f = used <= 0.5 ? 0.0 : used >= 1.0 ? 1.0 : 2.0 * used - 1.0;
  return alone + (busy - alone) * f;
}

// Tile shape, and how the tiles are dealt out: the cheapest of a few forms by that estimate.
inline Tiling choose_tiling(int M, int N, int K, int sm_count) {
  const int nk = K / BK, nst = (K + WK - 1) / WK;
  Tiling best;
  memset(&best, 0, sizeof(best));
  double best_cost = 1e300;
  for (int cg = 1; cg <= 2 && cg <= sm_count; ++cg) {
    const int P = sm_count / cg;
    const int tn = (N + cg * BN - 1) / (cg * BN);
    for (int bm = 32; bm <= (cg == 1 ? 128 : 256); bm += 32) {
      const int tm = (M + bm - 1) / bm;
      if (bm > 32 && tm == (M + bm - 33) / (bm - 32)) continue;      // the same number of tiles fit a lower tile
      const long long tiles = static_cast<long long>(tn) * tm;
      Tiling t;
      t.cg = cg; t.bm = bm; t.n_tiles_n = tn; t.n_tiles = static_cast<int>(tiles);
      t.nd = bm <= 128 ? 2 : 1;
      t.nas = bm <= 64 ? 3 : 2;
      const int per_cta = bm / cg;                    // rows of x a CTA stages
      t.nxs = per_cta <= 16 ? 6 : per_cta <= 32 ? 5 : per_cta <= 64 ? 3 : 2;
      t.nws = (227 * 1024 - 1024 - t.nxs * x_stage_bytes(bm, cg)) / WS_STAGE;
      if (t.nws > MAX_WS) t.nws = MAX_WS;
      const auto consider = [&](long long teams, long long sk, long long full, int tail, int split, double cost) {
        if (cost >= best_cost) return;
        best_cost = cost;
        t.teams = static_cast<int>(teams); t.sk_tiles = static_cast<int>(sk); t.split = split;
        t.full = static_cast<int>(full); t.tail = tail;
        best = t;
      };
      const auto step = [&](int rows, double teams) { return terms(K % WK != 0) * step_us(cg, rows, teams / P); };
      const double start = cg == 1 ? 4.5 : 5.5, epilogue = t.nd == 1 ? 0.0075 * bm : 0.0;   // one accumulator: its epilogue shows
      const long long waves = tiles / P, rem = tiles % P;
      const double full_waves = static_cast<double>(waves) * (nk * step(bm, P) + epilogue);
      // whole tiles
      consider(tiles < P ? tiles : P, 0, tiles, 1, 1, start + full_waves + (rem ? nk * step(bm, static_cast<double>(rem)) + epilogue : 0.0));
      if (rem == 0) continue;
      // the tiles of the last wave in pieces of fewer rows of x
      for (int tail = 2; tail <= 8; tail *= 2) {
        const int piece = bm / tail;
        if (piece < 32 || piece % mma_n_step(cg) != 0 || piece * tail != bm) continue;
        const long long pieces = rem * tail, last = (pieces + P - 1) / P;
        consider(waves == 0 && pieces < P ? pieces : P, 0, tiles - rem, tail, 1,
                 start + full_waves + last * nk * step(piece, static_cast<double>(pieces) / last) + 0.5);
      }
      if (cg == 2) continue;
      if (waves == 0) {
        // fewer tiles than SMs: a cluster per tile.  Clusters pack the ~16 SMs that are sure of each GPC
        // (18 SMs on average); more of them than fit at once take turns, at twice the time.
        for (int c = 2; c <= 6 && c <= nst; ++c) {
          if (tiles > static_cast<long long>(sm_count / 18) * (16 / c)) continue;
          consider(tiles * c, 0, tiles, 1, c, start + ((nst + c - 1) / c) * 4 * step(bm, static_cast<double>(tiles * c)) + 2.5);
        }
      } else {
        // equal shares of K for what does not fill all SMs, with a wave of whole tiles added when the shares
        // would be short (each contributor costs the one who adds up a round trip per 16 rows)
        const long long sk = rem * 3 >= P ? rem : rem + P;
        const long long share = (sk * nst + P - 1) / P;
        consider(P, sk, tiles, 1, 1, start + static_cast<double>((tiles - sk) / P) * (nk * step(bm, P) + epilogue) +
                                         share * 4 * step(bm, P) + (sk == rem ? 2.0 : 6.0));
      }
    }
  }
  return best;
}

inline bool supported(int M, int N, int K, int G, int x_dtype, int scale_dtype) {
  return M >= 1 && N >= 1 && K >= BK && (K % BK) == 0 && G == 32 &&
         (x_dtype == LCQ_F16 || x_dtype == LCQ_BF16) && scale_dtype == LCQ_F16;
}

inline size_t x_copy_bytes(int M, int K, int x_dtype) {
  return x_dtype == LCQ_BF16 ? ((static_cast<size_t>(M) * K * 2 + 255) & ~static_cast<size_t>(255)) : 0;
}
inline size_t partial_bytes(const Tiling& t) {
  return t.sk_tiles ? static_cast<size_t>(t.teams) * 2 * t.bm * BN * sizeof(float) : 0;
}
// [shared counter region][fp16 copy of bf16 activations][float partials of the tiles cut along K]
inline size_t workspace_bytes(const Tiling& t, int M, int K, int x_dtype) {
  const size_t scratch = x_copy_bytes(M, K, x_dtype) + partial_bytes(t);
  return scratch ? kWorkspaceCounterBytes + scratch : 0;
}
inline size_t workspace_bytes(int M, int N, int K, int x_dtype, int sm_count = 148) {
  return workspace_bytes(choose_tiling(M, N, K, sm_count), M, K, x_dtype);
}

inline void pdl_launch_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr, int grid, int block, size_t smem, cudaStream_t stream) {
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 1 : 0;
}

template <int CG, typename OT, bool PERM, bool RAGGED, bool HALVES = false>
int launch_t(const CUtensorMap* tm, const Params& p, cudaStream_t stream) {
  if constexpr (CG == 1 && !RAGGED && !HALVES) {
    if (p.bm > 64) return launch_t<CG, OT, PERM, RAGGED, true>(tm, p, stream);
  }
  auto kern = w4a16_gemm_kernel<CG, OT, PERM, RAGGED, HALVES>;
  static thread_local int configured_device = -1;
  int dev = 0;
  LCQ_CUDA_TRY(cudaGetDevice(&dev));
  if (configured_device != dev) {
    LCQ_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    configured_device = dev;
  }
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[2];
  pdl_launch_config(cfg, attr, CG * p.teams, NTHREADS, smem_map(p.bm, CG, p.nxs, p.nws).total, stream);
  const int cluster = CG == 2 ? 2 : p.split;
  if (cluster > 1) {
    cudaLaunchAttribute& a = attr[cfg.numAttrs++];
    a.id = cudaLaunchAttributeClusterDimension;
    a.val.clusterDim.x = cluster;
    a.val.clusterDim.y = 1;
    a.val.clusterDim.z = 1;
  }
  LCQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, tm[0], tm[1], tm[2], tm[3], p));
  return LCQ_OK;
}
template <int CG, typename OT>
int launch_by_kind(bool perm, bool ragged, const CUtensorMap* tm, const Params& p,
                   cudaStream_t stream) {
  if (perm) return ragged ? launch_t<CG, OT, true, true>(tm, p, stream) : launch_t<CG, OT, true, false>(tm, p, stream);
  return ragged ? launch_t<CG, OT, false, true>(tm, p, stream) : launch_t<CG, OT, false, false>(tm, p, stream);
}
template <typename OT>
int launch_by_team(int cg, bool perm, bool ragged, const CUtensorMap* tm, const Params& p,
                   cudaStream_t stream) {
  return cg == 2 ? launch_by_kind<2, OT>(perm, ragged, tm, p, stream) : launch_by_kind<1, OT>(perm, ragged, tm, p, stream);
}

inline Params make_params(const Tiling& t, int M, int N, int K) {
  Params p;
  memset(&p, 0, sizeof(p));
  p.M = M; p.N = N; p.K = K;
  p.bm = t.bm; p.n_tiles_n = t.n_tiles_n; p.n_tiles = t.n_tiles;
  p.nst = (K + WK - 1) / WK;
  p.teams = t.teams; p.sk_tiles = t.sk_tiles; p.full = t.full; p.tail = t.tail; p.split = t.split;
  p.nxs = t.nxs; p.nws = t.nws; p.nas = t.nas; p.nd = t.nd;
  return p;
}

inline int launch(const void* x, const void* w, const void* s, void* out, int M, int N, int K, int x_dtype,
                  int out_dtype, void* workspace, size_t ws_bytes, int sm_count, cudaStream_t stream) {
  if (!aligned(w, 16) || !aligned(s, 16) || !aligned(x, 16)) {
    set_error("w4a16 gemm: x, w_packed and scales must be 16-byte aligned");
    return LCQ_ERR_BAD_ARG;
  }
  const Tiling t = choose_tiling(M, N, K, sm_count);
  const size_t need = workspace_bytes(t, M, K, x_dtype);
  if (need && (workspace == nullptr || ws_bytes < need || !aligned(workspace, 256))) {
    set_error("w4a16 gemm: workspace of %zu bytes (256-byte aligned) required, got %zu", need, ws_bytes);
    return LCQ_ERR_WORKSPACE;
  }
  uint8_t* scratch = need ? static_cast<uint8_t*>(workspace) + kWorkspaceCounterBytes : nullptr;
  const bool perm = x_dtype == LCQ_BF16, ragged = K % WK != 0;
  const void* xh = x;
  // kind::f16 wants both operands in one 16-bit format and the weight tiles must be fp16, so bf16
  // activations are converted once into the workspace.
  if (perm) {
    const long long n16 = static_cast<long long>(M) * K / 8;
    long long blocks = (n16 + 255) / 256;
    if (blocks > static_cast<long long>(sm_count) * 8) blocks = static_cast<long long>(sm_count) * 8;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    pdl_launch_config(cfg, attr, static_cast<int>(blocks), 256, 0, stream);
    LCQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, bf16_to_f16_perm_kernel, static_cast<const uint4*>(x), reinterpret_cast<uint4*>(scratch), n16));
    xh = scratch;
  }
  Params p = make_params(t, M, N, K);
  p.out = out;
  p.scales = s;
  p.counters = static_cast<int*>(workspace);
  p.partials = reinterpret_cast<float*>(scratch + x_copy_bytes(M, K, x_dtype));
  CUtensorMap tm[4];    // x in whole tiles, x in pieces of a tile, weights, scales
  const uint64_t k64 = static_cast<uint64_t>(K), m64 = static_cast<uint64_t>(M), n64 = static_cast<uint64_t>(N);
  int rc = encode_tmap_2d(&tm[0], 1, xh, k64, m64, k64 * 2, BK, p.bm / t.cg, 3);
  if (rc != LCQ_OK) return rc;
  if (t.tail == 1) tm[1] = tm[0];
  else if ((rc = encode_tmap_2d(&tm[1], 1, xh, k64, m64, k64 * 2, BK, p.bm / t.tail / t.cg, 3)) != LCQ_OK) return rc;
  if ((rc = encode_tmap_2d(&tm[2], 0, w, k64 / 2, n64, k64 / 2, WK / 2, BN, 3)) != LCQ_OK) return rc;
  if (ragged) tm[3] = tm[2];                     // not used
  else if ((rc = encode_tmap_2d(&tm[3], 1, s, k64 / 32, n64, k64 / 16, WK / 32, BN, 0)) != LCQ_OK) return rc;
  switch (out_dtype) {
    case LCQ_F32: return launch_by_team<float>(t.cg, perm, ragged, tm, p, stream);
    case LCQ_F16: return launch_by_team<__half>(t.cg, perm, ragged, tm, p, stream);
    case LCQ_BF16: return launch_by_team<__nv_bfloat16>(t.cg, perm, ragged, tm, p, stream);
    default: break;
  }
  set_error("w4a16 gemm: bad out_dtype %d", out_dtype);
  return LCQ_ERR_BAD_ARG;
}

}  // namespace gemm_tc
}  // namespace lcq
