// One decode step of a Llama-style stack of quantized linears (M = 1, int4 weights in groups of 32) as ONE
// kernel: embedding, per layer {RMS norm, q|k|v and o projections, residual add + RMS norm, gate|up, SiLU *
// up, down, residual add}, final norm, lm_head and greedy argmax -- the chain that locomp_b200.DecodeStack
// runs as 8 launches a layer otherwise (examples/54_smollm2_inference.py:494-578 without the attention
// itself; o reads a prepared buffer, so it depends on nothing in its layer).  That makes two dependent
// exchanges a layer.  It is an order that only a step without attention has: a layer whose o reads the
// attention output has four (q|k|v, o, gate|up, down) and cannot take this schedule.
//
// What bounds it.  SmolLM2-135M has 30 layers of 2 MB: 12 us of HBM time for the whole token, but a chain
// of 60 dependent matvecs whose results every SM needs.  Latency is all there is to it: the round trip
// through L2 (0.9 us from storing a result to every CTA's having it) and the dependent instructions of a matvec, a norm and
// an activation.  As separate kernels 484 us a token, as one kernel with float32 FMAs 285 to 297, now 185 to 188 (over boxes).  Hence
//   * one CTA per SM stays for the whole step; a producer thread streams the CTA's rows of ALL layers
//     through one shared-memory ring (bulk copies), running ahead across layers, so that weights are there
//     when their input is;
//   * results that the next phase needs are published as words {fp16 value, 16-bit tag of the phase}: a
//     consumer polls the data itself until every tag is the one it expects.  No grid barrier, no fence, no
//     flag: one store and one load through L2 between dependent matvecs;
//   * every CTA keeps the hidden state and does the norms redundantly;
//   * the warps are two sets with roles of their own, so that what is not on the chain runs beside it: the first
//     set publishes the activation and the down projection and waits for the activations of the others, and computes o two layers ahead;
//     the second does the norms and q|k|v.  Both multiply gate|up and down;
//   * all of it is one loop body without calls: registers that a call saves go to the stack, and with all of L1 given to
//     shared memory that is a trip to L2 (one call a phase cost 60 us a step); and code beyond 32 KB is fetched at half the speed.
// A matvec runs on mma.sync: 16 rows x 32 k (one group) are two m16n8k16 MMAs whose A operand are the nibbles as q - 8
// in fp16 (exact) and whose B operand is x; the group's scale multiplies the float32 result.
// No shuffles: the tensor core adds up a group, a lane the groups of its rows, shared memory the warps.
//
// A set waits for the stages that it uses itself and skips the other's, up to more than a round of the ring.  A barrier's parity tells only
// neighbouring rounds apart, so before it a set waits for the producer's count of issued stages, which says which round a place of the ring is in.
//
// Every CTA has at least one unit of 4 rows in every phase on the chain.  So whoever has all results of a phase knows
// that all CTAs have read what they needed for it, and a buffer that is rewritten a layer later has no reader left.  The
// results of o take two buffers in turn: those of layer l + 2 are written after all activations of layer l have come in, which were
// published after the norms that read o of layer l.
//
// The CTAs wait for one another: the launch is cooperative, and every wait is bounded (on expiry the CTA
// records a status code and runs to its end without waiting).
//
// Arithmetic as in the separate kernels: exact products and float32 sums, each result rounded to fp16 where
// those kernels store it.  (A group of 32 is summed by the tensor core, which truncates, by about 1e-7 of it; the chain's matvec does the same.
// The sums run in other orders, so single fp16 results may turn: against 64 bits the logits after 30 layers of 576 / 1536 are off by 1.86e-3, those of the
// chain by 1.97e-3, of the kernel with FMAs by 1.92e-3, root mean square over eight inputs; 2 layers of 2048 / 8192 2.62e-4, 2.64e-4, 2.62e-4.)
#pragma once
#include "common.cuh"

namespace lcq {
namespace step {

// Two sets of SET consumer warps, and the producer; of a warp's share of a stage U groups of 32 columns at a time.
template <int SET> struct Threads {
  static constexpr int NCW = 2 * SET, NCT = NCW * 32, SET_T = SET * 32, ALL = NCT + 32;
};
constexpr int MAX_STAGES = 32;
enum { BAR_ALL = 1, BAR_SUMS, BAR_SET0, BAR_SET1 };   // named barriers: all consumers; a phase's sums are there; those of a set
constexpr int STATE_BYTES = 64;                // epoch, argmax counter, argmax key
constexpr int HEAD_SLABS = 32;                 // slabs of the lm_head whose sums are kept at a time (of the other parts: all of a CTA's, where they fit)
constexpr int COPIES = 8;                      // of the published words: a CTA polls copy b % 8.  (30 layers of width 576: 1 copy 420 us, 2 363, 4 337, 8 332, 16 325 in an early build)
constexpr int ROW_SUMS = 48;                   // bytes of a row's partial sums of a stage, one per warp of a set (eight at most; rows sit in different banks)
constexpr int STAGE_SUMS = 16 * ROW_SUMS;
constexpr int PART_INFO_BYTES = 16 + 8 * 16 + 8 * 4;

struct Shape { int hidden, inter, qkv, q_dim, vocab; };
enum { PART_O, PART_GATE, PART_QKV, PART_DOWN, PART_HEAD, N_PARTS };
// How a weight [n, K] is streamed: as [n * v, K / v], a matrix of the same bytes with shorter rows.  A stage is a slab of up to 16 of
// those, the rows of an MMA's A operand, as they lie in memory: one copy, and one of their scales.  gate|up: up to 8 rows of gate, then the same
// ones of up, so that both sums of a row end up in the same lane.
struct Part {
  int K, v, lg_v;       // lg: logarithms
  int groups;           // of 32 columns of a (short) row; 16 bytes each, so that a row is `groups` times 16 bytes
  int h1, slots;        // short rows of the first half of a slab (at most 8), of both
  int lg;               // short rows of a slab (gate|up: of a half) of a CTA that has more than one
  int per;              // rows that a slab advances by (gate|up: of each)
  int piece;            // slabs whose sums are kept at a time
};

// Offsets in shared memory.
struct Smem { int stages, xn, xq, xm, hid, gam, sums, side, red, info, bars, flags, rows, table, total; };

struct Params {
  lcq_decode_stack d;
  Shape sh;
  Part part[N_PARTS];
  Smem map;
  int n_layers, ctas;
  int stage_bytes, n_stages;
  float inv_hidden;
  uint32_t* o_buf;      // published words, first copy: o projection (two buffers), down projection [hidden], activation [inter]
  uint32_t* d_buf;
  uint32_t* m_buf;
};

// Rows of an [n, K] weight that CTA b streams: whole units of 4 (so that rows of scales start on 16 bytes).
__host__ __device__ inline int share(int n, int b, int ctas) { return static_cast<int>(static_cast<unsigned>(n / 4) * static_cast<unsigned>(b) / static_cast<unsigned>(ctas)) * 4; }
__host__ __device__ inline int max_share(int n, int ctas) { return (n / 4 + ctas - 1) / ctas * 4; }
__host__ __device__ inline int min2(int a, int b) { return a < b ? a : b; }
__host__ __device__ inline int max2(int a, int b) { return a > b ? a : b; }
__host__ __device__ inline int stages_of(const Part& q, int rows) { return (rows + q.per - 1) / q.per; }

inline Smem smem_map(const Params& p) {
  const Shape& s = p.sh;
  Smem m;
  m.stages = 0;
  m.xn = p.n_stages * p.stage_bytes;
  m.xq = m.xn + 2 * s.hidden * 2;              // both norms of a layer
  m.xm = m.xq + s.q_dim * 2;
  m.hid = m.xm + s.inter * 2;
  m.gam = m.hid + 2 * s.hidden * 2;            // before and after o
  m.sums = m.gam + 2 * s.hidden * 2;           // partial sums of the phases on the chain; of q|k|v, then of o
  const auto slabs = [&](int part, int n) { return min2(stages_of(p.part[part], max_share(n, p.ctas)), p.part[part].piece); };
  m.side = m.sums + max2(max2(slabs(PART_GATE, s.inter), slabs(PART_DOWN, s.hidden)), slabs(PART_HEAD, s.vocab)) * STAGE_SUMS;
  m.red = m.side + (slabs(PART_QKV, s.qkv) + slabs(PART_O, s.hidden)) * STAGE_SUMS;
  m.info = m.red + 32 * 8;
  m.bars = m.info + N_PARTS * PART_INFO_BYTES;
  m.flags = m.bars + 2 * MAX_STAGES * 8;
  m.rows = m.flags + 16;                       // (flags: a wait ran out; the epoch; stages issued) Rows
  m.table = m.rows + 64;                       // the layer records
  m.total = m.table + p.n_layers * static_cast<int>(sizeof(lcq_decode_layer));
  return m;
}

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ uint4 load_words(const uint32_t* p) {
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void publish(uint32_t* p, __half v, uint32_t tag) {
  const uint32_t word = (static_cast<uint32_t>(__half_as_ushort(v)) << 16) | tag;
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(word) : "memory");
}
__device__ __forceinline__ uint32_t nibbles(uint32_t w, uint32_t mask, uint32_t magic, uint32_t offset) {   // two q - 8 as fp16, exact
  uint32_t r;
  asm("{\n\t.reg .b32 t;\n\tlop3.b32 t, %1, %2, %3, 0xEA;\n\tsub.f16x2 %0, t, %4;\n\t}" : "=r"(r) : "r"(w), "r"(mask), "r"(magic), "r"(offset));
  return r;
}
// The 8 nibbles of a word as four operand registers: (0,4) (1,5) (2,6) (3,7).  x is staged in that order.
__device__ __forceinline__ void unpack(uint32_t w, uint32_t (&v)[4]) {
  const uint32_t w8 = w >> 8;
  v[0] = nibbles(w, 0x000F000Fu, 0x64006400u, 0x64086408u);
  v[1] = nibbles(w, 0x00F000F0u, 0x54005400u, 0x54805480u);
  v[2] = nibbles(w8, 0x000F000Fu, 0x64006400u, 0x64086408u);
  v[3] = nibbles(w8, 0x00F000F0u, 0x54005400u, 0x54805480u);
}

// The order of the stream: o of the first two layers; per layer gate|up, q|k|v, down, o of the layer after next; the lm_head.
struct Order {
  int layer, part;      // layer of the weight
  bool begun;
  __host__ __device__ inline void next(int n_layers) {
    if (part == PART_O) {
      if (begun) { --layer; part = PART_GATE; }
      else if (layer == 0 && n_layers > 1) layer = 1;
      else { layer = 0; part = PART_GATE; begun = true; }
    } else if (part == PART_GATE) part = PART_QKV;
    else if (part == PART_QKV) part = PART_DOWN;
    else if (part == PART_DOWN) {
      if (layer + 2 < n_layers) { layer += 2; part = PART_O; }
      else { ++layer; part = layer < n_layers ? PART_GATE : PART_HEAD; }
    } else part = N_PARTS;
  }
};
// The way of a set of warps through the stream: of gate|up, down and the lm_head each set takes every other stage; o is the first
// set's alone, q|k|v the second's.
struct Walk {
  int set, part, layer;
  int ahead;            // o is that of layer + ahead: of the first two layers before them, later of the layer after next
  int done;             // stages of the part that are done: it is taken in pieces
  __host__ __device__ inline explicit Walk(int set_) : set(set_), part(set_ == 0 ? PART_O : PART_GATE), layer(0), ahead(0), done(0) {}
  __host__ __device__ inline bool joint() const { return part == PART_GATE || part == PART_DOWN || part == PART_HEAD; }
  // The set's first of the n stages that are next, and the distance to the one after it.  (The set that has more to do besides takes the smaller half.)
  __host__ __device__ inline int first() const { return !joint() ? 0 : part == PART_DOWN ? 1 - set : set; }
  __host__ __device__ inline int step() const { return joint() ? 2 : 1; }
  __host__ __device__ inline int count(const int* stages, const Part* parts) const { return min2(stages[part] - done, parts[part].piece); }
  // The other set's stages before the first of this set's own.
  static __host__ __device__ inline int skipped_at_first(int set, int n_layers, const int* stages) { return set == 0 ? 0 : min2(n_layers, 2) * stages[PART_O]; }
  // On to what is next; returns how many stages of the stream in between are the other set's.  (The end: N_PARTS.)
  __host__ __device__ inline int next(int n_layers, const int* stages, const Part* parts) {
    int skipped = 0;
    done += parts[part].piece;
    if (done < stages[part]) return 0;
    done = 0;
    if (part == PART_GATE) {
      part = set == 0 ? PART_DOWN : PART_QKV;
      return set == 0 ? stages[PART_QKV] : 0;
    }
    if (part == PART_QKV) {
      part = PART_DOWN;
      return 0;
    }
    if (part == PART_HEAD) {
      part = N_PARTS;
      return 0;
    }
    if (part == PART_DOWN) {
      if (layer + 2 < n_layers) {
        if (set == 0) { part = PART_O; return 0; }
        skipped = stages[PART_O];
      }
      ++layer;
    } else {
      if (ahead == 0 && n_layers > 1) { ahead = 1; return 0; }
      if (ahead == 2) ++layer;
      ahead = 2;
    }
    part = layer < n_layers ? PART_GATE : PART_HEAD;
    return skipped;
  }
};

// The shares of a CTA: first row, rows (gate|up: of each), stages.
struct Rows { int row0[N_PARTS], rows[N_PARTS], stages[N_PARTS]; };
__host__ __device__ inline Rows rows_of(const Params& p, int b) {
  const int n[N_PARTS] = {p.sh.hidden, p.sh.inter, p.sh.qkv, p.sh.hidden, p.sh.vocab};
  Rows r;
  for (int i = 0; i < N_PARTS; ++i) {
    r.row0[i] = share(n[i], b, p.ctas);
    r.rows[i] = share(n[i], b + 1, p.ctas) - r.row0[i];
    r.stages[i] = stages_of(p.part[i], r.rows[i]);
  }
  return r;
}

// Shared memory by 32-bit addresses: generic pointers would take two registers each and a slower load.
__device__ __forceinline__ uint32_t ld32(uint32_t a) { uint32_t v; asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a)); return v; }
__device__ __forceinline__ uint4 ld128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ uint2 ld64(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ uint16_t ld16(uint32_t a) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a));
  return v;
}
// The sum of 4 or 8 floats.
template <int N> __device__ __forceinline__ float sum_words(uint32_t a) {
  const uint4 u = ld128(a);
  float t = (__uint_as_float(u.x) + __uint_as_float(u.y)) + (__uint_as_float(u.z) + __uint_as_float(u.w));
  if (N == 8) {
    const uint4 v = ld128(a + 16);
    t += (__uint_as_float(v.x) + __uint_as_float(v.y)) + (__uint_as_float(v.z) + __uint_as_float(v.w));
  }
  return t;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}
__device__ __forceinline__ void st128(uint32_t a, const uint4& v) { asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory"); }
__device__ __forceinline__ void st32(uint32_t a, float x) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(x) : "memory"); }
// Eight consecutive values of x, from index i (a multiple of 8), in the order that the operand registers want: (0,4) (1,5) (2,6) (3,7).
__device__ __forceinline__ void stage_x(uint32_t x, int i, const __half2 (&v)[4]) {
  uint32_t u[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) u[e] = *reinterpret_cast<const uint32_t*>(&v[e]);
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(x + i * 2), "r"(__byte_perm(u[0], u[2], 0x5410)), "r"(__byte_perm(u[0], u[2], 0x7632)),
               "r"(__byte_perm(u[1], u[3], 0x5410)), "r"(__byte_perm(u[1], u[3], 0x7632)) : "memory");
}

__device__ __forceinline__ bool try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
// Whether a wait that began with the first call has to end: another warp of the CTA has given up, or the limit has passed.
// (Inline, as all of this kernel: around a call registers go to the stack, and with all of L1 given to shared memory that is a trip to L2.)
__device__ __forceinline__ bool over(unsigned long long& t0, uint32_t flag_abort) {
  const unsigned long long now = global_timer_ns();
  if (t0 == 0) t0 = now;
  return ld32(flag_abort) != 0u || now - t0 > wait_limit_ns();
}
// Bounded wait for a phase of a stage's barrier; gives up when another warp of the CTA has, too.  A parity tells only neighbouring phases apart:
// who waits has to know that the phase before has completed.
__device__ __forceinline__ bool wait_stage(uint32_t bar, uint32_t parity, uint32_t flag_abort) {
  unsigned long long t0 = 0;
#pragma unroll 1
  while (!try_wait(bar, parity))
    if (over(t0, flag_abort)) return false;
  return true;
}

// Bounded wait until more than q stages of the stream have been issued.  A set does not see the other's stages, so this is how it knows which use of a place
// of the ring it waits for: stage q is issued once stage q - n_stages has been consumed, thus has landed.
// `issued` is what the warp knows already; the producer is mostly far ahead.
__device__ __forceinline__ void count_issued(uint32_t a, int n) { asm volatile("st.release.cta.shared.u32 [%0], %1;" ::"r"(a), "r"(n) : "memory"); }
__device__ __forceinline__ bool wait_issued(uint32_t a, int q, int& issued, uint32_t flag_abort) {
  unsigned long long t0 = 0;
#pragma unroll 1
  while (issued <= q) {
    asm volatile("ld.acquire.cta.shared.u32 %0, [%1];" : "=r"(issued) : "r"(a) : "memory");
    if (issued <= q && over(t0, flag_abort)) return false;
  }
  return true;
}

__device__ __forceinline__ void bar_arrive(int id, int threads) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// What a consumer needs to know of a part, in shared memory: one copy for the CTA, addresses inside a stage and of x per row of the MMA.
struct PartInfo { int groups, second, pad[2]; uint4 row[8]; uint32_t x[8]; };
static_assert(sizeof(PartInfo) == PART_INFO_BYTES, "PartInfo layout");
__device__ __forceinline__ void describe(const Part& q, PartInfo& info, int lane, bool turn) {
  if (lane < 8) {
    const int g = lane, ra = min2(g, q.h1 - 1), rb = q.h1 + min2(g, max2(q.slots - q.h1, 1) - 1), sc = q.slots * q.groups * 16;
    info.row[g] = make_uint4(ra * q.groups * 16, rb * q.groups * 16, sc + ra * q.groups * 2, sc + rb * q.groups * 2);
    info.x[g] = (g & (q.v - 1)) * q.groups * 64 + (turn && q.groups % 8 == 0 ? g : 0);      // (an offset of whole 64 bytes; below, how far its groups are turned)
  }
  if (lane == 0) { info.groups = q.groups; info.second = q.slots > q.h1; }
}

// The matvec of a part: the next n stages of the stream times x; a set of warps takes every step-th stage from `first`.  Its warps
// take the groups of a stage in turn.  Rows lie one behind the other; with eight warps, where they are a multiple of 8 groups (128 bytes) long, each row g takes
// another group of the eight, g further on, so that the eight rows that a quarter of the A operand takes sit in different banks.  Column g of the B
// operand is x at the group that row g takes (and row g + 8), so the sums of both are in column g of the result.
// What does not need x -- waiting for the stage, fetching up to U groups of weights -- is done before x is there (fetch).
template <int SET, int U>
struct Matvec {
  int q, end, step;                            // the set's next stage, counted over the whole stream; the end of its stages, their distance
  int i;                                       // its place in the ring
  uint32_t phase;
  int unit, units;                             // of the stage: this warp's next group, and how many it has
  bool second;
  uint4 at;                                    // addresses in a stage of the first group of both rows: weights, scales
  uint32_t xt;                                 // offset of its x
  // what has been fetched
  uint32_t a[U], b[U];                         // words of both rows, their scales
  uint32_t c[U];

  __device__ __forceinline__ void begin(const Params& p, uint32_t info, int n, int first, int step_, int pos, int turn) {
    const int w = (threadIdx.x >> 5) & (SET - 1), lane = threadIdx.x & 31;
    const int g = lane >> 2, t4 = lane & 3;
    const uint2 head = ld64(info);
    const uint32_t x = ld32(info + 16 + 128 + g * 4);
    at = ld128(info + 16 + g * 16);
    units = (static_cast<int>(head.x) - w + SET - 1) / SET;
    second = head.y != 0;
    const uint32_t r = SET == 8 ? (w + x) & 7 : w;         // (w where the rows do not turn)
    at.x += r * 16 + t4 * 4; at.y += r * 16 + t4 * 4; at.z += r * 2; at.w += r * 2;
    xt = (x & ~7u) + t4 * 16 + r * 64;
    q = pos + first; end = pos + n; step = step_; i = turn + first; phase = 0; unit = 0;
#pragma unroll 1
    while (i >= p.n_stages) { i -= p.n_stages; phase ^= 1u; }
  }
  // the next groups of stage q
  __device__ __forceinline__ void fetch(const Params& p, uint32_t base, int& issued, bool& dead, uint32_t flag_abort) {
    if (unit == 0 && !dead) {
      if (!wait_issued(base + p.map.flags + 8, q, issued, flag_abort) || !wait_stage(base + p.map.bars + i * 8, phase, flag_abort)) {
        dead = true;                           // (of this lane; the warp agrees on it where it polls next)
        st32(flag_abort, 1.0f);
        atomicExch(&g_device_status, 51);
      }
    }
    __syncwarp();                              // (no vote, here it costs more than what it guards: 30 layers of 576 / 1536 195 -> 185 us, 8 of 4096 / 11008 459 -> 467)
    const uint32_t st = base + i * p.stage_bytes;
    const uint32_t a0 = st + at.x + unit * (SET * 16), b0 = st + at.y + unit * (SET * 16), s0 = st + at.z + unit * (SET * 2), t0 = st + at.w + unit * (SET * 2);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      c[u] = 0u; b[u] = 0x88888888u; a[u] = 0x88888888u;           // nothing: zeros
      if (unit + u < units) {
        a[u] = ld32(a0 + u * (SET * 16));
        c[u] = ld16(s0 + u * (SET * 2));
        if (second) {
          b[u] = ld32(b0 + u * (SET * 16));
          c[u] |= static_cast<uint32_t>(ld16(t0 + u * (SET * 2))) << 16;
        }
      }
    }
  }
  // all of it, the first groups fetched before; the sums of stage q go to sums + q * STAGE_SUMS: [row][warp]
  __device__ __forceinline__ void run(const Params& p, uint32_t base, uint32_t x, uint32_t sums, int& issued, bool& dead, uint32_t flag_abort) {
    const int w = (threadIdx.x >> 5) & (SET - 1), lane = threadIdx.x & 31, g = lane >> 2;
    const bool odd = g & 1;
    float sum0 = 0.0f, sum1 = 0.0f;
#pragma unroll 1
    while (q < end) {
      const uint32_t x0 = x + xt + unit * (SET * 64);
      float d[U][4];
      uint4 xv[U];
#pragma unroll
      for (int u = 0; u < U; ++u) xv[u] = ld128(x0 + (unit + u < units ? u * (SET * 64) : 0));
#pragma unroll
      for (int u = 0; u < U; ++u) {
        uint32_t va[4], vb[4];
        unpack(a[u], va);
        unpack(b[u], vb);
        const float zero[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        mma_m16n8k16_f16(d[u], va[0], vb[0], va[1], vb[1], xv[u].x, xv[u].y, zero);
        mma_m16n8k16_f16(d[u], va[2], vb[2], va[3], vb[3], xv[u].z, xv[u].w, d[u]);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (unit + u < units) {                // (a group that does not exist is zeros times some x, which may be infinite)
          const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&c[u]));
          sum0 = fmaf(f.x, odd ? d[u][1] : d[u][0], sum0);
          sum1 = fmaf(f.y, odd ? d[u][3] : d[u][2], sum1);
        }
      }
      unit += U;
      if (unit >= units) {                     // the stage is done
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(base + p.map.bars + (MAX_STAGES + i) * 8) : "memory");
        if ((lane & 3) == (g >> 1)) {
          const uint32_t to = sums + static_cast<uint32_t>(q) * STAGE_SUMS + g * ROW_SUMS + w * 4;
          st32(to, sum0);
          st32(to + 8 * ROW_SUMS, sum1);
        }
        sum0 = 0.0f; sum1 = 0.0f;
        unit = 0; q += step; i += step;
#pragma unroll 1
        while (i >= p.n_stages) { i -= p.n_stages; phase ^= 1u; }
      }
      if (q < end) fetch(p, base, issued, dead, flag_abort);
    }
  }
};

// Polls eight published words until all carry `tag`.
struct Poll {
  const uint32_t* src;
  uint4 w[2];
  __device__ __forceinline__ void start(const uint32_t* p) { src = p; w[0] = load_words(p); w[1] = load_words(p + 4); }
  static __device__ __forceinline__ uint32_t differs(const uint4& w, uint32_t tag) { return (((w.x ^ tag) | (w.y ^ tag)) | ((w.z ^ tag) | (w.w ^ tag))) & 0xFFFFu; }
  __device__ __forceinline__ void finish(uint32_t tag, bool& dead, uint32_t flag_abort, __half2 (&v)[4]) {
    unsigned long long t0 = 0;
#pragma unroll 1
    for (uint32_t tries = 0; (differs(w[0], tag) | differs(w[1], tag)) != 0 && !dead; ++tries) {
      if ((tries & 255u) == 255u && over(t0, flag_abort)) { dead = true; st32(flag_abort, 1.0f); atomicExch(&g_device_status, 52); }
      w[0] = load_words(src);
      w[1] = load_words(src + 4);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t lo = __byte_perm(w[h].x, w[h].y, 0x7632), hi = __byte_perm(w[h].z, w[h].w, 0x7632);
      v[2 * h] = *reinterpret_cast<const __half2*>(&lo);
      v[2 * h + 1] = *reinterpret_cast<const __half2*>(&hi);
    }
  }
};

template <int SET, int U>
__global__ void __launch_bounds__(Threads<SET>::ALL, 1) decode_step_kernel(const __grid_constant__ Params p) {
  constexpr int NCW = Threads<SET>::NCW, NCT = Threads<SET>::NCT, SET_T = Threads<SET>::SET_T;
  extern __shared__ __align__(128) uint8_t smem[];
  const Shape& sh = p.sh;
  const Smem& L = p.map;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + L.bars);
  uint64_t* empty = full + MAX_STAGES;
  const uint32_t flag_abort = smem_u32(smem) + L.flags;     // set when a wait ran out
  uint32_t* smem_epoch = reinterpret_cast<uint32_t*>(smem + L.flags + 4);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31, tid = threadIdx.x, b = blockIdx.x;
  uint32_t* epoch = static_cast<uint32_t*>(p.d.state);
  unsigned int* finished = static_cast<unsigned int*>(p.d.state) + 1;
  unsigned long long* best_key = static_cast<unsigned long long*>(p.d.state) + 1;

  if (tid == 0) {
#pragma unroll 1
    for (int i = 0; i < p.n_stages; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], SET); }
    st32(flag_abort, 0.0f);
    count_issued(flag_abort + 8, 0);
    *smem_epoch = *reinterpret_cast<volatile uint32_t*>(epoch);
    *reinterpret_cast<Rows*>(smem + L.rows) = rows_of(p, b);
    fence_barrier_init();
  }
#pragma unroll 1
  for (int i = tid; i < p.n_layers * static_cast<int>(sizeof(lcq_decode_layer) / 8); i += Threads<SET>::ALL)
    reinterpret_cast<uint64_t*>(smem + L.table)[i] = static_cast<const uint64_t*>(p.d.layers)[i];
  if (warp < N_PARTS) describe(p.part[warp], reinterpret_cast<PartInfo*>(smem + L.info)[warp], lane, SET == 8);
  __syncthreads();
  const Rows& mine = *reinterpret_cast<const Rows*>(smem + L.rows);

  if (warp >= NCW) {
    // ------------------------------------------------------------ producer: one thread, the whole stream in order.  (A copy takes it 60 clocks
    // to issue, also where several lanes issue one each: with a copy per row that alone was 2000 a stage.)
    if (lane == 0) {
    int s = 0, issued = 0, in_flight = 0;      // the next stage; stages before it, and how many of them may be on their way
    uint32_t phase = 0;
    bool ok = true;
#pragma unroll 1
    for (Order o = {0, PART_O, false}; ok && o.part != N_PARTS; o.next(p.n_layers)) {
      const lcq_decode_layer* l = reinterpret_cast<const lcq_decode_layer*>(smem + L.table) + (o.part == PART_HEAD ? 0 : o.layer);
      const Part& q = p.part[o.part];
      const bool paired = o.part == PART_GATE;
      const uint8_t* w = static_cast<const uint8_t*>(o.part == PART_O ? l->o_w : paired ? l->gate_up_w : o.part == PART_QKV ? l->qkv_w : o.part == PART_DOWN ? l->down_w : p.d.head_w);
      const uint8_t* sc = static_cast<const uint8_t*>(o.part == PART_O ? l->o_s : paired ? l->gate_up_s : o.part == PART_QKV ? l->qkv_s : o.part == PART_DOWN ? l->down_s : p.d.head_s);
      const int n = mine.rows[o.part], row0 = mine.row0[o.part];
      const int row_w = q.K / 2, row_s = q.K / 16;
#pragma unroll 1
      for (int r = 0; r < n; r += q.per) {
        const int rows = min2(n - r, q.per);
        if (!wait_stage(smem_u32(&empty[s]), phase ^ 1u, flag_abort) || ld32(flag_abort) != 0u) {
          st32(flag_abort, 1.0f);                     // (the flag after the wait: consumers that gave up release stages whose copies have not landed)
          atomicExch(&g_device_status, 50);
          ok = false;
          break;
        }
        mbar_expect_tx(&full[s], static_cast<uint32_t>(rows * (row_w + row_s)) << (paired ? 1 : 0));
        count_issued(flag_abort + 8, ++issued);
        const uint32_t dst = smem_u32(smem) + s * p.stage_bytes, dst_s = dst + q.slots * q.groups * 16;
        bulk_load(dst, w + static_cast<long long>(row0 + r) * row_w, rows * row_w, &full[s]);
        bulk_load(dst_s, sc + static_cast<long long>(row0 + r) * row_s, rows * row_s, &full[s]);
        if (paired) {
          bulk_load(dst + q.h1 * q.groups * 16, w + static_cast<long long>(sh.inter + row0 + r) * row_w, rows * row_w, &full[s]);
          bulk_load(dst_s + q.h1 * q.groups * 2, sc + static_cast<long long>(sh.inter + row0 + r) * row_s, rows * row_s, &full[s]);
        }
        if (++s == p.n_stages) { s = 0; phase ^= 1u; }
        if (in_flight < p.n_stages) ++in_flight;
      }
    }
    // Consumers that gave up wait for no more stages, so the copies into the last ones are waited for here: none may
    // land after the CTA has left.  They read this GPU's memory and end by themselves, whatever the wait limit.
#pragma unroll 1
    for (; in_flight > 0; --in_flight) {
      if (--s < 0) { s = p.n_stages - 1; phase ^= 1u; }
      mbar_wait_landed(&full[s], phase);
    }
    }
  } else {
    // ------------------------------------------------------------ consumers
    // Both sets of warps multiply.  The first also puts together the activation (publishes it, waits for that of the others) and
    // publishes the down projection; the second does the norms, and q|k|v and o while the activation travels.
    const uint32_t base = smem_u32(smem);
    const int set = warp / SET, w = warp & (SET - 1), st = tid & (SET_T - 1);      // warp and thread of the set
    const uint32_t xn = base + L.xn, xq = base + L.xq, xm = base + L.xm;
    const uint32_t sums_c = base + L.sums, sums_s = base + L.side;
    const uint32_t tag0 = *smem_epoch * static_cast<uint32_t>(2 * p.n_layers + 1) + 1u;
    const int words = 3 * sh.hidden + sh.inter, copy = (b % COPIES) * words;       // the copy that is read here; warp w writes copy w
    int pos = 0, turn = 0;                     // stages of the stream that are behind, and these modulo two rounds of the ring
    int issued = 0;                            // stages that are known to have been issued
    bool dead = false;
    const auto pass = [&](int n) {
      pos += n;
      turn += n;
#pragma unroll 1
      while (turn >= 2 * p.n_stages) turn -= 2 * p.n_stages;
    };
    // the sum of row i of a slab (half: of its first or second half) whose sums begin at `sums`: v short rows of a partial sum per warp
    const auto row_sum = [&](uint32_t sums, int i, int v) {
      float t = 0.0f;
#pragma unroll 1
      for (uint32_t a = sums + i * v * ROW_SUMS; v > 0; --v, a += ROW_SUMS) {
        t += sum_words<SET>(a);
      }
      return t;
    };
    // row i of a piece of a part that is not gate|up
    const auto sum_of = [&](uint32_t sums, int i, const Part& q) { return row_sum(sums + (i << q.lg_v >> q.lg) * STAGE_SUMS, i & ((1 << (q.lg - q.lg_v)) - 1), q.v); };
    // A thread's share of the hidden state and of the next norms' weights, 8 values of every 8 * SET_T, lies in shared memory.
    const uint32_t hid = base + L.hid;
    const auto fetch_norms = [&](int of) {           // a layer ahead: they may come from HBM.  A thread fetches what it will use.
#pragma unroll 1
      for (int j = 0; j < 2 && 2 * of + j <= 2 * p.n_layers; ++j)
#pragma unroll 1
        for (int i = 8 * st; i < sh.hidden; i += 8 * SET_T)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(base + L.gam + 2 * (j * sh.hidden + i)), "l"(static_cast<const __half*>(p.d.norms) + static_cast<long long>(2 * of + j) * sh.hidden + i) : "memory");
    };
    const auto squares = [&](const __half2 (&h)[4], float ss) {
      float t[2] = {0.0f, 0.0f};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f = __half22float2(h[e]);
        t[e & 1] = fmaf(f.x, f.x, t[e & 1]);
        t[e & 1] = fmaf(f.y, f.y, t[e & 1]);
      }
      return ss + (t[0] + t[1]);
    };
    // hidden += the down projection; x = rms_norm(hidden); hidden += the o projection; x2 = rms_norm(hidden)
    // (the first layer has no down projection before it, the lm_head no o)
    const auto norms = [&](const uint32_t* down, const uint32_t* o, uint32_t tag) {
      float ss = 0.0f, ss2 = 0.0f;
#pragma unroll 1
      for (int i = 8 * st; i < sh.hidden; i += 8 * SET_T) {
        Poll pd, po;
        if (o != nullptr) po.start(o + i);
        if (down != nullptr) pd.start(down + i);
        __half2 h[4], v[4];
        *reinterpret_cast<uint4*>(h) = ld128(hid + 2 * i);
        if (down != nullptr) {
          pd.finish(tag, dead, flag_abort, v);
#pragma unroll
          for (int e = 0; e < 4; ++e) h[e] = __hadd2_rn(h[e], v[e]);       // (rounds as the float32 sum rounded to fp16 does)
        }
        st128(hid + 2 * i, *reinterpret_cast<const uint4*>(h));
        ss = squares(h, ss);
        if (o != nullptr) {
          po.finish(tag, dead, flag_abort, v);
#pragma unroll
          for (int e = 0; e < 4; ++e) h[e] = __hadd2_rn(h[e], v[e]);
          st128(hid + 2 * (sh.hidden + i), *reinterpret_cast<const uint4*>(h));
          ss2 = squares(h, ss2);
        }
      }
      dead = __any_sync(0xffffffffu, dead);
      ss = warp_sum(ss);
      ss2 = warp_sum(ss2);
      const uint32_t red = base + L.red;
      if (lane == 0) { st32(red + w * 4, ss); st32(red + SET * 4 + w * 4, ss2); }
      asm volatile("cp.async.wait_all;" ::: "memory");
      named_bar_sync(BAR_SET1, SET_T);
      if (8 * (st & ~31) < sh.hidden) {
        float total[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          total[j] = rsqrtf(fmaf(sum_words<SET>(red + j * SET * 4), p.inv_hidden, p.d.eps));
        }
#pragma unroll 1
        for (int i = 8 * st; i < sh.hidden; i += 8 * SET_T) {
#pragma unroll
          for (int j = 1; j >= 0; --j) {       // (gate|up wait for the second one)
            __half2 h[4], n[4], y[4];
            *reinterpret_cast<uint4*>(n) = ld128(base + L.gam + 2 * (j * sh.hidden + i));
            *reinterpret_cast<uint4*>(h) = ld128(hid + 2 * (j * sh.hidden + i));
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float2 hf = __half22float2(h[e]), nf = __half22float2(n[e]);
              y[e] = __floats2half2_rn(hf.x * total[j] * nf.x, hf.y * total[j] * nf.y);
            }
            stage_x(xn + j * sh.hidden * 2, i, y);
          }
          if (o != nullptr) st128(hid + 2 * i, ld128(hid + 2 * (sh.hidden + i)));
        }
      }
    };

    // embedding; the prepared input of the o projections
    if (set == 1) {
      fetch_norms(0);
      const int id = *static_cast<const int*>(p.d.token);
      const bool known = id >= 0 && id < sh.vocab;
      if (!known && b == 0 && st == 0) atomicExch(&g_device_status, 40);
      const __half* row = static_cast<const __half*>(p.d.table) + static_cast<long long>(known ? id : 0) * sh.hidden;
#pragma unroll 1
      for (int i = 8 * st; i < sh.hidden; i += 8 * SET_T)
        st128(hid + 2 * i, known ? *reinterpret_cast<const uint4*>(row + i) : make_uint4(0u, 0u, 0u, 0u));
    } else {
#pragma unroll 1
      for (int i = 8 * st; i < sh.q_dim; i += 8 * SET_T) {
        __half2 v[4];
        *reinterpret_cast<uint4*>(v) = *reinterpret_cast<const uint4*>(static_cast<const __half*>(p.d.x_q) + i);
        stage_x(xq, i, v);
      }
    }
    named_bar_sync(BAR_ALL, NCT);

    // Three matvecs a layer for each set: gate|up together, then the first one takes its half of down, and o of the layer after next; the
    // second one q|k|v and its half of down.  (Before the first layer: o of the first two layers.  At the end: the lm_head, in pieces.)
    // One loop body for all of them: it is small enough to stay in the instruction cache next to the schedulers.
    // tags: o of layer l 2 l, its activation 2 l + 1, its down projection 2 l + 2 (o has buffers of its own, the layers' in turn)
    const int layer_out = sh.qkv + 2 * sh.hidden + 2 * sh.inter;
    Walk to(set);
    unsigned long long* keys = reinterpret_cast<unsigned long long*>(smem + L.red);     // the best logit of each warp
    pass(Walk::skipped_at_first(set, p.n_layers, mine.stages));
#pragma unroll 1
    while (to.part != N_PARTS) {
      const int part = to.part, layer = to.layer;
      const uint32_t tag = tag0 + 2u * layer;
      __half* out = static_cast<__half*>(p.d.outputs) + static_cast<long long>(layer) * layer_out;     // the layer's q|k|v, o, gate|up, down
      const int n = to.count(mine.stages, p.part);
      const uint32_t sums = part == PART_QKV ? sums_s : part == PART_O ? sums_s + min2(mine.stages[PART_QKV], p.part[PART_QKV].piece) * STAGE_SUMS : sums_c;
      const int v = p.part[part].v, r0 = to.done * p.part[part].per, rows = min2(mine.rows[part] - r0, n * p.part[part].per);       // rows of this piece
      Matvec<SET, U> m;
      m.begin(p, base + L.info + part * PART_INFO_BYTES, n, to.first(), to.step(), pos, turn);
      if (m.q < m.end) m.fetch(p, base, issued, dead, flag_abort);
      const uint32_t sums_q = sums - static_cast<uint32_t>(pos) * STAGE_SUMS;
      pass(n);
      if (set == 0) {
        if (part == PART_DOWN && to.done == 0) {          // the activation
#pragma unroll 1
          for (int i = 8 * st; i < sh.inter; i += 2 * 8 * SET_T) {
            const int i2 = i + 8 * SET_T;      // two at a time
            Poll q, q2;
            __half2 y[4];
            q.start(p.m_buf + copy + i);
            if (i2 < sh.inter) q2.start(p.m_buf + copy + i2);
            q.finish((tag + 1u) & 0xFFFFu, dead, flag_abort, y);
            stage_x(xm, i, y);
            if (i2 < sh.inter) {
              q2.finish((tag + 1u) & 0xFFFFu, dead, flag_abort, y);
              stage_x(xm, i2, y);
            }
          }
          dead = __any_sync(0xffffffffu, dead);
        }
      } else if (to.done == 0 && (part == PART_GATE || part == PART_HEAD)) {
        norms(layer == 0 ? nullptr : p.d_buf + copy, part == PART_HEAD ? nullptr : p.o_buf + (layer & 1) * sh.hidden + copy, tag & 0xFFFFu);
      }
      if (to.joint()) named_bar_sync(BAR_ALL, NCT);
      else if (set == 0) named_bar_sync(BAR_SET0, SET_T);          // (the sums of the piece before have been read)
      else if (to.done != 0) named_bar_sync(BAR_SET1, SET_T);
      m.run(p, base, part == PART_DOWN ? xm : part == PART_O ? xq : part == PART_GATE ? xn + 2 * sh.hidden : xn, sums_q, issued, dead, flag_abort);

      if (part == PART_GATE || part == PART_DOWN) {
        if (set == 1) {
          bar_arrive(BAR_SUMS, NCT);
          pass(to.next(p.n_layers, mine.stages, p.part));
          continue;
        }
        named_bar_sync(BAR_SUMS, NCT);
      }
      if (part == PART_GATE) {
        const int lg_v = p.part[PART_GATE].lg_v, lg = p.part[PART_GATE].lg, mine0 = mine.row0[PART_GATE] + r0;
#pragma unroll 1
        for (int i = lane; i < rows; i += 32) {
          const uint32_t slab = sums + (i << lg_v >> lg) * STAGE_SUMS;
          const int r = i & ((1 << (lg - lg_v)) - 1);
          const __half gate = __float2half_rn(row_sum(slab, r, v)), up = __float2half_rn(row_sum(slab + 8 * ROW_SUMS, r, v));
          const float x = __half2float(gate);
          const __half y = __float2half_rn((x * (1.0f / (1.0f + expf(-x)))) * __half2float(up));
#pragma unroll
          for (int c = 0; c < COPIES / SET; ++c) publish(p.m_buf + (w + c * SET) * words + mine0 + i, y, (tag + 1u) & 0xFFFFu);
          if (w == 0) {                        // what the caller sees
            __half* o = out + sh.qkv + sh.hidden + mine0 + i;
            o[0] = gate;
            o[sh.inter] = up;
            if (layer + 1 == p.n_layers) static_cast<__half*>(p.d.mlp_out)[mine0 + i] = y;
          }
        }
      } else if (part == PART_DOWN || part == PART_O) {
        const bool down = part == PART_DOWN;
        if (!down) named_bar_sync(BAR_SET0, SET_T);
        uint32_t* words_out = (down ? p.d_buf : p.o_buf + ((layer + to.ahead) & 1) * sh.hidden) + w * words + mine.row0[part] + r0;
        __half* o = out + (down ? layer_out - sh.hidden : to.ahead * layer_out + sh.qkv) + mine.row0[part] + r0;
        const uint32_t t = (tag + (down ? 2u : 2u * to.ahead)) & 0xFFFFu;
#pragma unroll 1
        for (int i = lane; i < rows; i += 32) {
          const __half y = __float2half_rn(sum_of(sums, i, p.part[part]));
#pragma unroll
          for (int c = 0; c < COPIES / SET; ++c) publish(words_out + c * SET * words + i, y, t);
          if (w == 0) o[i] = y;
        }
      } else if (part == PART_QKV) {
        if (to.done == 0) fetch_norms(layer + 1);
        named_bar_sync(BAR_SET1, SET_T);
#pragma unroll 1
        for (int i = st; i < rows; i += SET_T) out[mine.row0[PART_QKV] + r0 + i] = __float2half_rn(sum_of(sums, i, p.part[part]));
      } else {
        // the key of a logit orders as np.argmax does: by value, NaN above all, the lowest index among equals
        named_bar_sync(BAR_ALL, NCT);
        const int v0 = mine.row0[PART_HEAD] + r0;
        unsigned long long key = 0;
#pragma unroll 1
        for (int i = tid; i < rows; i += NCT) {
          const __half y = __float2half_rn(sum_of(sums, i, p.part[part]));
          static_cast<__half*>(p.d.logits)[v0 + i] = y;
          const float f = __half2float(y) + 0.0f;        // -0 counts as 0
          uint32_t u = __float_as_uint(f);
          u = f != f ? 0xFFFFFFFFu : (u & 0x80000000u) ? ~u : (u | 0x80000000u);
          const unsigned long long k = (static_cast<unsigned long long>(u) << 32) | (0xFFFFFFFFu - static_cast<uint32_t>(v0 + i));
          if (k > key) key = k;
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
          const unsigned long long k = __shfl_xor_sync(0xffffffffu, key, off);
          if (k > key) key = k;
        }
        if (lane == 0 && (to.done == 0 || key > keys[warp])) keys[warp] = key;
      }
      pass(to.next(p.n_layers, mine.stages, p.part));
    }
    if (b == 0) {
#pragma unroll 1
      for (int i = tid; i < sh.hidden; i += NCT) {
        static_cast<__half*>(p.d.hidden_out)[i] = *reinterpret_cast<const __half*>(smem + L.hid + 2 * i);
        static_cast<__half*>(p.d.normed_out)[i] = *reinterpret_cast<const __half*>(smem + L.xn + (i >> 3) * 16 + 4 * (i & 3) + ((i >> 2) & 1) * 2);
      }
    }
    named_bar_sync(BAR_ALL, NCT);
    if (tid == 0) {
      unsigned long long key = keys[0];
#pragma unroll 1
      for (int i = 1; i < NCW; ++i) if (keys[i] > key) key = keys[i];
      atomicMax(best_key, key);
      __threadfence();
      if (atomicAdd(finished, 1u) == static_cast<unsigned int>(p.ctas) - 1u) {     // everybody's key is in
        __threadfence();
        const unsigned long long k = atomicExch(best_key, 0ull);
        *static_cast<int*>(p.d.next_token) = static_cast<int>(0xFFFFFFFFu - static_cast<uint32_t>(k));
        *finished = 0;
        *epoch = *smem_epoch + 1u;             // (every CTA has read it: all have published)
      }
    }
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------- host side
struct Plan { Params p; size_t smem, state_bytes; };
constexpr int CUT_ROW = 3584, LONG_ROW = 4096, MAX_STAGE = 40 * 1024;      // columns; bytes

// A weight of rows of K columns, of which a CTA has at most `rows`: cut into short rows where they would be longer than `whole_row` (then to CUT_ROW at
// most), or so few that they left rows of the MMA empty; fewer rows a slab where a stage would still be longer than max_bytes.  (Copies of scales are
// whole 16 bytes: 256 columns.)
// A stage costs a warp its rounds of U groups and about one more, so long rows are cheaper as long as the ring keeps three stages.  us a step with
// rows cut to 2560 at most / to 3584: 8 layers of 3072 / 8192 with 128,256 rows 291 / 272, 4 of 3200 / 8640 194 / 181, 6 of 3584 / 18944 603 / 423,
// 4 of 3072 / 24576 359 / 244; to 1536: 8 of 2048 / 8192 250 instead of 185.
inline Part make_part(int K, int rows, bool paired, int whole_row, int max_bytes) {
  Part q;
  q.K = K;
  q.lg_v = 0;
  q.lg = paired ? 3 : 4;
  const auto whole = [&](int lg, int lg_v) { return lg >= lg_v && K % (32 << lg_v) == 0 && (K << (lg - lg_v)) % 256 == 0; };
  const auto bytes = [&]() { return (paired ? 2 : 1) * (min2(1 << q.lg, rows << q.lg_v) * (K >> q.lg_v) / 32) * 18; };
  while (whole(q.lg, q.lg_v + 1) && ((K > whole_row && K >> q.lg_v > CUT_ROW) || rows << (q.lg_v + 1) <= 1 << q.lg)) ++q.lg_v;
  while (bytes() > max_bytes && whole(q.lg - 1, q.lg_v)) --q.lg;
  q.v = 1 << q.lg_v;
  q.groups = K / q.v / 32;
  const int n = min2(1 << q.lg, rows * q.v);
  q.h1 = min2(8, n);
  q.slots = paired ? 2 * n : n;
  q.per = n / q.v;
  q.piece = 1 << 30;
  return q;
}

// Four warps a set, which leave each more registers and fewer of them in each other's way, or eight, which hide each other's latencies when a
// stage is long.  us a step with four / eight: 30 layers of 576 / 1536 185 / 209, 12 of 256 / 768 85 / 96; 12 of 768 / 2048 105 / 95,
// 8 of 1024 / 3072 with 151,936 rows 129 / 118, 5 of 2048 / 8192 201 / 130.
inline bool narrow(const Params& p) { return p.sh.hidden <= 640; }

// Groups that a warp of eight takes at a time: two or three, whichever leaves fewer empty places in the stages of the stack.  A round costs
// as much as its groups and 0.85 of one more.  us a step with two / three: 8 layers of 2560 / 9728 (10 groups a warp and stage) 303 / 314, 5 of
// 5120 / 5120 (10) 210 / 218, 8 of 1024 / 3072 with 151,936 rows (4) 107 / 119; 5 of 4608 / 12288 (9) 308 / 274, 6 of 1536 / 8960 (6) 117 / 109.
inline int round_of(const Params& p) {
  if (narrow(p)) return 5;
  const int rows[N_PARTS] = {p.sh.hidden, p.sh.inter, p.sh.qkv, p.sh.hidden, p.sh.vocab};
  long long cost[2] = {0, 0};
  for (int i = 0; i < N_PARTS; ++i) {
    const Part& q = p.part[i];
    const int stages = stages_of(q, max_share(rows[i], p.ctas)), units = (q.groups + 7) / 8;
    const long long turns = static_cast<long long>(i == PART_O || i == PART_QKV ? stages : (stages + 1) / 2) * (i == PART_HEAD ? 1 : p.n_layers);      // (a set's)
    cost[0] += turns * ((units + 1) / 2) * (40 + 17);
    cost[1] += turns * ((units + 2) / 3) * (60 + 17);
  }
  return cost[0] < cost[1] ? 2 : 3;
}

inline bool make_plan(const lcq_decode_stack& d, int sm_count, Plan& pl) {
  const int H = d.hidden, I = d.inter;
  if (d.n_layers < 1 || H < 64 || I < 64 || d.qkv < 4 || d.q_dim < 64 || d.vocab < 4 || d.n_layers > 256) return false;
  if (H % 64 || I % 64 || d.q_dim % 64 || d.qkv % 4 || d.vocab % 4 || H > 8192 || I > (1 << 20) || d.q_dim > (1 << 20) || d.qkv > (1 << 24) || d.vocab > (1 << 24)) return false;
  Params& p = pl.p;
  memset(&p, 0, sizeof(p));
  p.d = d;
  p.sh = {H, I, d.qkv, d.q_dim, d.vocab};
  p.n_layers = d.n_layers;
  p.inv_hidden = 1.0f / static_cast<float>(H);
  // Four rows of the longest kind fit twice beside the vectors.  (Stages may be shorter; longer rows are the chain's.)
  const int longest = max2(max2(H, I), d.q_dim), vectors = (6 * H + d.q_dim + I) * 2;
  if (vectors + 2 * max2(24 * 1024, longest / 4 * 9) + d.n_layers * static_cast<int>(sizeof(lcq_decode_layer)) > 227 * 1024) return false;
  int units = H / 4;                           // every CTA needs a unit of 4 rows in every phase
  if (I / 4 < units) units = I / 4;
  if (d.vocab / 4 < units) units = d.vocab / 4;
  p.ctas = sm_count < units ? sm_count : units;
  const int hid = max_share(H, p.ctas), qkv = max_share(d.qkv, p.ctas);
  const auto cut = [&](int whole_row, int max_bytes) {
    p.part[PART_O] = make_part(d.q_dim, hid, false, whole_row, max_bytes);
    p.part[PART_GATE] = make_part(H, max_share(I, p.ctas), true, whole_row, max_bytes);
    p.part[PART_QKV] = make_part(H, qkv, false, whole_row, max_bytes);
    p.part[PART_DOWN] = make_part(I, hid, false, whole_row, max_bytes);
    p.part[PART_HEAD] = make_part(H, max_share(d.vocab, p.ctas), false, whole_row, max_bytes);
    p.part[PART_HEAD].piece = HEAD_SLABS;
    p.stage_bytes = 0;
    for (const Part& q : p.part) p.stage_bytes = max2(p.stage_bytes, (q.slots * q.groups * 18 + 127) & ~127);
  };
  // The longest stages and the largest pieces with which three stages fit, or two.
  for (int fit = 3, max_bytes = MAX_STAGE; p.n_stages < fit; max_bytes /= 2) {
    if (max_bytes < MAX_STAGE / 16) {
      if (--fit < 2) return false;
      max_bytes = MAX_STAGE;
    }
    cut(CUT_ROW, max_bytes);
    // (rows of up to 4096 whole where that makes the stages half as long again at most; cut / whole: 6 of 4096 / 14336 349 / 331, but 6 of 4096 / 4096 169 / 176)
    if (p.stage_bytes * 3 / 2 >= 16 * LONG_ROW / 32 * 18) cut(LONG_ROW, max_bytes);
    for (int piece = HEAD_SLABS; piece >= 2; piece /= 4) {
      if (piece < HEAD_SLABS) for (Part& q : p.part) q.piece = piece;
      p.n_stages = 0;
      p.n_stages = min2(MAX_STAGES, (227 * 1024 - smem_map(p).total) / p.stage_bytes);
      if (p.n_stages >= fit) break;
    }
  }
  p.map = smem_map(p);
  pl.smem = static_cast<size_t>(p.map.total);
  pl.state_bytes = STATE_BYTES + (static_cast<size_t>(3) * H + I) * 4 * COPIES;
  return true;
}

inline int launch(const lcq_decode_stack& d, int sm_count, cudaStream_t stream) {
  Plan pl;
  if (!make_plan(d, sm_count, pl)) { set_error("decode_step: this shape is not covered"); return LCQ_ERR_UNSUPPORTED; }
  if (d.state_bytes < pl.state_bytes) { set_error("decode_step: state of %zu bytes required, got %zu", pl.state_bytes, d.state_bytes); return LCQ_ERR_WORKSPACE; }
  const void* pointers[] = {d.layers, d.head_w, d.head_s, d.logits, d.norms, d.outputs, d.token, d.table, d.x_q, d.hidden_out, d.normed_out, d.mlp_out, d.next_token, d.state};
  for (const void* q : pointers)
    if (!q || !aligned(q, q == d.token || q == d.next_token ? 4 : 16)) { set_error("decode_step: null or misaligned pointer"); return LCQ_ERR_BAD_ARG; }
  Params& p = pl.p;
  p.o_buf = reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(d.state) + STATE_BYTES);
  p.d_buf = p.o_buf + 2 * d.hidden;
  p.m_buf = p.d_buf + d.hidden;
  static thread_local int configured_device = -1;
  int dev = 0;
  LCQ_CUDA_TRY(cudaGetDevice(&dev));
  if (configured_device != dev) {
    LCQ_CUDA_TRY(cudaFuncSetAttribute(decode_step_kernel<4, 5>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    LCQ_CUDA_TRY(cudaFuncSetAttribute(decode_step_kernel<8, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    LCQ_CUDA_TRY(cudaFuncSetAttribute(decode_step_kernel<8, 3>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    configured_device = dev;
  }
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(p.ctas);
  const int round = round_of(p);
  cfg.blockDim = dim3(round == 5 ? Threads<4>::ALL : Threads<8>::ALL);
  cfg.dynamicSmemBytes = pl.smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;           // all CTAs resident at once, or the launch fails
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  LCQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, round == 5 ? decode_step_kernel<4, 5> : round == 2 ? decode_step_kernel<8, 2> : decode_step_kernel<8, 3>, p));
  return LCQ_OK;
}

}  // namespace step
}  // namespace lcq
