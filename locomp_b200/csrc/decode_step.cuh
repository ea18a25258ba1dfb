// One decode step of a Llama-style stack of quantized linears (M = 1, int4 weights in groups of 32) as ONE
// kernel: embedding, per layer {RMS norm, q|k|v and o projections, residual add + RMS norm, gate|up, SiLU *
// up, down, residual add}, final norm, lm_head and greedy argmax -- the chain that locomp_b200.DecodeStack
// runs as 8 launches a layer otherwise (examples/54_smollm2_inference.py:494-578 without the attention
// itself; o reads a prepared buffer, so it depends on nothing in its layer and runs beside the down projection
// before it).  That makes two dependent phases a layer.  It is an order that only a step without attention has: a
// layer whose o reads the attention output has four (q|k|v, o, gate|up, down) and cannot take this schedule.
//
// What bounds it.  SmolLM2-135M has 30 layers of 2 MB: 12 us of HBM time for the whole token, but ~90
// dependent matvecs.  As separate kernels each costs ~2 us (launch, dependency wait, first loads, drain):
// 506 us a token, now 297; 5 layers of width 2048 167 us, now 135.  What is left is instruction latency: a phase
// is ~1000 dependent instructions of a warp (norm 1.2 us, tiles 1.3, publishing 0.9, waiting 1.3).  Here
//   * one CTA per SM stays for the whole step; a producer thread streams the CTA's rows of ALL layers
//     through one shared-memory ring (bulk copies), running ahead across layers, so that weights are there
//     when their input is;
//   * results that the next phase needs are published as words {fp16 value, 16-bit tag of the phase}: a
//     consumer polls the data itself until every tag is the one it expects.  No grid barrier, no fence, no
//     flag: one store and one load through L2 between dependent matvecs;
//   * every CTA keeps the hidden state and does the norms redundantly.
// Every CTA has at least one unit of 4 rows in every phase.  So whoever has all results of a phase knows
// that all CTAs have read what they needed for it, and a buffer that is rewritten two phases later (the
// next layer's) has no reader left.
//
// The CTAs wait for one another: the launch is cooperative, and every wait is bounded (on expiry the CTA
// records a status code and runs to its end without waiting).
//
// Arithmetic as in the separate kernels: products and sums in float32, each result rounded to fp16 where
// those kernels store it.
#pragma once
#include "common.cuh"

namespace lcq {
namespace step {

constexpr int NCW = 16;                        // consumer warps
constexpr int NCT = NCW * 32;
constexpr int NTHREADS = NCT + 32;             // + the producer warp
constexpr int MAX_STAGES = 32;
constexpr int BAR_C = 1;                       // named barrier of the consumers
constexpr int STATE_BYTES = 64;                // epoch, argmax counter, argmax key

struct Shape { int hidden, inter, qkv, q_dim, vocab; };

struct Params {
  lcq_decode_stack d;
  Shape sh;
  int n_layers, ctas;
  int stage_bytes, n_stages;
  int copies;           // of the published words: a CTA polls copy b % copies
  int copy_words;       // 2 * hidden + inter
  uint32_t* o_buf;      // published words, first copy: o projection, down projection [hidden], activation [inter]
  uint32_t* d_buf;
  uint32_t* m_buf;
};

// Rows of an [n, K] weight that CTA b streams: whole units of 4 (so that rows of scales start on 16 bytes).
__host__ __device__ inline int share(int n, int b, int ctas) { return static_cast<int>(static_cast<unsigned>(n / 4) * static_cast<unsigned>(b) / static_cast<unsigned>(ctas)) * 4; }
__host__ __device__ inline int row_bytes(int K) { return K / 2 + K / 16; }
__host__ __device__ inline int tile_rows(int stage_bytes, int K) { return (stage_bytes / row_bytes(K)) & ~3; }

struct Smem { int stages, xn, xq, xm, hid, gam, res, red, bars, flags, rows, table, total; };
__host__ __device__ inline int max2(int a, int b) { return a > b ? a : b; }
__host__ __device__ inline Smem smem_map(const Shape& s, int n_layers, int ctas, int stage_bytes, int n_stages) {
  Smem m;
  m.stages = 0;
  m.xn = n_stages * stage_bytes;
  m.xq = m.xn + 2 * s.hidden * 2;              // both norms of a layer
  m.xm = m.xq + s.q_dim * 2;
  m.hid = m.xm + s.inter * 2;
  m.gam = m.hid + 2 * s.hidden * 2;            // before and after o
  m.res = m.gam + 2 * s.hidden * 2;
  const int per = 4;                           // a share is at most one unit above the average
  const int rows = max2(max2((s.qkv + 2 * s.inter) / ctas + 6 * per, 2 * s.hidden / ctas + 4 * per), s.vocab / ctas + 2 * per);
  m.red = m.res + rows * 16;
  m.bars = m.red + 2 * NCW * 8;
  m.flags = m.bars + 2 * MAX_STAGES * 8;
  m.rows = m.flags + 16;                       // Rows
  m.table = m.rows + 32;                       // the layer records
  m.total = m.table + n_layers * static_cast<int>(sizeof(lcq_decode_layer));
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
// acc + a * b with float32 accumulation of the exact product; operands are halves of 32-bit registers
__device__ __forceinline__ float fma_lo(uint32_t a, uint32_t b, bool a_hi, bool b_hi, float acc) {
  const unsigned short x = static_cast<unsigned short>(a_hi ? a >> 16 : a), y = static_cast<unsigned short>(b_hi ? b >> 16 : b);
  asm("fma.rn.f32.f16 %0, %1, %2, %0;" : "+f"(acc) : "h"(x), "h"(y));
  return acc;
}
__device__ __forceinline__ uint32_t nibbles(uint32_t w, uint32_t mask, uint32_t magic, uint32_t offset) {   // two q - 8 as fp16, exact
  uint32_t r;
  asm("{\n\t.reg .b32 t;\n\tlop3.b32 t, %1, %2, %3, 0xEA;\n\tsub.f16x2 %0, t, %4;\n\t}" : "=r"(r) : "r"(w), "r"(mask), "r"(magic), "r"(offset));
  return r;
}
// sum of x[i] * (q[i] - 8) over the 8 nibbles of a word
__device__ __forceinline__ float dot8(uint32_t w, const uint4& x) {
  const uint32_t w8 = w >> 8;
  const uint32_t a = nibbles(w, 0x000F000Fu, 0x64006400u, 0x64086408u);     // q0, q4
  const uint32_t b = nibbles(w, 0x00F000F0u, 0x54005400u, 0x54805480u);     // q1, q5
  const uint32_t c = nibbles(w8, 0x000F000Fu, 0x64006400u, 0x64086408u);    // q2, q6
  const uint32_t d = nibbles(w8, 0x00F000F0u, 0x54005400u, 0x54805480u);    // q3, q7
  float p = 0.0f, q = 0.0f;
  p = fma_lo(a, x.x, false, false, p);
  q = fma_lo(a, x.z, true, false, q);
  p = fma_lo(b, x.x, false, true, p);
  q = fma_lo(b, x.z, true, true, q);
  p = fma_lo(c, x.y, false, false, p);
  q = fma_lo(c, x.w, true, false, q);
  p = fma_lo(d, x.y, false, true, p);
  q = fma_lo(d, x.w, true, true, q);
  return p + q;
}

// The phases of a step.  0: the first layer's o.  1 + 2 l: q|k|v, gate|up and the activation of layer l -- o
// depends on x_q alone, so it is there already and both norms of a layer follow from the down projection
// before it.  2 + 2 l: down of layer l, and o of the next layer.  1 + 2 n_layers: the lm_head.
enum { PART_QKV, PART_GATE, PART_UP, PART_DOWN, PART_O, PART_HEAD };
__device__ __forceinline__ int first_part(int ph, int n_layers) {
  return ph == 0 ? PART_O : ph > 2 * n_layers + 1 ? -1 : ph == 2 * n_layers + 1 ? PART_HEAD : (ph & 1) ? PART_QKV : PART_DOWN;
}
__device__ __forceinline__ int next_part(int part, int ph, int n_layers) {
  if (part == PART_QKV || part == PART_GATE) return part + 1;
  return part == PART_DOWN && ph < 2 * n_layers ? PART_O : -1;
}

// What a CTA streams for a part of a phase: rows of a weight and of its scales.
struct Rows { int qkv0, qkv, hid0, hid, int0, inter, voc0, voc; };   // this CTA's shares: first row, rows
struct Segment { const uint8_t* w; const uint8_t* s; int row0, rows, K; };
__device__ __forceinline__ Segment segment(const Params& p, const lcq_decode_layer* table, const Rows& r, int ph, int part) {
  const Shape& sh = p.sh;
  const lcq_decode_layer* l = table + (part == PART_O ? ph / 2 : (ph - 1) / 2);
  switch (part) {
    case PART_QKV: return {static_cast<const uint8_t*>(l->qkv_w), static_cast<const uint8_t*>(l->qkv_s), r.qkv0, r.qkv, sh.hidden};
    case PART_GATE: return {static_cast<const uint8_t*>(l->gate_up_w), static_cast<const uint8_t*>(l->gate_up_s), r.int0, r.inter, sh.hidden};
    case PART_UP: return {static_cast<const uint8_t*>(l->gate_up_w), static_cast<const uint8_t*>(l->gate_up_s), sh.inter + r.int0, r.inter, sh.hidden};
    case PART_DOWN: return {static_cast<const uint8_t*>(l->down_w), static_cast<const uint8_t*>(l->down_s), r.hid0, r.hid, sh.inter};
    case PART_O: return {static_cast<const uint8_t*>(l->o_w), static_cast<const uint8_t*>(l->o_s), r.hid0, r.hid, sh.q_dim};
    default: return {static_cast<const uint8_t*>(p.d.head_w), static_cast<const uint8_t*>(p.d.head_s), r.voc0, r.voc, sh.hidden};
  }
}

// Shared memory by 32-bit addresses: generic pointers would take two registers each and a slower load.
__device__ __forceinline__ uint32_t ld32(uint32_t a) { uint32_t v; asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a)); return v; }
__device__ __forceinline__ uint4 ld128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ float ld_half(uint32_t a) {
  unsigned short v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a));
  return __half2float(__ushort_as_half(v));
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}
__device__ __forceinline__ void st128(uint32_t a, float x, float y, float z, float w) {
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}
__device__ __forceinline__ void st32(uint32_t a, float x) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(x) : "memory"); }

// A lane's sums over the words word0, word0 + step, ... of NR rows that are NCW rows apart.
// w, sc, x: addresses of the first row's weights and scales and of the input.
template <int NR>
__device__ __forceinline__ void rows_dot(uint32_t w, uint32_t sc, uint32_t x, int K, int word0, int step, float (&acc)[NR]) {
  const int words = K / 8;
#pragma unroll
  for (int r = 0; r < NR; ++r) acc[r] = 0.0f;
#pragma unroll (NR == 1 ? 2 : 1)
  for (int j = word0; j < words; j += step) {
    const uint4 xv = ld128(x + j * 16);
#pragma unroll
    for (int r = 0; r < NR; ++r)
      acc[r] = fmaf(ld_half(sc + r * NCW * (K / 16) + (j >> 2) * 2), dot8(ld32(w + r * NCW * (K / 2) + j * 4), xv), acc[r]);
  }
}

// One tile (rows x K in shared memory) times x; row i's sum goes to res + 16 i as up to four parts.
__device__ __forceinline__ void tile_matvec(uint32_t stage, int rows, int K, uint32_t x, uint32_t res, int warp, int lane) {
  const uint32_t sc = stage + rows * (K / 2);
  if (rows <= 8) {                             // several warps a row
    const int shift = rows <= 4 ? 2 : 1, row = warp >> shift, part = warp & ((1 << shift) - 1);
    if (row >= rows) return;
    float acc[1];
    rows_dot<1>(stage + row * (K / 2), sc + row * (K / 16), x, K, part * 32 + lane, 32 << shift, acc);
    acc[0] = warp_sum(acc[0]);
    if (lane == 0) { st32(res + row * 16 + part * 4, acc[0]); if (shift == 1) st32(res + row * 16 + part * 4 + 8, 0.0f); }
    return;
  }
  int row = warp;
  for (; row + NCW < rows; row += 2 * NCW) {
    float acc[2];
    rows_dot<2>(stage + row * (K / 2), sc + row * (K / 16), x, K, lane, 32, acc);
    acc[0] = warp_sum(acc[0]);
    acc[1] = warp_sum(acc[1]);
    if (lane == 0) { st128(res + row * 16, acc[0], 0.0f, 0.0f, 0.0f); st128(res + (row + NCW) * 16, acc[1], 0.0f, 0.0f, 0.0f); }
  }
  if (row < rows) {
    float acc[1];
    rows_dot<1>(stage + row * (K / 2), sc + row * (K / 16), x, K, lane, 32, acc);
    acc[0] = warp_sum(acc[0]);
    if (lane == 0) st128(res + row * 16, acc[0], 0.0f, 0.0f, 0.0f);
  }
}

__global__ void __launch_bounds__(NTHREADS, 1) decode_step_kernel(const __grid_constant__ Params p) {
  extern __shared__ __align__(128) uint8_t smem[];
  const Shape& sh = p.sh;
  const Smem L = smem_map(sh, p.n_layers, p.ctas, p.stage_bytes, p.n_stages);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + L.bars);
  uint64_t* empty = full + MAX_STAGES;
  volatile int* flag_abort = reinterpret_cast<volatile int*>(smem + L.flags);
  uint32_t* smem_epoch = reinterpret_cast<uint32_t*>(smem + L.flags + 4);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x, b = blockIdx.x;
  uint32_t* epoch = static_cast<uint32_t*>(p.d.state);
  unsigned int* finished = static_cast<unsigned int*>(p.d.state) + 1;
  unsigned long long* best_key = static_cast<unsigned long long*>(p.d.state) + 1;

  if (tid == 0) {
    for (int i = 0; i < p.n_stages; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], NCW); }
    *flag_abort = 0;
    *smem_epoch = *reinterpret_cast<volatile uint32_t*>(epoch);
    Rows r;
    r.qkv0 = share(sh.qkv, b, p.ctas); r.qkv = share(sh.qkv, b + 1, p.ctas) - r.qkv0;
    r.hid0 = share(sh.hidden, b, p.ctas); r.hid = share(sh.hidden, b + 1, p.ctas) - r.hid0;
    r.int0 = share(sh.inter, b, p.ctas); r.inter = share(sh.inter, b + 1, p.ctas) - r.int0;
    r.voc0 = share(sh.vocab, b, p.ctas); r.voc = share(sh.vocab, b + 1, p.ctas) - r.voc0;
    *reinterpret_cast<Rows*>(smem + L.rows) = r;
    fence_barrier_init();
  }
  for (int i = tid; i < p.n_layers * static_cast<int>(sizeof(lcq_decode_layer) / 8); i += NTHREADS)
    reinterpret_cast<uint64_t*>(smem + L.table)[i] = static_cast<const uint64_t*>(p.d.layers)[i];
  __syncthreads();
  const Rows& mine = *reinterpret_cast<const Rows*>(smem + L.rows);
  const int step_h = tile_rows(p.stage_bytes, sh.hidden), step_q = tile_rows(p.stage_bytes, sh.q_dim), step_i = tile_rows(p.stage_bytes, sh.inter);

  if (warp >= NCW) {
    // ------------------------------------------------------------ producer: one thread, all phases in order
    if (lane == 0) {
      int s = 0, in_flight = 0;                // the next stage; stages before it whose copies may be on their way
      uint32_t phase = 0;
      bool ok = true;
      for (int ph = 0, part; ok && (part = first_part(ph, p.n_layers)) >= 0; ++ph) {
        for (; part >= 0 && ok; part = next_part(part, ph, p.n_layers)) {
          const Segment g = segment(p, reinterpret_cast<const lcq_decode_layer*>(smem + L.table), mine, ph, part);
          const int step = part == PART_O ? step_q : part == PART_DOWN ? step_i : step_h;
          for (int r = 0; r < g.rows; r += step) {
            const int rows = g.rows - r < step ? g.rows - r : step;
            // (the flag after the wait: consumers that gave up release stages whose copies have not landed)
            if (!mbar_wait_bounded(&empty[s], phase ^ 1u) || *flag_abort) { *flag_abort = 1; atomicExch(&g_device_status, 50); ok = false; break; }
            const uint32_t wb = static_cast<uint32_t>(rows) * (g.K / 2), sb = static_cast<uint32_t>(rows) * (g.K / 16);
            const uint32_t dst = smem_u32(smem) + s * p.stage_bytes;
            mbar_expect_tx(&full[s], wb + sb);
            bulk_load(dst, g.w + static_cast<long long>(g.row0 + r) * (g.K / 2), wb, &full[s]);
            bulk_load(dst + wb, g.s + static_cast<long long>(g.row0 + r) * (g.K / 16), sb, &full[s]);
            if (++s == p.n_stages) { s = 0; phase ^= 1u; }
            if (in_flight < p.n_stages) ++in_flight;
          }
        }
      }
      // Consumers that gave up wait for no more stages, so the copies into the last ones are waited for here: none may
      // land after the CTA has left.  They read this GPU's memory and end by themselves, whatever the wait limit.
      for (; in_flight > 0; --in_flight) {
        if (--s < 0) { s = p.n_stages - 1; phase ^= 1u; }
        mbar_wait_landed(&full[s], phase);
      }
    }
  } else {
    // ------------------------------------------------------------ consumers
    const uint32_t base = smem_u32(smem);
    const uint32_t xn = base + L.xn, xq = base + L.xq, xm = base + L.xm;
    __half* xn_p = reinterpret_cast<__half*>(smem + L.xn);
    float* red = reinterpret_cast<float*>(smem + L.red);
    const uint32_t tag0 = *smem_epoch * static_cast<uint32_t>(2 * p.n_layers + 1) + 1u;
    const int copy = (b % p.copies) * p.copy_words;
    int s = 0;
    uint32_t phase = 0;
    bool dead = false;

    // the next `n` rows of the stream (K columns, `step` rows a tile) times x
    const auto use_tiles = [&](int n, int K, int step, uint32_t x, int res0) {
      for (int r = 0; r < n; r += step) {
        const int rows = n - r < step ? n - r : step;
        if (!dead && (*flag_abort || !mbar_wait_bounded(&full[s], phase))) { dead = true; *flag_abort = 1; atomicExch(&g_device_status, 51); }
        dead = __any_sync(0xffffffffu, dead);
        if (!dead) tile_matvec(base + s * p.stage_bytes, rows, K, x, base + L.res + (res0 + r) * 16, warp, lane);
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[s]);
        if (++s == p.n_stages) { s = 0; phase ^= 1u; }
      }
    };
    // four published values, once they carry `tag`
    const auto take = [&](const uint32_t* src, uint32_t tag, __half (&v)[4]) {
      uint4 w = load_words(src);
      uint64_t t0 = 0;
      for (int i = 0; !dead && !(((w.x ^ tag) & 0xFFFFu) == 0 && ((w.y ^ tag) & 0xFFFFu) == 0 && ((w.z ^ tag) & 0xFFFFu) == 0 && ((w.w ^ tag) & 0xFFFFu) == 0); ++i) {
        if ((i & 1023) == 1023) {
          const uint64_t now = global_timer_ns();
          if (t0 == 0) t0 = now;
          if (*flag_abort || now - t0 > wait_limit_ns()) { dead = true; *flag_abort = 1; atomicExch(&g_device_status, 52); break; }
        }
        w = load_words(src);
      }
      v[0] = __ushort_as_half(static_cast<unsigned short>(w.x >> 16)); v[1] = __ushort_as_half(static_cast<unsigned short>(w.y >> 16));
      v[2] = __ushort_as_half(static_cast<unsigned short>(w.z >> 16)); v[3] = __ushort_as_half(static_cast<unsigned short>(w.w >> 16));
    };
    // A thread's share of the hidden state and of the next norms' weights, 4 values of every 4 * NCT, lies in
    // shared memory: in registers they cost the matvec loops theirs, and a spill goes to L2 here.
    __half* hid = reinterpret_cast<__half*>(smem + L.hid);
    const __half* next_norm = static_cast<const __half*>(p.d.norms);
    int norms_left = 2 * p.n_layers + 1;
    const auto fetch_norms = [&]() {           // a phase ahead: they may come from HBM
      const int two = norms_left > 1 ? 2 * sh.hidden : norms_left * sh.hidden;
      for (int i = 4 * tid; i < two; i += 4 * NCT)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(base + L.gam + 2 * i), "l"(next_norm + i) : "memory");
      next_norm += two;
      norms_left -= 2;
    };
    // hidden += the down projection; x = rms_norm(hidden); hidden += the o projection; x2 = rms_norm(hidden)
    // (the first phase has no down projection before it, the last one no o)
    const auto norms = [&](const uint32_t* down, const uint32_t* o, uint32_t tag) {
      float ss = 0.0f, ss2 = 0.0f;
      for (int i = 4 * tid; i < sh.hidden; i += 4 * NCT) {
        __half h[4], v[4];
        *reinterpret_cast<uint2*>(h) = *reinterpret_cast<const uint2*>(hid + i);
        if (down != nullptr) {
          take(down + i, tag, v);
#pragma unroll
          for (int e = 0; e < 4; ++e) h[e] = __float2half_rn(__half2float(h[e]) + __half2float(v[e]));
        }
        *reinterpret_cast<uint2*>(hid + i) = *reinterpret_cast<const uint2*>(h);
#pragma unroll
        for (int e = 0; e < 4; ++e) ss = fmaf(__half2float(h[e]), __half2float(h[e]), ss);
        if (o != nullptr) {
          take(o + i, tag, v);
#pragma unroll
          for (int e = 0; e < 4; ++e) h[e] = __float2half_rn(__half2float(h[e]) + __half2float(v[e]));
          *reinterpret_cast<uint2*>(hid + sh.hidden + i) = *reinterpret_cast<const uint2*>(h);
#pragma unroll
          for (int e = 0; e < 4; ++e) ss2 = fmaf(__half2float(h[e]), __half2float(h[e]), ss2);
        }
      }
      ss = warp_sum(ss);
      ss2 = warp_sum(ss2);
      if (lane == 0) { red[warp] = ss; red[NCW + warp] = ss2; }
      asm volatile("cp.async.wait_all;" ::: "memory");
      named_bar_sync(BAR_C, NCT);
      float total[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        total[j] = 0.0f;
#pragma unroll
        for (int i = 0; i < NCW / 4; ++i) {
          const float4 q = reinterpret_cast<const float4*>(red)[j * (NCW / 4) + i];
          total[j] += (q.x + q.y) + (q.z + q.w);
        }
        total[j] = rsqrtf(total[j] / static_cast<float>(sh.hidden) + p.d.eps);
      }
      for (int i = 4 * tid; i < sh.hidden; i += 4 * NCT) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          __half g[4], h[4], o4[4];
          *reinterpret_cast<uint2*>(g) = *reinterpret_cast<const uint2*>(smem + L.gam + 2 * (j * sh.hidden + i));
          *reinterpret_cast<uint2*>(h) = *reinterpret_cast<const uint2*>(hid + j * sh.hidden + i);
#pragma unroll
          for (int e = 0; e < 4; ++e) o4[e] = __float2half_rn(__half2float(h[e]) * total[j] * __half2float(g[e]));
          *reinterpret_cast<uint2*>(xn_p + j * sh.hidden + i) = *reinterpret_cast<const uint2*>(o4);
          if (j == 1 && o != nullptr) *reinterpret_cast<uint2*>(hid + i) = *reinterpret_cast<const uint2*>(h);
        }
      }
      named_bar_sync(BAR_C, NCT);
      fetch_norms();
    };
    const auto row_sum = [&](int i) {
      const uint4 v = ld128(base + L.res + i * 16);
      return (__uint_as_float(v.x) + __uint_as_float(v.y)) + (__uint_as_float(v.z) + __uint_as_float(v.w));
    };

    // embedding; the prepared input of the o projections
    fetch_norms();
    {
      const int id = *static_cast<const int*>(p.d.token);
      const bool known = id >= 0 && id < sh.vocab;
      if (!known && b == 0 && tid == 0) atomicExch(&g_device_status, 40);
      const __half* row = static_cast<const __half*>(p.d.table) + static_cast<long long>(known ? id : 0) * sh.hidden;
      for (int i = 4 * tid; i < sh.hidden; i += 4 * NCT)
        *reinterpret_cast<uint2*>(hid + i) = known ? *reinterpret_cast<const uint2*>(row + i) : make_uint2(0u, 0u);
      for (int i = 8 * tid; i < sh.q_dim; i += 8 * NCT)
        *reinterpret_cast<uint4*>(smem + L.xq + 2 * i) = *reinterpret_cast<const uint4*>(static_cast<const __half*>(p.d.x_q) + i);
    }

    // One loop body for all phases: code that runs once a phase is fetched anew each time.
    __half* out = static_cast<__half*>(p.d.outputs);     // this layer's q|k|v, o, gate|up, down
    const int layer_out = sh.qkv + 2 * sh.hidden + 2 * sh.inter, last = 2 * p.n_layers + 1;
    for (int ph = 0; ph <= last; ++ph) {
      const uint32_t tag = (tag0 + ph) & 0xFFFFu, before = (tag - 1u) & 0xFFFFu;
      const bool wide = (ph & 1) && ph != last;          // q|k|v, gate|up
      if (ph & 1) {
        norms(ph == 1 ? nullptr : p.d_buf + copy, ph == last ? nullptr : p.o_buf + copy, before);
      } else if (ph != 0) {
        for (int i = 4 * tid; i < sh.inter; i += 4 * NCT) {
          __half v[4];
          take(p.m_buf + copy + i, before, v);
          *reinterpret_cast<uint2*>(smem + L.xm + 2 * i) = *reinterpret_cast<const uint2*>(v);
        }
        named_bar_sync(BAR_C, NCT);
      } else {
        named_bar_sync(BAR_C, NCT);
      }
      int sums = 0;
      for (int part = first_part(ph, p.n_layers); part >= 0; part = next_part(part, ph, p.n_layers)) {
        const int n = part == PART_QKV ? mine.qkv : part == PART_HEAD ? mine.voc : part <= PART_UP ? mine.inter : mine.hid;
        use_tiles(n, part == PART_DOWN ? sh.inter : part == PART_O ? sh.q_dim : sh.hidden,
                  part == PART_DOWN ? step_i : part == PART_O ? step_q : step_h,
                  part == PART_DOWN ? xm : part == PART_O ? xq : part == PART_GATE || part == PART_UP ? xn + 2 * sh.hidden : xn, sums);
        sums += n;
      }
      named_bar_sync(BAR_C, NCT);
      if (ph == last) break;
      // warp w writes copies w, w + NCW, ... of what is published; the first also what the caller sees
      for (int c = warp; c < p.copies; c += NCW) {
        if (wide) {
          for (int i = lane; i < mine.inter; i += 32) {
            const __half gate = __float2half_rn(row_sum(mine.qkv + i)), up = __float2half_rn(row_sum(mine.qkv + mine.inter + i));
            const float x = __half2float(gate);
            const __half v = __float2half_rn((x * (1.0f / (1.0f + expf(-x)))) * __half2float(up));
            publish(p.m_buf + c * p.copy_words + mine.int0 + i, v, tag);
            if (c == 0) {
              __half* o = out + sh.qkv + sh.hidden + mine.int0 + i;
              o[0] = gate;
              o[sh.inter] = up;
              if (ph == last - 2) static_cast<__half*>(p.d.mlp_out)[mine.int0 + i] = v;
            }
          }
        } else {
          // down rows of this layer, then o rows of the next (phase 0: o rows only; the last layer: down only)
          const int n_down = ph == 0 ? 0 : mine.hid;
          for (int i = lane; i < sums; i += 32) {
            const __half v = __float2half_rn(row_sum(i));
            const bool down = i < n_down;
            const int row = mine.hid0 + (down ? i : i - n_down);
            publish((down ? p.d_buf : p.o_buf) + c * p.copy_words + row, v, tag);
            if (c == 0) (down ? out + layer_out - sh.hidden : (ph == 0 ? out : out + layer_out) + sh.qkv)[row] = v;
          }
        }
      }
      if (wide)
        for (int i = tid; i < mine.qkv; i += NCT) out[mine.qkv0 + i] = __float2half_rn(row_sum(i));
      if (!(ph & 1) && ph != 0) out += layer_out;
    }
    if (b == 0) {
      for (int i = 4 * tid; i < sh.hidden; i += 4 * NCT) {
        *reinterpret_cast<uint2*>(static_cast<__half*>(p.d.hidden_out) + i) = *reinterpret_cast<const uint2*>(hid + i);
        *reinterpret_cast<uint2*>(static_cast<__half*>(p.d.normed_out) + i) = *reinterpret_cast<const uint2*>(xn_p + i);
      }
    }
    const int v0 = mine.voc0, n = mine.voc;
    // the key of a logit orders as np.argmax does: by value, NaN above all, the lowest index among equals
    unsigned long long key = 0;
    for (int i = tid; i < n; i += NCT) {
      const __half v = __float2half_rn(row_sum(i));
      static_cast<__half*>(p.d.logits)[v0 + i] = v;
      const float f = __half2float(v) + 0.0f;            // -0 counts as 0
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
    unsigned long long* keys = reinterpret_cast<unsigned long long*>(red);
    if (lane == 0) keys[warp] = key;
    named_bar_sync(BAR_C, NCT);
    if (tid == 0) {
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
struct Plan { int ctas, stage_bytes, n_stages, copies; size_t smem, state_bytes; };

inline bool make_plan(const lcq_decode_stack& d, int sm_count, Plan& pl) {
  const int H = d.hidden, I = d.inter;
  if (d.n_layers < 1 || H < 64 || I < 64 || d.qkv < 4 || d.q_dim < 64 || d.vocab < 4 || d.n_layers > 256) return false;
  if (H % 64 || I % 64 || d.q_dim % 64 || d.qkv % 4 || d.vocab % 4 || H > 8192 || I > (1 << 20) || d.vocab > (1 << 24)) return false;
  int units = H / 4;                           // every CTA needs a unit of 4 rows in every phase
  if (I / 4 < units) units = I / 4;
  if (d.vocab / 4 < units) units = d.vocab / 4;
  pl.ctas = sm_count < units ? sm_count : units;
  // a stage holds at least 4 rows of the longest kind, and 24 KB of the others
  const int longest = max2(max2(row_bytes(H), row_bytes(I)), row_bytes(d.q_dim)) * 4;
  pl.stage_bytes = (max2(longest, 24 * 1024) + 127) & ~127;
  const Shape sh = {H, I, d.qkv, d.q_dim, d.vocab};
  const int rest = smem_map(sh, d.n_layers, pl.ctas, 0, 0).total;
  pl.n_stages = (227 * 1024 - rest) / pl.stage_bytes;
  if (pl.n_stages > MAX_STAGES) pl.n_stages = MAX_STAGES;
  if (pl.n_stages < 2) return false;
  pl.smem = static_cast<size_t>(smem_map(sh, d.n_layers, pl.ctas, pl.stage_bytes, pl.n_stages).total);
  pl.copies = 8;                               // 30 layers of width 576: 1 copy 420 us, 2 363, 4 337, 8 332, 16 325 (an earlier build)
  pl.state_bytes = STATE_BYTES + (static_cast<size_t>(2) * H + I) * 4 * pl.copies;
  return true;
}

inline int launch(const lcq_decode_stack& d, int sm_count, cudaStream_t stream) {
  Plan pl;
  if (!make_plan(d, sm_count, pl)) { set_error("decode_step: this shape is not covered"); return LCQ_ERR_UNSUPPORTED; }
  if (d.state_bytes < pl.state_bytes) { set_error("decode_step: state of %zu bytes required, got %zu", pl.state_bytes, d.state_bytes); return LCQ_ERR_WORKSPACE; }
  const void* pointers[] = {d.layers, d.head_w, d.head_s, d.logits, d.norms, d.outputs, d.token, d.table, d.x_q, d.hidden_out, d.normed_out, d.mlp_out, d.next_token, d.state};
  for (const void* q : pointers)
    if (!q || !aligned(q, q == d.token || q == d.next_token ? 4 : 16)) { set_error("decode_step: null or misaligned pointer"); return LCQ_ERR_BAD_ARG; }
  Params p;
  memset(&p, 0, sizeof(p));
  p.d = d;
  p.sh = {d.hidden, d.inter, d.qkv, d.q_dim, d.vocab};
  p.n_layers = d.n_layers;
  p.ctas = pl.ctas;
  p.copies = pl.copies;
  p.copy_words = 2 * d.hidden + d.inter;
  p.stage_bytes = pl.stage_bytes; p.n_stages = pl.n_stages;
  p.o_buf = reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(d.state) + STATE_BYTES);
  p.d_buf = p.o_buf + d.hidden;
  p.m_buf = p.d_buf + d.hidden;
  static thread_local int configured_device = -1;
  int dev = 0;
  LCQ_CUDA_TRY(cudaGetDevice(&dev));
  if (configured_device != dev) {
    LCQ_CUDA_TRY(cudaFuncSetAttribute(decode_step_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    configured_device = dev;
  }
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(p.ctas);
  cfg.blockDim = dim3(NTHREADS);
  cfg.dynamicSmemBytes = pl.smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;           // all CTAs resident at once, or the launch fails
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  LCQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, decode_step_kernel, p));
  return LCQ_OK;
}

}  // namespace step
}  // namespace lcq
