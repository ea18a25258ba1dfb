// One decode step of a Llama-style stack of quantized linears (M = 1, int4 weights in groups of 32) as ONE
// kernel: embedding, per layer {RMS norm, q|k|v and o projections, residual add + RMS norm, gate|up, SiLU *
// up, down, residual add}, final norm, lm_head and greedy argmax -- the chain that locomp_b200.DecodeStack
// runs as 8 launches a layer otherwise (examples/54_smollm2_inference.py:494-578 without the attention
// itself; o reads a prepared buffer, so it depends on nothing in its layer and runs beside q|k|v).
//
// What bounds it.  SmolLM2-135M has 30 layers of 2 MB: 12 us of HBM time for the whole token, but ~90
// dependent matvecs.  As separate kernels each costs ~2 us (launch, dependency wait, first loads, drain):
// 506 us a token.  Here
//   * one CTA per SM stays for the whole step; a producer thread streams the CTA's rows of ALL layers
//     through one shared-memory ring (bulk copies), running ahead across layers, so that weights are there
//     when their input is;
//   * results that the next phase needs are published as words {fp16 value, 16-bit tag of the phase}: a
//     consumer polls the data itself until every tag is the one it expects.  No grid barrier, no fence, no
//     flag: one store and one load through L2 between dependent matvecs;
//   * every CTA keeps the hidden state (in registers) and does the norms redundantly.
// Every CTA has at least one unit of 4 rows in every phase.  So whoever has all results of a phase knows
// that all CTAs have read what they needed for it, and a buffer that is rewritten three phases later (the
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
constexpr int MAX_STAGES = 16;
constexpr int BAR_C = 1;                       // named barrier of the consumers
constexpr int STATE_BYTES = 64;                // epoch, argmax counter, argmax key

struct Shape { int hidden, inter, qkv, q_dim, vocab; };

struct Params {
  lcq_decode_stack d;
  Shape sh;
  int n_layers, ctas;
  int stage_bytes, n_stages;
  uint32_t* o_buf;      // published words: o projection, down projection [hidden], activation [inter]
  uint32_t* d_buf;
  uint32_t* m_buf;
};

// Rows of an [n, K] weight that CTA b streams: whole units of 4 (so that rows of scales start on 16 bytes).
__host__ __device__ inline int share(int n, int b, int ctas) { return 4 * static_cast<int>(static_cast<long long>(n / 4) * b / ctas); }
__host__ __device__ inline int row_bytes(int K) { return K / 2 + K / 16; }
__host__ __device__ inline int tile_rows(int stage_bytes, int K) { return (stage_bytes / row_bytes(K)) & ~3; }

struct Smem { int stages, xn, xq, xm, res, red, bars, flags, total; };
__host__ __device__ inline int max2(int a, int b) { return a > b ? a : b; }
__host__ __device__ inline Smem smem_map(const Shape& s, int ctas, int stage_bytes, int n_stages) {
  Smem m;
  m.stages = 0;
  m.xn = n_stages * stage_bytes;
  m.xq = m.xn + s.hidden * 2;
  m.xm = m.xq + s.q_dim * 2;
  m.res = m.xm + s.inter * 2;
  const int per = 4;                           // a share is at most one unit above the average
  const int rows = max2(max2((s.qkv + s.hidden) / ctas + 4 * per, 2 * s.inter / ctas + 4 * per), s.vocab / ctas + 2 * per);
  m.red = m.res + rows * 16;
  m.bars = m.red + 2 * NCW * 8;
  m.flags = m.bars + 2 * MAX_STAGES * 8;
  m.total = m.flags + 16;
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
  float p = 0.0f;
  p = fma_lo(a, x.x, false, false, p);
  p = fma_lo(b, x.x, false, true, p);
  p = fma_lo(c, x.y, false, false, p);
  p = fma_lo(d, x.y, false, true, p);
  p = fma_lo(a, x.z, true, false, p);
  p = fma_lo(b, x.z, true, true, p);
  p = fma_lo(c, x.w, true, false, p);
  p = fma_lo(d, x.w, true, true, p);
  return p;
}

// The tiles of a CTA in the order in which the producer streams and the consumers use them: per layer q|k|v
// rows, o rows, gate rows, up rows, down rows; then the lm_head.
struct Segment { const uint8_t* w; const uint8_t* s; int row0, rows, K; };
__device__ __forceinline__ Segment segment(const Params& p, int layer, int part, int b) {
  Segment g;
  const Shape& sh = p.sh;
  int n, base = 0;
  if (layer == p.n_layers) {
    g.w = static_cast<const uint8_t*>(p.d.head_w); g.s = static_cast<const uint8_t*>(p.d.head_s);
    n = sh.vocab; g.K = sh.hidden;
  } else {
    const lcq_decode_layer* l = static_cast<const lcq_decode_layer*>(p.d.layers) + layer;
    if (part == 0) { g.w = static_cast<const uint8_t*>(l->qkv_w); g.s = static_cast<const uint8_t*>(l->qkv_s); n = sh.qkv; g.K = sh.hidden; }
    else if (part == 1) { g.w = static_cast<const uint8_t*>(l->o_w); g.s = static_cast<const uint8_t*>(l->o_s); n = sh.hidden; g.K = sh.q_dim; }
    else if (part == 4) { g.w = static_cast<const uint8_t*>(l->down_w); g.s = static_cast<const uint8_t*>(l->down_s); n = sh.hidden; g.K = sh.inter; }
    else { g.w = static_cast<const uint8_t*>(l->gate_up_w); g.s = static_cast<const uint8_t*>(l->gate_up_s); n = sh.inter; g.K = sh.hidden; base = part == 3 ? sh.inter : 0; }
  }
  const int r0 = share(n, b, p.ctas), r1 = share(n, b + 1, p.ctas);
  g.row0 = base + r0;
  g.rows = r1 - r0;
  return g;
}

// A lane's sums over the words lane, lane + step, ... of NR rows that are `row_step` rows apart.
template <int NR>
__device__ __forceinline__ void rows_dot(const uint8_t* w, const __half* sc, const uint4* x, int K, int row_step, int word0, int step, float (&acc)[4]) {
  const int words = K / 8, groups = K / 32;
#pragma unroll
  for (int r = 0; r < NR; ++r) acc[r] = 0.0f;
#pragma unroll 2
  for (int j = word0; j < words; j += step) {
    const uint4 xv = x[j];
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      const uint32_t word = *reinterpret_cast<const uint32_t*>(w + (static_cast<size_t>(r * row_step) * words + j) * 4);
      acc[r] = fmaf(__half2float(sc[r * row_step * groups + (j >> 2)]), dot8(word, xv), acc[r]);
    }
  }
}

// One tile (rows x K in shared memory) times x; row i's sum goes to res[4 i .. 4 i + 3] as up to four parts.
__device__ __forceinline__ void tile_matvec(const uint8_t* stage, int rows, int K, const uint4* x, float4* res, int warp, int lane) {
  const __half* sc = reinterpret_cast<const __half*>(stage + rows * (K / 2));
  if (rows <= 8) {                             // several warps a row
    const int parts = rows <= 4 ? 4 : 2, row = warp / parts, part = warp - row * parts;
    if (row >= rows) return;
    float acc[4];
    rows_dot<1>(stage + row * (K / 2), sc + row * (K / 32), x, K, 0, part * 32 + lane, parts * 32, acc);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], off);
    float* out = reinterpret_cast<float*>(res + row);
    if (lane == 0) { out[part] = acc[0]; if (parts == 2) out[part + 2] = 0.0f; }
    return;
  }
  for (int row = warp; row < rows; row += 4 * NCW) {
    float acc[4];
    const uint8_t* w = stage + row * (K / 2);
    const __half* s = sc + row * (K / 32);
    const int n = (rows - row + NCW - 1) / NCW;          // rows of this pass: 1 .. 4
    if (n >= 4) rows_dot<4>(w, s, x, K, NCW, lane, 32, acc);
    else if (n == 3) rows_dot<3>(w, s, x, K, NCW, lane, 32, acc);
    else if (n == 2) rows_dot<2>(w, s, x, K, NCW, lane, 32, acc);
    else rows_dot<1>(w, s, x, K, NCW, lane, 32, acc);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      if (r < n) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], off);
        if (lane == 0) res[row + r * NCW] = make_float4(acc[r], 0.0f, 0.0f, 0.0f);
      }
    }
  }
}

// CH: chunks of 4 * NCT hidden values (a thread keeps 4 of each in registers).
template <int CH>
__global__ void __launch_bounds__(NTHREADS, 1) decode_step_kernel(const __grid_constant__ Params p) {
  extern __shared__ __align__(128) uint8_t smem[];
  const Shape& sh = p.sh;
  const Smem L = smem_map(sh, p.ctas, p.stage_bytes, p.n_stages);
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
    fence_barrier_init();
  }
  __syncthreads();

  if (warp == NCW) {
    // ------------------------------------------------------------ producer: one thread, all layers in order
    if (lane == 0) {
      int s = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int layer = 0; layer <= p.n_layers && ok; ++layer) {
        for (int part = 0; part < (layer < p.n_layers ? 5 : 1) && ok; ++part) {
          const Segment g = segment(p, layer, part, b);
          const int step = tile_rows(p.stage_bytes, g.K);
          for (int r = 0; r < g.rows; r += step) {
            const int rows = g.rows - r < step ? g.rows - r : step;
            if (*flag_abort || !mbar_wait_bounded(&empty[s], phase ^ 1u)) { *flag_abort = 1; atomicExch(&g_device_status, 50); ok = false; break; }
            const uint32_t wb = static_cast<uint32_t>(rows) * (g.K / 2), sb = static_cast<uint32_t>(rows) * (g.K / 16);
            const uint32_t dst = smem_u32(smem) + s * p.stage_bytes;
            mbar_expect_tx(&full[s], wb + sb);
            bulk_load(dst, g.w + static_cast<long long>(g.row0 + r) * (g.K / 2), wb, &full[s]);
            bulk_load(dst + wb, g.s + static_cast<long long>(g.row0 + r) * (g.K / 16), sb, &full[s]);
            if (++s == p.n_stages) { s = 0; phase ^= 1u; }
          }
        }
      }
    }
  } else {
    // ------------------------------------------------------------ consumers
    __half* xn = reinterpret_cast<__half*>(smem + L.xn);
    __half* xq = reinterpret_cast<__half*>(smem + L.xq);
    __half* xm = reinterpret_cast<__half*>(smem + L.xm);
    float4* res = reinterpret_cast<float4*>(smem + L.res);
    float* red = reinterpret_cast<float*>(smem + L.red);
    const uint32_t tag0 = *smem_epoch * static_cast<uint32_t>(3 * p.n_layers) + 1u;
    int s = 0;
    uint32_t phase = 0;
    bool dead = false;

    const auto use_tiles = [&](int layer, int part, const __half* x, int res0) {
      const Segment g = segment(p, layer, part, b);
      const int step = tile_rows(p.stage_bytes, g.K);
      for (int r = 0; r < g.rows; r += step) {
        const int rows = g.rows - r < step ? g.rows - r : step;
        if (!dead && (*flag_abort || !mbar_wait_bounded(&full[s], phase))) { dead = true; *flag_abort = 1; atomicExch(&g_device_status, 51); }
        dead = __any_sync(0xffffffffu, dead);
        if (!dead) tile_matvec(smem + s * p.stage_bytes, rows, g.K, reinterpret_cast<const uint4*>(x), res + res0 + r, warp, lane);
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[s]);
        if (++s == p.n_stages) { s = 0; phase ^= 1u; }
      }
      return g.rows;
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
    __half h[CH][4];                           // the hidden state, values 4 * (c * NCT + tid) ..
    // hidden (+= what was published in src); xn = rms_norm(hidden) * weight
    // (the weights of the next norm are fetched a phase ahead: they may come from HBM)
    uint2 next_g[CH];
    int norm_index = 0;
    const auto fetch_norm = [&]() {
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        const int i = 4 * (c * NCT + tid);
        next_g[c] = make_uint2(0u, 0u);
        if (i < sh.hidden && norm_index <= 2 * p.n_layers)
          next_g[c] = __ldg(reinterpret_cast<const uint2*>(static_cast<const __half*>(p.d.norms) + static_cast<long long>(norm_index) * sh.hidden + i));
      }
      ++norm_index;
    };
    const auto norm = [&](const uint32_t* src, uint32_t tag) {
      float ss = 0.0f;
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        const int i = 4 * (c * NCT + tid);
        if (i < sh.hidden) {
          if (src != nullptr) {
            __half v[4];
            take(src + i, tag, v);
#pragma unroll
            for (int e = 0; e < 4; ++e) h[c][e] = __float2half_rn(__half2float(h[c][e]) + __half2float(v[e]));
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) ss = fmaf(__half2float(h[c][e]), __half2float(h[c][e]), ss);
        }
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
      if (lane == 0) red[warp] = ss;
      named_bar_sync(BAR_C, NCT);
      float total = 0.0f;
#pragma unroll
      for (int i = 0; i < NCW / 4; ++i) {
        const float4 q = reinterpret_cast<const float4*>(red)[i];
        total += (q.x + q.y) + (q.z + q.w);
      }
      const float rms = rsqrtf(total / static_cast<float>(sh.hidden) + p.d.eps);
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        const int i = 4 * (c * NCT + tid);
        if (i < sh.hidden) {
          __half o[4], g[4];
          *reinterpret_cast<uint2*>(g) = next_g[c];
#pragma unroll
          for (int e = 0; e < 4; ++e) o[e] = __float2half_rn(__half2float(h[c][e]) * rms * __half2float(g[e]));
          *reinterpret_cast<uint2*>(xn + i) = *reinterpret_cast<const uint2*>(o);
        }
      }
      named_bar_sync(BAR_C, NCT);
      fetch_norm();
    };
    const auto sum4 = [&](int i) { const float4 v = res[i]; return (v.x + v.y) + (v.z + v.w); };

    // embedding; the prepared input of the o projections
    fetch_norm();
    {
      const int id = *static_cast<const int*>(p.d.token);
      const bool known = id >= 0 && id < sh.vocab;
      if (!known && b == 0 && tid == 0) atomicExch(&g_device_status, 40);
      const __half* row = static_cast<const __half*>(p.d.table) + static_cast<long long>(known ? id : 0) * sh.hidden;
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        const int i = 4 * (c * NCT + tid);
        uint2 raw = make_uint2(0u, 0u);
        if (known && i < sh.hidden) raw = *reinterpret_cast<const uint2*>(row + i);
        *reinterpret_cast<uint2*>(h[c]) = raw;
      }
      for (int i = 8 * tid; i < sh.q_dim; i += 8 * NCT)
        *reinterpret_cast<uint4*>(xq + i) = *reinterpret_cast<const uint4*>(static_cast<const __half*>(p.d.x_q) + i);
    }

    for (int layer = 0; layer < p.n_layers; ++layer) {
      // this layer's outputs: q|k|v, o, gate|up, down
      __half* qkv_out = static_cast<__half*>(p.d.outputs) + static_cast<long long>(layer) * (sh.qkv + 2 * sh.hidden + 2 * sh.inter);
      __half *o_out = qkv_out + sh.qkv, *gate_up_out = o_out + sh.hidden, *down_out = gate_up_out + 2 * sh.inter;
      const uint32_t tag = (tag0 + 3u * layer) & 0xFFFFu, tag1 = (tag + 1u) & 0xFFFFu, tag2 = (tag + 2u) & 0xFFFFu;
      // ---- q|k|v and o
      norm(layer == 0 ? nullptr : p.d_buf, (tag - 1u) & 0xFFFFu);
      {
        const int q0 = share(sh.qkv, b, p.ctas), o0 = share(sh.hidden, b, p.ctas);
        const int n_q = use_tiles(layer, 0, xn, 0);
        const int n_o = use_tiles(layer, 1, xq, n_q);
        named_bar_sync(BAR_C, NCT);
        for (int i = tid; i < n_o + n_q; i += NCT) {
          if (i < n_o) {
            const __half v = __float2half_rn(sum4(n_q + i));
            publish(p.o_buf + o0 + i, v, tag);
            o_out[o0 + i] = v;
          } else {
            qkv_out[q0 + i - n_o] = __float2half_rn(sum4(i - n_o));
          }
        }
      }
      // ---- gate|up and the activation
      norm(p.o_buf, tag);
      {
        const int i0 = share(sh.inter, b, p.ctas);
        const int n = use_tiles(layer, 2, xn, 0);
        use_tiles(layer, 3, xn, n);
        named_bar_sync(BAR_C, NCT);
        for (int i = tid; i < n; i += NCT) {
          const __half g = __float2half_rn(sum4(i)), u = __float2half_rn(sum4(n + i));
          const float x = __half2float(g);
          const __half v = __float2half_rn((x * (1.0f / (1.0f + expf(-x)))) * __half2float(u));
          publish(p.m_buf + i0 + i, v, tag1);
          gate_up_out[i0 + i] = g;
          gate_up_out[sh.inter + i0 + i] = u;
          if (layer == p.n_layers - 1) static_cast<__half*>(p.d.mlp_out)[i0 + i] = v;
        }
      }
      // ---- down
      {
        for (int i = 4 * tid; i < sh.inter; i += 4 * NCT) {
          __half v[4];
          take(p.m_buf + i, tag1, v);
          *reinterpret_cast<uint2*>(xm + i) = *reinterpret_cast<const uint2*>(v);
        }
        const int d0 = share(sh.hidden, b, p.ctas);
        named_bar_sync(BAR_C, NCT);
        const int n = use_tiles(layer, 4, xm, 0);
        named_bar_sync(BAR_C, NCT);
        for (int i = tid; i < n; i += NCT) {
          const __half v = __float2half_rn(sum4(i));
          publish(p.d_buf + d0 + i, v, tag2);
          down_out[d0 + i] = v;
        }
      }
    }
    // ---- final norm, lm_head, argmax
    norm(p.d_buf, (tag0 + 3u * p.n_layers - 1u) & 0xFFFFu);
    if (b == 0) {
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        const int i = 4 * (c * NCT + tid);
        if (i < sh.hidden) {
          *reinterpret_cast<uint2*>(static_cast<__half*>(p.d.hidden_out) + i) = *reinterpret_cast<const uint2*>(h[c]);
          *reinterpret_cast<uint2*>(static_cast<__half*>(p.d.normed_out) + i) = *reinterpret_cast<const uint2*>(xn + i);
        }
      }
    }
    const int v0 = share(sh.vocab, b, p.ctas);
    const int n = use_tiles(p.n_layers, 0, xn, 0);
    named_bar_sync(BAR_C, NCT);
    // the key of a logit orders as np.argmax does: by value, NaN above all, the lowest index among equals
    unsigned long long key = 0;
    for (int i = tid; i < n; i += NCT) {
      const __half v = __float2half_rn(sum4(i));
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
struct Plan { int ctas, stage_bytes, n_stages, chunks; size_t smem, state_bytes; };

inline bool make_plan(const lcq_decode_stack& d, int sm_count, Plan& pl) {
  const int H = d.hidden, I = d.inter;
  if (d.n_layers < 1 || H < 64 || I < 64 || d.qkv < 4 || d.q_dim < 64 || d.vocab < 4) return false;
  if (H % 64 || I % 64 || d.q_dim % 64 || d.qkv % 4 || d.vocab % 4 || H > 8 * NCT || I > (1 << 20) || d.vocab > (1 << 28)) return false;
  int units = H / 4;                           // every CTA needs a unit of 4 rows in every phase
  if (I / 4 < units) units = I / 4;
  if (d.vocab / 4 < units) units = d.vocab / 4;
  pl.ctas = sm_count < units ? sm_count : units;
  pl.chunks = H <= 4 * NCT ? 1 : 2;
  // a stage holds at least 4 rows of the longest kind, and 16 KB of the others
  const int longest = max2(max2(row_bytes(H), row_bytes(I)), row_bytes(d.q_dim)) * 4;
  pl.stage_bytes = (max2(longest, 16 * 1024) + 127) & ~127;
  const Shape sh = {H, I, d.qkv, d.q_dim, d.vocab};
  const int rest = smem_map(sh, pl.ctas, 0, 0).total;
  pl.n_stages = (227 * 1024 - rest) / pl.stage_bytes;
  if (pl.n_stages > MAX_STAGES) pl.n_stages = MAX_STAGES;
  if (pl.n_stages < 2) return false;
  pl.smem = static_cast<size_t>(smem_map(sh, pl.ctas, pl.stage_bytes, pl.n_stages).total);
  pl.state_bytes = STATE_BYTES + (static_cast<size_t>(2) * H + I) * 4;
  return true;
}

template <int CH>
int launch_t(const Params& p, size_t smem, cudaStream_t stream) {
  static thread_local int configured_device = -1;
  int dev = 0;
  LCQ_CUDA_TRY(cudaGetDevice(&dev));
  if (configured_device != dev) {
    LCQ_CUDA_TRY(cudaFuncSetAttribute(decode_step_kernel<CH>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    configured_device = dev;
  }
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(p.ctas);
  cfg.blockDim = dim3(NTHREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;           // all CTAs resident at once, or the launch fails
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  LCQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, decode_step_kernel<CH>, p));
  return LCQ_OK;
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
  p.stage_bytes = pl.stage_bytes; p.n_stages = pl.n_stages;
  p.o_buf = reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(d.state) + STATE_BYTES);
  p.d_buf = p.o_buf + d.hidden;
  p.m_buf = p.d_buf + d.hidden;
  return pl.chunks == 1 ? launch_t<1>(p, pl.smem, stream) : launch_t<2>(p, pl.smem, stream);
}

}  // namespace step
}  // namespace lcq
