// Quantized matmul on CUDA cores, a warp per row (per four rows when M > 1): the general kernels (any K % G == 0, any
// dtype combination, float32 math end to end).  It is the path for the reference's own
// dtypes -- float32 x / scales / out, M = 1 (examples/38_quantized_matmul.py:30-134) --
// and the fallback for shapes the tensor-core kernels do not take.
//
//   out[m, n] = sum_k x[m, k] * wq(n, k) * scales[n, k / G]
//   wq = nibble - 8 (int4, low nibble = even k)  or  int8 value
//
// One warp owns one output row n and MT rows of x; lanes stride over K in chunks of 8
// weights (vector path) or single bytes (scalar path), accumulate in float32 and combine
// with a shuffle tree.  Within a chunk the scale is factored out of the 8 products.
#pragma once
#include "common.cuh"
#include "dequant.cuh"

namespace lcq {

template <typename XT> __device__ __forceinline__ void load8(const XT* p, float (&v)[8]);
template <> __device__ __forceinline__ void load8<float>(const float* p, float (&v)[8]) {
  const float4 a = __ldg(reinterpret_cast<const float4*>(p));
  const float4 b = __ldg(reinterpret_cast<const float4*>(p) + 1);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
template <> __device__ __forceinline__ void load8<__half>(const __half* p, float (&v)[8]) {
  const uint4 r = __ldg(reinterpret_cast<const uint4*>(p));
  const __half2* h = reinterpret_cast<const __half2*>(&r);
#pragma unroll
  for (int i = 0; i < 4; ++i) { const float2 f = __half22float2(h[i]); v[2 * i] = f.x; v[2 * i + 1] = f.y; }
}
template <> __device__ __forceinline__ void load8<__nv_bfloat16>(const __nv_bfloat16* p, float (&v)[8]) {
  const uint4 r = __ldg(reinterpret_cast<const uint4*>(p));
  const uint32_t* u = reinterpret_cast<const uint32_t*>(&r);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[2 * i] = __uint_as_float(u[i] << 16);
    v[2 * i + 1] = __uint_as_float(u[i] & 0xFFFF0000u);
  }
}

// Two float32 values in one 64-bit register: the FMA pipe takes them as one instruction, each rounded as by itself.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float sum2(f32x2 v) {
  float a, b;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
  return a + b;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// 8 values of x in pairs
__device__ __forceinline__ void load8_pairs(const float* p, f32x2 (&v)[4]) {
  const ulonglong2 a = __ldg(reinterpret_cast<const ulonglong2*>(p)), b = __ldg(reinterpret_cast<const ulonglong2*>(p) + 1);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
template <typename XT> __device__ __forceinline__ void load8_pairs(const XT* p, f32x2 (&v)[4]) {
  float f[8];
  load8<XT>(p, f);
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = pack2(f[2 * i], f[2 * i + 1]);
}
// An octet of int4 weights: bits of 2^23 + q, from which 2^23 + 8 is taken exactly.  By a mask per nibble parity and a byte permute
// a weight; a shift and a mask for each nibble take five more instructions.
__device__ __forceinline__ void int4_bits(uint32_t w, uint32_t (&v)[8]) {
  const uint32_t even = w & 0x0F0F0F0Fu, odd = (w >> 4) & 0x0F0F0F0Fu;
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __byte_perm(i & 1 ? odd : even, 0x4B000000u, 0x7540 + i / 2);
}
__device__ __forceinline__ void int4_pairs(uint32_t w, f32x2 (&v)[4]) {
  uint32_t bits[8];
  int4_bits(w, bits);
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = add2(pack2(__uint_as_float(bits[2 * i]), __uint_as_float(bits[2 * i + 1])), pack2(-8388616.0f, -8388616.0f));
}
// SHIFTS: by a shift and a mask for each nibble; else by permutes, which take fewer instructions and more registers.  Shifts for two rows of x, and for
// float32 scales with more: the forms in which permutes lost somewhere.  us, shifts / permutes.  Two rows, float32: 4096 -> 8192 13.5 / 17.3, 2048 -> 2000
// 2.8 / 3.2, 8192 -> 16000 51.0 / 54.1, but 1024 -> 12000 7.5 / 5.3; float16: 8192 -> 16000 52.7 / 53.9, but 4096 -> 8192 21.6 / 18.2, 1024 -> 12000 6.0 / 5.2.  Three and
// more, float32: M = 8, 3072 -> 3000 12.6 / 13.1, M = 3, 2048 -> 6000 9.7 / 9.9, but M = 8, 4096 -> 8192 35.5 / 31.2, 8192 -> 16000 123 / 111, M = 5, 1536 -> 3690 7.8 / 6.9;
// float16: M = 8, 4096 -> 8192 40.4 / 32.1, 8192 -> 16000 184 / 111.
template <bool SHIFTS> __device__ __forceinline__ void int4_floats(uint32_t w, float (&v)[8]) {
  if (SHIFTS) {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(0x4B000000u | ((w >> (4 * i)) & 15u)) - 8388616.0f;
  } else {
    uint32_t bits[8];
    int4_bits(w, bits);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(bits[i]) - 8388616.0f;
  }
}
// The sums of gemv_rows_kernel, in one register or as two halves.
template <bool PAIRS> struct RowSums { typedef float type; };
template <> struct RowSums<true> { typedef f32x2 type; };
__device__ __forceinline__ void scaled_sum(float& acc, float s, float p) { acc = fmaf(s, p, acc); }
__device__ __forceinline__ void scaled_sum(f32x2& acc, float s, f32x2 p) { acc = fma2(pack2(s, s), p, acc); }
__device__ __forceinline__ f32x2 dot8(const f32x2 (&x)[4], const f32x2 (&w)[4]) {
  f32x2 p = mul2(x[0], w[0]);
#pragma unroll
  for (int i = 1; i < 4; ++i) p = fma2(x[i], w[i], p);
  return p;
}
__device__ __forceinline__ float row_sum(float v) { return v; }
__device__ __forceinline__ float row_sum(f32x2 v) { return sum2(v); }

template <int WBITS, typename XT, typename ST, typename OT, int MT, bool VEC>
__global__ void __launch_bounds__(256) gemv_simt_kernel(const XT* __restrict__ x, const uint8_t* __restrict__ w,
                                                        const ST* __restrict__ scales, OT* __restrict__ out,
                                                        int M, int N, int K, int G) {
  const int lane = threadIdx.x & 31;
  const int n = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int m0 = blockIdx.y * MT;
  // Programmatic dependent launch.  Weights and scales are constants, so a lane fetches its first
  // chunk of them BEFORE waiting for the kernel ahead of it on the stream: that DRAM round trip then
  // runs under the other kernel's tail.  x (possibly that kernel's output) and out are touched only
  // after the wait.  A grid that fits on the machine at once lets the next kernel in right away
  // (its launch and its own weight prefetch then overlap this kernel entirely); a larger grid does so
  // only once its loads are issued, so that resident-but-waiting CTAs of the next kernel do not take
  // SM slots from this grid's later waves.
  const bool small_grid = gridDim.x * gridDim.y <= 296u;
  if (small_grid) griddep_launch_dependents();
  const bool row_ok = n < N;
  const int ns = K / G;
  const ST* srow = scales + static_cast<long long>(row_ok ? n : 0) * ns;
  float acc[MT];
#pragma unroll
  for (int m = 0; m < MT; ++m) acc[m] = 0.0f;

  if (VEC) {
    // K % 8 == 0, G % 8 == 0, all rows 16-byte (x) / 4- or 8-byte (w) aligned.
    const int nchunks = K >> 3;
    const uint8_t* wrow8 = w + static_cast<long long>(row_ok ? n : 0) * (WBITS == 4 ? (K >> 1) : K);
    constexpr int PRE = 4;       // chunks per lane fetched ahead of the wait (K <= 1024 is covered whole)
    uint32_t pre_w0[PRE], pre_w1[PRE];
    float pre_sc[PRE];
#pragma unroll
    for (int j = 0; j < PRE; ++j) {
      const int c = lane + 32 * j;
      pre_w0[j] = 0u; pre_w1[j] = 0u; pre_sc[j] = 0.0f;
      if (row_ok && c < nchunks) {
        if (WBITS == 4) {
          pre_w0[j] = __ldg(reinterpret_cast<const uint32_t*>(wrow8) + c);
        } else {
          const uint2 two = __ldg(reinterpret_cast<const uint2*>(wrow8) + c);
          pre_w0[j] = two.x; pre_w1[j] = two.y;
        }
        pre_sc[j] = to_f32<ST>(__ldg(srow + (c << 3) / G));
      }
    }
    griddep_wait();
    if (!row_ok) { if (!small_grid) griddep_launch_dependents(); return; }
    auto chunk = [&](int c, uint32_t w0, uint32_t w1, float sc) {
      const int k0 = c << 3;
      float wq[8];
      if (WBITS == 4) {
#pragma unroll
        for (int i = 0; i < 8; ++i) wq[i] = small_uint_to_f32((w0 >> (4 * i)) & 15u) - 8.0f;
      } else {
        float f[4];
        int8x4_to_f32(w0, f); wq[0] = f[0]; wq[1] = f[1]; wq[2] = f[2]; wq[3] = f[3];
        int8x4_to_f32(w1, f); wq[4] = f[0]; wq[5] = f[1]; wq[6] = f[2]; wq[7] = f[3];
      }
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        if (m0 + m < M) {
          float xv[8];
          load8<XT>(x + static_cast<long long>(m0 + m) * K + k0, xv);
          float p = 0.0f;
#pragma unroll
          for (int i = 0; i < 8; ++i) p = fmaf(xv[i], wq[i], p);
          acc[m] = fmaf(sc, p, acc[m]);
        }
      }
    };
#pragma unroll
    for (int j = 0; j < PRE; ++j) {
      const int c = lane + 32 * j;
      if (c < nchunks) chunk(c, pre_w0[j], pre_w1[j], pre_sc[j]);
    }
#pragma unroll 4
    for (int c = lane + 32 * PRE; c < nchunks; c += 32) {
      uint32_t w0, w1 = 0u;
      if (WBITS == 4) {
        w0 = __ldg(reinterpret_cast<const uint32_t*>(wrow8) + c);
      } else {
        const uint2 two = __ldg(reinterpret_cast<const uint2*>(wrow8) + c);
        w0 = two.x; w1 = two.y;
      }
      chunk(c, w0, w1, to_f32<ST>(__ldg(srow + (c << 3) / G)));
    }
    if (!small_grid) griddep_launch_dependents();
  } else {
    griddep_wait();
    if (!small_grid) griddep_launch_dependents();
    if (!row_ok) return;
    if (WBITS == 4) {
      const uint8_t* wrow = w + static_cast<long long>(n) * (K >> 1);
      for (int j = lane; j < (K >> 1); j += 32) {
        const uint32_t b = __ldg(wrow + j);
        const int k0 = 2 * j, k1 = 2 * j + 1;
        const float w0 = (small_uint_to_f32(b & 15u) - 8.0f) * to_f32<ST>(__ldg(srow + k0 / G));
        const float w1 = (small_uint_to_f32(b >> 4) - 8.0f) * to_f32<ST>(__ldg(srow + k1 / G));
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          if (m0 + m < M) {
            const XT* xr = x + static_cast<long long>(m0 + m) * K;
            acc[m] = fmaf(to_f32<XT>(xr[k0]), w0, acc[m]);
            acc[m] = fmaf(to_f32<XT>(xr[k1]), w1, acc[m]);
          }
        }
      }
    } else {
      const int8_t* wrow = reinterpret_cast<const int8_t*>(w) + static_cast<long long>(n) * K;
      for (int k = lane; k < K; k += 32) {
        const float wv = static_cast<float>(__ldg(wrow + k)) * to_f32<ST>(__ldg(srow + k / G));
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          if (m0 + m < M) acc[m] = fmaf(to_f32<XT>(x[static_cast<long long>(m0 + m) * K + k]), wv, acc[m]);
        }
      }
    }
  }

#pragma unroll
  for (int m = 0; m < MT; ++m) {
    float v = acc[m];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if (lane == 0 && m0 + m < M) out[static_cast<long long>(m0 + m) * N + n] = from_f32<OT>(v);
  }
}

// Several rows of x, or one and a weight beyond 2 Mi elements; float32 math end to end: a warp owns R = 4 weight rows and MT rows of x, lanes
// stride over K in chunks of 8.  With one weight row per warp every warp re-read all of x -- M * 4 bytes of
// it from L1 per half byte of weight -- and that bound the kernel; here a chunk of x serves four rows and a
// dequantised weight MT rows of x.  `splits` warps of a block share a row group's K when N alone gives too few
// warps, and add up in shared memory.
// M = 4, K = 2176, N = 8056, int8, f16: 23.8 us before, now 10.1; M = 8, K = 8192, N = 7000, int4, f32: 129, now 57;
// M = 1, K = 8192, N = 16000, int8, f32: 56.7, now 35.1, int4 47, now 29.7.  Scales stay in their type until they are used: a conversion
// of fp16 scales between the loads held the next load up (M = 4, 640 -> 12000, int4, f16: 9.1 -> 6.6).
template <int WBITS, typename XT, typename ST, typename OT, int MT, int C>
__global__ void __launch_bounds__(256) gemv_rows_kernel(const XT* __restrict__ x, const uint8_t* __restrict__ w,
                                                        const ST* __restrict__ scales, OT* __restrict__ out,
                                                        int M, int N, int K, int G, int gshift, int split_shift) {
  constexpr int R = 4;
  __shared__ float red[8][R * MT];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int splits = 1 << split_shift, part = warp & (splits - 1);
  const int n0 = (blockIdx.x * (8 >> split_shift) + (warp >> split_shift)) * R;
  const int m0 = blockIdx.y * MT;
  const int nchunks = K >> (2 + C), ns = K / G, row_bytes = WBITS == 4 ? (K >> 1) : K;
  const uint8_t* wrow[R];
  const ST* srow[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {                // (rows past N read the last one and are not written)
    const int n = n0 + r < N ? n0 + r : N - 1;
    wrow[r] = w + static_cast<long long>(n) * row_bytes;
    srow[r] = scales + static_cast<long long>(n) * ns;
  }
  const XT* xrow[MT];
#pragma unroll
  for (int m = 0; m < MT; ++m) xrow[m] = x + static_cast<long long>(m0 + m < M ? m0 + m : M - 1) * K;
  // C = 2 (int4, one row of x; where, launch_gemv_simt says): two octets a lane and load, so that as many bytes are on their way as with int8; even and
  // odd k add up in the halves of 64-bit registers.  M = 1, f32, groups of 32, us in a CUDA graph, one octet as it was / now: 4096 -> 8192 23.1 / 10.8, 8192 ->
  // 16000 46.6 / 29.7, 3072 -> 3000 5.1 / 3.5.
  // (int8 with two octets: 4096 -> 8192 10.7 -> 9.4, but 3072 -> 3000 4.5 -> 5.5; halves with two and four rows of x cost registers: M = 2,
  // 1024 -> 12000 5.4 -> 6.0, M = 8 33 -> 39.)
  static_assert(C == 1 || (C == 2 && MT == 1 && WBITS == 4), "two octets a lane: int4, one row of x");
  constexpr bool PAIRS = C == 2;
  typedef typename RowSums<PAIRS>::type Sum;
  Sum acc[MT][R];
#pragma unroll
  for (int m = 0; m < MT; ++m) {
#pragma unroll
    for (int r = 0; r < R; ++r) acc[m][r] = 0;
  }
  constexpr int NW = C * (WBITS / 4);          // words of a chunk
  uint32_t next[R][NW];                        // the next chunk, on its way (four chunks ahead cost occupancy: 37 -> 90 us for one case)
  ST sc[R];
  const auto fetch = [&](int c) {
    if (c >= nchunks) return;
    const int g = gshift >= 0 ? (c << (2 + C)) >> gshift : (c << (2 + C)) / G;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if constexpr (NW == 1) {
        next[r][0] = __ldg(reinterpret_cast<const uint32_t*>(wrow[r]) + c);
      } else {
        const uint2 v = __ldg(reinterpret_cast<const uint2*>(wrow[r]) + c);
        next[r][0] = v.x; next[r][1] = v.y;
      }
      sc[r] = __ldg(srow[r] + g);
    }
  };
  int c = part * 32 + lane;
  fetch(c);                                    // weights are constants: ahead of the wait for the preceding kernel
  griddep_launch_dependents();
  griddep_wait();
  for (; c < nchunks; c += 32 << split_shift) {
    if constexpr (PAIRS) {
      uint32_t now[R][NW];
      float s[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        s[r] = to_f32<ST>(sc[r]);
#pragma unroll
        for (int i = 0; i < NW; ++i) now[r][i] = next[r][i];
      }
      fetch(c + (32 << split_shift));
      f32x2 p[R];
#pragma unroll
      for (int h = 0; h < C; ++h) {
        f32x2 xv[4];
        load8_pairs(xrow[0] + (c * C + h) * 8, xv);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          f32x2 wq[4];
          int4_pairs(now[r][h], wq);
          const f32x2 octet = dot8(xv, wq);
          p[r] = h == 0 ? octet : add2(p[r], octet);
        }
      }
#pragma unroll
      for (int r = 0; r < R; ++r) scaled_sum(acc[0][r], s[r], p[r]);
    } else {
      float wq[R][8], s[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        s[r] = to_f32<ST>(sc[r]);
        if (WBITS == 4) {
          int4_floats<(MT == 2 || (MT > 1 && sizeof(ST) == 4))>(next[r][0], wq[r]);
        } else {
          int8x4_to_f32(next[r][0], wq[r]);
          int8x4_to_f32(next[r][NW - 1], wq[r] + 4);
        }
      }
      fetch(c + (32 << split_shift));
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        float xv[8];
        load8<XT>(xrow[m] + (c << 3), xv);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          float p = 0.0f;
#pragma unroll
          for (int i = 0; i < 8; ++i) p = fmaf(xv[i], wq[r][i], p);
          scaled_sum(acc[m][r], s[r], p);
        }
      }
    }
  }
  // Sums over the lanes: at each step a lane gives half of its values to its partner and keeps the other half, so V
  // values take V - 1 shuffles and log2(32 / V) more instead of 5 V. The high bits of the lane number say which value
  // (index = m * R + r) it ends with; its low log2(32 / V) bits tell copies apart. M = 5, 4-bit, 1536 -> 3690:
  // 8.15 -> 7.73 us; M = 3, 1024 -> 16000: 11.70 -> 11.24 us; M = 1, 8-bit, 8192 -> 16000: 36.8 -> 35.4 us.
  constexpr int V = R * MT;
  float v[V];
#pragma unroll
  for (int i = 0; i < V; ++i) v[i] = row_sum(acc[i / R][i % R]);
  int index = 0;
#pragma unroll
  for (int h = V / 2, off = 16; h > 0; h >>= 1, off >>= 1) {
    const bool upper = lane & off;
    if (upper) index += h;
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const float keep = upper ? v[i + h] : v[i], give = upper ? v[i] : v[i + h];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, off);
    }
  }
  float mine = v[0];
#pragma unroll
  for (int off = 16 / V; off > 0; off >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, off);
  const bool writer = (lane & (32 / V - 1)) == 0;
  if (splits > 1) {
    if (writer) red[warp][index] = mine;
    __syncthreads();
    if (part != 0) return;
    if (writer) {
      for (int q = 1; q < splits; ++q) mine += red[warp + q][index];
    }
  }
  const int m = m0 + index / R, n = n0 + index % R;
  if (writer && m < M && n < N) out[static_cast<long long>(m) * N + n] = from_f32<OT>(mine);
}

template <int WBITS, typename XT, typename ST, typename OT>
int launch_gemv_simt(const void* x, const void* w, const void* s, void* out, int M, int N, int K, int G,
                     int sm_count, cudaStream_t stream) {
  if (M == 0 || N == 0) return LCQ_OK;
  const bool vec = (K % 8 == 0) && (G % 8 == 0) && aligned(x, 16) && aligned(w, WBITS == 4 ? 4 : 8);
  const XT* xp = static_cast<const XT*>(x);
  const uint8_t* wp = static_cast<const uint8_t*>(w);
  const ST* sp = static_cast<const ST*>(s);
  OT* op = static_cast<OT*>(out);
  const int rows_per_block = 8;
  const unsigned gx = (N + rows_per_block - 1) / rows_per_block;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.blockDim = dim3(256);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 1 : 0;
#define LCQ_SIMT_LAUNCH(MT_, VEC_)                                                                   \
  do {                                                                                               \
    cfg.gridDim = dim3(gx, (M + MT_ - 1) / MT_);                                                     \
    LCQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, gemv_simt_kernel<WBITS, XT, ST, OT, MT_, VEC_>, xp, wp, sp, \
                                    op, M, N, K, G));                                                \
  } while (0)
  if (vec && (M > 1 || static_cast<long long>(N) * K > (1LL << 21))) {
    // 8 warps a block; the warps of a block share K while there are too few warps an SM and each of them still has a chunk per
    // lane: 12 warps, and with one row of x more where their shares stay long: int8 24 (4096 -> 8192 with 14 warps an SM 19.0 us, with
    // 28 10.5, but 1152 -> 5000 with 17 and with 34 3.9 / 4.5), int4 32.
    int split = 0;
    const long long groups = (N + 3) / 4;
    const int mt = M == 1 ? 1 : M == 2 ? 2 : 4, m_blocks = (M + mt - 1) / mt;
    bool two = WBITS == 4 && mt == 1 && K % 16 == 0 && G % 16 == 0 && aligned(w, 8) && K > 256;
    const long long wave_two = sm_count * 24LL, wave_one = sm_count * 32LL;      // warps that are resident, two octets a lane (80 registers) and one (64)
    if (two) {
      // Two octets a lane: as many shares as still make one wave, however short (1536 -> 2800 in 2 / 4 shares 3.2 / 2.4 us, 8 are two waves: 4.0;
      // 8000 rows of 1152 in 1 / 2 4.9 / 5.7).  Long shares are worth a second wave: 8192 -> 8000 in 1 / 4 20.4 / 17.4.
      while (split < 3 && (groups << (split + 1)) <= wave_two && K >= (256 << split)) ++split;
      const int next = groups > wave_two ? 0 : split + 1;
      const bool one_wave_of_one = next <= 3 && (groups << next) > wave_two && (groups << next) <= wave_one;
      if (one_wave_of_one && K < (sizeof(XT) == 4 ? 1536 : 1024) && (next == 0 || K > 512)) {
        // One octet: a wave of it holds 4/3 of the warps.  float32, one octet in one wave / two in two: 16000 rows of 512 3.3 / 4.0, of 1152 6.9 / 7.7, of
        // 1536 8.4 / 8.3; 2000 rows of 1152 in 8 shares 1.9, two octets in 4 2.4.  float16: 16000 rows of 768 4.6 / 5.4, of 1024 6.0 / 5.4.
        two = false;
        split = next;
      } else if (sizeof(XT) == 4 && K > 512 && K <= 768 && groups > wave_one * 5 / 4) {
        two = false;                           // three rounds of one octet against two of two, the second half empty: 768 -> 50000 11.5 / 12.0
      } else {
        while (split < 3 && (groups << split) < wave_one && K >= (1792 << split)) ++split;
      }
    } else {
      const long long few = sm_count * 12LL, more = mt > 1 ? few : sm_count * (WBITS == 4 ? 32LL : 24LL);
      while (split < 3 && ((((groups * m_blocks) << split) < few && K >= (512 << split)) || (((groups * m_blocks) << split) < more && K >= (2048 << split)))) ++split;
    }
    int gshift = -1;
    if ((G & (G - 1)) == 0) { gshift = 0; while ((1 << gshift) < G) ++gshift; }
    cfg.gridDim = dim3(static_cast<unsigned>((groups + (8 >> split) - 1) / (8 >> split)), m_blocks);
    if (two) LCQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, gemv_rows_kernel<4, XT, ST, OT, 1, 2>, xp, wp, sp, op, M, N, K, G, gshift, split));
    else if (mt == 1) LCQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, gemv_rows_kernel<WBITS, XT, ST, OT, 1, 1>, xp, wp, sp, op, M, N, K, G, gshift, split));
    else if (mt == 2) LCQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, gemv_rows_kernel<WBITS, XT, ST, OT, 2, 1>, xp, wp, sp, op, M, N, K, G, gshift, split));
    else LCQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, gemv_rows_kernel<WBITS, XT, ST, OT, 4, 1>, xp, wp, sp, op, M, N, K, G, gshift, split));
  } else if (vec) {
    LCQ_SIMT_LAUNCH(1, true);
  } else {
    if (M == 1) LCQ_SIMT_LAUNCH(1, false);
    else LCQ_SIMT_LAUNCH(4, false);
  }
#undef LCQ_SIMT_LAUNCH
  return LCQ_OK;
}

}  // namespace lcq
