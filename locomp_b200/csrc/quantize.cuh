// Weight quantisers: float weights -> packed int4 (or int8) + per-group float32 scales, with the
// reference's arithmetic reproduced bit for bit.
//
// Reference behaviour (Zyora-Dev/locomp v1.0.0), all in float32:
//   style 0  examples/38_quantized_matmul.py:248-271 (quantize_int4), :274-293 (quantize_int8)
//            amax  = max |w| over the group
//            scale = amax / 7  (int8: / 127), or 1.0 when the group is all zero
//            q     = clip(rint(w / scale) + 8, 0, 15)          (int8: clip(rint(w / scale), -128, 127))
//   style 1  examples/52_dequantize.py:110-126 (quantize_int4_ref), :162-165 (int8 self-check)
//            amax  = max(max |w|, 1e-10)   (int8: no floor)
//            scale = amax / 7  (int8: / 127)
//            q     = clip(rint(w / (scale + 1e-10)) + 8, 0, 15)
//   packing  byte j of a row = q[2j] | q[2j+1] << 4  (low nibble = even k)
// rint is round-half-to-even (np.round); both divisions are IEEE float32 divisions.
//
// Streaming kernel, HBM-bound: 4 B read per weight (float32 input), 0.5 B + 4/G B written.
// One thread owns one to four octets of 8 consecutive weights (one packed 32-bit word each) and has all of them on their way before
// it starts on the first; the G/8 threads of a group combine their maxima with warp shuffles, so loads are 32 B per thread and
// stores 4 B per thread, both coalesced.  Group sizes that are not 8, 16, 32, 64, 128 or 256 take a generic
// kernel with one thread per group.
//
// The rounded quotient without dividing.  t = w * (1 / denom) differs from the IEEE quotient by less than
// 2^-22 |t| (approximate reciprocal 2^-23, product 2^-24, the quotient's own rounding 2^-24), so both round
// to the same integer unless t lies that close to a half-integer.  Adding 1.5 * 2^23 rounds t to an integer
// (to even) and leaves it in the low bits of the sum; t minus that integer is exact, and when it comes
// within the bound of 1/2 (or t is no number) the thread divides.  Dividing every weight and converting
// with rint / min / max / float-to-int instructions bound the kernel.
//
// What it measured (4096 x 14336, us a call among others over three weights): int4 from float32 48.6 before, 47.3 now (235 MB
// read, 37 MB written; floor 41.6 at 6525 GB/s), from float16 49.1 / 38.6, from bfloat16 61.4 / 47.9 (its ties: one octet in a few
// divides); int8 from float32 52.4 / 50.6, from float16 50.9 / 41.4.  Before: one wave of blocks that looped with one octet ahead,
// converted as it arrived.
#pragma once
#include "common.cuh"
#include "gemv_simt.cuh"

namespace lcq {
namespace quant {

// 8 values read once (past L1, and not kept in it), as they are stored: all loads of a thread are issued before the first conversion.
// Float32 values in one 32-byte load where they are on 32 bytes.  ld.global and volatile, not .nc: the kernel before this one may write them
// while this one is already there (load_written, dequant.cuh).
template <typename XT> struct Raw8 {           // 16-bit types
  uint4 r;
  __device__ __forceinline__ void load(const XT* p, bool) {
    asm volatile("ld.global.cs.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p) : "memory");
  }
  __device__ __forceinline__ void zero() { r = make_uint4(0u, 0u, 0u, 0u); }
  __device__ __forceinline__ void get(float (&v)[8]) const;
};
template <> __device__ __forceinline__ void Raw8<__half>::get(float (&v)[8]) const {
  const __half2* h = reinterpret_cast<const __half2*>(&r);
#pragma unroll
  for (int i = 0; i < 4; ++i) { const float2 f = __half22float2(h[i]); v[2 * i] = f.x; v[2 * i + 1] = f.y; }
}
template <> __device__ __forceinline__ void Raw8<__nv_bfloat16>::get(float (&v)[8]) const {
  const uint32_t* u = reinterpret_cast<const uint32_t*>(&r);
#pragma unroll
  for (int i = 0; i < 4; ++i) { v[2 * i] = __uint_as_float(u[i] << 16); v[2 * i + 1] = __uint_as_float(u[i] & 0xFFFF0000u); }
}
template <> struct Raw8<float> {
  float f[8];
  __device__ __forceinline__ void load(const float* p, bool on_32) {
    if (on_32) {
      asm volatile("ld.global.L1::no_allocate.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                   : "=f"(f[0]), "=f"(f[1]), "=f"(f[2]), "=f"(f[3]), "=f"(f[4]), "=f"(f[5]), "=f"(f[6]), "=f"(f[7]) : "l"(p) : "memory");
    } else {
      asm volatile("ld.global.cs.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(f[0]), "=f"(f[1]), "=f"(f[2]), "=f"(f[3]) : "l"(p) : "memory");
      asm volatile("ld.global.cs.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(f[4]), "=f"(f[5]), "=f"(f[6]), "=f"(f[7]) : "l"(p + 4) : "memory");
    }
  }
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = 0.0f;
  }
  __device__ __forceinline__ void get(float (&v)[8]) const {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = f[i];
  }
};

__device__ __forceinline__ float group_scale(float amax, float qmax, int style, int wbits) {
  if (style == 0) return amax > 0.0f ? __fdiv_rn(amax, qmax) : 1.0f;
  if (wbits == 4) amax = fmaxf(amax, 1e-10f);
  return __fdiv_rn(amax, qmax);
}
__device__ __forceinline__ float group_denom(float scale, int style) {
  return style == 0 ? scale : __fadd_rn(scale, 1e-10f);
}
__device__ __forceinline__ uint32_t q4(float w, float denom) {
  const float r = rintf(__fdiv_rn(w, denom)) + 8.0f;
  return static_cast<uint32_t>(fminf(fmaxf(r, 0.0f), 15.0f));
}
__device__ __forceinline__ int q8(float w, float denom) {
  const float r = rintf(__fdiv_rn(w, denom));
  return static_cast<int>(fminf(fmaxf(r, -128.0f), 127.0f));
}

constexpr float ROUND_MAGIC = 12582912.0f;    // 1.5 * 2^23
// 1/2 minus a bound on |t - quotient|: |t| < 7.5 * 2^-22 = 1.8e-6 for int4, 127.5 * 2^-22 = 3.1e-5 for int8
template <int WBITS> __device__ __forceinline__ constexpr float round_limit() { return WBITS == 4 ? 0.5f - 4e-6f : 0.5f - 6e-5f; }
__device__ __forceinline__ float approx_rcp(float v) {
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}

// bits[i] = 0x4B400000 + q[i] (two's complement) as the bytes that are stored: one word (int4) or two (int8).
template <int WBITS>
__device__ __forceinline__ uint2 pack_octet(const uint32_t (&bits)[8]) {
  uint2 out = make_uint2(0u, 0u);
  if (WBITS == 4) {
    uint32_t word = 0;                        // sum of (0x4B400000 + q + 8) << 4 i, less the constant part
#pragma unroll
    for (int i = 7; i >= 0; --i) word = (word << 4) + bits[i];
    out.x = word - 0x4B400000u * 0x11111111u + 0x88888888u;
  } else {
    out.x = __byte_perm(__byte_perm(bits[0], bits[1], 0x0040), __byte_perm(bits[2], bits[3], 0x0040), 0x5410);
    out.y = __byte_perm(__byte_perm(bits[4], bits[5], 0x0040), __byte_perm(bits[6], bits[7], 0x0040), 0x5410);
  }
  return out;
}

template <int WBITS>
__device__ __forceinline__ uint2 quantize_octet(const float (&v)[8], float amax, float denom) {
  const float inv = approx_rcp(denom);
  // Outside this range the reciprocal may overflow, underflow or be flushed, and a quotient may need clipping;
  // inside it |quotient| <= 7 (127) but for the last bit.
  const bool plain = amax > 1e-30f && amax < 1e30f;
  bool sure = plain;
  uint32_t bits[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float t = v[i] * inv;
    const float m = t + ROUND_MAGIC;
    sure = sure && fabsf(t - (m - ROUND_MAGIC)) < round_limit<WBITS>();
    bits[i] = __float_as_uint(m);
  }
  if (!sure) {
    // (16-bit weights meet exact half-integers often: a scale that is a few bits long does it)
    bool numbers = plain;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float t = __fdiv_rn(v[i], denom);
      numbers = numbers && fabsf(t) < 130.0f;
      bits[i] = __float_as_uint(t + ROUND_MAGIC);
    }
    if (!numbers) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        bits[i] = 0x4B400000u + (WBITS == 4 ? q4(v[i], denom) - 8u : static_cast<uint32_t>(q8(v[i], denom)));
    }
  }
  return pack_octet<WBITS>(bits);
}

// Fast path: G in {8, ..., 256} (a power of two), K % 8 == 0, rows 16-byte aligned.
// total_oct = N*K/8 octets; octet e belongs to group e / (G/8).
// U octets a thread.
template <typename XT, int WBITS, int U>
__global__ void __launch_bounds__(256) quantize_octets_kernel(const XT* w, uint8_t* q, float* scales, long long total_oct,
                                                              int group_shift, int style, bool on_32) {
  griddep_wait();                              // (no early start for the next kernel, which may be a linear layer with these weights, see WaitingLaunch)
  const int lanes_per_group = 1 << group_shift;
  // whole blocks iterate together so the shuffles below are convergent
  for (long long first = static_cast<long long>(blockIdx.x) * (256 * U); first < total_oct; first += static_cast<long long>(gridDim.x) * (256 * U)) {
    Raw8<XT> raw[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long e = first + u * 256 + threadIdx.x;
      if (e < total_oct) raw[u].load(w + e * 8, on_32);
      else raw[u].zero();
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long e = first + u * 256 + threadIdx.x;
      float v[8];
      raw[u].get(v);
      float amax = 0.0f;
#pragma unroll
      for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(v[i]));
      for (int off = 1; off < lanes_per_group; off <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
      const float scale = group_scale(amax, WBITS == 4 ? 7.0f : 127.0f, style, WBITS);
      if (e >= total_oct) continue;
      if ((e & (lanes_per_group - 1)) == 0) scales[e >> group_shift] = scale;
      const uint2 out = quantize_octet<WBITS>(v, amax, group_denom(scale, style));
      if (WBITS == 4) reinterpret_cast<uint32_t*>(q)[e] = out.x;
      else reinterpret_cast<uint2*>(q)[e] = out;
    }
  }
}

// Generic path: one thread per group, any G dividing K (G even for int4).
template <typename XT, int WBITS>
__global__ void __launch_bounds__(256) quantize_groups_kernel(const XT* __restrict__ w, uint8_t* __restrict__ q,
                                                              float* __restrict__ scales, long long total_groups,
                                                              int G, int style) {
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  for (long long g = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; g < total_groups; g += stride) {
    const XT* src = w + g * G;
    float amax = 0.0f;
    for (int i = 0; i < G; ++i) amax = fmaxf(amax, fabsf(to_f32<XT>(src[i])));
    const float scale = group_scale(amax, WBITS == 4 ? 7.0f : 127.0f, style, WBITS);
    const float denom = group_denom(scale, style);
    scales[g] = scale;
    if (WBITS == 4) {
      uint8_t* dst = q + g * (G / 2);
      for (int i = 0; i < G; i += 2)
        dst[i / 2] = static_cast<uint8_t>(q4(to_f32<XT>(src[i]), denom) | (q4(to_f32<XT>(src[i + 1]), denom) << 4));
    } else {
      int8_t* dst = reinterpret_cast<int8_t*>(q) + g * G;
      for (int i = 0; i < G; ++i) dst[i] = static_cast<int8_t>(q8(to_f32<XT>(src[i]), denom));
    }
  }
}

template <typename XT, int WBITS>
int launch_quantize(const void* w, void* q, void* scales, long long N, long long K, int G, int style, int sm_count,
                    cudaStream_t st) {
  const long long total = N * K;
  if (total == 0) return LCQ_OK;
  const bool pow2 = G >= 8 && G <= 256 && (G & (G - 1)) == 0;
  const bool fast = pow2 && aligned(w, 16) && aligned(q, 8) && ((K * sizeof(XT)) % 16 == 0);
  if (fast) {
    const long long oct = total / 8;
    int shift = 0;
    while ((8 << shift) < G) ++shift;
    // Octets a thread: two of 16-bit weights (1 / 2 / 4: float16 42.9 / 38.6 / 37.9 us, bfloat16 52.7 / 47.9 / 48.2, 4096 x 14336, int4).  Float32
    // weights: one up to 32 Mi weights, where four make few and long blocks that leave SMs idle (int4, one / four: 192 x 576 1.33 / 2.40, 1536 x 576
    // 2.43 / 3.37, 2048 x 2048 4.89 / 6.28, 3000 x 4096 10.7 / 11.8, 7000 x 4096 22.4 / 22.8, 8192 x 4096 26.0 / 26.2), and four beyond (10240 x 4096 32.8 / 32.0,
    // 4096 x 14336 48.2 / 47.3).
    constexpr int FEW = sizeof(XT) == 4 ? 1 : 2, MANY = sizeof(XT) == 4 ? 4 : 2;
    const bool many = total > (1LL << 25);
    const long long per_block = 256 * (many ? MANY : FEW), need = (oct + per_block - 1) / per_block;
    const int grid = static_cast<int>(need < (1 << 30) ? need : (1 << 30));
    const WaitingLaunch launch(grid, 256, st);
    auto kern = many ? quantize_octets_kernel<XT, WBITS, MANY> : quantize_octets_kernel<XT, WBITS, FEW>;
    LCQ_CUDA_TRY(cudaLaunchKernelEx(&launch.cfg, kern, static_cast<const XT*>(w), static_cast<uint8_t*>(q), static_cast<float*>(scales), oct, shift, style, aligned(w, 32)));
  } else {
    const long long groups = total / G;
    long long blocks = (groups + 255) / 256;
    if (blocks > static_cast<long long>(sm_count) * 16) blocks = static_cast<long long>(sm_count) * 16;
    quantize_groups_kernel<XT, WBITS><<<static_cast<int>(blocks), 256, 0, st>>>(
        static_cast<const XT*>(w), static_cast<uint8_t*>(q), static_cast<float*>(scales), groups, G, style);
  }
  LCQ_CUDA_TRY(cudaGetLastError());
  return LCQ_OK;
}

}  // namespace quant
}  // namespace lcq
