// Streaming dequantize kernels: packed int4 / int8 weights -> f32 / f16 / bf16.
//
// Reference behaviour: examples/52_dequantize.py:27-53 (int4) and :60-74 (int8):
//   out[r, 2j]   = (float(b & 15) - 8) * scales[r, 2j / G]
//   out[r, 2j+1] = (float(b >> 4) - 8) * scales[r, (2j+1) / G]
// Because K % G == 0, the scale of flat element e = r*K + k is scales_flat[e / G], so the
// fast paths index everything flat and never need the row.
//
// HBM-bound (write dominated: 4 B out per 0.5 B in for f32).  The fast path gives a thread whole octets of weights: one word
// (int4) or two (int8) in, one scale, and one store of 32 bytes (f32) or 16 (16-bit outputs).
//
// What it measured (4096 x 14336, us a call among others over three weights; floor 41.1 for int4 -> f32 at 6525 GB/s): int4 -> f32 49.0
// before, 41.4 now, -> f16 32.7 / 27.0; int8 -> f32 56.1 / 46.3, -> f16 41.5 / 28.9.  Before: one wave of blocks that looped, int4
// words spread over the lanes by shuffles to get 16-byte stores, int8 one word a thread.  What gave it: blocks that end
// after one round of loads and stores instead of looping (a loop's next loads wait behind its stores; 53 -> 43 in a kernel by
// itself), fp16 scales converted only after all loads are issued (33.6 -> 27.0 for f16 outputs), and the programmatic attribute, without
// which a launch starts up to 2 us late whatever is in front of it (-2).  Octets a thread: f32 1 / 2 / 4 46.5 / 41.6 / 41.6, f16 1 / 2 / 4 39.2 / 29.4 / 27.0.
#pragma once
#include "common.cuh"

namespace lcq {

// Launch of a kernel that waits for its predecessor itself (griddep_wait before its first access).  Behind a kernel that lets its successor start
// early its blocks are there when that one ends; behind any other the attribute saves the up to 2 us by which a launch without it starts late.
// A kernel that writes packed weights or scales does not let its own successor start early (griddep_launch_dependents): a linear layer's kernel fetches
// those without waiting, and would do so while they are being written.  That does not free the caller from synchronising between writing
// weights and the first call of the layer (locomp_b200.h): that the stores of blocks which have ended are visible to a fetch ahead of the wait is not specified.
struct WaitingLaunch {
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[1];
  WaitingLaunch(int grid, int block, cudaStream_t stream) {
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.stream = stream;
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 1 : 0;
  }
  WaitingLaunch(const WaitingLaunch&) = delete;
};

template <typename OT> struct Out4;   // 4 consecutive outputs, one vector store
template <> struct Out4<float> {
  static __device__ __forceinline__ void store(float* p, float a, float b, float c, float d) {
    __stcs(reinterpret_cast<float4*>(p), make_float4(a, b, c, d));
  }
};
template <> struct Out4<__half> {
  static __device__ __forceinline__ void store(__half* p, float a, float b, float c, float d) {
    __half2 lo = __floats2half2_rn(a, b), hi = __floats2half2_rn(c, d);
    uint2 v = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
    __stcs(reinterpret_cast<uint2*>(p), v);
  }
};
template <> struct Out4<__nv_bfloat16> {
  static __device__ __forceinline__ void store(__nv_bfloat16* p, float a, float b, float c, float d) {
    __nv_bfloat162 lo = __floats2bfloat162_rn(a, b), hi = __floats2bfloat162_rn(c, d);
    uint2 v = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
    __stcs(reinterpret_cast<uint2*>(p), v);
  }
};

// Index of the scale of flat element e: a shift when G is a power of two (gshift >= 0), else a division.
__device__ __forceinline__ long long scale_index(long long e, int G, int gshift) {
  return gshift >= 0 ? (e >> gshift) : (e / G);
}

// 8 consecutive outputs: one 16-byte store of 16-bit values, one of 32 bytes of float32 values (or, where out is on 16 bytes only, two of 16).
template <typename OT> struct Out8;
template <> struct Out8<float> {
  static __device__ __forceinline__ void store(float* p, const float (&f)[8], bool on_32) {
    if (on_32) {
      asm volatile("st.global.L1::no_allocate.L2::evict_first.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                   ::"l"(p), "f"(f[0]), "f"(f[1]), "f"(f[2]), "f"(f[3]), "f"(f[4]), "f"(f[5]), "f"(f[6]), "f"(f[7]) : "memory");
    } else {
      Out4<float>::store(p, f[0], f[1], f[2], f[3]);
      Out4<float>::store(p + 4, f[4], f[5], f[6], f[7]);
    }
  }
};
template <> struct Out8<__half> {
  static __device__ __forceinline__ void store(__half* p, const float (&f)[8], bool) {
    __half2 h[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2half2_rn(f[2 * i], f[2 * i + 1]);
    __stcs(reinterpret_cast<uint4*>(p), *reinterpret_cast<const uint4*>(h));
  }
};
template <> struct Out8<__nv_bfloat16> {
  static __device__ __forceinline__ void store(__nv_bfloat16* p, const float (&f)[8], bool) {
    __nv_bfloat162 h[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
    __stcs(reinterpret_cast<uint4*>(p), *reinterpret_cast<const uint4*>(h));
  }
};

// float(int8) for the 4 bytes of a word without conversion instructions.
__device__ __forceinline__ void int8x4_to_f32(uint32_t v, float* f) {
  v ^= 0x80808080u;  // bias to unsigned: b + 128
  f[0] = __uint_as_float(__byte_perm(v, 0x4B000000u, 0x7540)) - 8388736.0f;
  f[1] = __uint_as_float(__byte_perm(v, 0x4B000000u, 0x7541)) - 8388736.0f;
  f[2] = __uint_as_float(__byte_perm(v, 0x4B000000u, 0x7542)) - 8388736.0f;
  f[3] = __uint_as_float(__byte_perm(v, 0x4B000000u, 0x7543)) - 8388736.0f;
}

// Loads of what the kernel before this one may have written while this one was already there (WaitingLaunch): ld.global, since ld.global.nc
// is for memory that nobody writes during the life of the kernel that reads, and volatile, so that none moves ahead of griddep_wait.
__device__ __forceinline__ uint32_t load_written(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint2 load_written(const uint2* p) {
  uint2 v;
  asm volatile("ld.global.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ float load_written(const float* p) { return __uint_as_float(load_written(reinterpret_cast<const uint32_t*>(p))); }
__device__ __forceinline__ unsigned short load_written(const unsigned short* p) {
  unsigned short v;
  asm volatile("ld.global.u16 %0, [%1];" : "=h"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ __half load_written(const __half* p) { return __ushort_as_half(load_written(reinterpret_cast<const unsigned short*>(p))); }
__device__ __forceinline__ __nv_bfloat16 load_written(const __nv_bfloat16* p) {
  return __ushort_as_bfloat16(load_written(reinterpret_cast<const unsigned short*>(p)));
}

// The 8 weights of an octet as they are stored: one word (int4), two (int8).
template <int WBITS> struct Octet;
template <> struct Octet<4> {
  uint32_t v;
  __device__ __forceinline__ void load(const void* w, long long i) { v = load_written(static_cast<const uint32_t*>(w) + i); }
  __device__ __forceinline__ void scaled(float s, float (&f)[8]) const {
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = (small_uint_to_f32((v >> (4 * i)) & 15u) - 8.0f) * s;
  }
};
template <> struct Octet<8> {
  uint2 v;
  __device__ __forceinline__ void load(const void* w, long long i) { v = load_written(static_cast<const uint2*>(w) + i); }
  __device__ __forceinline__ void scaled(float s, float (&f)[8]) const {
    int8x4_to_f32(v.x, f);
    int8x4_to_f32(v.y, f + 4);
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] *= s;
  }
};

// ---- fast path: K % 8 == 0, G % 8 == 0, w on the size of an octet and out on 16 bytes.  A thread has dq_unroll<OT>() octets, a block's
// width apart, and loads all of them and their scales before its first conversion.  (The loop is for more octets than a grid has
// threads; ordinary sizes take one round.)
template <typename OT> __host__ __device__ constexpr int dq_unroll() { return sizeof(OT) == 4 ? 2 : 4; }
template <int WBITS, typename ST, typename OT>
__global__ void __launch_bounds__(256) dequant_octets_kernel(const void* w, const ST* scales, OT* out,
                                                             long long octets, int G, int gshift, bool on_32) {
  constexpr int U = dq_unroll<OT>();
  griddep_wait();                              // (no early start for the next kernel: the outputs may be a linear layer's scales, see WaitingLaunch)
  for (long long i0 = static_cast<long long>(blockIdx.x) * (256 * U) + threadIdx.x; i0 < octets; i0 += static_cast<long long>(gridDim.x) * (256 * U)) {
    Octet<WBITS> q[U];
    ST s[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long i = i0 + u * 256;
      if (i < octets) {
        q[u].load(w, i);
        s[u] = load_written(scales + scale_index(i * 8, G, gshift));
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long i = i0 + u * 256;
      if (i < octets) {
        float f[8];
        q[u].scaled(to_f32<ST>(s[u]), f);
        Out8<OT>::store(out + i * 8, f, on_32);
      }
    }
  }
}

// ---- int4 generic path: one thread per packed byte; any even K, any G dividing K.
template <typename ST, typename OT>
__global__ void __launch_bounds__(256) dequant_w4_bytes_kernel(const uint8_t* __restrict__ w,
                                                               const ST* __restrict__ scales,
                                                               OT* __restrict__ out,
                                                               long long total_bytes, int K, int G) {
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  const int half_k = K >> 1, ns = K / G;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < total_bytes; i += stride) {
    const long long r = i / half_k;
    const int j = static_cast<int>(i - r * half_k);
    const uint32_t b = __ldg(w + i);
    const int k0 = 2 * j, k1 = 2 * j + 1;
    const float s0 = to_f32<ST>(__ldg(scales + r * ns + k0 / G));
    const float s1 = to_f32<ST>(__ldg(scales + r * ns + k1 / G));
    out[r * K + k0] = from_f32<OT>((small_uint_to_f32(b & 15u) - 8.0f) * s0);
    out[r * K + k1] = from_f32<OT>((small_uint_to_f32(b >> 4) - 8.0f) * s1);
  }
}

// ---- int8, K % 4 == 0, G % 4 == 0: one 32-bit word (4 weights) per thread and load.
template <typename ST, typename OT>
__global__ void __launch_bounds__(256) dequant_w8_words_kernel(const uint32_t* __restrict__ w,
                                                               const ST* __restrict__ scales,
                                                               OT* __restrict__ out,
                                                               long long total_words, int G, int gshift) {
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < total_words; i += stride) {
    const float s = to_f32<ST>(__ldg(scales + scale_index(i * 4, G, gshift)));
    float f[4];
    int8x4_to_f32(__ldg(w + i), f);
    Out4<OT>::store(out + i * 4, f[0] * s, f[1] * s, f[2] * s, f[3] * s);
  }
}

// ---- int8 generic path: one thread per weight.
template <typename ST, typename OT>
__global__ void __launch_bounds__(256) dequant_w8_elems_kernel(const int8_t* __restrict__ w,
                                                               const ST* __restrict__ scales,
                                                               OT* __restrict__ out,
                                                               long long total, int K, int G) {
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  const int ns = K / G;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += stride) {
    const long long r = i / K;
    const int k = static_cast<int>(i - r * K);
    const float sc = to_f32<ST>(__ldg(scales + r * ns + k / G));
    out[i] = from_f32<OT>(static_cast<float>(__ldg(w + i)) * sc);
  }
}

// Blocks of `kern` (256 threads, no dynamic shared memory) that are resident on the whole GPU at
// once: the grid-stride kernels are launched with exactly one wave, never more blocks than work.
template <auto kern>
int one_wave_grid(long long work_items, int per_block, int sm_count) {
  static thread_local int per_sm = 0;      // per (thread, kernel): the kernel is a template VALUE, not its type
  if (per_sm == 0) {
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, 256, 0) != cudaSuccess || nb < 1) nb = 4;
    per_sm = nb;
  }
  long long need = (work_items + per_block - 1) / per_block;
  const long long cap = static_cast<long long>(sm_count) * per_sm;
  if (need < 1) need = 1;
  return static_cast<int>(need < cap ? need : cap);
}

template <typename ST, typename OT>
int launch_dequant(int wbits, const void* w, const void* scales, void* out, long long N, long long K, int G,
                   int sm_count, cudaStream_t stream) {
  const long long total = N * K;
  if (total == 0) return LCQ_OK;
  const size_t out_vec_align = 4 * sizeof(OT);
  int gshift = -1;
  if (G > 0 && (G & (G - 1)) == 0) { gshift = 0; while ((1 << gshift) < G) ++gshift; }
  if (K % 8 == 0 && G % 8 == 0 && aligned(w, wbits) && aligned(out, 16)) {
    const long long octets = total / 8, per_block = 256 * dq_unroll<OT>(), need = (octets + per_block - 1) / per_block;
    const int grid = static_cast<int>(need < (1 << 30) ? need : (1 << 30));
    auto kern = wbits == 4 ? dequant_octets_kernel<4, ST, OT> : dequant_octets_kernel<8, ST, OT>;
    const WaitingLaunch launch(grid, 256, stream);
    LCQ_CUDA_TRY(cudaLaunchKernelEx(&launch.cfg, kern, w, static_cast<const ST*>(scales), static_cast<OT*>(out), octets, G, gshift, aligned(out, 32)));
  } else if (wbits == 4) {
    const long long bytes = total / 2;
    const int grid = one_wave_grid<dequant_w4_bytes_kernel<ST, OT>>(bytes, 256, sm_count);
    dequant_w4_bytes_kernel<ST, OT><<<grid, 256, 0, stream>>>(
        static_cast<const uint8_t*>(w), static_cast<const ST*>(scales), static_cast<OT*>(out), bytes,
        static_cast<int>(K), G);
  } else {
    const bool fast = (K % 4 == 0) && (G % 4 == 0) && aligned(w, 4) && aligned(out, out_vec_align);
    if (fast) {
      const long long words = total / 4;
      const int grid = one_wave_grid<dequant_w8_words_kernel<ST, OT>>(words, 256, sm_count);
      dequant_w8_words_kernel<ST, OT><<<grid, 256, 0, stream>>>(
          static_cast<const uint32_t*>(w), static_cast<const ST*>(scales), static_cast<OT*>(out), words, G, gshift);
    } else {
      const int grid = one_wave_grid<dequant_w8_elems_kernel<ST, OT>>(total, 256, sm_count);
      dequant_w8_elems_kernel<ST, OT><<<grid, 256, 0, stream>>>(
          static_cast<const int8_t*>(w), static_cast<const ST*>(scales), static_cast<OT*>(out), total,
          static_cast<int>(K), G);
    }
  }
  LCQ_CUDA_TRY(cudaGetLastError());
  return LCQ_OK;
}

}  // namespace lcq
