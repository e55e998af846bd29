// Register-tiled fp32 products over shared memory, shared by the fp32 attention kernels (simt.cu) and the fp32 form
// of the KV-cached block forward (cached.cu): 128 threads as 8 groups of 16, a group owning rows grp, grp + 8, ..,
// a thread of it the columns col, col + 16, col + 32, col + 48 of a score tile (so that its 16-byte reads along D
// fall on different banks) and D / 16 columns of an output.  Operands lie in shared memory as fp32 at a pitch of
// D + 4.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "ptx.cuh"

namespace nlfa {
namespace tiles {

constexpr int kThreads = 128;
constexpr int kBN = 64;                    // rows of a streamed tile
constexpr int kPPitch = kBN + 16;          // row pitch of the probability tile: neighbouring rows 16 banks apart

template <typename T>
__device__ __forceinline__ float to_f32(T x);
template <>
__device__ __forceinline__ float to_f32<float>(float x) { return x; }
template <>
__device__ __forceinline__ float to_f32<__half>(__half x) { return __half2float(x); }
template <>
__device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 x) { return __bfloat162float(x); }

template <typename T>
__device__ __forceinline__ T from_f32(float x);
template <>
__device__ __forceinline__ float from_f32<float>(float x) { return x; }
template <>
__device__ __forceinline__ __half from_f32<__half>(float x) { return __float2half_rn(x); }
template <>
__device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }

// `rows` rows of D values, `stride` elements apart, into shared memory as fp32 at a pitch of D + 4; rows from
// `valid` on become zeros.  fp32 goes by asynchronous copies (the caller commits and waits), 16-bit types are
// converted on the way.
template <typename T, int D>
__device__ __forceinline__ void load_rows(float* dst, const T* src, long long stride, int rows, int valid) {
  constexpr int kPitch = D + 4;
  if constexpr (sizeof(T) == 4) {
    constexpr int V = D / 4;
    for (int i = threadIdx.x; i < rows * V; i += kThreads) {
      const int r = i / V, c = 4 * (i % V);
      const bool in = r < valid;
      const T* s = in ? src + r * stride + c : src;
      const int bytes = in ? 16 : 0;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                   ::"r"(smem_u32(dst + r * kPitch + c)), "l"(s), "r"(bytes) : "memory");
    }
  } else {
    constexpr int V = D / 8;
    for (int i = threadIdx.x; i < rows * V; i += kThreads) {
      const int r = i / V, c = 8 * (i % V);
      uint4 w = make_uint4(0u, 0u, 0u, 0u);
      if (r < valid) w = *reinterpret_cast<const uint4*>(src + r * stride + c);
      T x[8];
      *reinterpret_cast<uint4*>(x) = w;
      float* d = dst + r * kPitch + c;
      *reinterpret_cast<float4*>(d) = make_float4(to_f32(x[0]), to_f32(x[1]), to_f32(x[2]), to_f32(x[3]));
      *reinterpret_cast<float4*>(d + 4) = make_float4(to_f32(x[4]), to_f32(x[5]), to_f32(x[6]), to_f32(x[7]));
    }
  }
}
__device__ __forceinline__ void load_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void load_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Pairs the mask hides must not touch an output, whatever stands in the hidden rows: a weight of zero does not do where
// the other factor is infinite or NaN.  Hidden weights are therefore written as -0 (a visible one never is: kHidden),
// and when a tile of a cut block holds such a value the output product leaves them out one by one (GUARD).  A
// thread looks through what it loaded itself, so the check needs no barrier of its own: cut blocks only, a few per cent.
constexpr float kHidden = -0.f;
template <typename T, int D>
__device__ __forceinline__ bool own_rows_finite(const float* tile, int rows) {
  constexpr int kPitch = D + 4, V = sizeof(T) == 4 ? D / 4 : D / 8;                // as load_rows shares them out
  float z = 0.f;
  for (int i = threadIdx.x; i < rows * V; i += kThreads) {
    const float* p = tile + (i / V) * kPitch + (D / V) * (i % V);
#pragma unroll
    for (int c = 0; c < D / V; c += 4) {
      const float4 x = ld4(p + c);
      z = fmaf(x.x, 0.f, fmaf(x.y, 0.f, fmaf(x.z, 0.f, fmaf(x.w, 0.f, z))));       // NaN once anything is not finite
    }
  }
  return z == z;
}

// s[i][j] = row (grp + 8 i) of A . row (col + 16 j) of B
template <int D, int RM>
__device__ __forceinline__ void score_product(const float* a, const float* b, int grp, int col, float (&s)[RM][4]) {
  constexpr int kPitch = D + 4;
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
  const float* ap = a + grp * kPitch;
  const float* bp = b + col * kPitch;
#pragma unroll 2
  for (int d = 0; d < D; d += 4) {
    float4 bv[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) bv[j] = ld4(bp + 16 * j * kPitch + d);
#pragma unroll
    for (int i = 0; i < RM; ++i) {
      const float4 av = ld4(ap + 8 * i * kPitch + d);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        s[i][j] = fmaf(av.w, bv[j].w, fmaf(av.z, bv[j].z, fmaf(av.y, bv[j].y, fmaf(av.x, bv[j].x, s[i][j]))));
    }
  }
}

// acc[i][.] += row (grp + 8 i) of the [rows][kBN] tile w times B [kBN][D]; a thread's D / 16 columns are 4 col ..
// (per 64 columns), or 2 col .. at D = 32; `guard`: see kHidden
template <int D, int RM, bool GUARD = false>
__device__ __forceinline__ void output_product(const float* w, const float* b, int grp, int col, float (&acc)[RM][D / 16]) {
  constexpr int kPitch = D + 4;
  const float* wp = w + grp * kPPitch;
#pragma unroll 2
  for (int k = 0; k < kBN; k += 4) {
    float wv[RM][4];
#pragma unroll
    for (int i = 0; i < RM; ++i) {
      const float4 t = ld4(wp + 8 * i * kPPitch + k);
      wv[i][0] = t.x; wv[i][1] = t.y; wv[i][2] = t.z; wv[i][3] = t.w;
    }
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      float bv[D / 16];
      const float* row = b + (k + x) * kPitch;
      if constexpr (D == 32) {
        const float2 t = *reinterpret_cast<const float2*>(row + 2 * col);
        bv[0] = t.x; bv[1] = t.y;
      } else {
#pragma unroll
        for (int h = 0; h < D / 64; ++h) {
          const float4 t = ld4(row + 64 * h + 4 * col);
          bv[4 * h] = t.x; bv[4 * h + 1] = t.y; bv[4 * h + 2] = t.z; bv[4 * h + 3] = t.w;
        }
      }
#pragma unroll
      for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int n = 0; n < D / 16; ++n)
          if (!GUARD || __float_as_uint(wv[i][x]) != __float_as_uint(kHidden)) acc[i][n] = fmaf(wv[i][x], bv[n], acc[i][n]);
    }
  }
}

template <int D, int RM>
__device__ __forceinline__ void output_product(const float* w, const float* b, int grp, int col, float (&acc)[RM][D / 16],
                                               bool guard) {
  if (guard) output_product<D, RM, true>(w, b, grp, col, acc);
  else output_product<D, RM, false>(w, b, grp, col, acc);
}

// one thread's D / 16 columns of an output row, times `mul`
template <typename T, int D>
__device__ __forceinline__ void store_row(T* row, int col, const float (&acc)[D / 16], float mul) {
  if constexpr (D == 32) {
    T x[2] = {from_f32<T>(acc[0] * mul), from_f32<T>(acc[1] * mul)};
    if constexpr (sizeof(T) == 4) *reinterpret_cast<float2*>(row + 2 * col) = make_float2(x[0], x[1]);
    else *reinterpret_cast<uint32_t*>(row + 2 * col) = *reinterpret_cast<uint32_t*>(x);
  } else {
#pragma unroll
    for (int h = 0; h < D / 64; ++h) {
      T x[4];
#pragma unroll
      for (int n = 0; n < 4; ++n) x[n] = from_f32<T>(acc[4 * h + n] * mul);
      if constexpr (sizeof(T) == 4) *reinterpret_cast<float4*>(row + 64 * h + 4 * col) = make_float4(x[0], x[1], x[2], x[3]);
      else *reinterpret_cast<uint2*>(row + 64 * h + 4 * col) = *reinterpret_cast<uint2*>(x);
    }
  }
}

}  // namespace tiles
}  // namespace nlfa
