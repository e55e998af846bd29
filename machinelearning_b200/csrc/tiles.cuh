// Register-tiled fp32 products over shared memory, shared by the fp32 attention kernels (simt.cu) and the fp32 form
// of the KV-cached block forward (cached.cu): 128 threads as 8 groups of 16, a group owning rows grp, grp + 8, ..,
// a thread of it the columns col, col + 16, col + 32, col + 48 of a score tile (so that its 16-byte reads along D
// fall on different banks) and D / 16 columns of an output.  Operands lie in shared memory as fp32 at a pitch of
// D + 4.
#pragma once

#include <type_traits>

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

// Sums are taken in short runs whose totals are added (eight products, the runs of a block, the blocks): the rounding error
// of one chain grows with the square root of half its length.  With chains of D products and of all keys the relative error
// against 64 bits was up to 1.35 times (attention) and 3.4 times (cached) that of the kernels with one warp lane per key;
// as it is, o of B=2 H=6/2 T=700 D=128: lanes 2.9e-7, chains 3.6e-7, runs 1.4e-7; of 64 queries over 16,448 keys at D = 128
// 3.7e-7, 9.3e-7, 2.2e-7.  RM = 8, where sums of runs would take the registers of a CTA per SM, keeps one chain over the
// keys, as the lanes had (B=8 H=12/4 T=1024 D=64: 3.3e-7, 3.3e-7, 2.7e-7).

// s[i][j] = row (grp + 8 i) of A . row (col + 16 j) of B.  Packed: even and odd elements in the two halves, D = 128 as two
// sums of 64.  At RM = 8 packed sums would take the registers of a CTA per SM: runs of eight, their halves added to one sum.
template <int D, int RM>
__device__ __forceinline__ void score_product(const float* a, const float* b, int grp, int col, float (&s)[RM][4]) {
  constexpr int kPitch = D + 4, kSpan = D < 64 ? D : 64;
  const float* ap = a + grp * kPitch;
  const float* bp = b + col * kPitch;
  auto ld2 = [](const float* p) { return *reinterpret_cast<const ulonglong2*>(p); };
  if constexpr (RM == 8) {
#pragma unroll
    for (int i = 0; i < RM; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 1
    for (int d = 0; d < D; d += 8) {
      ulonglong2 b0[4], b1[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        b0[j] = ld2(bp + 16 * j * kPitch + d);
        b1[j] = ld2(bp + 16 * j * kPitch + d + 4);
      }
#pragma unroll
      for (int i = 0; i < RM; ++i) {
        const ulonglong2 a0 = ld2(ap + 8 * i * kPitch + d), a1 = ld2(ap + 8 * i * kPitch + d + 4);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float x, y;
          unpack_f2(ffma2(a1.y, b1[j].y, ffma2(a1.x, b1[j].x, ffma2(a0.y, b0[j].y, fmul2(a0.x, b0[j].x)))), x, y);
          s[i][j] += x + y;
        }
      }
    }
    return;
  }
#pragma unroll
  for (int d0 = 0; d0 < D; d0 += kSpan) {
    uint64_t sum[RM][4];
#pragma unroll
    for (int i = 0; i < RM; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) sum[i][j] = 0ull;
#pragma unroll(RM <= 2 ? 2 : 1)
    for (int d = d0; d < d0 + kSpan; d += 8) {
      ulonglong2 b0[4], b1[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        b0[j] = ld2(bp + 16 * j * kPitch + d);
        b1[j] = ld2(bp + 16 * j * kPitch + d + 4);
      }
#pragma unroll
      for (int i = 0; i < RM; ++i) {
        const ulonglong2 a0 = ld2(ap + 8 * i * kPitch + d), a1 = ld2(ap + 8 * i * kPitch + d + 4);
#pragma unroll
        for (int j = 0; j < 4; ++j)
          sum[i][j] = fadd2(sum[i][j], ffma2(a1.y, b1[j].y, ffma2(a1.x, b1[j].x, ffma2(a0.y, b0[j].y, fmul2(a0.x, b0[j].x)))));
      }
    }
#pragma unroll
    for (int i = 0; i < RM; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float x, y;
        unpack_f2(sum[i][j], x, y);
        s[i][j] = d0 == 0 ? x + y : s[i][j] + (x + y);
      }
  }
}

// acc[i][.] = acc[i][.] mul[i] + row (grp + 8 i) of the [rows][kBN] tile w times B [kBN][D]; a thread's D / 16 columns are
// 4 col .. (per 64 columns), or 2 col .. at D = 32; `guard`: see kHidden
template <int D, int RM>
__device__ __forceinline__ void output_product(const float* w, const float* b, int grp, int col, float (&acc)[RM][D / 16],
                                               const float (&mul)[RM], bool guard) {
  constexpr int kPitch = D + 4, N = D / 16, kRun = RM == 8 ? 4 : 8;
  const float* wp = w + grp * kPPitch;
  auto columns = [&](const float* row, float (&v)[N]) {
    if constexpr (D == 32) {
      const float2 t = *reinterpret_cast<const float2*>(row + 2 * col);
      v[0] = t.x; v[1] = t.y;
    } else {
#pragma unroll
      for (int h = 0; h < D / 64; ++h) {
        const float4 t = ld4(row + 64 * h + 4 * col);
        v[4 * h] = t.x; v[4 * h + 1] = t.y; v[4 * h + 2] = t.z; v[4 * h + 3] = t.w;
      }
    }
  };
  auto product = [&](auto guarded, float (&sum)[RM][N]) {
#pragma unroll(RM <= 2 || RM == 8 ? 2 : 1)
    for (int k = 0; k < kBN; k += kRun) {
      float bv[kRun][N];
#pragma unroll
      for (int x = 0; x < kRun; ++x) columns(b + (k + x) * kPitch, bv[x]);
#pragma unroll
      for (int i = 0; i < RM; ++i) {
        float wv[kRun];
#pragma unroll
        for (int x = 0; x < kRun; x += 4) *reinterpret_cast<float4*>(wv + x) = ld4(wp + 8 * i * kPPitch + k + x);
#pragma unroll
        for (int n = 0; n < N; ++n) {
          constexpr int kPer = RM == 1 ? 2 : kRun;         // products in a chain; RM = 1 is all latency: pairs, as a tree
          float t[kRun / kPer];
#pragma unroll
          for (int x = 0; x < kRun; ++x) {
            const bool hidden = decltype(guarded)::value && __float_as_uint(wv[x]) == __float_as_uint(kHidden);
            float& c = t[x / kPer];
            if (x % kPer == 0 && RM < 8) c = hidden ? 0.f : wv[x] * bv[x][n];
            else if (x == 0) c = hidden ? sum[i][n] : fmaf(wv[0], bv[0][n], sum[i][n]);
            else c = hidden ? c : fmaf(wv[x], bv[x][n], c);
          }
          if constexpr (RM == 8) sum[i][n] = t[0];
          else if constexpr (RM == 1) sum[i][n] += (t[0] + t[1]) + (t[2] + t[3]);
          else sum[i][n] += t[0];
        }
      }
    }
  };
  auto add = [&](float (&sum)[RM][N]) {
    if (guard) product(std::true_type{}, sum);
    else product(std::false_type{}, sum);
  };
  if constexpr (RM == 8) {                                 // (sums of runs and blocks would take another CTA's registers: a chain)
#pragma unroll
    for (int i = 0; i < RM; ++i)
#pragma unroll
      for (int n = 0; n < N; ++n) acc[i][n] *= mul[i];
    add(acc);
  } else {
    float sum[RM][N];
#pragma unroll
    for (int i = 0; i < RM; ++i)
#pragma unroll
      for (int n = 0; n < N; ++n) sum[i][n] = 0.f;
    add(sum);
#pragma unroll
    for (int i = 0; i < RM; ++i)
#pragma unroll
      for (int n = 0; n < N; ++n) acc[i][n] = fmaf(acc[i][n], mul[i], sum[i][n]);
  }
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
