// What the two kernels of the KV-cached block forward share: the problem, the mask by absolute positions, and the
// combination of partial rows when the keys of a query tile are split over several CTAs.
#pragma once

#include "common.cuh"
#include "ptx.cuh"

namespace nlfa {
namespace cached {

struct CachedParams {
  int B, Tq, H, Hkv, L, D;
  int causal, window, sinks;
  float scale_log2;
  const void* qpos;      // nullptr: the block is the last Tq positions of a contiguous [0, L)
  const void* kpos;      // nullptr: contiguous
  int wide;              // positions are 64-bit integers (else 32-bit)
  int splits;            // CTAs per query tile (blockIdx.y, one cluster): each takes a share of the key blocks
  void* o;
  float* lse;            // or nullptr
  int loose;             // q or o is not 16-byte aligned (fp32 kernel only): one element at a time
};

// A position as the kernels use it; 64-bit ones are clamped into 32 bits (they are compared, and with a window
// subtracted from one another: sequence positions, far below the limits).
__device__ __forceinline__ int position(const void* p, int wide, int i) {
  if (!wide) return static_cast<const int*>(p)[i];
  const long long v = static_cast<const long long*>(p)[i];
  return v > 0x3fffffff ? 0x3fffffff : v < -0x3fffffff ? -0x3fffffff : static_cast<int>(v);
}
__device__ __forceinline__ int query_position(const CachedParams& p, int t) {
  return p.qpos ? position(p.qpos, p.wide, t) : p.L - p.Tq + t;
}
__device__ __forceinline__ int key_position(const CachedParams& p, int key) {
  return p.kpos ? position(p.kpos, p.wide, key) : key;
}

// With a window (causal by definition): kpos <= qpos and (kpos > qpos - (window - sinks) or kpos < sinks); causal:
// kpos <= qpos; otherwise every key.
__device__ __forceinline__ bool position_visible(const CachedParams& p, int qp, int kp) {
  bool vis = true;
  if (p.causal) vis = kp <= qp;
  if (p.window > 0) vis = vis && (kp > qp - (p.window - p.sinks) || kp < p.sinks);
  return vis;
}

// The key blocks of `rows` keys a tile of query positions t0 .. t1 has to visit: all of them when positions are
// given or nothing is masked, else sink blocks and the range its rows can reach.
struct KeyRange {
  int lo, extra, count;
  __host__ __device__ __forceinline__ int at(int n) const { return n < extra ? n : lo + (n - extra); }
};
__host__ __device__ inline KeyRange key_range(int Tq, int L, bool positions, int causal, int window, int sinks, int t0,
                                              int t1, int rows) {
  const int n_blocks = (L + rows - 1) / rows;
  KeyRange r{0, 0, n_blocks};
  if (positions || !causal) return r;
  const int hi = (L - Tq + t1) / rows;
  int sink_blocks = 0;
  if (window > 0) {
    const int first = L - Tq + t0 - (window - sinks) + 1;
    r.lo = first > 0 ? first / rows : 0;
    sink_blocks = (sinks + rows - 1) / rows;
  }
  r.extra = sink_blocks < r.lo ? sink_blocks : r.lo;
  r.count = r.extra + hi - r.lo + 1;
  return r;
}

// Whether every key of a block with positions [kp_min, kp_max] is visible to every query of a tile.
__device__ __forceinline__ bool all_visible(const CachedParams& p, int kp_min, int kp_max, int qp_min, int qp_max) {
  if (p.causal && kp_max > qp_min) return false;
  return p.window == 0 || kp_min > qp_max - (p.window - p.sinks) || kp_max < p.sinks;
}

template <typename T>
__device__ __forceinline__ void store4(T* dst, float4 v, bool loose = false) {
  if (loose) {
    const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) dst[i] = static_cast<T>(x[i]);
    return;
  }
  if constexpr (sizeof(T) == 4) {
    *reinterpret_cast<float4*>(dst) = v;
  } else {
    T x[4] = {static_cast<T>(v.x), static_cast<T>(v.y), static_cast<T>(v.z), static_cast<T>(v.w)};
    *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<uint2*>(x);
  }
}

// The most CTAs a query tile's keys may be split over: all clusters resident at once, `most` at most.
inline int cluster_splits(const void* kernel, int threads, int smem, long long tiles, int most) {
  if (most > kMostCluster) most = kMostCluster;
  for (int s = most; s > 1; --s)
    if (resident_clusters(kernel, threads, smem, s) >= tiles) return s;
  return 1;
}

}  // namespace cached
}  // namespace nlfa
