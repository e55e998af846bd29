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
__device__ __forceinline__ void store4(T* dst, float4 v) {
  if constexpr (sizeof(T) == 4) {
    *reinterpret_cast<float4*>(dst) = v;
  } else {
    T x[4] = {static_cast<T>(v.x), static_cast<T>(v.y), static_cast<T>(v.z), static_cast<T>(v.w)};
    *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<uint2*>(x);
  }
}

// Combines the partial rows of a query tile.  The CTAs of its cluster hold PARTS partial results each in shared
// memory: rows of D fp32 sums at a pitch of D + 4 (`rows`, `part_bytes` apart) and per row its (maximum, sum of
// exponentials) in base-2 units (`stats`, 128 rows apart).  CTA `rank` finishes rows rank, rank + splits, ..: a warp
// turns a row's maxima and sums into weights at once, then every thread adds up pieces of four columns with all
// the loads of a piece in flight.  Parts are added in order: the result does not depend on timing.  `weights` is
// room for 32 floats per own row, `sync` a barrier of the `threads` threads that take part (false: something
// gave up).  (Through global memory -- partial rows, a ticket, the last CTA combining -- this took 16 of 42 us at
// B=1 H=16 D=128, 64 queries over 16,448 keys, most of it L2 latency; a kernel of its own took 10.)
template <typename T, int D, int PARTS, class RowOf, class Sync>
__device__ __forceinline__ void merge_rows(const CachedParams& p, int n, RowOf out_row, uint32_t rows, uint32_t part_bytes,
                                           uint32_t stats, float* weights, int rank, Sync sync, int thread, int threads) {
  const int lane = thread & 31, splits = p.splits, parts = PARTS * splits;       // at most 32
  const int own = (n - rank + splits - 1) / splits;
  const uint32_t stat_addr = cluster_addr(stats, lane < parts ? lane / PARTS : 0) + (lane % PARTS) * 1024u;
  for (int i = thread >> 5; i < own; i += threads >> 5) {
    const int r = rank + i * splits;
    float2 ml = ld_cluster_f2(stat_addr + 8u * r);
    if (lane >= parts) ml = make_float2(-INFINITY, 0.f);
    float mx = ml.x;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    const float w = exp2f(ml.x - (mx == -INFINITY ? 0.f : mx));                  // a part that saw no key: 0
    float sum = w * ml.y;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    weights[32 * i + lane] = sum > 0.f ? w / sum : 0.f;                          // a row that sees no key gives zeros
    if (p.lse && lane == 0) {
      const long long row = out_row(r), t = (row / p.H) % p.Tq, h = row % p.H, b = row / (static_cast<long long>(p.H) * p.Tq);
      p.lse[(b * p.H + h) * p.Tq + t] = sum > 0.f ? (mx + log2f(sum)) * kLn2 : -INFINITY;
    }
  }
  if (!sync()) return;
  for (int i = thread; i < own * (D / 4); i += threads) {
    const int k = i / (D / 4), c = 4 * (i % (D / 4)), r = rank + k * splits;
    if (c >= p.D) continue;                                                      // head dim 32 on 64-wide tiles
    const uint32_t at = rows + (r * (D + 4) + c) * 4u;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int s = 0; s < splits; ++s) {
      const uint32_t a = cluster_addr(at, s);
#pragma unroll
      for (int x = 0; x < PARTS; ++x) {
        const float4 y = ld_cluster_f4(a + x * part_bytes);
        const float f = weights[32 * k + PARTS * s + x];
        if (f != 0.f)                                                            // (a part that saw no key left its rows unwritten)
          acc = make_float4(fmaf(f, y.x, acc.x), fmaf(f, y.y, acc.y), fmaf(f, y.z, acc.z), fmaf(f, y.w, acc.w));
      }
    }
    store4(static_cast<T*>(p.o) + out_row(r) * p.D + c, acc);
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
