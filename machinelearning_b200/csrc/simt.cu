// fp32 attention kernels on the FMA pipe: the accuracy path (fp32 inputs need 1e-5), for every dtype and head dim.
//
// Register-tiled: a CTA of 128 threads owns BM = 8 RM rows (queries in the forward and in dQ, keys in dK/dV) and
// streams tiles of 64 rows of the other side past them through shared memory, everything held as fp32.  The threads
// form 8 groups of 16: a group owns RM rows, a thread of it the columns c, c + 16, c + 32, c + 48 of a score tile
// (so that its 16-byte reads along D fall on different banks) and D / 16 columns of an output.  A score product
// takes RM + 4 vector loads for 16 RM multiply-adds: at RM = 8 the FMA pipe, not shared memory, is the bound.
// The group's probabilities go through shared memory to become the other operand of the output product; only the
// warp's own rows are involved, so that exchange needs no CTA-wide barrier.  No atomics: bit-reproducible.
//
// RM = 8, 4 or 2 by the number of row tiles (rows_per_thread).  The dQ pass runs beside the dK/dV pass.
// Measured, a row per warp before -> tiles: B=4 H=4 T=256 D=64 forward 82 -> 16 us, backward 174 -> 34 us
// (latency); B=8 H=12/4 T=2048 D=64 forward 14.9 -> 1.49 ms (35 TFLOP/s, half of
// what the FMA pipe can issue), backward 32.0 -> 4.63 ms.
//
// Algebra follows the reference's FMA kernels (nanolab/csrc/flash_attn_cuda.cu
// :147-281 forward, :1234-1262 Delta, :1265-1366 dQ, :1371-1482 dK/dV): softmax
// in base 2, L = m ln2 + log(l), P recomputed from L in the backward,
// dS = P (dP - Delta) scale, the GQA group summed inside the dK/dV kernel.
#include "tiles.cuh"

namespace nlfa {
namespace {

using namespace tiles;

// The 64-key blocks query rows [q_lo, q_hi] can see: block `it` of `count`, sink blocks first.
struct KeyBlocks {
  int lo, extra, count;
  __device__ __forceinline__ int at(int it) const { return it < extra ? it : lo + (it - extra); }
};
__device__ __forceinline__ KeyBlocks key_blocks(const Problem& p, int q_lo, int q_hi) {
  KeyBlocks r;
  int hi = last_key_of_query(q_hi < p.T ? q_hi : p.T - 1, p.block, p.T) / kBN;
  int lo = 0, sinks = 0;
  if (p.window > 0) {
    const int first = q_lo - (p.window - p.sinks) + 1;
    lo = first > 0 ? first / kBN : 0;
    sinks = (p.sinks + kBN - 1) / kBN;
  }
  r.lo = lo;
  r.extra = sinks < lo ? sinks : lo;
  r.count = r.extra + hi - lo + 1;
  return r;
}

template <typename T, int D, int RM>
__global__ void __launch_bounds__(kThreads, RM == 8 ? 3 : RM == 4 && D == 64 ? 4 : 1)
fwd_tile_kernel(Problem p, const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v,
                T* __restrict__ o, float* __restrict__ lse) {
  constexpr int BM = 8 * RM, kPitch = D + 4;
  extern __shared__ __align__(16) float smem[];
  float* qs = smem;
  float* ks = qs + BM * kPitch;
  float* vs = ks + kBN * kPitch;
  float* ps = vs + kBN * kPitch;
  const int grp = threadIdx.x >> 4, col = threadIdx.x & 15;
  const int BH = p.B * p.H, n_tiles = (p.T + BM - 1) / BM;
  const int rank = blockIdx.x / BH, bh = blockIdx.x - rank * BH;      // late (heavy) query tiles first
  const int b = bh / p.H, h = bh - b * p.H, hk = h / (p.H / p.Hkv);
  const int q0 = (n_tiles - 1 - rank) * BM;
  const long long q_stride = static_cast<long long>(p.H) * D, k_stride = static_cast<long long>(p.Hkv) * D;
  const T* kb = k + (static_cast<long long>(b) * p.T * p.Hkv + hk) * D;
  const T* vb = v + (static_cast<long long>(b) * p.T * p.Hkv + hk) * D;
  const KeyBlocks blocks = key_blocks(p, q0, q0 + BM - 1);
  auto load_kv = [&](float* dst, const T* src, int j) {
    load_rows<T, D>(dst, src + j * kBN * k_stride, k_stride, kBN, p.T - j * kBN);
    load_commit();
  };

  load_rows<T, D>(qs, q + ((static_cast<long long>(b) * p.T + q0) * p.H + h) * D, q_stride, BM, p.T - q0);
  load_kv(ks, kb, blocks.at(0));
  load_kv(vs, vb, blocks.at(0));

  const float scale2 = p.scale * kLog2e;
  float m[RM], l[RM], acc[RM][D / 16];
  int qlim[RM];
#pragma unroll
  for (int i = 0; i < RM; ++i) {
    m[i] = -INFINITY;
    l[i] = 0.f;
    qlim[i] = last_key_of_query(q0 + grp + 8 * i, p.block, p.T);
#pragma unroll
    for (int n = 0; n < D / 16; ++n) acc[i][n] = 0.f;
  }
  for (int it = 0; it < blocks.count; ++it) {
    const int k0 = blocks.at(it) * kBN;
    load_wait<1>();
    __syncthreads();                                   // K (and Q) are there; V may be on its way
    float s[RM][4];
    score_product<D, RM>(qs, ks, grp, col, s);
    __syncthreads();
    if (it + 1 < blocks.count) load_kv(ks, kb, blocks.at(it + 1));
    else load_commit();
    float alpha[RM];
    const bool full = rect_fully_visible(q0, q0 + BM - 1, k0, k0 + kBN - 1, p.window, p.sinks, p.block, p.T);
#pragma unroll
    for (int i = 0; i < RM; ++i) {
      const int qpos = q0 + grp + 8 * i;
      float mx = m[i];
      bool seen[4] = {true, true, true, true};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (!full) {
          const int kp = k0 + col + 16 * j;
          seen[j] = kp <= qlim[i] && (p.window == 0 || kp > qpos - (p.window - p.sinks) || kp < p.sinks);
        }
        mx = fmaxf(mx, seen[j] ? s[i][j] * scale2 : -INFINITY);
      }
#pragma unroll
      for (int off = 8; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
      const float ref = mx == -INFINITY ? 0.f : mx;    // nothing seen yet
      alpha[i] = exp2f(m[i] - ref);
      m[i] = mx;
      float e[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        e[j] = seen[j] ? exp2f(fmaf(s[i][j], scale2, -ref)) : kHidden;
        ps[(grp + 8 * i) * kPPitch + col + 16 * j] = e[j];
      }
      l[i] = fmaf(l[i], alpha[i], (e[0] + e[1]) + (e[2] + e[3]));
    }
    load_wait<1>();
    // V is there (and this warp's probabilities)
    const bool guard = __syncthreads_or(!full && !own_rows_finite<T, D>(vs, kBN)) != 0;
    output_product<D, RM>(ps, vs, grp, col, acc, alpha, guard);
    __syncthreads();
    if (it + 1 < blocks.count) load_kv(vs, vb, blocks.at(it + 1));
    else load_commit();
  }
#pragma unroll
  for (int i = 0; i < RM; ++i) {
    float sum = l[i];
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    const int t = q0 + grp + 8 * i;
    if (t >= p.T) continue;
    store_row<T, D>(o + ((static_cast<long long>(b) * p.T + t) * p.H + h) * D, col, acc[i], 1.f / sum);
    if (col == 0) lse[static_cast<long long>(bh) * p.T + t] = (m[i] + log2f(sum)) * kLn2;
  }
}

// dQ pass (DKV = false): stationary Q, dO, streamed K, V.  dK/dV pass: stationary K, V, streamed Q, dO of every
// head of the group.  T0 = X0 Y0^T, T1 = X1 Y1^T; P from T0 and the taped logsumexp, dS = P (T1 - Delta) scale;
// dV += P dO, dQ or dK += dS Y0.  NB: buffers of streamed tiles.
template <typename T, int D, int RM, bool DKV, int NB>
__global__ void __launch_bounds__(kThreads, RM == 8 && D == 32 ? 3 : 1)
bwd_tile_kernel(Problem p, const T* __restrict__ dout, const T* __restrict__ q, const T* __restrict__ k,
                const T* __restrict__ v, const float* __restrict__ lse, const float* __restrict__ delta,
                T* __restrict__ out0, T* __restrict__ out1, int wait_first) {
  constexpr int BM = 8 * RM, kPitch = D + 4;
  extern __shared__ __align__(16) float smem[];
  float* x0 = smem;
  float* x1 = x0 + BM * kPitch;
  float* ys = x1 + BM * kPitch;                                  // [NB][2][kBN * kPitch]
  float* ws = ys + NB * 2 * kBN * kPitch;
  float* vec = ws + BM * kPPitch;                                // [NB][2][kBN]: base-2 logsumexp, Delta of streamed queries
  const int grp = threadIdx.x >> 4, col = threadIdx.x & 15;
  const int group = p.H / p.Hkv;
  const int heads = DKV ? p.Hkv : p.H;
  const int BH = p.B * heads, n_tiles = (p.T + BM - 1) / BM;
  const int rank = blockIdx.x / BH, bh = blockIdx.x - rank * BH;
  const int b = bh / heads, xh = bh - b * heads, hk = DKV ? xh : xh / group;
  const int r0 = (DKV ? rank : n_tiles - 1 - rank) * BM;          // heavy tiles first: early keys, late queries
  const long long q_stride = static_cast<long long>(p.H) * D, k_stride = static_cast<long long>(p.Hkv) * D;
  const T* qb = q + (static_cast<long long>(b) * p.T * p.H) * D;
  const T* dob = dout + (static_cast<long long>(b) * p.T * p.H) * D;
  const T* kb = k + (static_cast<long long>(b) * p.T * p.Hkv + hk) * D;
  const T* vb = v + (static_cast<long long>(b) * p.T * p.Hkv + hk) * D;

  // what is streamed: key blocks of a query tile, or the query blocks that see a key tile, per head of the group
  KeyBlocks blocks{0, 0, 0};
  int y_first = 0, n_inner = 0;
  if (DKV) {
    y_first = first_query_of_key(r0, p.block) / kBN;
    int last = p.T - 1;
    if (p.window > 0 && r0 >= p.sinks) {
      const int w_last = r0 + BM - 1 + (p.window - p.sinks) - 1;
      last = w_last < last ? w_last : last;
    }
    n_inner = last / kBN - y_first + 1;
  } else {
    blocks = key_blocks(p, r0, r0 + BM - 1);
    n_inner = blocks.count;
  }
  const int n_iters = DKV ? n_inner * group : n_inner;
  auto load_y = [&](int it) {
    float* y = ys + (it % NB) * 2 * kBN * kPitch;
    if (DKV) {
      const int g = it / n_inner, y0 = (y_first + it - g * n_inner) * kBN, h = hk * group + g;
      load_rows<T, D>(y, qb + h * D + y0 * q_stride, q_stride, kBN, p.T - y0);
      load_rows<T, D>(y + kBN * kPitch, dob + h * D + y0 * q_stride, q_stride, kBN, p.T - y0);
      if (threadIdx.x < kBN) {
        const int t = y0 + threadIdx.x;
        const long long row = (static_cast<long long>(b) * p.H + h) * p.T + t;
        float* w = vec + (it % NB) * 2 * kBN + threadIdx.x;
        w[0] = t < p.T ? lse[row] * kLog2e : 0.f;
        w[kBN] = t < p.T ? delta[row] : 0.f;
      }
    } else {
      const int y0 = blocks.at(it) * kBN;
      load_rows<T, D>(y, kb + y0 * k_stride, k_stride, kBN, p.T - y0);
      load_rows<T, D>(y + kBN * kPitch, vb + y0 * k_stride, k_stride, kBN, p.T - y0);
    }
    load_commit();
  };

  if (wait_first) grid_dep_wait();
  grid_dep_release();
  if (DKV) {
    load_rows<T, D>(x0, kb + r0 * k_stride, k_stride, BM, p.T - r0);
    load_rows<T, D>(x1, vb + r0 * k_stride, k_stride, BM, p.T - r0);
  } else {
    load_rows<T, D>(x0, qb + xh * D + r0 * q_stride, q_stride, BM, p.T - r0);
    load_rows<T, D>(x1, dob + xh * D + r0 * q_stride, q_stride, BM, p.T - r0);
  }
  load_y(0);

  const float scale2 = p.scale * kLog2e;
  float acc0[RM][D / 16], acc1[DKV ? RM : 1][D / 16];
  float l2[RM], dl[RM];
  int edge[RM];                                                  // a query's last key, a key's first query
#pragma unroll
  for (int i = 0; i < RM; ++i) {
    const int r = r0 + grp + 8 * i;
    edge[i] = DKV ? first_query_of_key(r, p.block) : last_key_of_query(r, p.block, p.T);
    l2[i] = dl[i] = 0.f;
    if (!DKV && r < p.T) {
      l2[i] = lse[static_cast<long long>(bh) * p.T + r] * kLog2e;
      dl[i] = delta[static_cast<long long>(bh) * p.T + r];
    }
#pragma unroll
    for (int n = 0; n < D / 16; ++n) {
      acc0[i][n] = 0.f;
      if (DKV) acc1[i][n] = 0.f;
    }
  }
  float one[RM];
#pragma unroll
  for (int i = 0; i < RM; ++i) one[i] = 1.f;
  for (int it = 0; it < n_iters; ++it) {
    if (NB == 1 && it > 0) {
      __syncthreads();
      load_y(it);
    }
    const float* y0s = ys + (it % NB) * 2 * kBN * kPitch;
    const float* y1s = y0s + kBN * kPitch;
    const float* w = vec + (it % NB) * 2 * kBN;
    const int c0 = (DKV ? y_first + it % n_inner : blocks.at(it)) * kBN;
    const bool full = DKV ? c0 + kBN <= p.T && rect_fully_visible(c0, c0 + kBN - 1, r0, r0 + BM - 1, p.window, p.sinks, p.block, p.T)
                          : rect_fully_visible(r0, r0 + BM - 1, c0, c0 + kBN - 1, p.window, p.sinks, p.block, p.T);
    load_wait<0>();
    const bool guard = __syncthreads_or(!full && !(own_rows_finite<T, D>(y0s, kBN) &&
                                                   (!DKV || own_rows_finite<T, D>(y1s, kBN)))) != 0;
    if (NB == 2 && it + 1 < n_iters) load_y(it + 1);             // its buffer was last read before the barrier
    float s[RM][4], ds[RM][4];
    score_product<D, RM>(x0, y0s, grp, col, s);
    score_product<D, RM>(x1, y1s, grp, col, ds);
#pragma unroll
    for (int i = 0; i < RM; ++i) {
      const int r = r0 + grp + 8 * i;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int c = c0 + col + 16 * j;
        const float ref = DKV ? w[col + 16 * j] : l2[i], dlt = DKV ? w[kBN + col + 16 * j] : dl[i];
        float e = exp2f(fmaf(s[i][j], scale2, -ref)), de = e * (ds[i][j] - dlt) * p.scale;
        if (!full) {
          const int qp = DKV ? c : r, kp = DKV ? r : c;
          const bool vis = (DKV ? c >= edge[i] && c < p.T : c <= edge[i]) &&
                           (p.window == 0 || kp > qp - (p.window - p.sinks) || kp < p.sinks);
          e = vis ? e : kHidden;
          de = vis ? de + 0.f : kHidden;                         // (a visible -0 becomes +0)
        }
        s[i][j] = e;
        ds[i][j] = de;
      }
    }
    auto hand_over = [&](const float (&x)[RM][4]) {              // within this warp's rows
      __syncwarp();
#pragma unroll
      for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) ws[(grp + 8 * i) * kPPitch + col + 16 * j] = x[i][j];
      __syncwarp();
    };
    if constexpr (DKV) {
      hand_over(s);
      output_product<D, RM>(ws, y1s, grp, col, acc1, one, guard);
    }
    hand_over(ds);
    output_product<D, RM>(ws, y0s, grp, col, acc0, one, guard);
  }
#pragma unroll
  for (int i = 0; i < RM; ++i) {
    const int t = r0 + grp + 8 * i;
    if (t >= p.T) continue;
    const long long at = ((static_cast<long long>(b) * p.T + t) * heads + xh) * D;
    store_row<T, D>(out0 + at, col, acc0[i], 1.f);
    if constexpr (DKV) store_row<T, D>(out1 + at, col, acc1[i], 1.f);
  }
  // a pass that started beside its predecessor does not finish before it: what follows may rely on both
  if (!wait_first) grid_dep_wait();
}

// Delta = rowsum(dO * O): pure streaming.  A lane moves 16 bytes of dO and of O per row and has two rows in flight;
// D values are 16 bytes each of D sizeof(T) / 16 consecutive lanes, which combine with shuffles.
template <typename T, int D>
__global__ void __launch_bounds__(256)
delta_kernel(Problem p, const T* __restrict__ dout, const T* __restrict__ o, float* __restrict__ delta) {
  constexpr int kPer = 16 / sizeof(T);                     // values per lane and row
  constexpr int kLanesPerRow = D / kPer;                   // 4 .. 32
  constexpr int kRowsPerWarp = 32 / kLanesPerRow;
  constexpr int U = 2;
  grid_dep_wait();                                         // O comes from the stream's previous kernel
  grid_dep_release();
  const int lane = threadIdx.x & 31;
  const long long warp_id = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const long long rows = static_cast<long long>(p.B) * p.T * p.H;     // rows index [B,T,H]
  const long long row0 = warp_id * (kRowsPerWarp * U) + lane / kLanesPerRow;
  uint4 a[U], c[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const long long row = row0 + u * kRowsPerWarp;
    a[u] = c[u] = make_uint4(0u, 0u, 0u, 0u);
    if (row < rows) {
      a[u] = *reinterpret_cast<const uint4*>(dout + row * D + kPer * (lane % kLanesPerRow));
      c[u] = *reinterpret_cast<const uint4*>(o + row * D + kPer * (lane % kLanesPerRow));
    }
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    T x[kPer], y[kPer];
    *reinterpret_cast<uint4*>(x) = a[u];
    *reinterpret_cast<uint4*>(y) = c[u];
    float part = 0.f;
#pragma unroll
    for (int i = 0; i < kPer; ++i) part = fmaf(to_f32(x[i]), to_f32(y[i]), part);
#pragma unroll
    for (int off = kLanesPerRow / 2; off > 0; off >>= 1) part += __shfl_xor_sync(0xffffffffu, part, off);
    const long long row = row0 + u * kRowsPerWarp;
    if (row < rows && (lane % kLanesPerRow) == 0) {
      const int h = static_cast<int>(row % p.H);
      const long long bt = row / p.H;
      const int t = static_cast<int>(bt % p.T);
      const int b = static_cast<int>(bt / p.T);
      delta[(static_cast<long long>(b) * p.H + h) * p.T + t] = part;
    }
  }
}

// Rows per group of a CTA's tile: 8 (64-row tiles) when there are two tiles per SM, else 4, or 2 where 32-row tiles
// are fewer than `least` per SM: a CTA is four warps, so a lone one leaves its SM waiting on latency (B=4 H=4 T=256
// forward 20.6 -> 18.5 us).  At D = 128 never 8: the accumulators of both gradients and the tiles of
// 64 rows would leave one CTA of four warps per SM.
inline int rows_per_thread(const Problem& p, int heads, int least) {
  auto tiles = [&](int rows) { return static_cast<long long>(p.B) * heads * ((p.T + rows - 1) / rows); };
  if (p.D <= 64 && tiles(64) >= 2ll * sm_count()) return 8;
  return tiles(32) >= static_cast<long long>(least) * sm_count() ? 4 : 2;
}

int launched(cudaError_t e) {
  if (e == cudaSuccess) return NLFA_OK;
  (void)cudaGetLastError();
  return NLFA_ERR_CUDA;
}

template <typename T, int D, int RM>
int fwd_rm(const Problem& p, const T* q, const T* k, const T* v, T* o, float* lse, cudaStream_t s) {
  constexpr int BM = 8 * RM;
  constexpr int smem = ((BM + 2 * kBN) * (D + 4) + BM * kPPitch) * 4;
  auto kern = fwd_tile_kernel<T, D, RM>;
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem) != NLFA_OK) return NLFA_ERR_CUDA;
  const long long blocks = static_cast<long long>(p.B) * p.H * ((p.T + BM - 1) / BM);
  return launched(launch_kernel(kern, dim3(static_cast<unsigned>(blocks)), dim3(kThreads), smem, s, false, p, q, k, v, o, lse));
}

template <typename T, int D>
int fwd_t(const Problem& p, const void* q, const void* k, const void* v, void* o, float* lse, cudaStream_t s) {
  const T *q_ = static_cast<const T*>(q), *k_ = static_cast<const T*>(k), *v_ = static_cast<const T*>(v);
  const int rm = rows_per_thread(p, p.H, 2);
  if constexpr (D <= 64)
    if (rm == 8) return fwd_rm<T, D, 8>(p, q_, k_, v_, static_cast<T*>(o), lse, s);
  if (rm == 2) return fwd_rm<T, D, 2>(p, q_, k_, v_, static_cast<T*>(o), lse, s);
  return fwd_rm<T, D, 4>(p, q_, k_, v_, static_cast<T*>(o), lse, s);
}

template <typename T, int D>
int delta_t(const Problem& p, const void* dout, const void* o, float* delta, cudaStream_t s) {
  const long long rows = static_cast<long long>(p.B) * p.H * p.T;
  constexpr int kRowsPerBlock = 8 * 2 * (32 / (D * static_cast<int>(sizeof(T)) / 16));
  const unsigned blocks = static_cast<unsigned>((rows + kRowsPerBlock - 1) / kRowsPerBlock);
  if (launch_kernel(delta_kernel<T, D>, dim3(blocks), dim3(256), 0, s, overlap_launches(kOverlapDelta), p,
                    static_cast<const T*>(dout), static_cast<const T*>(o), delta) != cudaSuccess) {
    (void)cudaGetLastError();
    return NLFA_ERR_CUDA;
  }
  return NLFA_OK;
}

template <typename T, int D, int RM, bool DKV>
int bwd_rm(const Problem& p, const T* dout, const T* q, const T* k, const T* v, const float* lse, const float* delta,
           void* out0, void* out1, bool beside_previous, cudaStream_t s) {
  constexpr int BM = 8 * RM;
  constexpr int NB = RM <= 4 && D <= 64 ? 2 : 1;       // a second streamed buffer where two CTAs still fit an SM
  constexpr int smem = ((2 * BM + NB * 2 * kBN) * (D + 4) + BM * kPPitch + NB * 2 * kBN) * 4;
  auto kern = bwd_tile_kernel<T, D, RM, DKV, NB>;
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem) != NLFA_OK) return NLFA_ERR_CUDA;
  const long long blocks = static_cast<long long>(p.B) * (DKV ? p.Hkv : p.H) * ((p.T + BM - 1) / BM);
  const bool overlap = overlap_launches(DKV ? kOverlapDkv : kOverlapDq);
  return launched(launch_kernel(kern, dim3(static_cast<unsigned>(blocks)), dim3(kThreads), smem, s, overlap, p, dout, q, k, v,
                                lse, delta, static_cast<T*>(out0), static_cast<T*>(out1), overlap && beside_previous ? 0 : 1));
}

template <typename T, int D, bool DKV>
int bwd_pass(const Problem& p, const void* dout, const void* q, const void* k, const void* v, const float* lse,
             const float* delta, void* out0, void* out1, bool beside_previous, cudaStream_t s) {
  const T *g = static_cast<const T*>(dout), *q_ = static_cast<const T*>(q), *k_ = static_cast<const T*>(k),
          *v_ = static_cast<const T*>(v);
  const int rm = rows_per_thread(p, DKV ? p.Hkv : p.H, DKV ? 2 : 1);      // (the dQ pass has the dK/dV pass beside it)
  if constexpr (D <= 64)
    if (rm == 8) return bwd_rm<T, D, 8, DKV>(p, g, q_, k_, v_, lse, delta, out0, out1, beside_previous, s);
  if (rm == 2) return bwd_rm<T, D, 2, DKV>(p, g, q_, k_, v_, lse, delta, out0, out1, beside_previous, s);
  return bwd_rm<T, D, 4, DKV>(p, g, q_, k_, v_, lse, delta, out0, out1, beside_previous, s);
}

template <typename T, int D>
int bwd_t(const Problem& p, const void* dout, const void* q, const void* k, const void* v,
          const float* lse, void* dq, void* dk, void* dv, const float* delta, int passes,
          cudaStream_t s) {
  int st = NLFA_OK;
  // The dQ pass reads nothing of the dK/dV pass right before it and starts beside it.
  if (passes & NLFA_PASS_DKV) st = bwd_pass<T, D, true>(p, dout, q, k, v, lse, delta, dk, dv, false, s);
  if (st == NLFA_OK && (passes & NLFA_PASS_DQ))
    st = bwd_pass<T, D, false>(p, dout, q, k, v, lse, delta, dq, nullptr, (passes & NLFA_PASS_DKV) != 0, s);
  return st;
}

#define NLFA_DISPATCH(p, CALL)                                                        \
  do {                                                                                \
    switch ((p).dtype) {                                                              \
      case NLFA_DTYPE_F32:                                                            \
        switch ((p).D) {                                                              \
          case 32: return CALL(float, 32);                                            \
          case 64: return CALL(float, 64);                                            \
          case 128: return CALL(float, 128);                                          \
        }                                                                             \
        return NLFA_ERR_BAD_HEAD_DIM;                                                 \
      case NLFA_DTYPE_F16:                                                            \
        switch ((p).D) {                                                              \
          case 32: return CALL(__half, 32);                                           \
          case 64: return CALL(__half, 64);                                           \
          case 128: return CALL(__half, 128);                                         \
        }                                                                             \
        return NLFA_ERR_BAD_HEAD_DIM;                                                 \
      case NLFA_DTYPE_BF16:                                                           \
        switch ((p).D) {                                                              \
          case 32: return CALL(__nv_bfloat16, 32);                                    \
          case 64: return CALL(__nv_bfloat16, 64);                                    \
          case 128: return CALL(__nv_bfloat16, 128);                                  \
        }                                                                             \
        return NLFA_ERR_BAD_HEAD_DIM;                                                 \
    }                                                                                 \
    return NLFA_ERR_BAD_DTYPE;                                                        \
  } while (0)

}  // namespace

int launch_fwd_simt(const Problem& p, const void* q, const void* k, const void* v, void* o,
                    float* lse, cudaStream_t stream) {
#define CALL(T, DD) fwd_t<T, DD>(p, q, k, v, o, lse, stream)
  NLFA_DISPATCH(p, CALL);
#undef CALL
}

int launch_delta(const Problem& p, const void* dout, const void* o, float* delta,
                 cudaStream_t stream) {
#define CALL(T, DD) delta_t<T, DD>(p, dout, o, delta, stream)
  NLFA_DISPATCH(p, CALL);
#undef CALL
}

int launch_bwd_simt(const Problem& p, const void* dout, const void* q, const void* k,
                    const void* v, const void* o, const float* lse, void* dq, void* dk, void* dv,
                    float* delta, int passes, cudaStream_t stream) {
  if (passes & NLFA_PASS_DELTA) {
    int st = launch_delta(p, dout, o, delta, stream);
    if (st != NLFA_OK) return st;
  }
#define CALL(T, DD) bwd_t<T, DD>(p, dout, q, k, v, lse, dq, dk, dv, delta, passes, stream)
  NLFA_DISPATCH(p, CALL);
#undef CALL
}

}  // namespace nlfa
