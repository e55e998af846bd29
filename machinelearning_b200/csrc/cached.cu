// Forward attention of an active block of queries over [cache | block], masked by absolute
// positions: the attention core of nanolab's KV-cached block forward
// (nanolab/mixers.py:372-467, `Attention.forward_cached`), which nanolab runs as a
// `torch.cat`, a `repeat_interleave` and a masked SDPA per layer.
//
//   q [B,Tq,H,D]; k, v [B,Hkv,L,D] (nanolab's cache layout, the block's own keys last);
//   qpos [Tq], kpos [L]: absolute positions.  After window eviction the cached keys'
//   positions are no longer contiguous, so positions, not offsets, define the mask:
//     window > 0 : kpos <= qpos and (kpos > qpos - (window - sinks) or kpos < sinks)
//     causal     : kpos <= qpos              (full to the cache, lower-triangular in the block)
//     neither    : every key                 (block diffusion: a bidirectional block)
//
// Forward only (the cached path is inference).  This file has the entry points and the fp32 kernel; 16-bit inputs
// go to the tensor cores (cached_tc.cu).  The fp32 kernel: a CTA of 128 threads owns 8 RM query rows of one (batch, KV
// head) -- the rows (t, g) of every query head of the group, so K and V are fetched once for all of them -- and
// streams 64 keys at a time through shared memory, products in register tiles (tiles.cuh).  RM is the
// largest of 4, 2, 1 that leaves enough CTAs (launch_dim): more rows per thread take fewer shared-memory reads per
// multiply-add, but a block of a few rows needs CTAs.  Key blocks no row of the CTA can see (contiguous positions)
// are skipped without being read; with few row tiles the key blocks are split over the CTAs of a cluster, which
// combine the partial rows through distributed shared memory in a fixed order.  No atomics: bit-reproducible.
// A warp of lanes over the keys of 8 rows before -> tiles: B=2 H=8 T=32 L=2048 D=64 in fp32 56 -> 25 us,
// B=4 H=16/4 T=100 L=4096 848 -> 367 us.
#include "cached.cuh"
#include "tiles.cuh"

namespace nlfa {
namespace {

using namespace tiles;
using cached::CachedParams;
using cached::KeyRange;

// Combines the partial rows of a query tile, one part in the shared memory of each CTA of the cluster: rows of D
// sums at a pitch of D + 4 (`rows`) and per row its (maximum, sum of exponentials) in base-2 units (`stats`).  CTA
// `rank` finishes rows rank, rank + splits, ..: a warp turns a row's maxima and sums into weights at once (`weights`:
// 32 floats per own row), then every thread adds up pieces of four columns with the loads of eight parts in flight,
// its own CTA's first: in the same order everywhere, all CTAs would read one CTA's memory at a time, whose 38 bytes
// per clock were the limit.
template <typename T, int D, class RowOf>
__device__ __forceinline__ void merge_rows(const CachedParams& p, int n, RowOf out_row, uint32_t rows, uint32_t stats,
                                           float* weights, int rank) {
  constexpr int kBatch = 8;
  const int lane = threadIdx.x & 31, splits = p.splits;                          // at most 16
  const int own = (n - rank + splits - 1) / splits;
  const uint32_t stat_addr = cluster_addr(stats, lane < splits ? lane : 0);
  for (int i = threadIdx.x >> 5; i < own; i += kThreads / 32) {
    const int r = rank + i * splits;
    float2 ml = ld_cluster_f2(stat_addr + 8u * r);
    if (lane >= splits) ml = make_float2(-INFINITY, 0.f);
    float mx = ml.x;
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    mx = __shfl_sync(0xffffffffu, mx, 0);
    const float w = exp2f(ml.x - (mx == -INFINITY ? 0.f : mx));                  // a part that saw no key: 0
    float sum = w * ml.y;
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    sum = __shfl_sync(0xffffffffu, sum, 0);
    weights[32 * i + lane] = sum > 0.f ? w / sum : 0.f;                          // a row that sees no key gives zeros
    if (p.lse && lane == 0) {
      const long long row = out_row(r), t = (row / p.H) % p.Tq, h = row % p.H, b = row / (static_cast<long long>(p.H) * p.Tq);
      p.lse[(b * p.H + h) * p.Tq + t] = sum > 0.f ? (mx + log2f(sum)) * kLn2 : -INFINITY;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < own * (D / 4); i += kThreads) {
    const int k = i / (D / 4), c = 4 * (i % (D / 4)), r = rank + k * splits;
    const uint32_t at = rows + (r * (D + 4) + c) * 4u;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s0 = 0; s0 < splits; s0 += kBatch) {
      float4 y[kBatch];
      float f[kBatch];
#pragma unroll
      for (int x = 0; x < kBatch; ++x) {
        const bool is = s0 + x < splits;
        int s = is ? s0 + x + rank : rank;
        s = s < splits ? s : s - splits;
        y[x] = ld_cluster_f4(cluster_addr(at, s));
        if (!is) y[x] = make_float4(0.f, 0.f, 0.f, 0.f);                          // (0 times an infinity would be NaN)
        f[x] = is ? weights[32 * k + s] : 0.f;
      }
#pragma unroll
      for (int x = 0; x < kBatch; ++x)
        acc = make_float4(fmaf(f[x], y[x].x, acc.x), fmaf(f[x], y[x].y, acc.y), fmaf(f[x], y[x].z, acc.z), fmaf(f[x], y[x].w, acc.w));
    }
    cached::store4(static_cast<T*>(p.o) + out_row(r) * D + c, acc, p.loose);
  }
}

// HIDES: positions are given and the mask goes by them, so any block may be one that no row sees.
template <typename T, int D, int RM, bool HIDES>
__global__ void __launch_bounds__(kThreads, RM == 1 && D == 64 ? 5 : 1)
fwd_cached_kernel(CachedParams p, const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v) {
  constexpr int BM = 8 * RM, kPitch = D + 4;
  extern __shared__ __align__(16) float smem[];
  __shared__ unsigned words[kThreads / 32];
  float* qs = smem;
  float* ks = qs + BM * kPitch;
  float* vs = ks + kBN * kPitch;
  float* ps = vs + kBN * kPitch;
  const int grp = threadIdx.x >> 4, col = threadIdx.x & 15;
  const int G = p.H / p.Hkv;
  const int head_rows = p.Tq * G;                          // query rows that share this KV head: (t, g)
  const int chunks = (head_rows + BM - 1) / BM;
  const int chunk = blockIdx.x % chunks, bh = blockIdx.x / chunks;
  const int hk = bh % p.Hkv, b = bh / p.Hkv;
  const int r0 = chunk * BM, rows = head_rows - r0 < BM ? head_rows - r0 : BM;
  const int t0 = r0 / G, t1 = (r0 + rows - 1) / G;
  // row r of the tile in q / o [B,Tq,H]
  auto out_row = [&](int r) -> long long {
    const int t = (r0 + r) / G, g = (r0 + r) - t * G;
    return (static_cast<long long>(b) * p.Tq + t) * p.H + hk * G + g;
  };
  const bool given = p.qpos != nullptr || p.kpos != nullptr;
  const KeyRange range = cached::key_range(p.Tq, p.L, given, p.causal, p.window, p.sinks, t0, t1, kBN);
  const int per = (range.count + p.splits - 1) / p.splits;
  const int n_begin = static_cast<int>(blockIdx.y) * per;
  const int n_stop = n_begin + per < range.count ? n_begin + per : range.count;

  for (int i = threadIdx.x; i < BM * (D / 4); i += kThreads) {
    const int r = i / (D / 4), c = 4 * (i % (D / 4));
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < rows) {
      const T* src = q + out_row(r) * D + c;
      if (sizeof(T) == 4 && !p.loose) x = *reinterpret_cast<const float4*>(src);
      else x = make_float4(to_f32(src[0]), to_f32(src[1]), to_f32(src[2]), to_f32(src[3]));
    }
    *reinterpret_cast<float4*>(qs + r * kPitch + c) = x;
  }
  const T* kb = k + (static_cast<long long>(b) * p.Hkv + hk) * p.L * D;
  const T* vb = v + (static_cast<long long>(b) * p.Hkv + hk) * p.L * D;
  auto load_kv = [&](float* dst, const T* src, int n) {
    const long long j = range.at(n);
    load_rows<T, D>(dst, src + j * kBN * D, D, kBN, p.L - static_cast<int>(j) * kBN);
    load_commit();
  };
  float m[RM], l[RM], acc[RM][D / 16];
  int qp[RM];
#pragma unroll
  for (int i = 0; i < RM; ++i) {
    m[i] = -INFINITY;
    l[i] = 0.f;
    const int r = grp + 8 * i;
    qp[i] = r < rows ? cached::query_position(p, (r0 + r) / G) : 0;
#pragma unroll
    for (int n = 0; n < D / 16; ++n) acc[i][n] = 0.f;
  }
  // The first block from n on that may hold a key some row sees.  Contiguous positions leave only such blocks in the
  // range; given ones are looked over, 32 blocks (8 a warp) at a time, where a CTA has more than a few: a window of 256 over
  // 16,384 keys that were not compacted, 1 query, H=12 D=64 87 -> 19.5 us.  The look costs 1.5 us, as much as four blocks.
  const bool look = HIDES && n_stop - n_begin > 4;
  int qp_min = 0, qp_max = 0;
  if (look) {
    const int qp_lane = cached::query_position(p, t0 + static_cast<int>(threadIdx.x & 31) <= t1 ? t0 + static_cast<int>(threadIdx.x & 31) : t0);
    qp_min = __reduce_min_sync(0xffffffffu, qp_lane);
    qp_max = __reduce_max_sync(0xffffffffu, qp_lane);
  }
  unsigned shown = 0u;                                     // of blocks shown_end - 32 ..
  int shown_end = n_begin;
  auto next = [&](int n) -> int {
    while (look && n < n_stop) {
      if (n >= shown_end) {
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        unsigned bits = 0u;
#pragma unroll
        for (int x = 0; x < 8; ++x) {
          const int block = n + 8 * warp + x;
          bool any = false;
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int key = block < n_stop ? range.at(block) * kBN + lane + 32 * e : p.L;
            if (key >= p.L) continue;
            const int at = cached::key_position(p, key);
            any = any || (at <= qp_max && (p.window == 0 || at > qp_min - (p.window - p.sinks) || at < p.sinks));
          }
          if (__any_sync(0xffffffffu, any)) bits |= 1u << (8 * warp + x);
        }
        if (lane == 0) words[warp] = bits;
        __syncthreads();
        shown = words[0] | words[1] | words[2] | words[3];
        shown_end = n + 32;
        __syncthreads();                                   // (read before they are written again)
      }
      const unsigned rest = shown >> (32 - (shown_end - n));
      if (rest != 0u) return n + __ffs(rest) - 1;
      n = shown_end;
    }
    return n;
  };
  int n = next(n_begin);
  if (n < n_stop) {
    load_kv(ks, kb, n);
    load_kv(vs, vb, n);
  }
  for (int n_next; n < n_stop; n = n_next) {
    n_next = next(n + 1);
    const int k0 = range.at(n) * kBN;
    int kp[4];
    bool in[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int key = k0 + col + 16 * j;
      in[j] = key < p.L;
      kp[j] = in[j] ? cached::key_position(p, key) : 0;
    }
    const bool full = !given && k0 + kBN <= p.L &&
                      cached::all_visible(p, k0, k0 + kBN - 1, p.L - p.Tq + t0, p.L - p.Tq + t1);
    load_wait<1>();
    __syncthreads();                                       // K (and Q) are there; V may be on its way
    float s[RM][4], alpha[RM];
    score_product<D, RM>(qs, ks, grp, col, s);
    __syncthreads();
    if (n_next < n_stop) load_kv(ks, kb, n_next);
    else load_commit();
#pragma unroll
    for (int i = 0; i < RM; ++i) {
      float mx = m[i];
      bool seen[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        seen[j] = full || (in[j] && cached::position_visible(p, qp[i], kp[j]));
        mx = fmaxf(mx, seen[j] ? s[i][j] * p.scale_log2 : -INFINITY);
      }
#pragma unroll
      for (int off = 8; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
      const float ref = mx == -INFINITY ? 0.f : mx;        // nothing seen yet
      alpha[i] = exp2f(m[i] - ref);
      m[i] = mx;
      float e[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        e[j] = seen[j] ? exp2f(fmaf(s[i][j], p.scale_log2, -ref)) : kHidden;
        ps[(grp + 8 * i) * kPPitch + col + 16 * j] = e[j];
      }
      l[i] = fmaf(l[i], alpha[i], (e[0] + e[1]) + (e[2] + e[3]));
    }
    load_wait<1>();
    // V is there (and this warp's probabilities)
    const bool guard = __syncthreads_or(!full && !own_rows_finite<T, D>(vs, kBN)) != 0;
    output_product<D, RM>(ps, vs, grp, col, acc, alpha, guard);
    __syncthreads();
    if (n_next < n_stop) load_kv(vs, vb, n_next);
    else load_commit();
  }
#pragma unroll
  for (int i = 0; i < RM; ++i) {
    float sum = l[i];
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    const int r = grp + 8 * i;
    if (r >= rows) continue;
    if (p.splits > 1) {                                    // (K's and V's tiles are dead: the last product has read them)
      store_row<float, D>(ks + r * kPitch, col, acc[i], 1.f);
      if (col == 0) reinterpret_cast<float2*>(vs)[r] = make_float2(m[i], sum);
      continue;
    }
    const long long row = out_row(r);
    const float inv = sum > 0.f ? 1.f / sum : 0.f;         // a row that sees no key gives zeros
    T* out = static_cast<T*>(p.o) + row * D;
    if (!p.loose) {
      store_row<T, D>(out, col, acc[i], inv);
    } else {
      constexpr int kRun = D == 32 ? 2 : 4;                // columns of a thread that stand together (store_row)
#pragma unroll
      for (int n = 0; n < D / 16; ++n) out[64 * (n / 4) + kRun * col + n % 4] = from_f32<T>(acc[i][n] * inv);
    }
    if (p.lse && col == 0) {
      const long long t = (row / p.H) % p.Tq, h = row % p.H;
      p.lse[(static_cast<long long>(b) * p.H + h) * p.Tq + t] = sum > 0.f ? (m[i] + log2f(sum)) * kLn2 : -INFINITY;
    }
  }
  if (p.splits > 1) {
    cluster_arrive();
    cluster_wait();
    merge_rows<T, D>(p, rows, out_row, smem_u32(ks), smem_u32(vs), ps, static_cast<int>(blockIdx.y));
    cluster_arrive();                                      // no CTA leaves while another reads its shared memory
    cluster_wait();
  }
}

template <typename T, int D, int RM, bool HIDES>
int launch_kern(CachedParams p, const void* q, const void* k, const void* v, int splits, cudaStream_t st) {
  constexpr int BM = 8 * RM;
  constexpr int smem = ((BM + 2 * kBN) * (D + 4) + BM * kPPitch) * 4;
  auto kern = fwd_cached_kernel<T, D, RM, HIDES>;
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem) != NLFA_OK) return NLFA_ERR_CUDA;
  const long long head_rows = static_cast<long long>(p.Tq) * (p.H / p.Hkv);
  const long long grid = static_cast<long long>(p.B) * p.Hkv * ((head_rows + BM - 1) / BM);
  if (grid >= (1ll << 31)) return NLFA_ERR_BAD_SHAPE;
  p.splits = splits > 1 ? cached::cluster_splits(reinterpret_cast<const void*>(kern), kThreads, smem, grid, splits) : 1;
  if (launch_cluster(kern, dim3(static_cast<unsigned>(grid), static_cast<unsigned>(p.splits)), dim3(kThreads), smem, st, false,
                     p.splits, p, static_cast<const T*>(q), static_cast<const T*>(k), static_cast<const T*>(v)) != cudaSuccess) {
    (void)cudaGetLastError();
    return NLFA_ERR_CUDA;
  }
  return NLFA_OK;
}

template <typename T, int D, int RM>
int launch_rm(const CachedParams& p, const void* q, const void* k, const void* v, int splits, cudaStream_t st) {
  return p.causal && (p.qpos || p.kpos) ? launch_kern<T, D, RM, true>(p, q, k, v, splits, st)
                                        : launch_kern<T, D, RM, false>(p, q, k, v, splits, st);
}

template <typename T, int D>
int launch_dim(const CachedParams& p, const void* q, const void* k, const void* v, cudaStream_t st) {
  const long long head_rows = static_cast<long long>(p.Tq) * (p.H / p.Hkv), heads = static_cast<long long>(p.B) * p.Hkv;
  const long long want = 2ll * sm_count(), pairs = ((p.L + kBN - 1) / kBN + 1) / 2;      // two key blocks per CTA at least
  // the taller tile first, its keys split as far as it takes to fill the GPU; only then shorter ones
  auto splits = [&](int rm) {
    const long long tiles = heads * ((head_rows + 8 * rm - 1) / (8 * rm));
    long long s = (2 * want + tiles - 1) / tiles;
    if (tiles >= want) s = 1;
    if (s > kMostCluster) s = kMostCluster;
    if (s > pairs) s = pairs;
    return static_cast<int>(s < 1 ? 1 : s);
  };
  auto ctas = [&](int rm) { return heads * ((head_rows + 8 * rm - 1) / (8 * rm)) * splits(rm); };
  // Half the height takes well over half the time: two rows a thread win over one as soon as they occupy most of the SMs (108
  // to 216 CTAs, D = 32 / 64 / 128: H=12, 32 over 1,056 13.5 / 19.8 / 35.0 -> 12.5 / 16.5 / 25.3 us; H=8, 16 over 4,096 at
  // D = 128 45.2 -> 41.0), not with a few dozen (H=4, 20 over 300: 10.4 / 12.4).
  if (head_rows > 16 && ctas(4) >= want) return launch_rm<T, D, 4>(p, q, k, v, splits(4), st);
  if (head_rows > 8 && 3 * ctas(2) >= want) return launch_rm<T, D, 2>(p, q, k, v, splits(2), st);
  return launch_rm<T, D, 1>(p, q, k, v, splits(1), st);
}

template <typename T>
int launch_simt(const CachedParams& p, const void* q, const void* k, const void* v, cudaStream_t st) {
  if (p.D == 32) return launch_dim<T, 32>(p, q, k, v, st);
  if (p.D == 64) return launch_dim<T, 64>(p, q, k, v, st);
  return launch_dim<T, 128>(p, q, k, v, st);
}

}  // namespace

// tensor-core form (cached_tc.cu)
bool cached_tc_applies(int Tq, int H, int Hkv, int L, int D, int dtype);
bool cached_tc_can(int H, int Hkv, int D, int dtype);
int launch_fwd_cached_tc(CachedParams p, const void* q, const void* k_cache, const void* v_cache, int dtype, bool split_p,
                         unsigned* status, cudaStream_t stream);
unsigned* status_block();      // api.cu

}  // namespace nlfa

// Nothing is kept in scratch: the partial rows of a split stay in the cluster's shared memory.
extern "C" size_t nlfa_fwd_cached_scratch_bytes(int, int, int, int, int, int) { return 0; }

extern "C" int nlfa_fwd_cached(const void* q, const void* k_cache, const void* v_cache, void* o, float* lse,
                               const int* qpos, const int* kpos, int B, int Tq, int H, int Hkv, int L, int D,
                               float scale, int causal, int window, int sinks, int dtype, void* scratch,
                               size_t scratch_bytes, void* stream) {
  return nlfa_fwd_cached_path(q, k_cache, v_cache, o, lse, qpos, kpos, B, Tq, H, Hkv, L, D, scale, causal, window,
                              sinks, dtype, NLFA_PATH_AUTO, scratch, scratch_bytes, stream);
}

extern "C" int nlfa_fwd_cached_path(const void* q, const void* k_cache, const void* v_cache, void* o, float* lse,
                                    const int* qpos, const int* kpos, int B, int Tq, int H, int Hkv, int L, int D,
                                    float scale, int causal, int window, int sinks, int dtype, int path,
                                    void* scratch, size_t scratch_bytes, void* stream) {
  return nlfa_fwd_cached_positions(q, k_cache, v_cache, o, lse, qpos, kpos, 4, B, Tq, H, Hkv, L, D, scale, causal, window,
                                   sinks, dtype, path, scratch, scratch_bytes, stream);
}

extern "C" int nlfa_fwd_cached_positions(const void* q, const void* k_cache, const void* v_cache, void* o, float* lse,
                                         const void* qpos, const void* kpos, int position_bytes, int B, int Tq, int H,
                                         int Hkv, int L, int D, float scale, int causal, int window, int sinks, int dtype,
                                         int path, void* scratch, size_t scratch_bytes, void* stream) {
  using namespace nlfa;
  (void)scratch;
  (void)scratch_bytes;
  if (path != NLFA_PATH_AUTO && path != NLFA_PATH_SIMT && path != NLFA_PATH_TENSOR) return NLFA_ERR_UNSUPPORTED_PATH;
  if (position_bytes != 4 && position_bytes != 8) return NLFA_ERR_BAD_ARGUMENT;
  if (B < 0 || Tq < 0 || H < 0 || L < 0 || Hkv <= 0 || H % Hkv != 0 || !(scale == scale)) return NLFA_ERR_BAD_SHAPE;
  if (D != 32 && D != 64 && D != 128) return NLFA_ERR_BAD_HEAD_DIM;
  if (dtype != NLFA_DTYPE_F32 && dtype != NLFA_DTYPE_F16 && dtype != NLFA_DTYPE_BF16) return NLFA_ERR_BAD_DTYPE;
  if (window < 0 || sinks < 0 || (window == 0 && sinks != 0) || (window > 0 && sinks >= window))
    return NLFA_ERR_BAD_WINDOW;
  if (window > 0 && !causal) return NLFA_ERR_BAD_WINDOW;           // a window is defined on distance to the query
  if (qpos == nullptr && Tq > L) return NLFA_ERR_BAD_SHAPE;
  const long long rows = static_cast<long long>(B) * Tq * H;
  if (rows == 0) return NLFA_OK;
  if (rows / 4 >= (1ll << 31)) return NLFA_ERR_BAD_SHAPE;
  if (!q || !o || (L > 0 && (!k_cache || !v_cache))) return NLFA_ERR_NULL_POINTER;
  // a window that cuts nothing of a contiguous cache (and sinks next to 2^31 would overflow when rounded up to blocks)
  if (window > 0 && qpos == nullptr && kpos == nullptr && (window - sinks >= L || sinks >= L)) window = sinks = 0;
  CachedParams p{B, Tq, H, Hkv, L, D, causal ? 1 : 0, window, sinks, scale * kLog2e, qpos, kpos, position_bytes == 8,
                       1, o, lse, 0};
  cudaStream_t st = (cudaStream_t)stream;
  auto off = [](const void* x) { return (reinterpret_cast<uintptr_t>(x) & 15u) != 0; };
  const bool kv_aligned = L == 0 || !(off(k_cache) || off(v_cache));
  p.loose = off(q) || off(o);
  // 16-bit inputs: the products run on the tensor cores, whatever the block's size, because the cache's
  // bandwidth is what counts.  Blocks a caller cannot force onto them (fewer than 16 rows per KV head, or under
  // 256 keys) keep the fp32 kernel's precision there (SPLIT_P).
  const bool applies = cached_tc_applies(Tq, H, Hkv, L, D, dtype);
  if (kv_aligned && !p.loose && L > 0 && scale > 0.f && nlfa_device_supported() &&
      (path == NLFA_PATH_TENSOR ? applies : path == NLFA_PATH_AUTO && cached_tc_can(H, Hkv, D, dtype))) {
    if (nlfa_peek_status() != NLFA_OK) return NLFA_ERR_DEVICE_TIMEOUT;
    unsigned* status = status_block();
    if (!status) return NLFA_ERR_CUDA;
    return launch_fwd_cached_tc(p, q, k_cache, v_cache, dtype, !applies, status, st);
  }
  if (path == NLFA_PATH_TENSOR) return NLFA_ERR_UNSUPPORTED_PATH;
  if (!kv_aligned) return NLFA_ERR_MISALIGNED;             // K and V come by 16-byte copies in this kernel, too
  if (dtype == NLFA_DTYPE_BF16) return launch_simt<__nv_bfloat16>(p, q, k_cache, v_cache, st);
  if (dtype == NLFA_DTYPE_F16) return launch_simt<__half>(p, q, k_cache, v_cache, st);
  return launch_simt<float>(p, q, k_cache, v_cache, st);
}
