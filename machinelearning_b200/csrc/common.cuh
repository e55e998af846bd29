// Shared host/device definitions for the attention library.
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda.h>
#include <cuda_runtime.h>

#include "../../include/nlfa.h"

namespace nlfa {

constexpr int kTile = 128;          // query rows per tile and keys per block
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

// One attention problem.  Layouts follow the reference kernel's contract
// (nanolab/csrc/flash_attn_cuda.cu:1628-1650): q, o, dout, dq are contiguous
// [B,T,H,D]; k, v, dk, dv are contiguous [B,T,Hkv,D]; lse and delta are fp32
// [B,H,T]; lse is a natural-log logsumexp.
struct Problem {
  int B, T, H, Hkv, D;
  int window, sinks;     // window == 0: plain causal
  float scale;
  int dtype;             // NLFA_DTYPE_*
  int block = 0;         // > 0: block-causal (bidirectional inside blocks of this many positions); needs window == 0
};

// Block-causal attention (nanolab/mixers.py:78-93, `block_causal_mask`): a query sees every
// position of its own block and of all earlier blocks, i.e. query q sees the keys up to the end
// of its block, and key k is seen by the queries from the start of its block on.  block == 0
// (or 1) is plain causal attention.  A block may reach past the end of the sequence (`t_len`
// positions): the keys stop there.
__host__ __device__ inline int last_key_of_query(int q, int block, int t_len = 1 << 30) {
  if (block <= 1) return q;
  const int last = (q / block + 1) * block - 1;
  return last < t_len - 1 ? last : t_len - 1;
}
__host__ __device__ inline int first_query_of_key(int k, int block) {
  return block > 1 ? (k / block) * block : k;
}

// Division of a non-negative int by a divisor the host knows: q = (mulhi(n, mul) + n) >> shift with 2^shift >= d and
// mul = floor(2^32 (2^shift - d) / d) + 1 (Granlund and Montgomery, "Division by Invariant Integers using Multiplication",
// PLDI 1994, figure 4.1), exact for every n < 2^31.
struct FastDiv {
  unsigned mul, shift;
  int d;
  FastDiv() = default;
  explicit FastDiv(int divisor) : mul(0), shift(0), d(divisor) {
    while ((1ull << shift) < static_cast<unsigned long long>(divisor)) ++shift;
    mul = static_cast<unsigned>(((1ull << 32) * ((1ull << shift) - divisor)) / divisor + 1);
  }
  __host__ __device__ __forceinline__ int div(int n) const {
#ifdef __CUDA_ARCH__
    return static_cast<int>((__umulhi(static_cast<unsigned>(n), mul) + static_cast<unsigned>(n)) >> shift);
#else
    return static_cast<int>(((static_cast<unsigned long long>(n) * mul >> 32) + n) >> shift);
#endif
  }
};

// Which key blocks a 128-row query tile must visit.  Block j covers keys
// [w j, w j + w - 1], w = `width`.  The mask is the reference's sliding_window_mask
// (nanolab/mixers.py:125-132): keep k <= q and (k > q - (window - sinks) or
// k < sinks).
struct TileRange {
  int lo, hi;            // contiguous range of recent blocks, inclusive
  int sink_blocks;       // blocks [0, sink_blocks) hold sink keys
};

// `block` > 0 (block-causal; window must be 0) lets a tile see past the diagonal, up to the end
// of its last row's block; `n_blocks` key blocks bound that.
__host__ __device__ inline TileRange tile_range(int tile, int window, int sinks, int block = 0,
                                                int n_blocks = 1 << 30, int width = kTile) {
  TileRange r;
  r.hi = last_key_of_query(tile * kTile + kTile - 1, block) / width;
  r.hi = r.hi < n_blocks - 1 ? r.hi : n_blocks - 1;
  r.lo = 0;
  r.sink_blocks = 0;
  if (window > 0) {
    const int span = window - sinks;
    const int first_key = tile * kTile - span + 1;     // lowest recent key of the tile's first row
    r.lo = first_key > 0 ? first_key / width : 0;
    r.sink_blocks = (sinks + width - 1) / width;
  }
  return r;
}

// Whether every (query, key) of a rectangle of query positions [q_lo, q_hi] x key positions [k_lo, k_hi] survives the mask,
// so that the element-wise predicate can be skipped, and which edges of the mask cut through one that is not fully visible: only the causal edge k <= q (plain
// causal, or windows whose lower edge stays below it), only the window's lower edge k > q - (window - sinks) (below the
// diagonal, no sink keys), or both / sinks involved.  With one edge a compare per element against a per-thread limit does.
enum { EDGE_CAUSAL = 0, EDGE_WINDOW = 1, EDGE_BOTH = 2 };
__host__ __device__ inline bool rect_fully_visible(int q_lo, int q_hi, int k_lo, int k_hi,
                                                   int window, int sinks, int block = 0, int t_len = 1 << 30) {
  if (k_hi > last_key_of_query(q_lo, block, t_len)) return false;          // causal edge cuts in
  if (window > 0 && k_lo <= q_hi - (window - sinks)) return false;         // lower window edge cuts in
  return true;
}
__host__ __device__ inline int rect_edges(int q_lo, int q_hi, int k_lo, int k_hi, int window,
                                          int sinks) {
  if (window == 0) return EDGE_CAUSAL;
  if (k_lo > q_hi - (window - sinks)) return EDGE_CAUSAL;                  // lower edge below the rectangle
  if (k_hi <= q_lo && k_lo >= sinks) return EDGE_WINDOW;                   // causal edge above, no sink keys
  return EDGE_BOTH;
}

// Key-block-stationary passes (dK/dV, fused): the last streamed query tile (of `rows` rows each,
// `n_ytiles` in all) that reaches 128-key block `block`; the first is block * (128 / rows).
__host__ __device__ inline int last_query_tile_of_block(int block, int n_ytiles, int rows, int window,
                                                        int sinks) {
  int hi = n_ytiles - 1;
  if (window > 0 && block >= (sinks + kTile - 1) / kTile) {      // blocks with sink keys are seen by all
    const int last_q = block * kTile + kTile - 1 + (window - sinks) - 1;
    hi = last_q / rows < hi ? last_q / rows : hi;
  }
  return hi;
}

// Iterations (128-row query tiles, of one query head) of the dK/dV pass over one (batch, KV head) pair under a window: of its
// longest unit, and of all.  A block with sink keys is streamed past by every tile from its own on, one behind the sinks by
// those a window further.
struct DkvWork {
  long long longest, total;
};
inline DkvWork dkv_work(int T, int window, int sinks) {
  const long long n = (static_cast<long long>(T) + kTile - 1) / kTile, span = static_cast<long long>(window) - sinks;
  const long long with_sinks = (static_cast<long long>(sinks) + kTile - 1) / kTile, ns = with_sinks < n ? with_sinks : n;
  const long long reach = (span + kTile - 2) / kTile + 1, rest = n - ns;               // of a block without sinks, inside the row
  const long long behind = rest <= reach ? rest * (rest + 1) / 2 : reach * (reach + 1) / 2 + (rest - reach) * reach;
  return {ns > 0 ? n : rest < reach ? rest : reach, ns * n - ns * (ns - 1) / 2 + behind};
}

// Fused backward: key block `block`'s place in the fixed order in which the blocks that see
// 128-row query tile `tile` add their dQ shares (ascending block index: sink blocks below the
// window first, then the window's blocks up to the last one the tile sees -- the diagonal, or
// beyond it under a block-causal mask of `mask_block` positions).  *count is the number of such blocks.
__host__ __device__ inline int dq_turn_of_block(int block, int tile, int window, int sinks, int* count,
                                                int mask_block = 0, int n_tiles = 1 << 30) {
  const TileRange r = tile_range(tile, window, sinks, mask_block, n_tiles);
  const int extra = r.sink_blocks < r.lo ? r.sink_blocks : r.lo;
  *count = extra + (r.hi - r.lo + 1);
  return block < extra ? block : extra + (block - r.lo);
}

// Where the dK/dV pass leaves dS for the dQ pass (bwd_dq.cu): one 32 KB tile of 16-bit values per
// (query head, query tile, key block the tile sees), a query tile's blocks side by side in the order
// of dq_turn_of_block.  Tile `i`'s blocks start at slot ds_tile_offset(i) of its head.  In 64 bits where the host sizes
// the scratch (the square of the number of tiles leaves 32 bits at T = 5.9 million); a kernel addresses tiles that
// exist, whose numbers fit an int.
constexpr int kDsTileBytes = kTile * kTile * 2;
struct DsLayout {
  int n_tiles;
  int stride;            // > 0 (windows): every query tile has this many slots
  int ahead;             // otherwise: tile i has min(n_tiles, i + 1 + ahead) of them (block-causal: ahead > 0)
};
template <typename Int = int>
__host__ __device__ inline Int ds_tile_offset(const DsLayout& l, int tile) {
  const Int i = tile;
  if (l.stride > 0) return i * l.stride;
  const Int full = l.n_tiles - 1 - l.ahead > 0 ? l.n_tiles - 1 - l.ahead : 0;    // first tile that sees every block
  return i <= full ? i * (i + 1) / 2 + i * l.ahead : full * (full + 1) / 2 + full * l.ahead + (i - full) * l.n_tiles;
}
inline DsLayout ds_layout(int T, int window, int sinks, int block) {
  DsLayout l{(T + kTile - 1) / kTile, 0, 0};
  if (window > 0) {
    for (int t = 0; t < l.n_tiles; ++t) {
      int count = 0;
      (void)dq_turn_of_block(t, t, window, sinks, &count, block, l.n_tiles);
      if (count > l.stride) l.stride = count;
    }
  } else if (block > 1) {
    l.ahead = (block - 1 + kTile - 1) / kTile;      // blocks past the diagonal a tile's last row can reach
    if (l.ahead > l.n_tiles - 1) l.ahead = l.n_tiles - 1;
  }
  return l;
}

__host__ __device__ inline bool key_visible(int q, int k, int window, int sinks, int block = 0,
                                            int t_len = 1 << 30) {
  if (k > last_key_of_query(q, block, t_len)) return false;
  if (window == 0) return true;
  return (k > q - (window - sinks)) || (k < sinks);
}

// Host-side launchers (one per translation unit); all return an NLFA_* status.
int launch_fwd_simt(const Problem& p, const void* q, const void* k, const void* v, void* o,
                    float* lse, cudaStream_t stream);
int launch_bwd_simt(const Problem& p, const void* dout, const void* q, const void* k,
                    const void* v, const void* o, const float* lse, void* dq, void* dk, void* dv,
                    float* delta, int passes, cudaStream_t stream);
int launch_delta(const Problem& p, const void* dout, const void* o, float* delta,
                 cudaStream_t stream);
int fwd_key_block(const Problem& p);            // keys per block of the tensor-core forward
int launch_fwd_tc(const Problem& p, const void* q, const void* k, const void* v, void* o,
                  float* lse, unsigned* status, cudaStream_t stream);
// Scratch of the fused backward pass (head dim <= 64), behind the Delta tape in the caller's
// buffer: per (batch, head, 128-row query tile) a turn counter and 128 x 64 fp32 partial sums.
struct FusedScratch {
  float* dq_acc;
  unsigned* dq_turn;
};
// Room for dS behind the Delta tape in the caller's buffer, in whole (batch, KV head) pairs.
struct DsScratch {
  void* tiles;
  int pairs;
};
int launch_bwd_tc(const Problem& p, const void* dout, const void* q, const void* k, const void* v,
                  const void* o, const float* lse, void* dq, void* dk, void* dv, float* delta,
                  int passes, unsigned* status, cudaStream_t stream, const FusedScratch* fused,
                  const DsScratch* ds);
// dQ of the query heads of (batch, KV head) pairs [first_pair, first_pair + pairs) from their dS tiles.
int launch_dq_from_ds(const Problem& p, const void* k, const void* ds, const DsLayout& layout, int first_pair, int pairs,
                      void* dq, unsigned* sched, unsigned* status, cudaStream_t stream);
int launch_selftest_tiles(int dtype, int head_dim, const void* q, const void* k, const void* v,
                          float* s_out, float* o_out, unsigned* status, cudaStream_t stream);

// Encodes a 4-D tensor map over a contiguous [B,T,heads,D] 16-bit tensor with a
// box of 64 elements x 1 head x `rows` rows x 1 batch and 128-byte swizzle.  Encoded maps are
// kept in a small host-side table keyed by (base, dtype, shape, rows): a training loop calls
// with the same buffers step after step, and the driver's encoder costs a microsecond or two
// per map (ten maps per forward + backward).
int make_tile_map(CUtensorMap* map, const void* base, int dtype, int B, int T, int heads, int D,
                  int rows);
// The same for any 4-D tensor of 16-bit elements: extents, byte strides of dimensions 1-3, box.
int make_map(CUtensorMap* map, const void* base, int dtype, const unsigned long long dims[4],
             const unsigned long long strides[3], const unsigned box[4]);

// Two work counters for one launch of a persistent kernel ([0] next unit, [1] CTAs finished;
// the last CTA of a launch zeroes them again).  Launches on a capturing stream draw from a
// range of their own whose entries are never handed out twice, because a captured graph keeps
// the address for as long as it is replayed; eager launches take turns on a ring.  Returns an
// NLFA_* status (NLFA_ERR_GRAPH_SLOTS when the graph range is used up).
int sched_counters(cudaStream_t stream, unsigned** out);

// A ticket for one launch whose CTAs count themselves off and leave it at zero (rowwise.cuh, last_cta): of a ring for
// ordinary launches; under capture `own`, in the caller's scratch, zeroed by a node of the graph in front of the launch,
// so that captures are not limited (the launch then follows a memset: not overlapped).
int launch_ticket(cudaStream_t stream, unsigned* own, unsigned** out, bool* captured);

// cudaFuncSetAttribute(MaxDynamicSharedMemorySize), once per kernel and device.
int ensure_dynamic_smem(const void* kernel, int bytes);

int sm_count();
long long l2_bytes();

// How many clusters of `size` CTAs (up to kMostCluster, along y) of a kernel can be resident at once; asked of the
// driver once per kernel and device.
constexpr int kMostCluster = 16;
int resident_clusters(const void* kernel, int threads, int smem, int size);

// Which kernels are launched with programmatic stream serialization, so that their set-up
// (barriers, TMEM, descriptors) overlaps the predecessor's last CTAs.  NLFA_PDL=<mask> overrides
// the default (0: none).
enum { kOverlapFwd = 1, kOverlapDelta = 2, kOverlapDkv = 4, kOverlapDq = 8, kOverlapRowwise = 16, kOverlapDefault = 31 };
bool overlap_launches(int kernel);

// Whether the tensor-core backward forms Delta inside its dQ pass for this problem and mask
// (bwd_tc.cu); then it launches two kernels instead of three.
bool bwd_delta_in_dq(const Problem& p, int passes);

// One launch through cudaLaunchKernelEx, with the programmatic-serialization attribute when
// `overlap` is set and, given `cluster_y` > 1, in clusters of that many CTAs along y.  The kernel must then call grid_dep_wait() before it reads anything an earlier
// kernel of the stream wrote.
template <typename... Params, typename... Args>
cudaError_t launch_cluster(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                           bool overlap, int cluster_y, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  unsigned n = 0;
  if (overlap) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster_y > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = 1;
    attr[n].val.clusterDim.y = static_cast<unsigned>(cluster_y);
    attr[n++].val.clusterDim.z = 1;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}
template <typename... Params, typename... Args>
cudaError_t launch_kernel(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                          bool overlap, Args&&... args) {
  return launch_cluster(kernel, grid, block, smem, stream, overlap, 1, static_cast<Args&&>(args)...);
}

}  // namespace nlfa
