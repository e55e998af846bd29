// Tensor-core form of the KV-cached block forward (cached.cu has the fp32 one): attention of an
// active block of Tq queries over [cache | block] with the mask taken from absolute positions --
// the attention core of nanolab's `Attention.forward_cached` (nanolab/mixers.py:372-467).
//
// A CTA owns up to 128 query rows of one (batch, KV head): the rows (t, g) of every query head g
// of the group for a run of block positions t, so K and V are fetched once for the whole group.
// One TMA box (64 columns x group heads x positions) brings them in as consecutive 128-byte rows,
// which is the layout the S = Q K^T product wants.  The keys go past in blocks of 128, loaded by
// TMA from nanolab's cache layout [B,Hkv,L,D]; S lands in TMEM, softmax warps (one thread per row)
// mask it from the positions, exponentiate and hand P back through TMEM for O += P V.
//
// What bounds it is streaming K and V, so everything else has to hide behind the loads.  Two softmax
// warpgroups take alternate key blocks, each with S / P and O columns and a running maximum of its own:
// while one exponentiates, the products of the other's block run and K, V of the next blocks arrive (a
// single one, strictly in order, spent twice the load time per block).
//
// COPIES: up to 64 rows leave half or more of a tile's 128 lanes empty, and with them warps of either softmax
// warpgroup.  The rows then stand in the tile two or four times, and each copy's warps exponentiate their share of a
// block's columns (and put zeros where the other copies' probabilities stand): a block takes a half or a
// quarter of the time, 1,900 -> 600 clocks, and the copies' sums are parts like the others.  B=8 H=12 D=64, 32 over 8,192:
// 59 -> 41 us (4.9 TB/s); B=14 H=12 D=32, 8 over 3,000: 60 -> 39; B=1 H=12 D=64, 32 over 1,056: 8.8 -> 7.3.
//
// With few (batch, KV head) pairs the key blocks are split over the CTAs of a cluster (up to 16, as many as can be
// resident).  At the end a CTA's parts of a row become one, each CTA sends every other one the rows that one finishes (a bulk
// copy per pair, counted by a barrier there), and a row's parts are added in the order of the CTAs: no scratch, no second
// kernel, no wait for a remote read.  (Remote reads took 4.5 of 14.8 us of B=1 H=16 D=128, 64 queries over 2,048 keys; through
// global memory with a ticket it was more still; 16-byte remote stores, 2,800 clocks where the copies take 1,100.)
//
// Of a small block this end is half of the time, and it is a chain of short steps by few warps, so what counts is its length:
// the parts' statistics are exchanged, and their weights formed, while the last products run; the two warpgroups' sums of a
// row stand in one TMEM lane, so each warpgroup adds up half of the columns in registers and only copies go through shared
// memory; no element has a branch of its own (a condition on the number of blocks inside the loop over columns cost 34 clocks
// a column); a thread finishing a row loads all of its parts at once.  Before / after (us): B=1 H=12 D=64, 32 over 1,056
// 6.3 / 5.7; B=1 H=16 D=128, 64 over 2,048 10.5 / 9.5, 64 over 16,448 31.0 / 28.0 (4.8 TB/s of K, V), 128 over 4,096 17.6 / 15.1;
// B=1 H=2 D=64, 100 over 129 13.4 / 9.7; one query over 1,057 (SPLIT_P) 6.8 / 6.1.  It costs registers: every variant spills (12 to
// 84 bytes stored and 96 to 480 loaded a thread; 0 to 68 and 0 to 252 with the former end), since a thread is compiled for the 168
// that 384 threads start with, and the softmax warps' 216 come later.
//
// SPLIT_P: blocks so small that the fp32 kernel used to take them keep its precision: P goes in as the sum of two
// 16-bit values (its rounding error is then below the accumulator's), at the price of a second P V product,
// which the loads hide.  It also keeps what that kernel does with infinities and NaN in V.  Of a key the mask hides they
// reach no row: warps 10 and 11 go over the V tiles of blocks the mask cuts before the product reads them and put zeros for the
// rows no query sees and for values that are not finite.  An infinity that a row does see stays one: what was replaced, and
// what the product made NaN (zero times an infinity: the other copies' columns, a second part that is zero), is
// put right at the end by a walk over the cache that only then happens.  Blocks the mask leaves whole cost nothing (going
// over every tile: B=1 H=16 D=128, 1 query over 16,385, 30.5 -> 44.9 us).
//
// Warps 0-3 and 4-7 softmax, 8 TMA producer, 9 MMA issuer and TMEM owner, 10-11 idle or (SPLIT_P) looking through V; they
// complete the warpgroup that gives its registers to the softmax warps.  Every wait bounded.
#include <climits>
#include <type_traits>

#include "cached.cuh"

namespace nlfa {
namespace {

using cached::CachedParams;
using cached::KeyRange;

constexpr int kNoKey = INT_MAX;          // position written for keys past the end of the cache

struct TileParams {
  int group, tq_tile, n_qtiles;          // query heads per KV head; block positions per CTA; tiles per (b, hk)
  FastDiv by_group, by_qtiles, by_heads, by_splits;
  unsigned* status;
  const void* v;
};

template <int D, int STAGES, int COPIES>
struct CachedSmem {
  static constexpr int kTileBytes = kTile * D * 2;
  static constexpr int kK = 0;                                   // later: the rows to send, then those received
  static constexpr int kV = kK + STAGES * kTileBytes;
  static constexpr int kQ = kV + STAGES * kTileBytes;
  static constexpr int kPos = kQ + kTileBytes;                   // per K stage: 128 key positions
  static constexpr int kFull = kPos + STAGES * 512;              // per K stage: every key visible to every row
  // Rows of sums on their way together, four floats of padding apart (lanes a row apart hit different banks) in which the
  // maximum, the sum of exponentials and whether V held a value that is not finite travel: what the copies hand over, the
  // tile's rows, and what the CTAs of a split tile send, one row each for every row this CTA finishes.
  static constexpr int kPitch = 4 * (D + 4);
  static constexpr int kRows = kK + (COPIES > 1 ? kTile * kPitch : 0);
  static constexpr int kReceived = kRows + kTile / COPIES * kPitch;
  static constexpr int kBar = kFull + (STAGES * 4 + 15) / 16 * 16;
  // barriers: q_full, s_full[2], p_full[2], o_done, group, received, k_full[S], k_empty[S], v_full[S], v_empty[S], v_clean[S], scanned
  static constexpr int kNumBars = 9 + 5 * STAGES;
  static constexpr int kTmemSlot = kBar + 8 * kNumBars;
  static constexpr int kAbort = kTmemSlot + 4;
  static constexpr int kSpoilt = kAbort + 4;                     // V held a value that is not finite
  static constexpr int kTotal = kSpoilt + 4;
  static constexpr int kDynamic = kTotal + 1024;
  static_assert(STAGES * 2 * kTileBytes >= kReceived + (kTile / COPIES + kMostCluster) * kPitch && kTileBytes >= 256 * 8,
                "the combination lies over dead tiles");
};

// N columns of a row whose V held values that are not finite: what the row sees of them, as it is (`vr`: the columns of
// the first key).  A call: rare, and long.
template <typename T, int N>
__device__ __noinline__ void put_right(const CachedParams& p, const T* vr, int t, float (&x)[N]) {
  const int q_at = cached::query_position(p, t);
  float odd[N] = {};
  for (int key = 0; key < p.L; ++key, vr += p.D) {
    if (!cached::position_visible(p, q_at, cached::key_position(p, key))) continue;
#pragma unroll
    for (int e = 0; e < N; ++e) {
      const float y = static_cast<float>(vr[e]);
      if (!isfinite(y)) odd[e] += y;
    }
  }
#pragma unroll
  for (int e = 0; e < N; ++e)
    if (odd[e] != 0.f) x[e] = odd[e];
}

template <typename T, int D, int STAGES, int COPIES, bool SPLIT_P>
__global__ void __launch_bounds__(384, 1)
cached_tc_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                 const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CachedParams p,
                 const __grid_constant__ TileParams tp) {
  using L = CachedSmem<D, STAGES, COPIES>;
  constexpr int kLanes = kTile / COPIES, kCols = kTile / COPIES;   // of a copy: its TMEM lanes, its columns of S
  constexpr int kBoxes = D / 64;
  constexpr int kBoxBytes = kTile * 128;
  constexpr bool kBf16 = Pack2<T>::kIsBf16;
  constexpr uint32_t kTmemCols = 512;            // S_w at 128 w (P over it), O_w at 256 + D w
  constexpr int kRegsLaunch = 168, kRegsCompute = 216, kRegsOther = 72;

  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  auto bar = [&](int i) -> uint32_t { return base + L::kBar + 8u * i; };
  constexpr int Q_FULL = 0, S_FULL = 1, P_FULL = 3, O_DONE = 5, GROUP = 6, RECEIVED = 7, K_FULL = 8,
                K_EMPTY = K_FULL + STAGES, V_FULL = K_EMPTY + STAGES, V_EMPTY = V_FULL + STAGES, V_CLEAN = V_EMPTY + STAGES,
                SCANNED = V_CLEAN + STAGES;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gen + L::kAbort);
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gen + L::kTmemSlot);
  volatile int* spoilt_flag = reinterpret_cast<volatile int*>(gen + L::kSpoilt);
  volatile int* full_flag = reinterpret_cast<volatile int*>(gen + L::kFull);
  const WaitCtx wctx{abort_flag, tp.status};

  // this CTA's tile and its share of the key blocks the tile sees
  const int unit = blockIdx.x, bh = tp.by_qtiles.div(unit), qt = unit - bh * tp.n_qtiles;
  const int b = tp.by_heads.div(bh), hk = bh - b * p.Hkv;
  const int t0 = qt * tp.tq_tile;
  const int t1 = (t0 + tp.tq_tile < p.Tq ? t0 + tp.tq_tile : p.Tq) - 1;
  const KeyRange range = cached::key_range(p.Tq, p.L, p.qpos != nullptr || p.kpos != nullptr, p.causal, p.window, p.sinks,
                                           t0, t1, kTile);
  const int per = tp.by_splits.div(range.count + p.splits - 1);
  const int n_begin = static_cast<int>(blockIdx.y) * per;
  const int n_stop = n_begin + per < range.count ? n_begin + per : range.count;
  const int n_blocks = n_stop > n_begin ? n_stop - n_begin : 0;            // block i of this CTA: range.at(n_begin + i)
  const int n_rows = tp.group * (t1 - t0 + 1);
  // of these this CTA finishes rows_each, from own_first on (fewer at the end)
  const int rank = static_cast<int>(blockIdx.y);
  const int rows_each = tp.by_splits.div(n_rows + p.splits - 1), own_first = rank * rows_each;
  const int own = own_first >= n_rows ? 0 : own_first + rows_each < n_rows ? rows_each : n_rows - own_first;
  // Set-up by different warps at once: the barriers, and behind them the loads of Q and of the first block, whose latency then
  // passes under the rest of it (B=1 H=16 D=128, 64 over 16,448: 31.5 -> 29.6 us; every stage's loads there would hold up the
  // others: B=14 H=12 D=32, 8 over 3,000, 39.9 -> 43 us).
  const int ahead = n_blocks < 1 ? 0 : 1;
  auto load_k = [&](int i) {
    const int s = i % STAGES, j = range.at(n_begin + i);
    mbar_expect_tx(bar(K_FULL + s), L::kTileBytes);
    for (int x = 0; x < kBoxes; ++x)
      tma_load_4d(base + L::kK + s * L::kTileBytes + x * kBoxBytes, &tm_k, bar(K_FULL + s), 64 * x, j * kTile, hk, b);
  };
  auto load_v = [&](int i) {
    const int s = i % STAGES, j = range.at(n_begin + i);
    mbar_arrive_expect_tx(bar(V_FULL + s), L::kTileBytes);
    for (int x = 0; x < kBoxes; ++x)
      tma_load_4d(base + L::kV + s * L::kTileBytes + x * kBoxBytes, &tm_v, bar(V_FULL + s), 64 * x, j * kTile, hk, b);
  };
  if (warp == 8) {
    if (lane < 3) tma_prefetch_desc(lane == 0 ? &tm_q : lane == 1 ? &tm_k : &tm_v);
    for (int i = lane; i < L::kNumBars; i += 32)
      mbar_init(bar(i), i >= P_FULL && i < P_FULL + 2 ? 128u : i == GROUP ? 256u : i >= V_CLEAN ? 2u : 1u);
    fence_mbar_init();
    __syncwarp();
    grid_dep_wait();
    if (lane == 0) {
      if (p.splits > 1) mbar_arrive_expect_tx(bar(RECEIVED), p.splits * own * L::kPitch);
      mbar_arrive_expect_tx(bar(Q_FULL), COPIES * kBoxes * tp.group * tp.tq_tile * 128);
      for (int x = 0; x < COPIES * kBoxes; ++x)
        tma_load_4d(base + L::kQ + x / COPIES * kBoxBytes + x % COPIES * kLanes * 128, &tm_q, bar(Q_FULL), 64 * (x / COPIES), hk * tp.group, t0, b);
      for (int i = 0; i < ahead; ++i) {
        load_k(i);
        load_v(i);
      }
    }
    __syncwarp();
  }
  if (threadIdx.x == 0) {
    *spoilt_flag = 0;
    *abort_flag = (*reinterpret_cast<volatile unsigned*>(tp.status) != STATUS_OK) ? 1 : 0;
  }
  if (warp == 9) {
    tmem_alloc(base + L::kTmemSlot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const bool dead = *abort_flag != 0;
  // the tile's query positions, as a range (every lane of a warp)
  auto tile_positions = [&](int& qp_min, int& qp_max) {
    if (!p.qpos) {
      qp_min = p.L - p.Tq + t0;
      qp_max = p.L - p.Tq + t1;
      return;
    }
    qp_min = INT_MAX;
    qp_max = -INT_MAX;
    for (int t = t0 + lane; t <= t1; t += 32) {
      const int x = cached::query_position(p, t);
      qp_min = x < qp_min ? x : qp_min;
      qp_max = x > qp_max ? x : qp_max;
    }
    qp_min = __reduce_min_sync(0xffffffffu, qp_min);
    qp_max = __reduce_max_sync(0xffffffffu, qp_max);
  };

  grid_dep_wait();
  grid_dep_release();

  if (warp >= 8) {
    setmaxnreg_dec<kRegsOther>();
    static_assert((kRegsLaunch - kRegsOther) * 4 >= (kRegsCompute - kRegsLaunch) * 8, "register reallocation does not balance");
    if (dead) {
      // A give-up recorded earlier makes this launch a no-op.  Its loads are in flight: they land before the CTA leaves.
      if (warp == 8 && lane == 0) {
        const unsigned long long t0 = globaltimer_ns();
        auto landed = [&](uint32_t bb) {
          while (!mbar_try_wait(bb, 0))
            if (globaltimer_ns() - t0 > wctx.limit()) break;
        };
        landed(bar(Q_FULL));
        for (int i = 0; i < ahead; ++i) {
          mbar_arrive(bar(K_FULL + i));                          // (the arrival that brings the block's positions)
          landed(bar(K_FULL + i));
          landed(bar(V_FULL + i));
        }
      }
    } else if (!SPLIT_P && warp >= 10) {
      // spare warps
    } else if (warp >= 10) {
      // ============ V of blocks the mask cuts: no hidden infinities and NaN ====
      int qp_min, qp_max;
      tile_positions(qp_min, qp_max);
      for (int i = 0; i < n_blocks; ++i) {
        const int s = i % STAGES;
        const uint32_t ph = (i / STAGES) & 1;
        if (!__all_sync(0xffffffffu, mbar_wait(bar(K_FULL + s), ph, wctx, 71))) break;      // the block's positions
        if (full_flag[s] == 0) {
          if (!__all_sync(0xffffffffu, mbar_wait(bar(V_FULL + s), ph, wctx, 72))) break;
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            const int r = 64 * (warp - 10) + 32 * half + lane;
            const int kp = *reinterpret_cast<const int*>(gen + L::kPos + s * 512 + 4 * r);
            if (kp == kNoKey) continue;                                      // past the end: zeros already
            const bool shown = (!p.causal || kp <= qp_max) &&                // to some query, perhaps
                               (p.window == 0 || kp > qp_min - (p.window - p.sinks) || kp < p.sinks);
            uint4* tile_row = reinterpret_cast<uint4*>(gen + L::kV + s * L::kTileBytes + r * 128);
#pragma unroll
            for (int x = 0; x < kBoxes; ++x) {
              uint4* piece = tile_row + x * (kBoxBytes / 16);                // [8], met in another order by each lane: banks
              if (!shown) {
#pragma unroll
                for (int n = 0; n < 8; ++n) piece[n ^ (lane & 7)] = make_uint4(0u, 0u, 0u, 0u);
                continue;
              }
              bool finite = true;
#pragma unroll
              for (int n = 0; n < 8; ++n) finite &= Pack2<T>::finite(piece[n ^ (lane & 7)]);
              if (finite) continue;
              *spoilt_flag = 1;
              T* e = reinterpret_cast<T*>(piece);
              for (int c = 0; c < 64; ++c)
                if (!isfinite(static_cast<float>(e[c]))) e[c] = static_cast<T>(0.f);
            }
          }
          fence_proxy_async_smem();
          __syncwarp();
        }
        if (lane == 0) mbar_arrive(bar(V_CLEAN + s));
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(SCANNED));                  // the flag is final
    } else if (warp == 8) {
      // =============================== TMA producer ============================
      int qp_min, qp_max;
      tile_positions(qp_min, qp_max);
      bool ok = true;
      for (int i = 0; ok && i < n_blocks; ++i) {
        const int j = range.at(n_begin + i);
        const int s = i % STAGES;
        const uint32_t ph = (i / STAGES) & 1;
        if (i >= ahead) {
          if (lane == 0) {
            ok = mbar_wait(bar(K_EMPTY + s), ph ^ 1, wctx, 60);
            if (ok) {
              load_k(i);
              ok = mbar_wait(bar(V_EMPTY + s), ph ^ 1, wctx, 61);
            }
            if (ok) load_v(i);
          }
          ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
          if (!ok) break;
        }
        // positions of the block's keys (a key past the end of the cache gets the "no key" mark), and whether
        // the mask cuts the block at all
        int kp_min = j * kTile, kp_max = j * kTile + kTile - 1;
        const bool whole = (j + 1) * kTile <= p.L;
        if (p.kpos || !whole || !cached::all_visible(p, kp_min, kp_max, qp_min, qp_max)) {
          int* pos = reinterpret_cast<int*>(gen + L::kPos + s * 512);
          kp_min = INT_MAX;
          kp_max = -INT_MAX;
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int c = 4 * lane + e, key = j * kTile + c;
            // (without a mask by positions they may be anything, the mark for "no key" among them)
            const int x = key >= p.L ? kNoKey : p.causal ? cached::key_position(p, key) : 0;
            pos[c] = x;
            kp_min = x < kp_min ? x : kp_min;
            kp_max = x > kp_max ? x : kp_max;
          }
          kp_min = __reduce_min_sync(0xffffffffu, kp_min);
          kp_max = __reduce_max_sync(0xffffffffu, kp_max);
        }
        if (lane == 0) full_flag[s] = whole && cached::all_visible(p, kp_min, kp_max, qp_min, qp_max) ? 1 : 0;
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(K_FULL + s));              // both travel with the K tile
      }
    } else {
      // ================================ MMA issuer =============================
      const uint32_t leader = elect_one() ? 1u : 0u;
      const uint32_t tmem_u = __shfl_sync(0xffffffffu, *tmem_slot, 0);
      auto wait_all = [&](uint32_t bb, uint32_t parity, unsigned where) -> bool {
        return __all_sync(0xffffffffu, mbar_wait(bb, parity, wctx, where));
      };
      constexpr uint32_t idesc_qk = make_idesc(kBf16, 128, 128, false, false);
      constexpr uint32_t idesc_pv = make_idesc(kBf16, 128, D, false, true);
      bool ok = wait_all(bar(Q_FULL), 0, 62);
      auto do_s = [&](int i) {
        const int s = i % STAGES;
        if (!(ok = wait_all(bar(K_FULL + s), (i / STAGES) & 1, 63))) return;
        tc_fence_after();
        const uint32_t qa = base + L::kQ, ka = base + L::kK + s * L::kTileBytes;
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          const uint32_t off = (kk >> 2) * kBoxBytes + (kk & 3) * 32;
          umma_ss(leader, tmem_u + 128 * (i & 1), make_smem_desc(qa + off, 16, 1024), make_smem_desc(ka + off, 16, 1024),
                  idesc_qk, kk > 0 ? 1u : 0u);
        }
        umma_commit(leader, bar(S_FULL + (i & 1)));
        umma_commit(leader, bar(K_EMPTY + s));
      };
      auto do_pv = [&](int i) {
        const int s = i % STAGES, w = i & 1;
        if (!(ok = wait_all(bar(P_FULL + w), (i >> 1) & 1, 64))) return;
        if (!(ok = wait_all(bar(V_FULL + s), (i / STAGES) & 1, 65))) return;
        if (SPLIT_P && !(ok = wait_all(bar(V_CLEAN + s), (i / STAGES) & 1, 68))) return;
        tc_fence_after();
        const uint32_t va = base + L::kV + s * L::kTileBytes;
#pragma unroll
        for (int part = 0; part < (SPLIT_P ? 2 : 1); ++part) {
#pragma unroll
          for (int kk = 0; kk < kTile / 16; ++kk)
            umma_ts(leader, tmem_u + 256 + D * w, tmem_u + 128 * w + 64 * part + 8 * kk,
                    make_smem_desc(va + kk * 2048, kBoxBytes, 1024), idesc_pv, (i > 1 || part > 0 || kk > 0) ? 1u : 0u);
        }
        umma_commit(leader, bar(V_EMPTY + s));
      };
      // S of block i goes out before P V of block i - 1 (the other warpgroup's); it overwrites the P that block
      // i - 2's product, issued before it, reads
      for (int i = 0; ok && i < n_blocks; ++i) {
        do_s(i);
        if (ok && i > 0) do_pv(i - 1);
      }
      if (ok && n_blocks > 0) do_pv(n_blocks - 1);
      if (ok) umma_commit(leader, bar(O_DONE));
    }
    __syncwarp();
    for (int i = 0; i < 2; ++i) {
      cluster_arrive_relaxed();
      cluster_wait();
    }
  } else {
    // ================================= softmax ===============================
    setmaxnreg_inc<kRegsCompute>();
    if (!dead) {
    const int w = warp >> 2;                                     // warpgroup: blocks w, w + 2, ...
    const int copy = (threadIdx.x & 127) / kLanes;               // the same for the whole warp
    const int row = threadIdx.x % kLanes;                        // row of the tile; its TMEM lane is kLanes * copy + row
    const uint32_t lane_base = 32u * (warp & 3);
    const uint32_t p_addr = tmem_addr(tmem, lane_base, 128 * w), s_addr = p_addr + kCols * copy;
    const uint32_t o_addr = tmem_addr(tmem, lane_base, 256 + D * w);
    const bool valid = row < n_rows;
    const bool warp_rows = row - lane < n_rows;                  // some row of this warp belongs to a query
    const int qp = valid ? cached::query_position(p, t0 + tp.by_group.div(row)) : 0;
    const int span = p.window - p.sinks;
    const uint64_t scale2 = pack_f2(p.scale_log2, p.scale_log2);
    float m_ref = -INFINITY, l = 0.f;
    bool ok = true;
    for (int i = w; i < n_blocks; i += 2) {
      const int s = i % STAGES;
      ok = mbar_wait(bar(S_FULL + w), (i >> 1) & 1, wctx, 66);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      if (!warp_rows) {                                          // nothing of this warp's is ever read
        mbar_arrive(bar(P_FULL + w));
        continue;
      }
      tc_fence_after();
      uint32_t sv[kCols / 32][32];
#pragma unroll
      for (int c = 0; c < kCols / 32; ++c) tmem_ld32(s_addr + 32 * c, sv[c]);
      // (the stage's positions and flag stay: the producer rewrites them only once V_EMPTY says that this block's
      // P V product, which waits for this warpgroup, has completed)
      const bool full = full_flag[s] != 0;
      tc_wait_ld();
      if (!full) {
        const int4* pos4 = reinterpret_cast<const int4*>(gen + L::kPos + s * 512) + kCols / 4 * copy;
#pragma unroll
        for (int c = 0; c < kCols / 32; ++c) {
#pragma unroll
          for (int e = 0; e < 32; e += 4) {
            const int4 kp = pos4[8 * c + e / 4];
            const int k4[4] = {kp.x, kp.y, kp.z, kp.w};
#pragma unroll
            for (int x = 0; x < 4; ++x) {
              bool vis = k4[x] != kNoKey;
              if (p.causal) vis = vis && k4[x] <= qp;
              if (p.window > 0) vis = vis && (k4[x] > qp - span || k4[x] < p.sinks);
              if (!vis) sv[c][e + x] = __float_as_uint(-INFINITY);
            }
          }
        }
      }
      float b0 = -INFINITY, b1 = -INFINITY;
#pragma unroll
      for (int c = 0; c < kCols / 32; ++c) {
#pragma unroll
        for (int e = 0; e < 32; e += 4) {
          b0 = fmax3(b0, __uint_as_float(sv[c][e]), __uint_as_float(sv[c][e + 1]));
          b1 = fmax3(b1, __uint_as_float(sv[c][e + 2]), __uint_as_float(sv[c][e + 3]));
        }
      }
      const float mx = fmaxf(b0, b1) * p.scale_log2;
      // Online softmax in base 2 with a reference exponent that is only raised (with O and l
      // rescaled) when a block's maximum exceeds it by more than 2^8.
      float alpha = 1.f;
      bool rescale = false;
      if (mx > m_ref + 8.f || m_ref == -INFINITY) {
        if (m_ref != -INFINITY) {
          alpha = fast_exp2(m_ref - mx);
          rescale = true;
          l *= alpha;
        }
        m_ref = mx;                                                // may still be -inf: nothing seen yet
      }
      // this warpgroup's previous P V product is complete (it was issued before this block's S, whose
      // completion S_FULL reports): O may be rescaled, S and P overwritten
      if (i > 1 && __any_sync(0xffffffffu, rescale)) {
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
          uint32_t orr[32];
          tmem_ld32(o_addr + 32 * c, orr);
          tc_wait_ld();
#pragma unroll
          for (int e = 0; e < 32; ++e) orr[e] = __float_as_uint(__uint_as_float(orr[e]) * alpha);
          tmem_st32(o_addr + 32 * c, orr);
        }
      }
      const float m_use = (m_ref == -INFINITY) ? 0.f : m_ref;
      const uint64_t negm2 = pack_f2(-m_use, -m_use);
      uint64_t acc0 = 0ull, acc1 = 0ull;
#pragma unroll
      for (int c = 0; c < kCols / 32; ++c) {
        uint32_t pk[16], lo[16];
#pragma unroll
        for (int e = 0; e < 32; e += 4) {
          float e0, e1, e2, e3;
          unpack_f2(ffma2(pack_f2(__uint_as_float(sv[c][e]), __uint_as_float(sv[c][e + 1])), scale2, negm2), e0, e1);
          unpack_f2(ffma2(pack_f2(__uint_as_float(sv[c][e + 2]), __uint_as_float(sv[c][e + 3])), scale2, negm2), e2, e3);
          e0 = fast_exp2(e0); e1 = fast_exp2(e1); e2 = fast_exp2(e2); e3 = fast_exp2(e3);
          acc0 = fadd2(acc0, pack_f2(e0, e1));
          acc1 = fadd2(acc1, pack_f2(e2, e3));
          pk[e / 2] = Pack2<T>::pack(e0, e1);
          pk[e / 2 + 1] = Pack2<T>::pack(e2, e3);
          if constexpr (SPLIT_P) {                                 // what the rounding left
            T r[4];
            *reinterpret_cast<uint32_t*>(r) = pk[e / 2];
            *reinterpret_cast<uint32_t*>(r + 2) = pk[e / 2 + 1];
            lo[e / 2] = Pack2<T>::pack(e0 - static_cast<float>(r[0]), e1 - static_cast<float>(r[1]));
            lo[e / 2 + 1] = Pack2<T>::pack(e2 - static_cast<float>(r[2]), e3 - static_cast<float>(r[3]));
          }
        }
        tmem_st16(p_addr + kCols / 2 * copy + 16 * c, pk);
        if constexpr (SPLIT_P) tmem_st16(p_addr + 64 + kCols / 2 * copy + 16 * c, lo);
      }
      // the other copies' keys: nothing here
      if constexpr (COPIES > 1) {
        const uint32_t zero[16] = {};
#pragma unroll
        for (int c = 0; c < (COPIES - 1) * kCols / 32; ++c) {
          const uint32_t at = p_addr + (kCols / 2 * (copy + 1) + 16 * c) % 64;
          tmem_st16(at, zero);
          if constexpr (SPLIT_P) tmem_st16(at + 64, zero);
        }
      }
      {
        float x, y;
        unpack_f2(fadd2(acc0, acc1), x, y);
        l += x + y;
      }
      tc_wait_st();
      tc_fence_before();
      mbar_arrive(bar(P_FULL + w));
    }
    // A row's parts -- of either warpgroup and every copy -- become one.  Their statistics are exchanged first, over Q, while the
    // last products run: Q is dead when both warpgroups' last score products have completed.
    constexpr int kParts = 2 * COPIES, kSlice = D / kParts;
    const bool split = p.splits > 1;
    const int part = w * COPIES + copy;
    const bool any = w < n_blocks;
    auto group_sync = [&](uint32_t parity) {
      mbar_arrive(bar(GROUP));
      const bool met = mbar_wait(bar(GROUP), parity, wctx, 69);
      ok = __all_sync(0xffffffffu, ok && met && *abort_flag == 0);
    };
    ok = ok && mbar_wait(bar(Q_FULL), 0, wctx, 73);
    if (ok && (w ^ 1) < n_blocks) {
      const int last = n_blocks - 1 - ((n_blocks - 1 - (w ^ 1)) & 1);        // the other warpgroup's
      ok = mbar_wait(bar(S_FULL + (w ^ 1)), (last >> 1) & 1, wctx, 74);
    }
    float2* stats = reinterpret_cast<float2*>(gen + L::kQ) + row;            // [kParts][kLanes]
    if (warp_rows) stats[part * kLanes] = any ? make_float2(m_ref, l) : make_float2(-INFINITY, 0.f);
    group_sync(0);
    float mx = -INFINITY, sum = 0.f;
#pragma unroll
    for (int x = 0; x < kParts; ++x) mx = fmaxf(mx, stats[x * kLanes].x);
    const float ref = mx == -INFINITY ? 0.f : mx;
#pragma unroll
    for (int x = 0; x < kParts; ++x) {
      const float2 ml = stats[x * kLanes];
      sum = fmaf(exp2f(ml.x - ref), ml.y, sum);                              // a part that saw no key: 0
    }
    const float f_first = exp2f(stats[copy * kLanes].x - ref), f_second = exp2f(stats[(COPIES + copy) * kLanes].x - ref);
    if (ok) ok = mbar_wait(bar(O_DONE), 0, wctx, 67);
    if constexpr (SPLIT_P) {
      const bool met = mbar_wait(bar(SCANNED), 0, wctx, 72);
      ok = ok && met;
    }
    ok = __all_sync(0xffffffffu, ok);
    if (ok) tc_fence_after();
    // Every product that read the tiles in shared memory is complete: the other CTAs may write there.
    __syncwarp();
    cluster_arrive_relaxed();
    // Both warpgroups' sums of a row stand in the same TMEM lane: each warpgroup adds up its half of the columns.  With
    // copies, each thread hands its sums over and adds up one slice of the half.
    constexpr int kHalf = D / 2;
    float sums[kHalf];
#pragma unroll
    for (int c = 0; c < kHalf; ++c) sums[c] = 0.f;
    const bool has_columns = warp_rows && kHalf * w < p.D;                   // (head dim 32 on 64-wide tiles: the first half)
    if (ok && has_columns) {
      const uint32_t at = tmem_addr(tmem, lane_base, 256 + kHalf * w);
      auto add = [&](uint32_t from, float weight) {
#pragma unroll
        for (int c = 0; c < kHalf; c += 32) {
          uint32_t x[32];
          tmem_ld32(from + c, x);
          tc_wait_ld();
#pragma unroll
          for (int e = 0; e < 32; ++e) sums[c + e] = fmaf(weight, __uint_as_float(x[e]), sums[c + e]);
        }
      };
      if (n_blocks > 0) add(at, f_first);
      if (n_blocks > 1) add(at + D, f_second);                               // (what no product wrote may be anything)
    }
    auto put = [&](uint8_t* to, const float* v, int n) {
#pragma unroll
      for (int c = 0; c < n; c += 4) *reinterpret_cast<float4*>(to + 4 * c) = make_float4(v[c], v[c + 1], v[c + 2], v[c + 3]);
    };
    const int col = kHalf * w + kSlice * copy;                               // first column of this thread's slice
    if constexpr (COPIES > 1) {
      if (ok && has_columns) put(gen + L::kK + (kLanes * copy + row) * L::kPitch + 4 * kHalf * w, sums, kHalf);
      group_sync(1);
      if (ok && has_columns) {
        const uint8_t* from = gen + L::kK + row * L::kPitch + 4 * col;
#pragma unroll
        for (int c = 0; c < kSlice; c += 4) {
          float4 acc = *reinterpret_cast<const float4*>(from + 4 * c);
#pragma unroll
          for (int x = 1; x < COPIES; ++x) {
            const float4 y = *reinterpret_cast<const float4*>(from + x * kLanes * L::kPitch + 4 * c);
            acc = make_float4(acc.x + y.x, acc.y + y.y, acc.z + y.z, acc.w + y.w);
          }
          sums[c] = acc.x; sums[c + 1] = acc.y; sums[c + 2] = acc.z; sums[c + 3] = acc.w;
        }
      }
    }
    const float spoilt = SPLIT_P && *spoilt_flag != 0 ? 1.f : 0.f;           // values were taken out of V
    // `n` columns (a multiple of four) of a row of the tile, from its sums, its maximum and its sum of exponentials
    auto finish = [&](int r, int c, const float* v, auto n, float mx, float sum, bool odd) {
      constexpr int N = decltype(n)::value < 8 ? 4 : 8;
      const int at = tp.by_group.div(r), t = t0 + at, h = hk * tp.group + (r - at * tp.group);
      const float inv = sum > 0.f ? 1.f / sum : 0.f;                         // a row that sees no key gives zeros
      T* out = static_cast<T*>(p.o) + ((static_cast<long long>(b) * p.Tq + t) * p.H + h) * p.D + c;
#pragma unroll
      for (int e = 0; e < decltype(n)::value; e += N) {
        if (c + e >= p.D) break;                                             // head dim 32 on 64-wide tiles
        float x[N], total = 0.f;
#pragma unroll
        for (int i = 0; i < N; ++i) {
          x[i] = v[e + i] * inv;
          total += x[i];
        }
        if constexpr (SPLIT_P) {
          // (a row whose own sum is NaN stays NaN)
          if (sum > 0.f && (odd || isnan(total)))
            put_right<T, N>(p, static_cast<const T*>(tp.v) + (static_cast<long long>(b) * p.Hkv + hk) * p.L * p.D + c + e, t, x);
        }
        uint32_t packed[N / 2];
#pragma unroll
        for (int i = 0; i < N; i += 2) packed[i / 2] = Pack2<T>::pack(x[i], x[i + 1]);
        if constexpr (N == 8) *reinterpret_cast<uint4*>(out + e) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
        else *reinterpret_cast<uint2*>(out + e) = make_uint2(packed[0], packed[1]);
      }
      if (p.lse && c == 0)
        p.lse[(static_cast<long long>(b) * p.H + h) * p.Tq + t] = sum > 0.f ? (mx + log2f(sum)) * kLn2 : -INFINITY;
    };
    if (split) {
      if (ok && warp_rows) {
        uint8_t* to = gen + L::kRows + row * L::kPitch;
        if (has_columns) put(to + 4 * col, sums, kSlice);
        if (part == 0) *reinterpret_cast<float4*>(to + 4 * D) = make_float4(mx, 0.f, sum, spoilt);
      }
      fence_proxy_async_smem();
      group_sync(COPIES > 1 ? 0 : 1);
      cluster_wait();                              // every CTA's tiles are dead
      // each CTA of the cluster gets the rows it finishes
      if (ok && warp == 0 && lane < p.splits) {
        const int first = lane * rows_each, count = first + rows_each < n_rows ? rows_each : n_rows - first;
        if (count > 0)
          bulk_copy_cluster(cluster_addr(base + L::kReceived + rank * rows_each * L::kPitch, lane),
                            base + L::kRows + first * L::kPitch, count * L::kPitch, cluster_addr(bar(RECEIVED), lane));
      }
      __syncwarp();
      if (ok) ok = mbar_wait(bar(RECEIVED), 0, wctx, 70);
      ok = __all_sync(0xffffffffu, ok);
      if (ok) {
        // one thread per eight columns of the rows this CTA finishes, or where that leaves threads enough per four; the parts
        // in the order of the CTAs
        auto rows = [&](auto n) {
          constexpr int N = decltype(n)::value;
          for (int i = threadIdx.x; i < own * (D / N); i += 256) {
            const int k = i / (D / N), c = N * (i % (D / N));
            if (c >= p.D) continue;                                          // head dim 32 on 64-wide tiles
            const uint8_t* at = gen + L::kReceived + k * L::kPitch;
            const int step = rows_each * L::kPitch;
            // (all loads of a kind at once: one after another their latency was most of this)
            float m[kMostCluster], mx = -INFINITY, sum = 0.f;
#pragma unroll
            for (int s = 0; s < kMostCluster; ++s) m[s] = s < p.splits ? *reinterpret_cast<const float*>(at + s * step + 4 * D) : -INFINITY;
#pragma unroll
            for (int s = 0; s < kMostCluster; ++s) mx = fmaxf(mx, m[s]);
            const float ref = mx == -INFINITY ? 0.f : mx;
            float v[N] = {};
            bool odd = false;
#pragma unroll
            for (int s = 0; s < kMostCluster; ++s) {
              if (s >= p.splits) break;
              const float2 l = *reinterpret_cast<const float2*>(at + s * step + 4 * D + 8);
              const float f = exp2f(m[s] - ref);
              sum = fmaf(f, l.x, sum);
#pragma unroll
              for (int e = 0; e < N; e += 4) {
                const float4 y = *reinterpret_cast<const float4*>(at + s * step + 4 * (c + e));
                v[e] = fmaf(f, y.x, v[e]); v[e + 1] = fmaf(f, y.y, v[e + 1]);
                v[e + 2] = fmaf(f, y.z, v[e + 2]); v[e + 3] = fmaf(f, y.w, v[e + 3]);
              }
              if (SPLIT_P) odd |= l.y != 0.f;
            }
            finish(own_first + k, c, v, n, mx, sum, odd);
          }
        };
        if (own * (D / 4) > 256) rows(std::integral_constant<int, 8>{});
        else rows(std::integral_constant<int, 4>{});
      }
      __syncwarp();
      cluster_arrive_relaxed();                    // what the others sent is here
    } else {
      cluster_wait();
      cluster_arrive_relaxed();
      if (ok && valid) finish(row, col, sums, std::integral_constant<int, kSlice>{}, mx, sum, spoilt != 0.f);
    }
    } else {
      cluster_arrive_relaxed();
      cluster_wait();
      cluster_arrive_relaxed();
    }
    __syncwarp();
    cluster_wait();                                // what this CTA sent has arrived
  }

  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    tc_fence_after();
    tmem_dealloc(tmem, kTmemCols);
  }
}

template <typename T, int D, int STAGES, int COPIES, bool SPLIT_P>
int launch_t(CachedParams p, TileParams tp, int n_blocks, const CUtensorMap& mq, const CUtensorMap& mk,
             const CUtensorMap& mv, cudaStream_t stream) {
  using L = CachedSmem<D, STAGES, COPIES>;
  static_assert(L::kDynamic <= 232448, "over the shared memory a CTA can have");
  auto kern = cached_tc_kernel<T, D, STAGES, COPIES, SPLIT_P>;
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(kern), L::kDynamic) != NLFA_OK) return NLFA_ERR_CUDA;
  // As many CTAs per query tile as can be resident at once, with at least two key blocks (one per softmax
  // warpgroup) each.
  const int tiles = p.B * p.Hkv * tp.n_qtiles;
  p.splits = cached::cluster_splits(reinterpret_cast<const void*>(kern), 384, L::kDynamic, tiles, (n_blocks + 1) / 2);
  tp.by_splits = FastDiv(p.splits);
  const dim3 grid(static_cast<unsigned>(tiles), static_cast<unsigned>(p.splits));
  if (launch_cluster(kern, grid, dim3(384), L::kDynamic, stream, overlap_launches(kOverlapFwd), p.splits, mq, mk, mv, p, tp) !=
      cudaSuccess) {
    (void)cudaGetLastError();
    return NLFA_ERR_CUDA;
  }
  return NLFA_OK;
}

template <typename T, int D, int STAGES, bool SPLIT_P>
int launch_copies(const CachedParams& p, const TileParams& tp, int n_blocks, const CUtensorMap& mq, const CUtensorMap& mk,
                  const CUtensorMap& mv, cudaStream_t stream) {
  const int rows = tp.group * tp.tq_tile;
  if (rows <= kTile / 4) return launch_t<T, D, STAGES, 4, SPLIT_P>(p, tp, n_blocks, mq, mk, mv, stream);
  if (rows <= kTile / 2) return launch_t<T, D, STAGES, 2, SPLIT_P>(p, tp, n_blocks, mq, mk, mv, stream);
  return launch_t<T, D, STAGES, 1, SPLIT_P>(p, tp, n_blocks, mq, mk, mv, stream);
}

template <typename T>
int launch_for(const CachedParams& p, const TileParams& tp, int n_blocks, bool split_p, const CUtensorMap& mq,
               const CUtensorMap& mk, const CUtensorMap& mv, cudaStream_t stream) {
  if (p.D <= 64)
    return split_p ? launch_copies<T, 64, 5, true>(p, tp, n_blocks, mq, mk, mv, stream)
                   : launch_copies<T, 64, 5, false>(p, tp, n_blocks, mq, mk, mv, stream);
  return split_p ? launch_copies<T, 128, 3, true>(p, tp, n_blocks, mq, mk, mv, stream)
                 : launch_copies<T, 128, 3, false>(p, tp, n_blocks, mq, mk, mv, stream);
}

int positions_per_tile(int Tq, int group) { return Tq < kTile / group ? Tq : kTile / group; }

}  // namespace

bool cached_tc_can(int H, int Hkv, int D, int dtype);

// What a caller may force: blocks of at least 16 rows per KV head over at least 256 keys.
bool cached_tc_applies(int Tq, int H, int Hkv, int L, int D, int dtype) {
  if (!cached_tc_can(H, Hkv, D, dtype)) return false;
  return positions_per_tile(Tq, H / Hkv) * (H / Hkv) >= 16 && L >= 2 * kTile;
}
// What the kernel can run: any block.
bool cached_tc_can(int H, int Hkv, int D, int dtype) {
  return (dtype == NLFA_DTYPE_F16 || dtype == NLFA_DTYPE_BF16) && (D == 32 || D == 64 || D == 128) && H / Hkv <= kTile;
}

int launch_fwd_cached_tc(CachedParams p, const void* q, const void* k_cache, const void* v_cache, int dtype, bool split_p,
                         unsigned* status, cudaStream_t stream) {
  TileParams tp;
  tp.group = p.H / p.Hkv;
  tp.by_group = FastDiv(tp.group);
  tp.tq_tile = positions_per_tile(p.Tq, tp.group);
  tp.n_qtiles = (p.Tq + tp.tq_tile - 1) / tp.tq_tile;
  tp.by_qtiles = FastDiv(tp.n_qtiles);
  tp.by_heads = FastDiv(p.Hkv);
  tp.status = status;
  tp.v = v_cache;
  int n_blocks = 0;                                         // key blocks of the tile that sees the most
  for (int qt = 0; qt < tp.n_qtiles; ++qt) {
    const int t0 = qt * tp.tq_tile, t1 = (t0 + tp.tq_tile < p.Tq ? t0 + tp.tq_tile : p.Tq) - 1;
    const KeyRange r = cached::key_range(p.Tq, p.L, p.qpos != nullptr || p.kpos != nullptr, p.causal, p.window, p.sinks, t0, t1, kTile);
    n_blocks = r.count > n_blocks ? r.count : n_blocks;
  }
  // q [B,Tq,H,D]: box = 64 columns x the group's heads x tq_tile positions -> rows (t, g) of 128 bytes
  // k, v [B,Hkv,L,D]: box = 64 columns x 128 keys
  const unsigned long long e = 2, D = p.D, H = p.H, Hkv = p.Hkv, Tq = p.Tq, L = p.L;
  const unsigned long long q_dims[4] = {D, H, Tq, static_cast<unsigned long long>(p.B)};
  const unsigned long long q_str[3] = {D * e, H * D * e, Tq * H * D * e};
  const unsigned q_box[4] = {64u, static_cast<unsigned>(tp.group), static_cast<unsigned>(tp.tq_tile), 1u};
  const unsigned long long k_dims[4] = {D, L, Hkv, static_cast<unsigned long long>(p.B)};
  const unsigned long long k_str[3] = {D * e, L * D * e, Hkv * L * D * e};
  const unsigned k_box[4] = {64u, static_cast<unsigned>(kTile), 1u, 1u};
  CUtensorMap mq, mk, mv;
  int st = make_map(&mq, q, dtype, q_dims, q_str, q_box);
  if (st == NLFA_OK) st = make_map(&mk, k_cache, dtype, k_dims, k_str, k_box);
  if (st == NLFA_OK) st = make_map(&mv, v_cache, dtype, k_dims, k_str, k_box);
  if (st != NLFA_OK) return st;
  return dtype == NLFA_DTYPE_BF16 ? launch_for<__nv_bfloat16>(p, tp, n_blocks, split_p, mq, mk, mv, stream)
                                  : launch_for<__half>(p, tp, n_blocks, split_p, mq, mk, mv, stream);
}

}  // namespace nlfa
