// dQ from the dS tiles the dK/dV pass leaves behind (bwd_tc.cu, MODE_DKV_DS): dQ_i = scale * sum_j dS_ij K_j,
// one product per (query tile, key block) where recomputing dS takes three and a second exponent phase.
// Head dim 128 (see launch_both in bwd_tc.cu for why).
//
// A work unit is two consecutive 128-row query tiles of one (batch, head); the CTA streams, per 64 keys, their
// two dS half tiles (16 KB each, contiguous in the scratch: one untiled bulk copy) and the K rows (TMA), and
// accumulates both tiles in TMEM.  The accumulators are double buffered, so the epilogue of a unit runs under
// the next one's products.  Bound by reading dS: 2.18 GB (B=2 H=16 T=8192) in 0.41 ms = 5.3 TB/s, 81% of the
// measured copy bandwidth; two query tiles per unit, because each K row is then read half as often.  dS lies in the scratch exactly as the product reads it: [64 keys][8 queries] pieces
// of 16 bytes, i.e. an MN-major operand without swizzle (its core matrices, 8 keys x 8 queries, are 128
// contiguous bytes), which is also what lets the dK/dV pass store it with fully coalesced 16-byte stores.
//
// Warps: 0 scheduler + producer, 1 MMA issuer and TMEM owner, 2-3 idle, 4-7 epilogue.
// Every wait is bounded (ptx.cuh); no multicast.
#include "common.cuh"
#include "ptx.cuh"

namespace nlfa {
namespace {

constexpr int kNT = 2;                             // query tiles per unit
constexpr int kHalfTile = kDsTileBytes / 2;        // 64 keys x 128 queries, 16 bit

struct DqParams {
  int H, Hkv;
  int window, sinks, block;
  int n_tiles, n_units, heads, total_units;        // heads: query heads of this launch
  int first_head;                                  // b * H + h of the first one
  int sched_group;                                 // query heads whose units are handed out together
  DsLayout layout;
  int per_head;                                    // dS tiles per head
  const uint8_t* ds;
  float scale;
  unsigned* status;
  unsigned* sched;
};

constexpr int D = 128;

struct DqSmem {
  static constexpr int kKBytes = 64 * D * 2;
  static constexpr int kStage = kNT * kHalfTile + kKBytes;
  static constexpr int kOut = 128 * D * 2;                     // one output tile, staged for its TMA store
  static constexpr int STAGES = 4;
  static constexpr int kBar = STAGES * kStage + kOut;
  // full[S], empty[S], acc_full[2], acc_empty[2], group, sched_full[kRing]
  static constexpr int kRing = 8;
  static constexpr int kNumBars = 2 * STAGES + 5 + kRing;
  static constexpr int kSched = (kBar + 8 * kNumBars + 15) / 16 * 16;
  static constexpr int kTmemSlot = kSched + 64 * kRing;
  static constexpr int kAbort = kTmemSlot + 4;
  static constexpr int kTotal = kAbort + 4;
  static constexpr int kDynamic = kTotal + 1024;
};

struct DqUnit {
  int head, b, h, hk, tile0, lo, extra, n_iters;
  TileRange tr[kNT];
  bool valid1;                                     // the second tile exists (the first always does)
  __device__ __forceinline__ int block_at(int it) const { return it < extra ? it : lo + (it - extra); }
  __device__ __forceinline__ bool sees(int t, int j) const {
    return (t == 0 || valid1) && j <= tr[t].hi && (j >= tr[t].lo || j < tr[t].sink_blocks);
  }
};

__device__ __forceinline__ DqUnit make_dq_unit(int u, const DqParams& p) {
  DqUnit w;
  // Groups of heads, the last ones first: their dS tiles were written last and are the likeliest to be in L2
  // still.  Inside a group the longest units (late query tiles) first.
  const int per_group = p.sched_group * p.n_units;
  const int last0 = p.heads - p.sched_group * (u / per_group);              // one past the group's last head
  const int size = last0 < p.sched_group ? last0 : p.sched_group;
  const int v = u - (u / per_group) * per_group;
  const int rank = v / size;
  w.head = last0 - size + (v - rank * size);
  const int bh = p.first_head + w.head;
  w.b = bh / p.H;
  w.h = bh - w.b * p.H;
  w.hk = w.h / (p.H / p.Hkv);
  w.tile0 = (p.n_units - 1 - rank) * kNT;
  w.valid1 = w.tile0 + 1 < p.n_tiles;
  w.tr[0] = tile_range(w.tile0, p.window, p.sinks, p.block, p.n_tiles);
  w.tr[1] = tile_range(w.valid1 ? w.tile0 + 1 : w.tile0, p.window, p.sinks, p.block, p.n_tiles);
  w.lo = w.tr[0].lo;
  w.extra = w.tr[0].sink_blocks < w.lo ? w.tr[0].sink_blocks : w.lo;
  w.n_iters = w.extra + (w.tr[1].hi - w.lo + 1);
  return w;
}

template <typename T>
__global__ void __launch_bounds__(256, 1)
dq_from_ds_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_dq, const DqParams p) {
  using L = DqSmem;
  constexpr int STAGES = L::STAGES;
  constexpr int kBoxes = D / 64;
  constexpr int kKBoxBytes = 64 * 128;
  constexpr int kOutBoxBytes = kTile * 128;
  constexpr bool kBf16 = Pack2<T>::kIsBf16;
  constexpr uint32_t kTmemCols = 2 * kNT * D;
  constexpr int kRing = L::kRing;

  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto bar = [&](int i) -> uint32_t { return base + L::kBar + 8u * i; };
  constexpr int FULL = 0, EMPTY = STAGES, ACC_FULL = 2 * STAGES, ACC_EMPTY = ACC_FULL + 2, GROUP = ACC_EMPTY + 2,
                SCHED_FULL = GROUP + 1;
  volatile int* sched_ring = reinterpret_cast<volatile int*>(gen + L::kSched);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gen + L::kAbort);
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gen + L::kTmemSlot);
  const WaitCtx wctx{abort_flag, p.status};

  if (threadIdx.x == 0) {
    *abort_flag = (*reinterpret_cast<volatile unsigned*>(p.status) != STATUS_OK) ? 1 : 0;
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(bar(FULL + s), 1);
      mbar_init(bar(EMPTY + s), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar(ACC_FULL + i), 1);
      mbar_init(bar(ACC_EMPTY + i), 128);
    }
    mbar_init(bar(GROUP), 128);
    for (int i = 0; i < kRing; ++i) mbar_init(bar(SCHED_FULL + i), 1);
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(base + L::kTmemSlot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const bool dead = *abort_flag != 0;
  grid_dep_wait();                                 // the dS tiles come from the stream's previous kernel
  grid_dep_release();

  // the uc-th unit of this CTA, as published by the producer: {u, head, b, h | hk << 16, tile0 | valid1 << 30, lo, extra,
  // n_iters, tr[0], tr[1]}
  auto next_unit = [&](int uc, bool& ok, DqUnit& w) -> int {
    ok = mbar_wait(bar(SCHED_FULL + (uc % kRing)), (uc / kRing) & 1, wctx, 70);
    if (!ok) return -1;
    const int4* e = reinterpret_cast<const int4*>(const_cast<const int*>(sched_ring) + 16 * (uc % kRing));
    const int4 a = e[0], b = e[1], c = e[2], d = e[3];
    w.head = a.y; w.b = a.z; w.h = a.w & 0xffff; w.hk = a.w >> 16;
    w.tile0 = b.x & 0x3fffffff; w.valid1 = (b.x >> 30) != 0;
    w.lo = b.y; w.extra = b.z; w.n_iters = b.w;
    w.tr[0].lo = c.x; w.tr[0].hi = c.y; w.tr[0].sink_blocks = c.z;
    w.tr[1].lo = d.x; w.tr[1].hi = d.y; w.tr[1].sink_blocks = d.z;
    return a.x;
  };

  if (dead) {
    // a give-up recorded earlier makes this launch a no-op
  } else if (warp == 0) {
    // ========================= scheduler + producer ==========================
    if (lane == 0) {
      tma_prefetch_desc(&tm_k);
      bool ok = true;
      int git = 0;
      for (int uc = 0; ok; ++uc) {
        int u = static_cast<int>(atomicAdd(&p.sched[0], 1u));
        if (u >= p.total_units) u = -1;
        DqUnit w{};
        if (u >= 0) w = make_dq_unit(u, p);
        // (a slot of the ring is free again once its unit's accumulators are: see the wait below)
        volatile int* e = sched_ring + 16 * (uc % kRing);
        e[0] = u; e[1] = w.head; e[2] = w.b; e[3] = w.h | (w.hk << 16);
        e[4] = w.tile0 | (w.valid1 ? 1 << 30 : 0); e[5] = w.lo; e[6] = w.extra; e[7] = w.n_iters;
        e[8] = w.tr[0].lo; e[9] = w.tr[0].hi; e[10] = w.tr[0].sink_blocks;
        e[12] = w.tr[1].lo; e[13] = w.tr[1].hi; e[14] = w.tr[1].sink_blocks;
        mbar_arrive(bar(SCHED_FULL + (uc % kRing)));
        if (u < 0) break;
        const uint8_t* head_tiles = p.ds + static_cast<long long>(w.head) * p.per_head * kDsTileBytes;
        const uint8_t* src[kNT];
#pragma unroll
        for (int t = 0; t < kNT; ++t)
          src[t] = head_tiles + static_cast<long long>(ds_tile_offset(p.layout, w.tile0 + t)) * kDsTileBytes;
        for (int it = 0; ok && it < w.n_iters; ++it) {
          const int j = w.block_at(it);
          const bool s0 = w.sees(0, j), s1 = w.sees(1, j);
          for (int half = 0; half < 2; ++half, ++git) {
            const int s = git % STAGES;
            if (!(ok = mbar_wait(bar(EMPTY + s), ((git / STAGES) & 1) ^ 1, wctx, 71))) break;
            const uint32_t st = base + s * L::kStage;
            mbar_arrive_expect_tx(bar(FULL + s), ((s0 ? 1 : 0) + (s1 ? 1 : 0)) * kHalfTile + L::kKBytes);
            if (s0) bulk_load(st, src[0] + half * kHalfTile, kHalfTile, bar(FULL + s));
            if (s1) bulk_load(st + kHalfTile, src[1] + half * kHalfTile, kHalfTile, bar(FULL + s));
            for (int x = 0; x < kBoxes; ++x)
              tma_load_4d(st + kNT * kHalfTile + x * kKBoxBytes, &tm_k, bar(FULL + s), 64 * x, w.hk, j * kTile + 64 * half,
                          w.b);
          }
          // a tile's blocks lie side by side in the order it meets them
          if (s0) src[0] += kDsTileBytes;
          if (s1) src[1] += kDsTileBytes;
        }
      }
    }
  } else if (warp == 1) {
    // ================================ MMA issuer =============================
    const uint32_t leader = elect_one() ? 1u : 0u;
    const uint32_t tmem_u = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    auto wait_all = [&](uint32_t bb, uint32_t parity, unsigned where) -> bool {
      return __all_sync(0xffffffffu, mbar_wait(bb, parity, wctx, where));
    };
    constexpr uint32_t idesc = make_idesc(kBf16, 128, D, true, true);
    bool ok = true;
    int git = 0;
    for (int uc = 0; ok; ++uc) {
      DqUnit w{};
      const int u = __shfl_sync(0xffffffffu, next_unit(uc, ok, w), 0);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok || u < 0) break;
      w.lo = __shfl_sync(0xffffffffu, w.lo, 0);
      w.extra = __shfl_sync(0xffffffffu, w.extra, 0);
      w.n_iters = __shfl_sync(0xffffffffu, w.n_iters, 0);
      w.valid1 = __shfl_sync(0xffffffffu, w.valid1 ? 1 : 0, 0) != 0;
#pragma unroll
      for (int t = 0; t < kNT; ++t) {
        w.tr[t].lo = __shfl_sync(0xffffffffu, w.tr[t].lo, 0);
        w.tr[t].hi = __shfl_sync(0xffffffffu, w.tr[t].hi, 0);
        w.tr[t].sink_blocks = __shfl_sync(0xffffffffu, w.tr[t].sink_blocks, 0);
      }
      const int buf = uc & 1;
      if (!(ok = wait_all(bar(ACC_EMPTY + buf), ((uc >> 1) & 1) ^ 1, 72))) break;
      bool started[kNT] = {false, false};
      for (int it = 0; ok && it < w.n_iters; ++it) {
        const int j = w.block_at(it);
        for (int half = 0; half < 2; ++half, ++git) {
          const int s = git % STAGES;
          if (!(ok = wait_all(bar(FULL + s), (git / STAGES) & 1, 73))) break;
          tc_fence_after();
          const uint32_t st = base + s * L::kStage, ka = st + kNT * kHalfTile;
#pragma unroll
          for (int t = 0; t < kNT; ++t) {
            if (!w.sees(t, j)) continue;
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              umma_ss(leader, tmem_u + (buf * kNT + t) * D, make_smem_desc_plain_mn(st + t * kHalfTile + kk * 256, 128, 1024),
                      make_smem_desc(ka + kk * 2048, kKBoxBytes, 1024), idesc, (started[t] || kk > 0) ? 1u : 0u);
            started[t] = true;
          }
          umma_commit(leader, bar(EMPTY + s));
        }
      }
      if (ok) umma_commit(leader, bar(ACC_FULL + buf));
    }
  } else if (warp >= 4) {
    // ================================ epilogue ===============================
    const uint32_t lane_base = 32u * (warp & 3);
    const int row = 32 * (warp & 3) + lane;
    const uint32_t sw = static_cast<uint32_t>(row & 7);
    const uint32_t stage = base + STAGES * L::kStage;
    uint32_t group_phase = 0;
    bool ok = true;
    auto group_sync = [&]() {
      mbar_arrive(bar(GROUP));
      const bool done = mbar_wait(bar(GROUP), group_phase & 1u, wctx, 74);
      ++group_phase;
      ok = __all_sync(0xffffffffu, done && *abort_flag == 0);
    };
    for (int uc = 0; ok; ++uc) {
      DqUnit w;
      const int u = next_unit(uc, ok, w);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok || u < 0) break;
      const int buf = uc & 1;
      ok = mbar_wait_idle(bar(ACC_FULL + buf), (uc >> 1) & 1, wctx, 75);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const int nt = w.valid1 ? 2 : 1;
      for (int t = 0; t < nt && ok; ++t) {
        // the previous store has finished reading the staging tile
        if (warp == 4 && lane == 0) tma_store_wait_read();
        group_sync();
        if (!ok) break;
#pragma unroll
        for (int c = 0; c < D; c += 32) {
          uint32_t r[32];
          tmem_ld32(tmem_addr(tmem, lane_base, (buf * kNT + t) * D + c), r);
          tc_wait_ld();
          if (c + 32 >= D && t + 1 == nt) {
            tc_fence_before();
            mbar_arrive(bar(ACC_EMPTY + buf));
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int col = c + 8 * i;
            const uint32_t addr = stage + static_cast<uint32_t>(col >> 6) * kOutBoxBytes + static_cast<uint32_t>(row) * 128u +
                                  ((static_cast<uint32_t>((col & 63) >> 3) ^ sw) << 4);
            st_shared_v4(addr,
                         Pack2<T>::pack(__uint_as_float(r[8 * i + 0]) * p.scale, __uint_as_float(r[8 * i + 1]) * p.scale),
                         Pack2<T>::pack(__uint_as_float(r[8 * i + 2]) * p.scale, __uint_as_float(r[8 * i + 3]) * p.scale),
                         Pack2<T>::pack(__uint_as_float(r[8 * i + 4]) * p.scale, __uint_as_float(r[8 * i + 5]) * p.scale),
                         Pack2<T>::pack(__uint_as_float(r[8 * i + 6]) * p.scale, __uint_as_float(r[8 * i + 7]) * p.scale));
          }
        }
        fence_proxy_async_smem();
        group_sync();
        if (!ok) break;
        if (warp == 4 && lane == 0) {
          for (int x = 0; x < kBoxes; ++x)
            tma_store_4d(&tm_dq, stage + x * kOutBoxBytes, 64 * x, w.h, (w.tile0 + t) * kTile, w.b);
          tma_store_commit();
        }
      }
    }
    // the CTA's shared memory outlives its last store's reads
    if (warp == 4 && lane == 0) tma_store_wait_read();
  }

  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, kTmemCols);
  }
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned done = atomicAdd(&p.sched[1], 1u);
    if (done == gridDim.x - 1) {
      p.sched[0] = 0u;
      p.sched[1] = 0u;
      __threadfence();
    }
  }
}

template <typename T>
int launch_t(const CUtensorMap& mk, const CUtensorMap& mdq, DqParams dp, cudaStream_t stream) {
  using L = DqSmem;
  static_assert(L::kDynamic <= 232448, "over the shared memory a CTA can have");
  auto kern = dq_from_ds_kernel<T>;
  if (ensure_dynamic_smem(reinterpret_cast<const void*>(kern), L::kDynamic) != NLFA_OK) return NLFA_ERR_CUDA;
  const int grid = dp.total_units < sm_count() ? dp.total_units : sm_count();
  dp.sched_group = dp.heads < grid ? dp.heads : grid;
  if (launch_kernel(kern, dim3(grid), dim3(256), L::kDynamic, stream, overlap_launches(kOverlapDq), mk, mdq, dp) !=
      cudaSuccess) {
    (void)cudaGetLastError();
    return NLFA_ERR_CUDA;
  }
  return NLFA_OK;
}

}  // namespace

int launch_dq_from_ds(const Problem& p, const void* k, const void* ds, const DsLayout& layout, int first_pair, int pairs,
                      void* dq, unsigned* sched, unsigned* status, cudaStream_t stream) {
  CUtensorMap mk, mdq;
  int st = make_tile_map(&mk, k, p.dtype, p.B, p.T, p.Hkv, p.D, 64);
  if (st == NLFA_OK) st = make_tile_map(&mdq, dq, p.dtype, p.B, p.T, p.H, p.D, kTile);
  if (st != NLFA_OK) return st;
  DqParams dp{};
  const int group = p.H / p.Hkv;
  dp.H = p.H; dp.Hkv = p.Hkv;
  dp.window = p.window; dp.sinks = p.sinks; dp.block = p.block;
  dp.n_tiles = layout.n_tiles;
  dp.n_units = (dp.n_tiles + kNT - 1) / kNT;
  dp.heads = pairs * group;
  dp.first_head = first_pair * group;
  dp.total_units = dp.heads * dp.n_units;
  dp.layout = layout;
  dp.per_head = ds_tile_offset(layout, layout.n_tiles);
  dp.ds = static_cast<const uint8_t*>(ds);
  dp.scale = p.scale;
  dp.sched = sched;
  dp.status = status;
  return p.dtype == NLFA_DTYPE_BF16 ? launch_t<__nv_bfloat16>(mk, mdq, dp, stream) : launch_t<__half>(mk, mdq, dp, stream);
}

}  // namespace nlfa
