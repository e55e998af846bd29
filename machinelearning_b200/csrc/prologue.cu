// Load-side prologue of the attention core for q or k, fused into one pass:
// per-head RMSNorm -> rotary embedding -> cast to the kernel dtype, and its backward.
//
// In nanolab these are separate tensor passes in front of every attention call:
// q_norm / k_norm (nanolab/mixers.py:287-289, RMSNorm at :46-56), apply_rope
// (:290-292, :68-75) and the cast + contiguous of flash_attn
// (nanolab/flash_cuda.py:263-266).  Here a row of D elements is read once and
// written once: HBM-bound, 2 + 2 bytes per element for 16-bit in and out.
//
// Thread mapping: a lane owns elements 4 s .. 4 s + 3 of each half of a row, so a row is D/8 lanes, a warp
// holds 256/D rows, and the rotary partner of an element (e +- D/2) is the lane's own: no exchange.  A lane's U rows
// are consecutive, so its position (row / H) % T is divided out once and stepped from there, and the cos / sin entries
// are fetched again only when the position changes (H heads share it).  Bound by HBM; with eight elements in a
// row per lane, the partner by shuffle and two divisions per row, instruction issue was in the way:
// [64,1024,12,64] bf16 forward 48.1 -> 36.5 us (5.5 TB/s), backward 77.7 -> 65.8 us (4.6 TB/s: half of the issue
// slots and half of the DRAM bandwidth, waiting on loads; fetching an iteration ahead cost registers, 78 us).
//
// The weight's gradient: a row of partial sums per CTA; the CTA that finishes last adds them up in a fixed order, so
// there is no second kernel.
//
// Rounding follows torch's path for 16-bit input under autocast: the normalised,
// weighted row is rounded to the input type (rms_norm returns the input's type), the
// rotation runs in fp32, the result is rounded to the output type.
#include "rowwise.cuh"

namespace nlfa {
namespace {

using namespace rowwise;

// Rows are indexed with 32 bits (the host refuses B*T*H >= 2^31): the position of a row, (row / H) % T,
// would otherwise cost two 64-bit divisions per row group.

// A lane's place in the sequence: position and head of its first row, stepped row by row.
struct Place {
  unsigned t, h;
  __device__ Place(unsigned row, unsigned T, unsigned H) {
    const unsigned q = row / H;
    h = row - q * H;
    t = q % T;
  }
  __device__ bool step(unsigned T, unsigned H) {           // true: another position
    if (++h < H) return false;
    h = 0;
    if (++t == T) t = 0;
    return true;
  }
};

// x [rows, D] (rows = B*T*H, position t = (row / H) % T) -> y [rows, D]; rstd [rows] when weight != nullptr.
template <typename TIn, typename TOut, int D>
__global__ void __launch_bounds__(kThreads)
qk_prologue_fwd_kernel(const TIn* __restrict__ x, const float* __restrict__ weight, const float* __restrict__ cosT,
                       const float* __restrict__ sinT, TOut* __restrict__ y, float* __restrict__ rstd,
                       unsigned rows, unsigned T, unsigned H, float eps) {
  constexpr int LPR = D / kVec;              // lanes per row
  constexpr int RPW = 32 / LPR;              // rows per warp and group
  constexpr int U = Elem<TIn>::kInFlight;    // rows a lane has in flight
  constexpr int kHalf = D / 2;
  grid_dep_wait();
  grid_dep_release();
  const unsigned lane = threadIdx.x & 31;
  const unsigned e0 = 4 * (lane % LPR);      // first element in the low half
  const unsigned warp = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
  const unsigned r0 = warp * (RPW * U) + (lane / LPR) * U;
  typename Elem<TIn>::Raw raw[U];
#pragma unroll
  for (int u = 0; u < U; ++u)                // every load first; the whole warp stays for the shuffles
    raw[u] = r0 + u < rows ? Elem<TIn>::load_halves(x + (size_t)(r0 + u) * D + e0, kHalf) : Elem<TIn>::zero();
  float w[kVec], c[kVec], s[kVec];
#pragma unroll
  for (int i = 0; i < kVec; ++i) w[i] = weight ? weight[e0 + (i & 3) + (i >> 2) * kHalf] : 1.f;
  Place at(r0 < rows ? r0 : 0u, T, H);
  bool fresh = true;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const unsigned row = r0 + u;
    const bool live = row < rows;
    float v[kVec];
    Elem<TIn>::unpack(raw[u], v);
    if (weight) {
      float ss = 0.f;
#pragma unroll
      for (int i = 0; i < kVec; ++i) ss = fmaf(v[i], v[i], ss);
      const float r = rsqrtf(row_sum<LPR>(ss) * (1.f / D) + eps);
      if (live && e0 == 0) rstd[row] = r;
#pragma unroll
      for (int i = 0; i < kVec; ++i) v[i] = Elem<TIn>::round(v[i] * r * w[i]);
    }
    if (cosT) {
      if (u > 0 && at.step(T, H)) fresh = true;
      if (fresh) {
        Elem<float>::unpack(Elem<float>::load_halves(cosT + (size_t)at.t * D + e0, kHalf), c);
        Elem<float>::unpack(Elem<float>::load_halves(sinT + (size_t)at.t * D + e0, kHalf), s);
        fresh = false;
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {          // rot = (-hi, lo)
        const float lo = v[i], hi = v[i + 4];
        v[i] = lo * c[i] - hi * s[i];
        v[i + 4] = hi * c[i + 4] + lo * s[i + 4];
      }
    }
    if (live) Elem<TOut>::store_halves(y + (size_t)row * D + e0, kHalf, v);
  }
}

// gy [rows, D] (gradient of the prologue's output), x and rstd from the forward -> gx [rows, D]; gweight [D] by way of
// one row of partial sums per CTA (partial [gridDim.x, D]).
template <typename TIn, typename TG, int D>
__global__ void __launch_bounds__(kThreads, 2)
qk_prologue_bwd_kernel(const TG* __restrict__ gy, const TIn* __restrict__ x, const float* __restrict__ weight,
                       const float* __restrict__ cosT, const float* __restrict__ sinT,
                       const float* __restrict__ rstd, TIn* __restrict__ gx, float* __restrict__ partial,
                       float* __restrict__ gweight, unsigned* ticket, unsigned rows, unsigned T, unsigned H) {
  constexpr int LPR = D / kVec;
  constexpr int RPW = 32 / LPR;
  constexpr int U = Elem<TIn>::kInFlight;
  constexpr int kHalf = D / 2;
  __shared__ __align__(16) float red[kThreads * 4];        // [warp][D] sums, then [thread][4] for the last CTA
  __shared__ int last;
  grid_dep_wait();
  grid_dep_release();
  const unsigned lane = threadIdx.x & 31;
  const unsigned e0 = 4 * (lane % LPR);
  const unsigned warp = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
  const unsigned stride = gridDim.x * (kThreads / 32) * (RPW * U);
  float w[kVec], dw[kVec];
#pragma unroll
  for (int i = 0; i < kVec; ++i) {
    w[i] = weight ? weight[e0 + (i & 3) + (i >> 2) * kHalf] : 1.f;
    dw[i] = 0.f;
  }

  for (unsigned r1 = warp * (RPW * U); r1 < rows; r1 += stride) {
    const unsigned r0 = r1 + (lane / LPR) * U;
    typename Elem<TG>::Raw graw[U];
    typename Elem<TIn>::Raw xraw[U];
    float r[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const unsigned row = r0 + u;
      graw[u] = Elem<TG>::zero();
      xraw[u] = Elem<TIn>::zero();
      r[u] = 0.f;
      if (row < rows) {
        graw[u] = Elem<TG>::load_halves(gy + (size_t)row * D + e0, kHalf);
        if (weight) { xraw[u] = Elem<TIn>::load_halves(x + (size_t)row * D + e0, kHalf); r[u] = rstd[row]; }
      }
    }
    float c[kVec], s[kVec];                  // table entries, kept while the position stays the same
    Place at(r0 < rows ? r0 : 0u, T, H);
    bool fresh = true;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const unsigned row = r0 + u;
      float g[kVec], v[kVec];
      Elem<TG>::unpack(graw[u], g);
      Elem<TIn>::unpack(xraw[u], v);
      if (cosT) {
        if (u > 0 && at.step(T, H)) fresh = true;
        if (fresh) {
          Elem<float>::unpack(Elem<float>::load_halves(cosT + (size_t)at.t * D + e0, kHalf), c);
          Elem<float>::unpack(Elem<float>::load_halves(sinT + (size_t)at.t * D + e0, kHalf), s);
          fresh = false;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {        // transpose of the rotation
          const float lo = g[i], hi = g[i + 4];
          g[i] = lo * c[i] + hi * s[i + 4];
          g[i + 4] = hi * c[i + 4] - lo * s[i];
        }
      }
      if (weight) {
        float dot = 0.f;
#pragma unroll
        for (int i = 0; i < kVec; ++i) {
          g[i] = Elem<TIn>::round(g[i]);     // the gradient passes back through rms_norm's output cast
          v[i] *= r[u];                      // normalised row
          dw[i] = fmaf(g[i], v[i], dw[i]);
          g[i] *= w[i];
          dot = fmaf(g[i], v[i], dot);
        }
        const float c = row_sum<LPR>(dot) * (1.f / D);
#pragma unroll
        for (int i = 0; i < kVec; ++i) g[i] = r[u] * (g[i] - v[i] * c);
      }
      if (row < rows) Elem<TIn>::store_halves(gx + (size_t)row * D + e0, kHalf, g);
    }
  }

  if (!weight) return;
  // CTA-wide sum of dw, then the last CTA's sum over all CTAs: both in a fixed order
#pragma unroll
  for (int i = 0; i < kVec; ++i) {
#pragma unroll
    for (int off = LPR; off < 32; off <<= 1) dw[i] += __shfl_xor_sync(0xffffffffu, dw[i], off);
  }
  if (lane < LPR) {
#pragma unroll
    for (int i = 0; i < kVec; ++i) red[(threadIdx.x >> 5) * D + e0 + (i & 3) + (i >> 2) * kHalf] = dw[i];
  }
  __syncthreads();
  if (threadIdx.x < D) {
    float sum = 0.f;
#pragma unroll
    for (int wi = 0; wi < kThreads / 32; ++wi) sum += red[wi * D + threadIdx.x];
    partial[(size_t)blockIdx.x * D + threadIdx.x] = sum;
  }
  if (!last_cta(ticket, gridDim.x, &last)) return;
  // thread (g, e4): rows g, g + G, .. of four columns, past L1 (other SMs wrote them); then the G sums of a column
  constexpr int E = D / 4, G = kThreads / E;
  const int e4 = threadIdx.x % E, g = threadIdx.x / E, n = gridDim.x;
  float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
  for (int i = g; i < n; i += G) {
    const float4 p = __ldcg(reinterpret_cast<const float4*>(partial + (size_t)i * D) + e4);
    sum = make_float4(sum.x + p.x, sum.y + p.y, sum.z + p.z, sum.w + p.w);
  }
  reinterpret_cast<float4*>(red)[threadIdx.x] = sum;
  __syncthreads();
  if (threadIdx.x < D) {
    float t = 0.f;
#pragma unroll
    for (int j = 0; j < G; ++j) t += red[j * D + threadIdx.x];
    gweight[threadIdx.x] = t;
  }
}

int grid_for(long long rows, int D, long long cap, int in_flight) {
  const long long rows_per_cta = (long long)(kThreads / 32) * (32 / (D / kVec)) * in_flight;
  long long need = (rows + rows_per_cta - 1) / rows_per_cta;
  if (need < 1) need = 1;
  return (int)(need < cap ? need : cap);
}

template <typename TIn, typename TOut>
int fwd_for_dim(int D, const void* x, const float* w, const float* c, const float* s, void* y, float* rstd,
                long long rows, int T, int H, float eps, cudaStream_t st) {
  const int grid = grid_for(rows, D, 1ll << 31, Elem<TIn>::kInFlight);          // one pass per warp
  cudaError_t e;
#define NLFA_GO(DD)                                                                                               \
  e = launch_kernel(qk_prologue_fwd_kernel<TIn, TOut, DD>, dim3(grid), dim3(kThreads), 0, st,                     \
                    overlap_launches(kOverlapRowwise), (const TIn*)x, w, c, s, (TOut*)y, rstd, (unsigned)rows,    \
                    (unsigned)T, (unsigned)H, eps)
  if (D == 32) NLFA_GO(32); else if (D == 64) NLFA_GO(64); else NLFA_GO(128);
#undef NLFA_GO
  if (e != cudaSuccess) (void)cudaGetLastError();
  return e == cudaSuccess ? NLFA_OK : NLFA_ERR_CUDA;
}

template <typename TIn, typename TG>
int bwd_for_dim(int D, const void* gy, const void* x, const float* w, const float* c, const float* s,
                const float* rstd, void* gx, float* partial, float* gweight, long long rows, int T, int H,
                cudaStream_t st) {
  // (the scratch's last row is the ticket's)
  const int grid = grid_for(rows, D, 2 * sm_count() < kMaxPartials - 1 ? 2 * sm_count() : kMaxPartials - 1, Elem<TIn>::kInFlight);
  unsigned* ticket = nullptr;
  bool captured = false;
  if (w != nullptr) {
    const int rc = launch_ticket(st, reinterpret_cast<unsigned*>(partial + (size_t)(kMaxPartials - 1) * D), &ticket, &captured);
    if (rc != NLFA_OK) return rc;
  }
  cudaError_t e;
#define NLFA_GO(DD)                                                                                               \
  e = launch_kernel(qk_prologue_bwd_kernel<TIn, TG, DD>, dim3(grid), dim3(kThreads), 0, st,                       \
                    !captured && overlap_launches(kOverlapRowwise), (const TG*)gy, (const TIn*)x, w, c, s, rstd, (TIn*)gx,     \
                    partial, gweight, ticket, (unsigned)rows, (unsigned)T, (unsigned)H)
  if (D == 32) NLFA_GO(32); else if (D == 64) NLFA_GO(64); else NLFA_GO(128);
#undef NLFA_GO
  if (e != cudaSuccess) (void)cudaGetLastError();
  return e == cudaSuccess ? NLFA_OK : NLFA_ERR_CUDA;
}


}  // namespace
}  // namespace nlfa

extern "C" {

size_t nlfa_qk_prologue_scratch_bytes(int D) {
  return (size_t)nlfa::kMaxPartials * (size_t)(D > 0 ? D : 0) * sizeof(float);
}

int nlfa_qk_prologue_fwd(const void* x, int x_dtype, const float* weight, const float* cos_table,
                         const float* sin_table, void* y, int y_dtype, float* rstd, int B, int T, int H, int D,
                         float eps, void* stream) {
  using namespace nlfa;
  if (B < 0 || T < 0 || H < 0) return NLFA_ERR_BAD_SHAPE;
  if (D != 32 && D != 64 && D != 128) return NLFA_ERR_BAD_HEAD_DIM;
  if (!dtype_ok(x_dtype) || !dtype_ok(y_dtype)) return NLFA_ERR_BAD_DTYPE;
  const long long rows = (long long)B * T * H;
  if (rows >= (1ll << 31)) return NLFA_ERR_BAD_SHAPE;
  if (rows == 0) return NLFA_OK;
  if (!x || !y || (weight && !rstd) || ((cos_table == nullptr) != (sin_table == nullptr))) return NLFA_ERR_NULL_POINTER;
  if (!aligned16(x) || !aligned16(y) || !aligned16(cos_table) || !aligned16(sin_table)) return NLFA_ERR_MISALIGNED;
  cudaStream_t st = (cudaStream_t)stream;
#define NLFA_OUT(TIn)                                                                                              \
  (y_dtype == NLFA_DTYPE_BF16 ? fwd_for_dim<TIn, __nv_bfloat16>(D, x, weight, cos_table, sin_table, y, rstd, rows, T, H, eps, st) \
   : y_dtype == NLFA_DTYPE_F16 ? fwd_for_dim<TIn, __half>(D, x, weight, cos_table, sin_table, y, rstd, rows, T, H, eps, st)       \
                               : fwd_for_dim<TIn, float>(D, x, weight, cos_table, sin_table, y, rstd, rows, T, H, eps, st))
  if (x_dtype == NLFA_DTYPE_BF16) return NLFA_OUT(__nv_bfloat16);
  if (x_dtype == NLFA_DTYPE_F16) return NLFA_OUT(__half);
  return NLFA_OUT(float);
#undef NLFA_OUT
}

int nlfa_qk_prologue_bwd(const void* gy, int gy_dtype, const void* x, int x_dtype, const float* weight,
                         const float* cos_table, const float* sin_table, const float* rstd, void* gx,
                         float* gweight, void* scratch, size_t scratch_bytes, int B, int T, int H, int D,
                         void* stream) {
  using namespace nlfa;
  if (B < 0 || T < 0 || H < 0) return NLFA_ERR_BAD_SHAPE;
  if (D != 32 && D != 64 && D != 128) return NLFA_ERR_BAD_HEAD_DIM;
  if (!dtype_ok(x_dtype) || !dtype_ok(gy_dtype)) return NLFA_ERR_BAD_DTYPE;
  const long long rows = (long long)B * T * H;
  if (rows >= (1ll << 31)) return NLFA_ERR_BAD_SHAPE;
  cudaStream_t st = (cudaStream_t)stream;
  if (rows == 0) {
    if (weight && gweight && cudaMemsetAsync(gweight, 0, D * sizeof(float), st) != cudaSuccess) return NLFA_ERR_CUDA;
    return NLFA_OK;
  }
  if (!gy || !gx || (weight && (!x || !rstd || !gweight || !scratch)) ||
      ((cos_table == nullptr) != (sin_table == nullptr)))
    return NLFA_ERR_NULL_POINTER;
  if (weight && scratch_bytes < nlfa_qk_prologue_scratch_bytes(D)) return NLFA_ERR_SCRATCH_TOO_SMALL;
  if (!aligned16(gy) || !aligned16(gx) || !aligned16(x) || !aligned16(cos_table) || !aligned16(sin_table))
    return NLFA_ERR_MISALIGNED;
  // (the kernel reads the partial sums 16 bytes at a time; the scratch's last row, the ticket's, has room to spare)
  scratch = reinterpret_cast<void*>((reinterpret_cast<uintptr_t>(scratch) + 15u) & ~static_cast<uintptr_t>(15u));
#define NLFA_G(TIn)                                                                                               \
  (gy_dtype == NLFA_DTYPE_BF16 ? bwd_for_dim<TIn, __nv_bfloat16>(D, gy, x, weight, cos_table, sin_table, rstd, gx, (float*)scratch, gweight, rows, T, H, st) \
   : gy_dtype == NLFA_DTYPE_F16 ? bwd_for_dim<TIn, __half>(D, gy, x, weight, cos_table, sin_table, rstd, gx, (float*)scratch, gweight, rows, T, H, st)       \
                                : bwd_for_dim<TIn, float>(D, gy, x, weight, cos_table, sin_table, rstd, gx, (float*)scratch, gweight, rows, T, H, st))
  if (x_dtype == NLFA_DTYPE_BF16) return NLFA_G(__nv_bfloat16);
  if (x_dtype == NLFA_DTYPE_F16) return NLFA_G(__half);
  return NLFA_G(float);
#undef NLFA_G
}

}  // extern "C"
