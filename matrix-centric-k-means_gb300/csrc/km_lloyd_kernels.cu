// Lloyd k-means kernels for sm_103a: point/centroid preparation, the SIMT FP32
// distance stage with fused candidate lists, exact near-tie refinement, the
// stable label sort (one-hot V as a label-sorted permutation), the exact
// centroid update V.X, and the per-iteration finalize kernel (whose last block
// takes the loop decision).
//
// Reference counterparts (HicrestLaboratory/Matrix-Centric-K-Means):
//   distance + argmin     comparisons/CPU_Kmeans/src/kmeans.cpp:86-122;
//                         src/kmeans.cu:847-936 (popcorn SpMM + RAFT argmin)
//   counts                src/kmeans.cu:941-947 (RAFT reduce_cols_by_key)
//   V rebuild             src/kmeans.cu:987-1031, src/kernels/kernels.cuh:296-314
//   centroid update       comparisons/CPU_Kmeans/src/kmeans.cpp:131-148
//   convergence           comparisons/CPU_Kmeans/src/kmeans.cpp:170-200;
//                         src/kmeans.cu:1054-1073 (score rule)
#include "km_lloyd.cuh"
#include "km_simt.cuh"
#include "km_sums.cuh"

#include <algorithm>
#include <cmath>
#include <cfloat>
#include <type_traits>

namespace km {

static __device__ __forceinline__ float f_inf() { return __int_as_float(0x7f800000); }

// ---------------------------------------------------------------------------
// Preparation
// ---------------------------------------------------------------------------

// h + l += a + al, the first addition by TwoSum (the FP64 units of this GPU are a
// small fraction of its FP32 rate): a sum of squares split exactly by an FMA each is
// within a few units of 2^-48 of the exact value, and float(h + l) is the correctly
// rounded norm.
static __device__ __forceinline__ void two_sum(float& h, float& l, float a, float al) {
  const float t = __fadd_rn(h, a), bp = __fsub_rn(t, h);
  const float err = __fadd_rn(__fsub_rn(h, __fsub_rn(t, bp)), __fsub_rn(a, bp));
  h = t;
  l = __fadd_rn(l, __fadd_rn(al, err));
}

// Per row: ||x||^2 (an FP32 pair, stored as float and as a per-row double for the
// deterministic total), non-finite check, the row's copy (only when Xc != nullptr) and
// its BF16 hi/lo copies padded with zeros to dp columns (only when Xb != nullptr).
// NaN/Inf and non-BF16 coordinates are flagged once per warp (after its rows), not once
// per row: an atomic per row on one word serialises.
// VEC: the widest of 4, 2 and 1 columns that d divides by and X (and Xc) are aligned
// to.  A row is taken by G lanes, VEC columns each and a step of G * VEC columns; four steps' loads (of four
// rows, or of one row that has more columns than a step) are in flight per warp.
// Bound by HBM: n = 1,048,576 d = 128 with the copy, Xb and Xlo 433 us (a copy, then a warp
// a row and a column a lane) -> 277 (5.8 TB/s); n = 200,000 d = 100 with the copy 81 -> 36;
// n = 300,007 d = 50 with Xb and Xlo 40 (84 with a column a lane).
template <int VEC, int G, bool ONE>
__global__ void __launch_bounds__(256, 4)
prep_points_kernel(const float* __restrict__ X, uint64_t n, uint32_t d, uint32_t dp, float* __restrict__ xn2,
                   double* __restrict__ xn2d, float* __restrict__ Xc, __nv_bfloat16* __restrict__ Xb,
                   __nv_bfloat16* __restrict__ Xlo, DevState* st) {
  constexpr int U = 4, R = 32 / G;
  constexpr uint32_t STEP = G * VEC;
  const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t col0 = (uint32_t)(lane % G) * VEC;
  const uint32_t cols = Xb ? dp : d;
  constexpr int NR = ONE ? U : 1;              // rows per lane and round; ONE: a row is one step
  constexpr uint64_t rows = R * NR;
  uint32_t top = 0, low = 0;                   // largest |x| as bits; bits below BF16's
  for (uint64_t base = warp * rows; base < n; base += nw * rows) {
    const uint64_t row0 = base + lane / G;
    float sh[NR], sl[NR];
#pragma unroll
    for (int u = 0; u < NR; ++u) sh[u] = sl[u] = 0.0f;
    for (uint32_t j0 = 0; j0 < cols; j0 += ONE ? STEP : STEP * U) {
      float v[U][VEC];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint64_t r = ONE ? row0 + (uint64_t)u * R : row0;
        const uint32_t j = j0 + col0 + (ONE ? 0u : u * STEP);
        const bool in = r < n && j < d;
        if constexpr (VEC == 4) {
          const float4 t = in ? *reinterpret_cast<const float4*>(X + r * d + j) : make_float4(0.f, 0.f, 0.f, 0.f);
          v[u][0] = t.x; v[u][1] = t.y; v[u][2] = t.z; v[u][3] = t.w;
        } else if constexpr (VEC == 2) {
          const float2 t = in ? *reinterpret_cast<const float2*>(X + r * d + j) : make_float2(0.f, 0.f);
          v[u][0] = t.x; v[u][1] = t.y;
        } else {
          v[u][0] = in ? X[r * d + j] : 0.0f;
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint64_t r = ONE ? row0 + (uint64_t)u * R : row0;
        const uint32_t j = j0 + col0 + (ONE ? 0u : u * STEP);
        alignas(8) __nv_bfloat16 hi[VEC], lo[VEC];
#pragma unroll
        for (int e = 0; e < VEC; ++e) {
          const float x = v[u][e];
          top = max(top, __float_as_uint(x) & 0x7fffffffu);
          low |= __float_as_uint(x);
          const float p = __fmul_rn(x, x);
          two_sum(sh[ONE ? u : 0], sl[ONE ? u : 0], p, fmaf(x, x, -p));
          hi[e] = __float2bfloat16_rn(x);
          if (Xlo) lo[e] = __float2bfloat16_rn(x - __bfloat162float(hi[e]));
        }
        if (Xc && r < n && j < d) {
          if constexpr (VEC == 4) *reinterpret_cast<float4*>(Xc + r * d + j) = make_float4(v[u][0], v[u][1], v[u][2], v[u][3]);
          else if constexpr (VEC == 2) *reinterpret_cast<float2*>(Xc + r * d + j) = make_float2(v[u][0], v[u][1]);
          else Xc[r * d + j] = v[u][0];
        }
        if (Xb && r < n && j < dp) {            // dp is a multiple of 64
          if constexpr (VEC == 4) {
            *reinterpret_cast<uint2*>(Xb + r * dp + j) = *reinterpret_cast<const uint2*>(hi);
            if (Xlo) *reinterpret_cast<uint2*>(Xlo + r * dp + j) = *reinterpret_cast<const uint2*>(lo);
          } else if constexpr (VEC == 2) {
            *reinterpret_cast<uint32_t*>(Xb + r * dp + j) = *reinterpret_cast<const uint32_t*>(hi);
            if (Xlo) *reinterpret_cast<uint32_t*>(Xlo + r * dp + j) = *reinterpret_cast<const uint32_t*>(lo);
          } else {
            Xb[r * dp + j] = hi[0];
            if (Xlo) Xlo[r * dp + j] = lo[0];
          }
        }
      }
    }
    // Over the G lanes: while a lane holds several rows' sums, each exchange leaves it
    // half of them (6 additions for four rows of a warp instead of 20).
    int o = G / 2, u = 0;                      // u: the row that this lane ends with
    auto add_from = [&](float& h, float& l, float oh, float ol, int off) {
      oh = __shfl_xor_sync(0xffffffffu, oh, off);
      ol = __shfl_xor_sync(0xffffffffu, ol, off);
      two_sum(h, l, oh, ol);
    };
    if constexpr (NR == 4) {
      const bool up = lane & o, up2 = lane & (o >> 1);
#pragma unroll
      for (int i = 0; i < 2; ++i) {            // keeps rows i (lower lanes) or i + 2 (upper)
        const float gh = up ? sh[i] : sh[i + 2], gl = up ? sl[i] : sl[i + 2];
        if (up) { sh[i] = sh[i + 2]; sl[i] = sl[i + 2]; }
        add_from(sh[i], sl[i], gh, gl, o);
      }
      const float gh = up2 ? sh[0] : sh[1], gl = up2 ? sl[0] : sl[1];
      if (up2) { sh[0] = sh[1]; sl[0] = sl[1]; }
      add_from(sh[0], sl[0], gh, gl, o >> 1);
      u = (up ? 2 : 0) + (up2 ? 1 : 0);
      o >>= 2;
    }
    const int holders = o;                     // lanes l % (2 * holders) == 0 write a row each
#pragma unroll
    for (; o > 0; o >>= 1) add_from(sh[0], sl[0], sh[0], sl[0], o);
    const uint64_t r = row0 + (uint64_t)u * R;
    if (lane % max(2 * holders, 1) == 0 && r < n) {
      const double s = (double)sh[0] + (double)sl[0];
      xn2[r] = (float)s;
      if (xn2d) xn2d[r] = s;
    }
  }
  const bool bad = top >= 0x7f800000u, inexact = (low & 0xffffu) != 0u;
  if (__any_sync(0xffffffffu, bad) && lane == 0) atomicOr(&st->err, KM_DEVERR_NONFINITE);
  if (__any_sync(0xffffffffu, inexact) && lane == 0) atomicOr(&st->x_not_bf16, 1u);
}

// The narrowest group of lanes that takes a row in one step, at most a warp (a warp a row
// leaves 28 of 32 lanes idle at d = 16).  sms: one wave of four blocks on each.
void launch_prep_points(const float* X, uint64_t n, uint32_t d, uint32_t dp, float* xn2, double* xn2d, float* Xc,
                        __nv_bfloat16* Xb, __nv_bfloat16* Xlo, DevState* st, int sms, cudaStream_t s) {
  const uint32_t cols = Xb ? dp : d;
  const uintptr_t at = reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(Xc);
  const int vec = d % 4 == 0 && at % 16 == 0 ? 4 : d % 2 == 0 && at % 8 == 0 ? 2 : 1;
  auto go = [&](auto kernel, uint64_t rows) {            // rows: per warp and round
    const int blocks = (int)std::min<uint64_t>((n + 8 * rows - 1) / (8 * rows), (uint64_t)sms * 4);
    kernel<<<blocks, 256, 0, s>>>(X, n, d, dp, xn2, xn2d, Xc, Xb, Xlo, st);
  };
  if (vec == 1) cols <= 8 ? go(prep_points_kernel<1, 8, true>, 16) : go(prep_points_kernel<1, 32, false>, 1);
  else if (vec == 2) cols <= 64 ? go(prep_points_kernel<2, 32, true>, 4) : go(prep_points_kernel<2, 32, false>, 1);
  else if (cols <= 16) go(prep_points_kernel<4, 4, true>, 32);
  else if (cols <= 64) go(prep_points_kernel<4, 16, true>, 8);
  else if (cols <= 128) go(prep_points_kernel<4, 32, true>, 4);
  else go(prep_points_kernel<4, 32, false>, 1);
}

// Deterministic FP64 sum: fixed-shape tree per block, block partials summed in
// index order by a second single-block pass.
__global__ void reduce_f64_partial_kernel(const double* __restrict__ v, uint64_t n,
                                          double* __restrict__ part) {
  __shared__ double sh[256];
  double s = 0.0;
  const uint64_t per = (n + gridDim.x - 1) / gridDim.x;
  const uint64_t b = per * blockIdx.x, e = min(n, b + per);
  for (uint64_t i = b + threadIdx.x; i < e; i += blockDim.x) s += v[i];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = sh[0];
}

// One block of 256 threads, np <= 256: a fixed tree (an FP64 addition takes about 40
// ns here, so 256 of them in turn were 10 us).
__global__ void reduce_f64_final_kernel(const double* __restrict__ part, int np, double* out) {
  __shared__ double sh[256];
  sh[threadIdx.x] = (int)threadIdx.x < np ? part[threadIdx.x] : 0.0;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = sh[0];
}

// One warp per centroid: ||c||^2 in FP64 (stored as float), BF16 hi/lo copies
// padded to (kp, dp), +inf norms for the padding centroids, and max ||c||.
__global__ void prep_centroids_kernel(const float* __restrict__ C, uint32_t k, uint32_t kp,
                                      uint32_t d, uint32_t dp, float* __restrict__ cn2,
                                      __nv_bfloat16* __restrict__ Cb,
                                      __nv_bfloat16* __restrict__ Clo, float* __restrict__ Ct,
                                      DevState* st, uint32_t kp64) {
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= kp) {
    // +inf norms up to whole 64-column groups (read by the distance epilogue)
    if (warp < kp64 && lane == 0) cn2[warp] = f_inf();
    return;
  }
  const uint32_t c = warp;
  double s = 0.0;
  for (uint32_t j = lane; j < dp; j += 32) {
    float v = (c < k && j < d) ? C[(uint64_t)c * d + j] : 0.0f;
    if (c < k && j < d) Ct[(uint64_t)j * k + c] = v;
    s += (double)v * (double)v;
    if (Cb) {
      __nv_bfloat16 hi = __float2bfloat16_rn(v);
      Cb[(uint64_t)c * dp + j] = hi;
      if (Clo) Clo[(uint64_t)c * dp + j] = __float2bfloat16_rn(v - __bfloat162float(hi));
    }
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) {
    float f = (c < k) ? (float)s : f_inf();
    cn2[c] = f;
    if (c < k) atomicMax(reinterpret_cast<unsigned int*>(&st->cmax), __float_as_uint(sqrtf(f)));
  }
}

// ---------------------------------------------------------------------------
// (a)+(b) SIMT FP32 distances with the argmin fused (km_simt.cuh has the product).
// A CTA takes ROWS rows and walks all centroids, COLS at a time.  After each
// column tile a row's minimum over its TX threads (exchanged by shuffles) joins
// the row's running minimum m, and every centroid with v(c) <= tau(m) (tie_tau)
// goes to the row's list of up to F32_LIST (index, value) pairs in shared memory,
// which drops the entries above the current tau between tiles.  tau only falls with
// m, so the entries with v(c) <= tau(m_final) are the whole candidate set: one is the
// proven argmin, 2..4 go to the short re-score queue, more (or a full list, or values that
// are not finite) to the full re-score.
//
// Bound by the FP32 pipes.  The tile is as wide as k asks (32, 48, 64, 96 or 128
// centroids), so that k = 64 pays for 64.  Measured, distance kernel: n = 200,000
// d = 100 k = 64 161 -> 75 us, k = 20 159 -> 55 us, k = 90 162 -> 109 us; n = 1M d =
// 128 k = 256 1571 -> 1568 us = 22 T FMA/s (16 columns a thread instead, or 16 rows,
// left eight warps an SM, 44 % of the issue slots used and 21 T).  With few coordinates what
// follows a tile's product counts as much: one lane works out a row's minimum and tau
// for all (every lane on its own: n = 2M d = 16 k = 1000 2905 us, now 2410; n = 625,000 d =
// 64 k = 1000 2173 and 2023).
// ---------------------------------------------------------------------------
constexpr int F32_NT = 128, F32_RT = 8, F32_LIST = 8;
constexpr int F32_GATHER_RUN = 64;       // (GATHER) coordinates summed on their own
template <int TX, int CT>
using F32Tile = SimtTile<F32_NT, F32_RT, TX, CT, TX == 16 && CT == 8 ? 16 : 8>;
// Shared memory after the product's stages: per row m, tau's row terms, the
// squared norm, the list and its length; per column the centroid's squared norm.
struct F32Row {
  float m, tau, x2;
  TauRow tr;
  uint32_t cnt;
  uint32_t row;                 // row of X
};
template <class T, bool GATHER>
constexpr size_t f32_smem() {
  return T::SMEM + (GATHER ? T::TOT_BYTES : 0) + T::ROWS * (sizeof(F32Row) + F32_LIST * sizeof(uint2)) +
         T::COLS * sizeof(float);
}

// GATHER: logical row li of the tiles is row ridx[li] of X, for li < *nidx; queue
// segments are taken over the logical rows.  These rows have many near ties (the
// chunked tensor-core kernel found more than its lists hold), so their lists are the
// global ones (rq.wl, L entries a row), filtered by a warp a row, and rows with
// 5..L candidates go to the wide queue instead of the full re-score.  Their products are
// summed in runs of F32_GATHER_RUN coordinates, which makes the near-tie bound (tb)
// narrower by as much as the chains are shorter: n = 4M d = 256 k = 4096 (BF16 points,
// Zipf sizes), an iteration: full re-score 57 (lists of 8) -> 24 (lists of 256) -> none
// (runs of 64; runs of 32 took this pass 22.9 ms for 21.7, and no row less to the queues).
template <int TX, int CT, bool DOUT, bool GATHER>
__global__ void __launch_bounds__(F32_NT, CT == 8 ? 3 : 4)
assign_f32_kernel(const float* __restrict__ X, const float* __restrict__ C, bool v4,
                  const float* __restrict__ cn2, const float* __restrict__ xn2, uint64_t n,
                  uint32_t d, uint32_t k, TieBound tb, DevState* st,
                  uint32_t* __restrict__ labels, float* __restrict__ mindist,
                  RefineQueues rq, float* __restrict__ Dout, const uint32_t* __restrict__ ridx,
                  const uint32_t* __restrict__ nidx) {
  using T = F32Tile<TX, CT>;
  griddep_wait();
  if (st->done) return;
  const uint64_t n_log = GATHER ? (uint64_t)*nidx : n;
  const uint64_t m0 = (uint64_t)blockIdx.x * T::ROWS;
  // (Without a gather the grid covers every segment of the queues, whose counts
  // all have to be written; a gather's start at zero.)
  if (GATHER && m0 >= n_log) return;
  extern __shared__ __align__(16) float f32_smem_raw[];
  uint2* const list = reinterpret_cast<uint2*>(f32_smem_raw + (T::SMEM + (GATHER ? T::TOT_BYTES : 0)) / sizeof(float));   // [ROWS][F32_LIST]
  F32Row* const rs = reinterpret_cast<F32Row*>(list + T::ROWS * F32_LIST);
  float* const cns = reinterpret_cast<float*>(rs + T::ROWS);
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  const float cmax = st->cmax;
  const uint32_t cap = GATHER ? rq.L : (uint32_t)F32_LIST;   // entries a list holds
  auto list_of = [&](int r) -> uint2* { return GATHER ? rq.wl + (uint64_t)rs[r].row * rq.L : list + r * F32_LIST; };
  // Drops a row's entries above tau (by the warp): the entries kept.
  auto filter = [&](uint2* l, uint32_t cnt, float tau) -> uint32_t {
    const int lane = tid & 31;
    uint32_t kept = 0;
    for (uint32_t q0 = 0; q0 < cnt; q0 += 32u) {
      const uint32_t q = q0 + (uint32_t)lane;
      const uint2 en = q < cnt ? l[q] : make_uint2(0u, 0u);
      const bool keep = q < cnt && __uint_as_float(en.y) <= tau;
      const unsigned b = __ballot_sync(0xffffffffu, keep);
      if (keep) l[kept + (uint32_t)__popc(b & ((1u << lane) - 1u))] = en;    // at or before q: read already
      kept += (uint32_t)__popc(b);
      __syncwarp();
    }
    return kept;
  };
  for (int r = tid; r < T::ROWS; r += F32_NT) {
    const uint64_t li = m0 + (uint64_t)r;
    F32Row w{};
    if (li < n_log) {
      w.row = GATHER ? ridx[li] : (uint32_t)li;
      w.x2 = xn2[w.row];
    }
    w.m = f_inf();
    w.tr = tie_tau_row(w.x2, cmax, tb);
    rs[r] = w;
  }
  __syncthreads();
  for (uint32_t c0 = 0; c0 < k; c0 += T::COLS) {
    for (int c = tid; c < T::COLS; c += F32_NT) cns[c] = c0 + (uint32_t)c < k ? cn2[c0 + c] : f_inf();
    float2 acc[F32_RT / 2][CT];
    simt_product<T, GATHER ? F32_GATHER_RUN : 0>(
        f32_smem_raw, d, v4,
        [&](int r) { return m0 + (uint64_t)r < n_log ? X + (uint64_t)rs[r].row * d : (const float*)nullptr; },
        [&](int c) { return c0 + (uint32_t)c < k ? C + (uint64_t)(c0 + c) * d : (const float*)nullptr; }, acc,
        reinterpret_cast<float4*>(f32_smem_raw + T::SMEM / sizeof(float)));
    // v = ||c||^2 - 2 x.c in place; columns at or past k hold +inf (or NaN)
    float cn[CT];
#pragma unroll
    for (int j = 0; j < CT; ++j) cn[j] = cns[T::col(tx, j)];
    float mine[F32_RT];
#pragma unroll
    for (int i = 0; i < F32_RT / 2; ++i) {
      mine[2 * i] = mine[2 * i + 1] = f_inf();
#pragma unroll
      for (int j = 0; j < CT; ++j) {
        acc[i][j] = __ffma2_rn(make_float2(-2.0f, -2.0f), acc[i][j], make_float2(cn[j], cn[j]));
        mine[2 * i] = fminf(mine[2 * i], acc[i][j].x);
        mine[2 * i + 1] = fminf(mine[2 * i + 1], acc[i][j].y);
      }
    }
    // The rows' minima over their TX lanes: each exchange leaves a lane half of the rows it
    // goes on with, so that a lane ends with one row (lanes of 8 and above with a copy),
    // whose tau it works out for all.
    {
      float red[F32_RT];
      int own = 0;
#pragma unroll
      for (int i = 0; i < F32_RT; ++i) red[i] = mine[i];
#pragma unroll
      for (int o = 1, live = F32_RT; o < TX; o <<= 1) {
        const bool up = (tx & o) != 0;
        const int h = live / 2;
#pragma unroll
        for (int i = 0; i < (h ? h : 1); ++i) {
          const float give = h ? (up ? red[i] : red[i + h]) : red[i], hold = h && up ? red[i + h] : red[i];
          red[i] = fminf(hold, __shfl_xor_sync(0xffffffffu, give, o));
        }
        if (h) { own += up ? h : 0; live = h; }
      }
      if (tx < F32_RT) {
        F32Row& w = rs[ty * F32_RT + own];
        const float before = w.m, m = fminf(red[0], before), tau = tie_tau_at(w.tr, m, tb);
        // every entry so far is at least the minimum before: past tau the list starts
        // again, overflowed or not (many equal centroids that were the nearest so far)
        if (before > tau) w.cnt = 0u;
        w.m = m;
        w.tau = tau;
      }
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < F32_RT; ++i) {
      const int r = ty * F32_RT + i;
      const float tau = rs[r].tau;
      auto val = [&](int j) { return (i & 1) ? acc[i / 2][j].y : acc[i / 2][j].x; };
      if (DOUT && m0 + (uint64_t)r < n_log) {
#pragma unroll
        for (int j = 0; j < CT; ++j) {
          const uint32_t c = c0 + (uint32_t)T::col(tx, j);
          if (c < k) Dout[(uint64_t)rs[r].row * k + c] = val(j) + rs[r].x2;
        }
      }
      // this thread holds candidates of the row (whose list has not overflowed)
      if (mine[i] <= tau && *(volatile uint32_t*)&rs[r].cnt <= cap && m0 + (uint64_t)r < n_log) {
        uint32_t mask = 0;
#pragma unroll
        for (int j = 0; j < CT; ++j) mask |= (val(j) <= tau ? 1u : 0u) << j;
        while (mask) {
          const int b = __ffs(mask) - 1;
          mask &= mask - 1u;
          float v = val(0);
#pragma unroll
          for (int j = 1; j < CT; ++j) v = j == b ? val(j) : v;
          const uint32_t c = c0 + (uint32_t)T::col(tx, b);
          if (c < k) {
            const uint32_t at = atomicAdd(&rs[r].cnt, 1u);
            if (at < cap) list_of(r)[at] = make_uint2(c, __float_as_uint(v));
          }
        }
      }
    }
    __syncthreads();
    // Lists that another tile might fill drop the entries that m has left behind
    // (the product's barriers come before the next entries).
    if (c0 + T::COLS < k) {
      const uint32_t high = max(cap / 2u, cap > (uint32_t)T::COLS ? cap - (uint32_t)T::COLS : 0u);
      if (GATHER) {
        for (int r = tid >> 5; r < T::ROWS; r += F32_NT / 32) {
          const uint32_t cnt = rs[r].cnt;
          if (cnt <= high || cnt > cap) continue;
          const uint32_t kept = filter(list_of(r), cnt, tie_tau_at(rs[r].tr, rs[r].m, tb));
          if ((tid & 31) == 0) rs[r].cnt = kept;
        }
      } else {
        for (int r = tid; r < T::ROWS; r += F32_NT) {
          const uint32_t cnt = rs[r].cnt;
          if (cnt <= high || cnt > cap) continue;
          const float tau = tie_tau_at(rs[r].tr, rs[r].m, tb);
          uint2* const l = list_of(r);
          uint32_t kept = 0;
          for (uint32_t q = 0; q < cnt; ++q) {
            const uint2 en = l[q];
            if (__uint_as_float(en.y) <= tau) l[kept++] = en;
          }
          rs[r].cnt = kept;
        }
      }
    }
  }

  if (GATHER) {
    for (int r = tid >> 5; r < T::ROWS; r += F32_NT / 32) {
      const uint32_t cnt = rs[r].cnt;
      if (cnt > cap) continue;
      const uint32_t kept = filter(list_of(r), cnt, tie_tau_at(rs[r].tr, rs[r].m, tb));
      if ((tid & 31) == 0) rs[r].cnt = kept;
    }
    __syncthreads();
  }
  // One thread per row: the candidates in index order, classify, queue near ties.
  for (int r = tid; r < T::ROWS; r += F32_NT) {
    const F32Row w = rs[r];
    const uint64_t li = m0 + (uint64_t)r, seg = li >> 5;
    if (seg >= rq.nseg) break;                             // whole segments past the queues' end
    const bool valid = li < n_log;
    const float tau = tie_tau_at(w.tr, w.m, tb);
    uint32_t got = 0, e[4] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu};
    // (a gathered row's list is filtered already: only a short one is looked at)
    const bool wide = GATHER && w.cnt > 4u && w.cnt <= cap;
    const uint32_t nl = wide ? 0u : min(w.cnt, cap);
    const uint2* const l = list_of(r);
    for (uint32_t q = 0; q < nl && got <= 4u; ++q) {
      const uint2 en = l[q];
      if (!(__uint_as_float(en.y) <= tau)) continue;
      ++got;
      uint32_t c = en.x;                                   // insert, smallest index first
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const uint32_t lo = min(c, e[a]);
        c = max(c, e[a]);
        e[a] = lo;
      }
    }
    // values that are not finite prove nothing: such rows take the full path
    const bool fin = isfinite(w.tr.T + w.m + w.tr.Em);
    const bool full = !fin || w.cnt > cap || (!wide && (got == 0u || got > 4u));
    if (valid) {
      labels[w.row] = got ? e[0] : 0u;
      if (mindist) mindist[w.row] = w.m + w.x2;
    }
    RefineEntry en{w.row, got, {e[0], e[1], e[2], e[3]}};
    seg_push(rq.cand, rq.ccnt, seg, valid && !full && !wide && got >= 2u, en);
    if (GATHER) {
      if (valid && wide) rq.wlc[w.row] = w.cnt;
      seg_push(rq.wide, rq.wcnt, seg, valid && !full && wide, w.row);
    }
    seg_push(rq.full, rq.fcnt, seg, valid && full, w.row);
  }
}

namespace {
// The narrowest tile that holds k (chunks of 128 above, of 96 where two of them
// hold k): the product's time goes with the tile's width.
template <class F>
void f32_shape(uint32_t k, F f) {
  if (k <= 32u) f(std::integral_constant<int, 8>{}, std::integral_constant<int, 4>{});
  else if (k <= 48u) f(std::integral_constant<int, 8>{}, std::integral_constant<int, 6>{});
  else if (k <= 64u) f(std::integral_constant<int, 8>{}, std::integral_constant<int, 8>{});
  else if (k <= 96u || (k > 128u && k <= 192u)) f(std::integral_constant<int, 16>{}, std::integral_constant<int, 6>{});
  else f(std::integral_constant<int, 16>{}, std::integral_constant<int, 8>{});
}
void launch_f32(const float* X, const float* C, const float* cn2, const float* xn2, uint64_t n, uint32_t d, uint32_t k,
                TieBound tb, DevState* st, uint32_t* labels, float* mindist, const RefineQueues& rq, float* Dout,
                const uint32_t* ridx, const uint32_t* nidx, cudaStream_t s) {
  const bool v4 = (d % 4 == 0) && (reinterpret_cast<uintptr_t>(X) % 16 == 0) &&
                  (reinterpret_cast<uintptr_t>(C) % 16 == 0);
  f32_shape(k, [&](auto tx, auto ct) {
    using T = F32Tile<tx(), ct()>;
    const uint64_t rows = rq.nseg * 32;                    // whole segments of the queues
    const unsigned blocks = (unsigned)((rows + T::ROWS - 1) / T::ROWS);
    auto kern = ridx   ? assign_f32_kernel<tx(), ct(), false, true>
                : Dout ? assign_f32_kernel<tx(), ct(), true, false>
                       : assign_f32_kernel<tx(), ct(), false, false>;
    (void)launch_pdl(kern, blocks, F32_NT, ridx ? f32_smem<T, true>() : f32_smem<T, false>(), s, X, C, v4, cn2, xn2, n, d, k, tb, st, labels, mindist, rq,
                     Dout, ridx, nidx);
  });
}
}  // namespace

km_status launch_assign_f32(const float* X, const float* C, const float* cn2, const float* xn2,
                            uint64_t n, uint32_t d, uint32_t k, TieBound tb, DevState* st,
                            uint32_t* labels, float* mindist, const RefineQueues& rq,
                            float* Dout, cudaStream_t s) {
  launch_f32(X, C, cn2, xn2, n, d, k, tb, st, labels, mindist, rq, Dout, nullptr, nullptr, s);
  KM_CUDA_TRY(cudaGetLastError());
  return KM_OK;
}

// Exact re-score of rows with 2..4 candidates, for rows that are not 16-byte
// aligned or d % 4 != 0 (refine_staged_kernel below is the vector path): four
// lanes per row, one candidate per lane, the reference's CPU distance (float,
// j ascending); smallest distance wins, lowest index on ties.  The candidate
// set provably holds the reference argmin over all k (tie_tau).
// One warp per RC_SEGS consecutive queue segments, their entries flattened so
// that every pass keeps eight rows in flight; the grid covers all segments at
// once (no loop over segments, so a warp pays one count load and its rows).
constexpr int RC_SEGS = 2;
constexpr int RC_WARPS = 8;

__global__ void __launch_bounds__(32 * RC_WARPS)
refine_cands_kernel(const float* __restrict__ X, const float* __restrict__ C, uint32_t d,
                    DevState* st, RefineQueues rq, uint32_t* __restrict__ labels,
                    float* __restrict__ mindist, bool count) {
  griddep_wait();
  if (st->done) return;
  __shared__ uint32_t block_rows;
  if (threadIdx.x == 0) block_rows = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t seg0 = warp * RC_SEGS;
  // inclusive prefix of the RC_SEGS segment counts, kept in every lane
  const uint32_t c = (lane < RC_SEGS && seg0 + (uint64_t)lane < rq.nseg) ? rq.ccnt[seg0 + lane] : 0u;
  uint32_t pre[RC_SEGS];
  uint32_t run = 0;
#pragma unroll
  for (int q = 0; q < RC_SEGS; ++q) {
    run += __shfl_sync(0xffffffffu, c, q);
    pre[q] = run;
  }
  const uint32_t total = run;
  const uint32_t slot = (uint32_t)lane & 3u;
  for (uint32_t base = 0; base < total; base += 8) {
    const uint32_t qi = base + (uint32_t)(lane >> 2);
    float bv = f_inf();
    uint32_t bi = 0xffffffffu;
    uint32_t row = 0;
    if (qi < total) {
      uint32_t sg = 0, before = 0;
#pragma unroll
      for (int q = 0; q < RC_SEGS - 1; ++q)
        if (qi >= pre[q]) { sg = (uint32_t)q + 1u; before = pre[q]; }
      const RefineEntry en = rq.cand[(seg0 + sg) * 32 + (qi - before)];
      row = en.row;
      if (slot < en.cnt) {
        const uint32_t cc = en.c[slot];
        const float* x = X + (uint64_t)row * d;
        const float* cr = C + (uint64_t)cc * d;
        const float v = cpu_dist(x, cr, d);
        if (v < bv) { bv = v; bi = cc; }
      }
    }
#pragma unroll
    for (int o = 1; o <= 2; o <<= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
      const uint32_t oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov < bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
    }
    if (qi < total && slot == 0) {
      labels[row] = (bi == 0xffffffffu) ? 0u : bi;
      if (mindist) mindist[row] = bv;
    }
  }
  if (count && lane == 0 && total) atomicAdd(&block_rows, total);
  __syncthreads();
  if (count && threadIdx.x == 0 && block_rows)
    atomicAdd(&st->refined_total, (unsigned long long)block_rows);
}

// Exact re-score of a group of up to FULL_ROWS rows (row ids rows[0..nr))
// against all k centroids by one warp: lanes over centroids (eight chains per
// lane and row), centroids read from the transposed copy Ct (d x k) so that
// every load of the warp is one coalesced 128-byte line and serves all rows of
// the group.  Per lane the centroids are visited in ascending order with a
// strict '<' and the warp reduction keeps the lowest index on ties: the
// reference's argmin (kmeans.cpp:106-122).
constexpr int FULL_ROWS = 4;

__device__ __forceinline__ void full_rescore_group(const float* __restrict__ X, const float* __restrict__ Ct,
                                                   uint32_t d, uint32_t k, const uint32_t* rows, uint32_t nr,
                                                   uint32_t* __restrict__ labels, float* __restrict__ mindist) {
  const int lane = threadIdx.x & 31;
  uint32_t row[FULL_ROWS];
  const float* x[FULL_ROWS];
#pragma unroll
  for (int r = 0; r < FULL_ROWS; ++r) {
    row[r] = rows[min((uint32_t)r, nr - 1)];   // pad with the last row
    x[r] = X + (uint64_t)row[r] * d;
  }
  float bv[FULL_ROWS];
  uint32_t bi[FULL_ROWS];
#pragma unroll
  for (int r = 0; r < FULL_ROWS; ++r) { bv[r] = f_inf(); bi[r] = 0xffffffffu; }
  for (uint32_t cb = 0; cb < k; cb += 256) {
    float s[FULL_ROWS][8];
#pragma unroll
    for (int r = 0; r < FULL_ROWS; ++r)
#pragma unroll
      for (int t = 0; t < 8; ++t) s[r][t] = 0.0f;
    // Four j steps per group: all their loads (the rows' x_j, the lanes'
    // centroid columns from Ct) are issued before the group's arithmetic,
    // which keeps 48 loads in flight per lane instead of one step's.
    for (uint32_t j0 = 0; j0 < d; j0 += 4) {
      float xj[4][FULL_ROWS], cv[4][8];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t j = j0 + (uint32_t)q;
        const bool jin = j < d;
#pragma unroll
        for (int r = 0; r < FULL_ROWS; ++r) xj[q][r] = jin ? x[r][j] : 0.0f;
        const float* ct = Ct + (uint64_t)(jin ? j : 0u) * k + cb + lane;
#pragma unroll
        for (int t = 0; t < 8; ++t) cv[q][t] = (jin && cb + lane + 32 * t < k) ? ct[32 * t] : 0.0f;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (j0 + (uint32_t)q >= d) break;
#pragma unroll
        for (int t = 0; t < 8; ++t) {
#pragma unroll
          for (int r = 0; r < FULL_ROWS; ++r) {
            const float tt = __fsub_rn(xj[q][r], cv[q][t]);
            s[r][t] = __fadd_rn(s[r][t], __fmul_rn(tt, tt));
          }
        }
      }
    }
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const uint32_t c = cb + lane + 32 * t;
#pragma unroll
      for (int r = 0; r < FULL_ROWS; ++r)
        if (c < k && s[r][t] < bv[r]) { bv[r] = s[r][t]; bi[r] = c; }
    }
  }
#pragma unroll
  for (int r = 0; r < FULL_ROWS; ++r) {
    float v = bv[r];
    uint32_t i = bi[r];
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, v, o);
      const uint32_t oi = __shfl_xor_sync(0xffffffffu, i, o);
      if (ov < v || (ov == v && oi < i)) { v = ov; i = oi; }
    }
    if (lane == 0 && (uint32_t)r < nr) {
      labels[row[r]] = (i == 0xffffffffu) ? 0u : i;
      if (mindist) mindist[row[r]] = v;
    }
  }
}

// Rows of the full queue, warp by warp: segments warp, warp + nw, warp + 2 nw,
// ... (a dense queue spreads over all warps); 32 of their counts per load,
// only the non-empty ones visited.
__global__ void __launch_bounds__(256, 2)
refine_full_kernel(const float* __restrict__ X, const float* __restrict__ Ct, uint32_t d, uint32_t k,
                   DevState* st, RefineQueues rq, uint32_t* __restrict__ labels,
                   float* __restrict__ mindist, bool count) {
  griddep_wait();
  if (st->done) return;
  const int lane = threadIdx.x & 31;
  const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  uint32_t done_rows = 0;
  for (uint64_t g0 = warp; g0 < rq.nseg; g0 += nw * 32) {
    const uint64_t sgl = g0 + (uint64_t)lane * nw;
    const uint32_t cl = (sgl < rq.nseg) ? rq.fcnt[sgl] : 0u;
    uint32_t nz = __ballot_sync(0xffffffffu, cl != 0u);
    while (nz) {
      const int sl = __ffs(nz) - 1;
      nz &= nz - 1u;
      const uint64_t seg = g0 + (uint64_t)sl * nw;
      const uint32_t cnt = __shfl_sync(0xffffffffu, cl, sl);
      done_rows += cnt;
      for (uint32_t e0 = 0; e0 < cnt; e0 += FULL_ROWS)
        full_rescore_group(X, Ct, d, k, rq.full + seg * 32 + e0, min(cnt - e0, (uint32_t)FULL_ROWS), labels,
                           mindist);
    }
  }
  if (count && lane == 0 && done_rows) {
    atomicAdd(&st->refined_total, (unsigned long long)done_rows);
    atomicAdd(&st->full_total, (unsigned long long)done_rows);
  }
}

// Exact re-score of the candidate queue with its operands staged in shared
// memory (d % 4 == 0, 16-byte aligned rows).  Each warp owns ranges of `span`
// (<= 32) consecutive queue segments, one segment count per lane, and walks a
// range's entries in passes.  A pass takes the leading entries whose point
// rows and candidate centroid rows fit RS_ROWS staged rows: the entries' point
// rows at [0, ne), the pairs' centroid rows at [ne, ne + np), pair p on lane p.
// The rows are copied by the TMA engine, one bulk copy per row issued by the
// lane that owns the row, RS_CH columns per round trip (all of d when d <=
// RS_CH), completing on the warp's mbarrier; the loads of the next pass's
// entries are issued before the copies are waited on.  (16-byte cp.async per
// lane, one row per instruction, spent most of the pass issuing the copies.)  Every lane then runs the reference's ordered
// chain (float, j ascending, no contraction) from shared memory.  A lane that
// loads its own rows straight from global memory touches up to 32 lines per
// instruction, and the L1 wavefronts, not DRAM, then set the time.  The
// entry's lane picks the smallest distance over its candidates in ascending
// index order with a strict '<' (lowest index on ties).  The candidate set
// provably holds the reference argmin over all k (tie_tau).
// FULL: the grid's warps then re-score the full queue against all k
// (full_rescore_group), so that one launch covers the whole refinement.
constexpr int RS_WARPS = 5;
constexpr int RS_ROWS = 40;              // staged rows per pass (at most 32 pairs)
constexpr uint32_t RS_CH = 128;          // staged columns per round trip
constexpr int RS_BLOCKS_PER_SM = 2;
constexpr uint64_t RS_WAIT_NS = 2000000000ull;   // bound of a wait for the warp's copies
// Shared row stride in floats for chunks of ch columns, with (stride / 4) odd
// so that float4 reads of eight consecutive rows cover the 32 banks.
__host__ __device__ constexpr uint32_t rs_ld(uint32_t ch) { return ((ch + 4u) / 4u) % 2u ? ch + 4u : ch + 8u; }
constexpr size_t RS_SMEM_MAX = (size_t)RS_WARPS * RS_ROWS * rs_ld(RS_CH) * sizeof(float);

template <bool FULL>
__global__ void __launch_bounds__(32 * RS_WARPS, RS_BLOCKS_PER_SM)
refine_staged_kernel(const float* __restrict__ X, const float* __restrict__ C, const float* __restrict__ Ct,
                     uint32_t d, uint32_t k, uint32_t span, DevState* st, RefineQueues rq,
                     uint32_t* __restrict__ labels, float* __restrict__ mindist, bool count) {
  griddep_wait();
  if (st->done) return;
  extern __shared__ __align__(16) float rs_smem[];
  __shared__ __align__(8) uint64_t rs_bar[RS_WARPS];
  __shared__ int rs_no_abort[RS_WARPS];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const uint32_t ch = min(d, RS_CH), ld = rs_ld(ch);
  float* const stg = rs_smem + (size_t)wib * RS_ROWS * ld;
  uint64_t* const bar = &rs_bar[wib];   // this warp's copies
  if (lane == 0) {
    mbar_init(bar, 1);
    rs_no_abort[wib] = 0;
    mbar_fence_init();
  }
  __syncwarp();
  uint32_t ph = 0;   // parity of the barrier phase the next wait completes
  const uint64_t nranges = (rq.nseg + span - 1) / span;
  const uint64_t nw = (uint64_t)gridDim.x * RS_WARPS;
  uint32_t cand_rows = 0, full_rows = 0;
  for (uint64_t rg = (uint64_t)blockIdx.x * RS_WARPS + wib; rg < nranges; rg += nw) {
    const uint64_t seg0 = rg * span;
    const bool segok = (uint32_t)lane < span && seg0 + (uint64_t)lane < rq.nseg;
    const uint32_t c = segok ? rq.ccnt[seg0 + lane] : 0u;
    uint32_t pre = c;   // inclusive prefix of the segment counts over the lanes
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, pre, o);
      if (lane >= o) pre += y;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, pre, 31);
    cand_rows += total;
    // Entry t of the range (all lanes call; loads only for t < total): its
    // segment is the number of lanes whose prefix is <= t.
    auto load_entry = [&](uint32_t t) {
      uint32_t sg = 0;
#pragma unroll
      for (int step = 16; step > 0; step >>= 1) {
        const uint32_t pv = __shfl_sync(0xffffffffu, pre, (int)(sg + (uint32_t)step - 1u));
        if (pv <= t) sg += (uint32_t)step;
      }
      const uint32_t before = __shfl_sync(0xffffffffu, pre, (int)((sg + 31u) & 31u));
      RefineEntry r{0u, 0u, {0u, 0u, 0u, 0u}};
      if (t < total) r = rq.cand[(seg0 + sg) * 32 + (t - (sg ? before : 0u))];
      return r;
    };
    RefineEntry en = load_entry((uint32_t)lane);
    for (uint32_t e0 = 0; e0 < total;) {
      const bool has = e0 + (uint32_t)lane < total;
      const uint32_t cl = has ? max(1u, min(en.cnt, 4u)) : 0u;
      uint32_t incl = cl;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      // entries of this pass: the leading lanes whose rows (one point row per
      // entry, one centroid row per pair) fit RS_ROWS and whose pairs fit the
      // 32 lanes (at least eight entries, cl <= 4)
      const uint32_t ne = (uint32_t)__popc(
          __ballot_sync(0xffffffffu, has && incl <= 32u && (uint32_t)lane + 1u + incl <= (uint32_t)RS_ROWS));
      const uint32_t np = __shfl_sync(0xffffffffu, incl, (int)ne - 1);
      const uint32_t off = incl - cl;
      // pair p = lane: its entry e (the last entry lane with off <= p)
      const uint32_t p = (uint32_t)lane;
      uint32_t e = 0;
#pragma unroll
      for (int step = 16; step > 0; step >>= 1) {
        const uint32_t t = e + (uint32_t)step;
        const uint32_t ot = __shfl_sync(0xffffffffu, off, (int)(t & 31u));
        if (t < ne && ot <= p) e = t;
      }
      const uint32_t m = p - __shfl_sync(0xffffffffu, off, (int)e);
      const uint32_t q0 = __shfl_sync(0xffffffffu, en.c[0], (int)e);
      const uint32_t q1 = __shfl_sync(0xffffffffu, en.c[1], (int)e);
      const uint32_t q2 = __shfl_sync(0xffffffffu, en.c[2], (int)e);
      const uint32_t q3 = __shfl_sync(0xffffffffu, en.c[3], (int)e);
      const uint32_t cand = m == 0 ? q0 : m == 1 ? q1 : m == 2 ? q2 : q3;   // meaningful for p < np
      const uint32_t nrows = ne + np;
      // Source rows of the staged rows: lane r holds staged row r (r < 32) and
      // lane r - 32 holds staged row r >= 32 (16-byte aligned: d % 4 == 0).
      const uint32_t crl = __shfl_sync(0xffffffffu, cand, (int)(((uint32_t)lane - ne) & 31u));
      const uint32_t crh = __shfl_sync(0xffffffffu, cand, (int)(((uint32_t)lane + 32u - ne) & 31u));
      const uint64_t srcl = (uint32_t)lane < ne ? reinterpret_cast<uint64_t>(X + (uint64_t)en.row * d)
                                                : reinterpret_cast<uint64_t>(C + (uint64_t)crl * d);
      const uint64_t srch = reinterpret_cast<uint64_t>(C + (uint64_t)crh * d);
      // columns [j0, j0 + nc) of the pass's rows: one bulk copy per row (a
      // multiple of 16 bytes between 16-byte aligned addresses)
      auto stage = [&](uint32_t j0) {
        const uint32_t bytes = min(ch, d - j0) * 4u;
        // Every earlier read of the rows has returned its value (the chain's
        // sums went through the lane reduction) before any lane gets here.
        if (lane == 0) mbar_arrive_expect_tx(bar, nrows * bytes);
        __syncwarp();
        if ((uint32_t)lane < nrows)
          bulk_copy_g2s(stg + lane * ld, reinterpret_cast<const float*>(srcl) + j0, bytes, bar);
        if ((uint32_t)lane + 32u < nrows)
          bulk_copy_g2s(stg + (32u + lane) * ld, reinterpret_cast<const float*>(srch) + j0, bytes, bar);
      };
      stage(0);
      const uint32_t e0n = e0 + ne;
      const RefineEntry enn = load_entry(e0n + (uint32_t)lane);   // in flight during this pass
      float s = 0.0f;
      auto step4 = [&](const float4 a, const float4 b) {
        float t = __fsub_rn(a.x, b.x); s = __fadd_rn(s, __fmul_rn(t, t));
        t = __fsub_rn(a.y, b.y); s = __fadd_rn(s, __fmul_rn(t, t));
        t = __fsub_rn(a.z, b.z); s = __fadd_rn(s, __fmul_rn(t, t));
        t = __fsub_rn(a.w, b.w); s = __fadd_rn(s, __fmul_rn(t, t));
      };
      for (uint32_t j0 = 0; j0 < d; j0 += ch) {
        if (j0) stage(j0);
        const bool okw = mbar_wait_bounded(bar, ph, &rs_no_abort[wib], RS_WAIT_NS);
        ph ^= 1u;
        if (!__all_sync(0xffffffffu, okw)) {
          // copies that never landed: flag, give the ones in flight a bounded
          // second wait, and end this warp (no block barrier follows)
          if (lane == 0) atomicOr(&st->err, KM_DEVERR_TIMEOUT);
          mbar_wait_bounded(bar, ph ^ 1u, &rs_no_abort[wib], RS_WAIT_NS);
          return;
        }
        if (p < np) {
          const float4* xs = reinterpret_cast<const float4*>(stg + e * ld);
          const float4* cs = reinterpret_cast<const float4*>(stg + (ne + p) * ld);
          const uint32_t nc4 = min(ch, d - j0) / 4u;
          if (nc4 == RS_CH / 4u) {
#pragma unroll 8
            for (uint32_t q = 0; q < RS_CH / 4u; ++q) step4(xs[q], cs[q]);
          } else {
            for (uint32_t q = 0; q < nc4; ++q) step4(xs[q], cs[q]);
          }
        }
        __syncwarp();   // the rows are restaged only after every lane's chain
      }
      // entry lane: the smallest of its cl candidates (pairs off .. off+cl-1)
      float bv = 0.0f;
      uint32_t bi = 0u;
#pragma unroll
      for (uint32_t mm = 0; mm < 4; ++mm) {
        const int src = (int)((off + mm) & 31u);
        const float v = __shfl_sync(0xffffffffu, s, src);
        const uint32_t ci = __shfl_sync(0xffffffffu, cand, src);
        if (mm == 0 || (mm < cl && v < bv)) { bv = v; bi = ci; }
      }
      if ((uint32_t)lane < ne) {
        labels[en.row] = bi;
        if (mindist) mindist[en.row] = bv;
      }
      en = enn;
      e0 = e0n;
    }
  }
  if (FULL) {
    // The full queue, interleaved over every warp of the grid as in
    // refine_full_kernel (its rows can be many and bunched: e.g. the FP32 pass
    // at very large k); 32 segment counts per load, only non-empty ones visited.
    for (uint64_t g0 = (uint64_t)blockIdx.x * RS_WARPS + wib; g0 < rq.nseg; g0 += nw * 32) {
      const uint64_t sgl = g0 + (uint64_t)lane * nw;
      const uint32_t fl = (sgl < rq.nseg) ? rq.fcnt[sgl] : 0u;
      uint32_t nz = __ballot_sync(0xffffffffu, fl != 0u);
      while (nz) {
        const int sl = __ffs(nz) - 1;
        nz &= nz - 1u;
        const uint64_t seg = g0 + (uint64_t)sl * nw;
        const uint32_t cnt = __shfl_sync(0xffffffffu, fl, sl);
        full_rows += cnt;
        for (uint32_t f0 = 0; f0 < cnt; f0 += FULL_ROWS)
          full_rescore_group(X, Ct, d, k, rq.full + seg * 32 + f0, min(cnt - f0, (uint32_t)FULL_ROWS), labels,
                             mindist);
      }
    }
  }
  if (count && lane == 0 && cand_rows + full_rows)
    atomicAdd(&st->refined_total, (unsigned long long)(cand_rows + full_rows));
  if (count && lane == 0 && full_rows) atomicAdd(&st->full_total, (unsigned long long)full_rows);
}

// Launch shape of refine_staged_kernel: a persistent grid, each warp a range
// of `span` consecutive segments.
struct StagedShape {
  unsigned blocks;
  uint32_t span;
  size_t smem;
};
static StagedShape staged_shape(int num_sms, uint64_t nseg, uint32_t d) {
  const uint64_t max_warps = (uint64_t)num_sms * RS_BLOCKS_PER_SM * RS_WARPS;
  const uint32_t span = (uint32_t)std::min<uint64_t>(32, std::max<uint64_t>(1, (nseg + max_warps - 1) / max_warps));
  const uint64_t ranges = (nseg + span - 1) / span;
  StagedShape sh;
  sh.blocks = (unsigned)std::max<uint64_t>(
      1, std::min<uint64_t>((uint64_t)num_sms * RS_BLOCKS_PER_SM, (ranges + RS_WARPS - 1) / RS_WARPS));
  sh.span = span;
  sh.smem = (size_t)RS_WARPS * RS_ROWS * rs_ld(std::min<uint32_t>(d, RS_CH)) * sizeof(float);
  return sh;
}

static void launch_refine_cands(bool v4, int num_sms, const float* X, const float* C, uint32_t d,
                                DevState* st, const RefineQueues& rq, uint32_t* labels, float* mindist,
                                bool count, cudaStream_t s) {
  if (v4) {
    const StagedShape sh = staged_shape(num_sms, rq.nseg, d);
    (void)launch_pdl(refine_staged_kernel<false>, sh.blocks, 32 * RS_WARPS, sh.smem, s, X, C,
                     (const float*)nullptr, d, 0u, sh.span, st, rq, labels, mindist, count);
  } else {
    const uint64_t warps = (rq.nseg + RC_SEGS - 1) / RC_SEGS;
    const unsigned blocks = (unsigned)std::max<uint64_t>(1, (warps + RC_WARPS - 1) / RC_WARPS);
    (void)launch_pdl(refine_cands_kernel, blocks, 32 * RC_WARPS, 0, s, X, C, d, st, rq, labels, mindist, count);
  }
}

// Rows of the full queue gathered into one list (order irrelevant: every row
// is re-scored on its own), counted as fully re-scored rows.
__global__ void full_compact_kernel(DevState* st, RefineQueues rq, uint32_t* __restrict__ out,
                                    uint32_t* __restrict__ nout) {
  griddep_wait();
  if (st->done) return;
  const int lane = threadIdx.x & 31;
  const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  uint32_t done_rows = 0;
  for (uint64_t seg = warp; seg < rq.nseg; seg += nw) {
    const uint32_t cnt = rq.fcnt[seg];
    if (cnt == 0u) continue;
    done_rows += cnt;
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(nout, cnt);
    base = __shfl_sync(0xffffffffu, base, 0);
    if ((uint32_t)lane < cnt) out[base + lane] = rq.full[seg * 32 + lane];
  }
  if (lane == 0 && done_rows) {
    atomicAdd(&st->refined_total, (unsigned long long)done_rows);
    atomicAdd(&st->full_total, (unsigned long long)done_rows);
  }
}

// Exact re-score of rows with 5..L candidates (chunked distance kernel), for rows that are
// not 16-byte aligned or d % 4 != 0 (refine_wide_staged_kernel below is the vector path):
// one warp per row, lanes stride over the row's candidates, the reference's CPU distance;
// smallest distance wins, lowest index on ties.
__global__ void __launch_bounds__(256, 2)
refine_wide_kernel(const float* __restrict__ X, const float* __restrict__ C, uint32_t d,
                   DevState* st, RefineQueues rq, uint32_t* __restrict__ labels,
                   float* __restrict__ mindist, bool count) {
  griddep_wait();
  if (st->done) return;
  const int lane = threadIdx.x & 31;
  const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  uint32_t done_rows = 0;
  for (uint64_t seg = warp; seg < rq.nseg; seg += nw) {
    const uint32_t cnt = rq.wcnt[seg];
    done_rows += cnt;
    for (uint32_t e = 0; e < cnt; ++e) {
      const uint32_t row = rq.wide[seg * 32 + e];
      const uint32_t nc = min(rq.wlc[row], rq.L);
      float bv = f_inf();
      uint32_t bi = 0xffffffffu;
      const float* x = X + (uint64_t)row * d;
      for (uint32_t e = (uint32_t)lane; e < nc; e += 32u) {
        const uint32_t c = rq.wl[(uint64_t)row * rq.L + e].x;
        const float v = cpu_dist(x, C + (uint64_t)c * d, d);
        if (v < bv || (v == bv && c < bi)) { bv = v; bi = c; }
      }
      for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const uint32_t oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov < bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
      }
      if (lane == 0) {
        labels[row] = (bi == 0xffffffffu) ? 0u : bi;
        if (mindist) mindist[row] = bv;
      }
    }
  }
  if (count && lane == 0 && done_rows) atomicAdd(&st->refined_total, (unsigned long long)done_rows);
}

// The same with the operands staged in shared memory by bulk copies, as in
// refine_staged_kernel (d % 4 == 0, 16-byte aligned rows).  A warp takes a segment's
// rows (one per lane) and walks their (row, candidate) pairs in passes of up to 32, one
// pair per lane, of up to RW_ENTRIES rows: a lane's distance joins its row's over the
// pass by a segmented scan, and the row's lane keeps the best over the passes (a row's
// candidates can span several).  A lane that reads its candidate's row from global memory
// itself touches 32 lines per instruction, whose L1 wavefronts set the time; now bound by
// the copies' bytes out of L2.  n = 4M d = 256 k = 4096 (BF16 points, Zipf sizes): 22.5 ->
// 10.9 ms an iteration, both queues.
constexpr int RW_ENTRIES = RS_ROWS - 32;      // point rows of a pass, staged before the candidates'
__global__ void __launch_bounds__(32 * RS_WARPS, RS_BLOCKS_PER_SM)
refine_wide_staged_kernel(const float* __restrict__ X, const float* __restrict__ C, uint32_t d, DevState* st,
                          RefineQueues rq, uint32_t* __restrict__ labels, float* __restrict__ mindist, bool count) {
  griddep_wait();
  if (st->done) return;
  extern __shared__ __align__(16) float rs_smem[];
  __shared__ __align__(8) uint64_t rw_bar[RS_WARPS];
  __shared__ int rw_no_abort[RS_WARPS];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const uint32_t ch = min(d, RS_CH), ld = rs_ld(ch);
  float* const stg = rs_smem + (size_t)wib * RS_ROWS * ld;
  uint64_t* const bar = &rw_bar[wib];   // this warp's copies
  if (lane == 0) {
    mbar_init(bar, 1);
    rw_no_abort[wib] = 0;
    mbar_fence_init();
  }
  __syncwarp();
  uint32_t ph = 0;
  const uint64_t warp = (uint64_t)blockIdx.x * RS_WARPS + wib, nw = (uint64_t)gridDim.x * RS_WARPS;
  uint32_t done_rows = 0;
  auto better = [](float v, uint32_t i, float bv, uint32_t bi) { return v < bv || (v == bv && i < bi); };
  for (uint64_t g0 = warp; g0 < rq.nseg; g0 += nw * 32) {
    const uint64_t sgl = g0 + (uint64_t)lane * nw;
    const uint32_t cl = sgl < rq.nseg ? rq.wcnt[sgl] : 0u;
    uint32_t nz = __ballot_sync(0xffffffffu, cl != 0u);
    while (nz) {
      const int sl = __ffs(nz) - 1;
      nz &= nz - 1u;
      const uint64_t seg = g0 + (uint64_t)sl * nw;
      const uint32_t cnt = __shfl_sync(0xffffffffu, cl, sl);
      done_rows += cnt;
      // lane e: row e of the segment, its candidates [incl - nc, incl) of the pairs
      const bool mine = (uint32_t)lane < cnt;
      const uint32_t row = mine ? rq.wide[seg * 32 + lane] : 0u;
      const uint32_t nc = mine ? min(rq.wlc[row], rq.L) : 0u;
      uint32_t incl = nc;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
      float bv = f_inf();
      uint32_t bi = 0xffffffffu;
      for (uint32_t p0 = 0; p0 < total;) {
        const uint32_t p = p0 + (uint32_t)lane;
        uint32_t e = 0;                          // the pair's row: the lanes whose incl is <= p
#pragma unroll
        for (int step = 16; step > 0; step >>= 1) {
          const uint32_t pv = __shfl_sync(0xffffffffu, incl, (int)(e + (uint32_t)step - 1u));
          if (pv <= p) e += (uint32_t)step;
        }
        const uint32_t first = __shfl_sync(0xffffffffu, e, 0);
        const uint32_t np = (uint32_t)__popc(__ballot_sync(0xffffffffu, p < total && e - first < (uint32_t)RW_ENTRIES));
        const uint32_t ne = __shfl_sync(0xffffffffu, e, (int)np - 1) - first + 1u;
        const bool has = (uint32_t)lane < np;
        const uint32_t row_e = __shfl_sync(0xffffffffu, row, (int)e);
        const uint32_t excl_e = __shfl_sync(0xffffffffu, incl - nc, (int)e);
        const uint32_t cand = has ? rq.wl[(uint64_t)row_e * rq.L + (p - excl_e)].x : 0u;
        const uint32_t xrow = __shfl_sync(0xffffffffu, row, (int)((first + (uint32_t)lane) & 31u));
        const float* xp = X + (uint64_t)xrow * d;            // lane < ne
        const float* cp = C + (uint64_t)cand * d;            // lane < np
        const float4* xs = reinterpret_cast<const float4*>(stg + (has ? e - first : 0u) * ld);
        const float4* cs = reinterpret_cast<const float4*>(stg + (RW_ENTRIES + lane) * ld);
        float s = 0.0f;
        auto step4 = [&](const float4 a, const float4 b) {
          float t = __fsub_rn(a.x, b.x); s = __fadd_rn(s, __fmul_rn(t, t));
          t = __fsub_rn(a.y, b.y); s = __fadd_rn(s, __fmul_rn(t, t));
          t = __fsub_rn(a.z, b.z); s = __fadd_rn(s, __fmul_rn(t, t));
          t = __fsub_rn(a.w, b.w); s = __fadd_rn(s, __fmul_rn(t, t));
        };
        for (uint32_t j0 = 0; j0 < d; j0 += ch) {
          const uint32_t cols = min(ch, d - j0), bytes = cols * 4u;
          // every lane's reads of the rows before were ordered by the barrier below
          if (lane == 0) mbar_arrive_expect_tx(bar, (np + ne) * bytes);
          __syncwarp();
          if ((uint32_t)lane < ne) bulk_copy_g2s(stg + lane * ld, xp + j0, bytes, bar);
          if (has) bulk_copy_g2s(stg + (RW_ENTRIES + lane) * ld, cp + j0, bytes, bar);
          const bool okw = mbar_wait_bounded(bar, ph, &rw_no_abort[wib], RS_WAIT_NS);
          ph ^= 1u;
          if (!__all_sync(0xffffffffu, okw)) {
            // copies that never landed: flag, give the ones in flight a bounded
            // second wait, and end this warp (no block barrier follows)
            if (lane == 0) atomicOr(&st->err, KM_DEVERR_TIMEOUT);
            mbar_wait_bounded(bar, ph ^ 1u, &rw_no_abort[wib], RS_WAIT_NS);
            return;
          }
          if (has) {
            if (cols == RS_CH) {
#pragma unroll 8
              for (uint32_t q = 0; q < RS_CH / 4u; ++q) step4(xs[q], cs[q]);
            } else {
              for (uint32_t q = 0; q < cols / 4u; ++q) step4(xs[q], cs[q]);
            }
          }
          __syncwarp();   // the rows are restaged only after every lane's chain
        }
        // smallest distance per row over the pass, in the row's last lane; a distance
        // that is not a number is never chosen
        uint32_t i = has && s == s ? cand : 0xffffffffu;
        float v = has && s == s ? s : f_inf();
        const uint32_t key = has ? e : 64u + (uint32_t)lane;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const float ov = __shfl_up_sync(0xffffffffu, v, o);
          const uint32_t oi = __shfl_up_sync(0xffffffffu, i, o), ok = __shfl_up_sync(0xffffffffu, key, o);
          if (lane >= o && ok == key && better(ov, oi, v, i)) { v = ov; i = oi; }
        }
        const uint32_t last = min(incl, p0 + np) - 1u - p0;
        const float rv = __shfl_sync(0xffffffffu, v, (int)(last & 31u));
        const uint32_t ri = __shfl_sync(0xffffffffu, i, (int)(last & 31u));
        if (mine && incl > p0 && incl - nc < p0 + np && better(rv, ri, bv, bi)) { bv = rv; bi = ri; }
        p0 += np;
      }
      if (mine) {
        labels[row] = (bi == 0xffffffffu) ? 0u : bi;
        if (mindist) mindist[row] = bv;
      }
    }
  }
  if (count && lane == 0 && done_rows) atomicAdd(&st->refined_total, (unsigned long long)done_rows);
}

km_status refine_prepare() {
  cudaError_t err = cudaSuccess;
  for (uint32_t k : {32u, 48u, 64u, 96u, 128u})            // every shape of the FP32 distance kernel
    f32_shape(k, [&](auto tx, auto ct) {
      for (auto kern : {assign_f32_kernel<tx(), ct(), true, false>, assign_f32_kernel<tx(), ct(), false, false>,
                        assign_f32_kernel<tx(), ct(), false, true>})
        if (err == cudaSuccess)
          err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)f32_smem<F32Tile<tx(), ct()>, true>());
    });
  KM_CUDA_TRY(err);
  KM_CUDA_TRY(cudaFuncSetAttribute(refine_staged_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)RS_SMEM_MAX));
  KM_CUDA_TRY(cudaFuncSetAttribute(refine_staged_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)RS_SMEM_MAX));
  KM_CUDA_TRY(cudaFuncSetAttribute(refine_wide_staged_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)RS_SMEM_MAX));
  return KM_OK;
}

km_status launch_refine(bool v4, int num_sms, const float* X, const float* C, const float* Ct,
                        uint32_t d, uint32_t k, DevState* st, const RefineQueues& rq,
                        uint32_t* labels, float* mindist, cudaStream_t s) {
  // Every row sits in one queue at most, so the queues are re-scored in any order.
  if (v4) {
    // candidate and full queues in one launch
    const StagedShape sh = staged_shape(num_sms, rq.nseg, d);
    KM_CUDA_TRY(launch_pdl(refine_staged_kernel<true>, sh.blocks, 32 * RS_WARPS, sh.smem, s, X, C, Ct, d, k,
                           sh.span, st, rq, labels, mindist, true));
  } else {
    launch_refine_cands(false, num_sms, X, C, d, st, rq, labels, mindist, true, s);
    KM_CUDA_TRY(launch_pdl(refine_full_kernel, num_sms * 4, 256, 0, s, X, Ct, d, k, st, rq, labels, mindist, true));
  }
  KM_CUDA_TRY(cudaGetLastError());
  return KM_OK;
}

uint32_t f32_gather_terms(uint32_t d) {
  return std::min<uint32_t>(d, F32_GATHER_RUN) + (d + F32_GATHER_RUN - 1) / F32_GATHER_RUN;
}

km_status launch_refine_gemm(bool v4, int num_sms, const float* X, const float* C, const float* Ct,
                             const float* cn2, const float* xn2, uint64_t n, uint32_t d, uint32_t k,
                             TieBound tb32, DevState* st, const RefineQueues& rq,
                             const RefineQueues& rq2, uint32_t* fidx, uint32_t* nfull,
                             uint32_t* labels, float* mindist, cudaStream_t s) {
  launch_refine_cands(v4, num_sms, X, C, d, st, rq, labels, mindist, true, s);
  auto wide = [&](const RefineQueues& q, bool count) {
    if (v4)
      refine_wide_staged_kernel<<<num_sms * RS_BLOCKS_PER_SM, 32 * RS_WARPS,
                                  (size_t)RS_WARPS * RS_ROWS * rs_ld(std::min(d, RS_CH)) * sizeof(float), s>>>(
          X, C, d, st, q, labels, mindist, count);
    else refine_wide_kernel<<<num_sms * 8, 256, 0, s>>>(X, C, d, st, q, labels, mindist, count);
  };
  wide(rq, true);
  // rows of the full queue: FP32 distance pass over all k on those rows alone,
  // then the exact re-score of its own near ties
  KM_CUDA_TRY(cudaMemsetAsync(nfull, 0, sizeof(uint32_t), s));
  // the gather pass writes the counts of the segments its rows reach only:
  // every other segment of rq2 must read as empty
  KM_CUDA_TRY(cudaMemsetAsync(rq2.ccnt, 0, sizeof(uint32_t) * rq2.nseg, s));
  KM_CUDA_TRY(cudaMemsetAsync(rq2.fcnt, 0, sizeof(uint32_t) * rq2.nseg, s));
  KM_CUDA_TRY(cudaMemsetAsync(rq2.wcnt, 0, sizeof(uint32_t) * rq2.nseg, s));   // (rq's wide queue is done with)
  full_compact_kernel<<<num_sms * 4, 256, 0, s>>>(st, rq, fidx, nfull);
  launch_f32(X, C, cn2, xn2, n, d, k, tb32, st, labels, mindist, rq2, nullptr, fidx, nfull, s);
  launch_refine_cands(v4, num_sms, X, C, d, st, rq2, labels, mindist, false, s);
  wide(rq2, false);
  refine_full_kernel<<<num_sms * 4, 256, 0, s>>>(X, Ct, d, k, st, rq2, labels, mindist, false);
  KM_CUDA_TRY(cudaGetLastError());
  return KM_OK;
}

// ---------------------------------------------------------------------------
// (c) One-hot V as a stable label-sorted permutation.
// Segments of `seg` rows, one warp per segment.  seghist is cluster-major
// (k x nseg) so that each cluster's segment counts are contiguous.
// ---------------------------------------------------------------------------
__global__ void seg_hist_kernel(const uint32_t* __restrict__ labels, uint64_t n, uint32_t k,
                                uint32_t seg, uint32_t nseg, uint32_t* __restrict__ seghist,
                                DevState* st) {
  griddep_wait();
  if (st->done) return;
  extern __shared__ uint32_t sh_cnt[];
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wpb = blockDim.x >> 5;
  uint32_t* cnt = sh_cnt + (uint64_t)wib * k;
  const uint32_t s = blockIdx.x * wpb + wib;
  for (uint32_t c = lane; c < k; c += 32) cnt[c] = 0;
  __syncwarp();
  if (s < nseg) {
    const uint64_t r0 = (uint64_t)s * seg, r1 = min(n, r0 + seg);
    bool bad = false;
    for (uint64_t g = r0; g < r1; g += 32u * 32u) {
      uint32_t lv[32];
#pragma unroll
      for (int q = 0; q < 32; ++q) {
        const uint64_t r = g + (uint64_t)q * 32u + (uint64_t)lane;
        lv[q] = (r < r1) ? labels[r] : 0u;
      }
#pragma unroll
      for (int q = 0; q < 32; ++q) {
        if (g + (uint64_t)q * 32u + (uint64_t)lane >= r1) break;
        const uint32_t l = lv[q];
        if (l < k) atomicAdd(&cnt[l], 1u); else bad = true;
      }
    }
    if (bad) atomicOr(&st->err, KM_DEVERR_OVERFLOW);
    __syncwarp();
    for (uint32_t c = lane; c < k; c += 32) seghist[(uint64_t)c * nseg + s] = cnt[c];
  }
}

// Clusters of fewer rows are summed by a warp alone where most are small
// (launch_update_sums).
constexpr uint32_t SUMS_WARP_ROWS = 256;

// Exclusive scan of the k counts -> cstart[0..k] (CSR row pointers of V) by one
// block (any size up to 1024 threads); order (nullable): clusters by descending count,
// ties by index, if ranked and k <= 1024 (k^2 comparisons); else those of at least
// SUMS_WARP_ROWS rows first, each part by index.  Counts are read from L2 (other blocks may
// have written them in the same launch); null: scnt holds them, followed by zeros up to a
// multiple of 4 (k <= 1024).  sstart (nullable): cstart in shared memory as well.
__device__ void cluster_scan_block(const uint32_t* counts, uint32_t k, uint32_t* __restrict__ cstart,
                                   uint32_t* __restrict__ order, uint32_t* part, uint32_t* scnt,
                                   uint32_t* sstart = nullptr, bool ranked = true) {
  const bool cached = k <= 1024u;
  if (cached && counts) {
    for (uint32_t c = threadIdx.x; c < ((k + 3u) & ~3u); c += blockDim.x) scnt[c] = c < k ? __ldcg(counts + c) : 0u;
    __syncthreads();
  }
  if (order && cached && ranked) {
    // largest cluster first, so that the longest ordered sums start first
    for (uint32_t c = threadIdx.x; c < k; c += blockDim.x) {
      const uint32_t v = scnt[c];
      uint32_t rank = 0;
      for (uint32_t o = 0; o < k; o += 4) {          // the zeros after the last count precede nothing
        const uint4 w = *reinterpret_cast<const uint4*>(scnt + o);
        rank += (w.x > v || (w.x == v && o < c)) ? 1u : 0u;
        rank += (w.y > v || (w.y == v && o + 1 < c)) ? 1u : 0u;
        rank += (w.z > v || (w.z == v && o + 2 < c)) ? 1u : 0u;
        rank += (w.w > v || (w.w == v && o + 3 < c)) ? 1u : 0u;
      }
      order[rank] = c;
    }
  }
  auto count = [&](uint32_t i) { return cached ? scnt[i] : __ldcg(counts + i); };
  const uint32_t per = (k + blockDim.x - 1) / blockDim.x;
  const uint32_t b = threadIdx.x * per, e = min(k, b + per);
  uint32_t s = 0;
  for (uint32_t i = b; i < e; ++i) s += count(i);
  // exclusive block scan of s: warp shuffles, then the warp totals
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t x = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) part[wid] = x;
  __syncthreads();
  if (wid == 0) {
    const uint32_t nw = blockDim.x >> 5;
    uint32_t t = (uint32_t)lane < nw ? part[lane] : 0u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += y;
    }
    if ((uint32_t)lane < nw) part[lane] = t;       // inclusive warp totals
  }
  __syncthreads();
  uint32_t acc = x - s + (wid > 0 ? part[wid - 1] : 0u);
  for (uint32_t i = b; i < e; ++i) {
    cstart[i] = acc;
    if (sstart) sstart[i] = acc;
    acc += count(i);
  }
  if (e == k && b < e) cstart[k] = acc;
  if (k == 0 && threadIdx.x == 0) cstart[0] = 0;
  if (order && !(cached && ranked)) {
    uint32_t large = 0;
    for (uint32_t i = b; i < e; ++i) large += count(i) >= SUMS_WARP_ROWS ? 1u : 0u;
    __syncthreads();                                 // part has been read
    if (threadIdx.x < 32u) part[threadIdx.x] = 0u;
    __syncthreads();
    uint32_t y = large;                              // inclusive over the warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t z = __shfl_up_sync(0xffffffffu, y, o);
      if (lane >= o) y += z;
    }
    if (lane == 31) part[wid] = y;
    __syncthreads();
    uint32_t before = 0, all = 0;
    for (uint32_t w = 0; w < 32u; ++w) {
      if ((int)w < wid) before += part[w];
      all += part[w];
    }
    before += y - large;                             // large clusters before b
    for (uint32_t i = b; i < e; ++i) {
      if (count(i) >= SUMS_WARP_ROWS) order[before++] = i;
      else order[all + i - before] = i;
    }
  }
}

// One warp per cluster: exclusive scan over its segments, total -> counts.
// With cstart, the block that finishes last (a ticket in DevState) then runs
// the cluster scan, which saves a dependent launch.  At most 512 threads per
// block (80 registers a thread); 128 for k <= 256, which spreads the warps' shuffles,
// which bound it, over the SMs (beyond, the last block's ranks take longer than that
// saves): k = 64, 196 -> 782 segments 7.4 -> 6.7 us, k = 10 6.1 -> 4.1.
__global__ void __launch_bounds__(512) seg_scan_kernel(uint32_t* __restrict__ seghist, uint32_t k, uint32_t nseg,
                                uint32_t* __restrict__ counts, DevState* st, uint32_t* __restrict__ cstart,
                                uint32_t* __restrict__ order) {
  griddep_wait();
  if (st->done) return;
  const uint32_t c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (c < k) {
    uint32_t* h = seghist + (uint64_t)c * nseg;
    uint32_t carry = 0;
    // groups of 32 coalesced chunks: every load of a group is issued before the
    // scans that use them
    for (uint32_t g = 0; g < nseg; g += 32u * 32u) {
      uint32_t v[32];
#pragma unroll
      for (int q = 0; q < 32; ++q) {
        const uint32_t i = g + (uint32_t)q * 32u + (uint32_t)lane;
        v[q] = (i < nseg) ? h[i] : 0u;
      }
#pragma unroll
      for (int q0 = 0; q0 < 32; q0 += 8) {      // eight chunks' scans interleave
        if (g + (uint32_t)q0 * 32u >= nseg) break;
#pragma unroll
        for (int q = q0; q < q0 + 8; ++q) {
          const uint32_t i = g + (uint32_t)q * 32u + (uint32_t)lane;
          uint32_t x = v[q];
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
          }
          if (i < nseg) h[i] = carry + x - v[q];
          carry += __shfl_sync(0xffffffffu, x, 31);
        }
      }
    }
    if (lane == 0) counts[c] = carry;
  }
  if (!cstart) return;
  __shared__ uint32_t part[32];
  __shared__ __align__(16) uint32_t scnt[1024];
  __shared__ int is_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) is_last = (atomicAdd(&st->scan_ticket, 1u) == gridDim.x - 1u) ? 1 : 0;
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  cluster_scan_block(counts, k, cstart, order, part, scnt);
  if (threadIdx.x == 0) reinterpret_cast<volatile DevState*>(st)->scan_ticket = 0u;
}

// Single block: cluster_scan_block as a kernel of its own, its order not ranked (for k =
// 1000 the ranks alone take one block 25 us).
__global__ void cluster_scan_kernel(const uint32_t* __restrict__ counts, uint32_t k,
                                    uint32_t* __restrict__ cstart, DevState* st,
                                    uint32_t* __restrict__ order) {
  griddep_wait();
  if (st->done) return;
  __shared__ uint32_t part[32];
  __shared__ __align__(16) uint32_t scnt[1024];
  cluster_scan_block(counts, k, cstart, order, part, scnt, nullptr, false);
}

// One warp per segment: stable scatter of row ids into perm.
__global__ void seg_scatter_kernel(const uint32_t* __restrict__ labels, uint64_t n, uint32_t k,
                                   uint32_t seg, uint32_t nseg, const uint32_t* __restrict__ seghist,
                                   const uint32_t* __restrict__ cstart,
                                   uint32_t* __restrict__ perm, DevState* st) {
  griddep_wait();
  if (st->done) return;
  extern __shared__ uint32_t sh_pos[];
  const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wpb = blockDim.x >> 5;
  uint32_t* pos = sh_pos + (uint64_t)wib * k;
  const uint32_t s = blockIdx.x * wpb + wib;
  if (s >= nseg) return;
  for (uint32_t c = lane; c < k; c += 32) pos[c] = cstart[c] + seghist[(uint64_t)c * nseg + s];
  __syncwarp();
  const uint64_t r0 = (uint64_t)s * seg, r1 = min(n, r0 + seg);
  // labels of up to 32 chunks into registers first (one load latency per group)
  for (uint64_t g = r0; g < r1; g += 32u * 32u) {
   uint32_t lv[32];
#pragma unroll
   for (int q = 0; q < 32; ++q) {
     const uint64_t r = g + (uint64_t)q * 32u + (uint64_t)lane;
     lv[q] = (r < r1) ? labels[r] : 0xffffffffu;
   }
#pragma unroll
   for (int q = 0; q < 32; ++q) {
    const uint64_t rb = g + (uint64_t)q * 32u;
    if (rb >= r1) break;
    const uint64_t r = rb + lane;
    const bool valid = r < r1;
    const uint32_t l = lv[q];
    const bool ok = valid && l < k;
    const unsigned m = __match_any_sync(0xffffffffu, ok ? l : 0xffffffffu);
    const uint32_t rank = __popc(m & ((1u << lane) - 1u));
    uint32_t base = ok ? pos[l] : 0u;
    __syncwarp();
    if (ok) {
      perm[base + rank] = (uint32_t)r;
      if (rank == 0) pos[l] = base + __popc(m);
    }
    __syncwarp();
   }
  }
}

// The whole sort by one block of 32 warps, up to ONE_BLOCK_ROWS rows and 256 clusters: a
// warp takes consecutive rows, 32 a step, and keeps each row's rank among the warp's rows
// of its cluster; the warps' counts are scanned per cluster, then over the clusters.
// Bound by latency, as the three kernels above are, without two launches between them:
// the sort of an iteration at n = 4096 / 4100 (one block / three kernels) is 10.2 / 14.1 us
// with k = 10, 14.2 / 16.2 with 100 and 16.5 / 19.5 with 256; at 8192 12.3 / 13.8 with 10
// and 22.8 / 22.2 with 256, at 16,384 16.5 / 14.2 and 34.8 / 20.2.
constexpr uint32_t OB_STEPS = ONE_BLOCK_ROWS / 1024;
__global__ void __launch_bounds__(1024)
one_block_sort_kernel(const uint32_t* __restrict__ labels, uint32_t n, uint32_t k, uint32_t* __restrict__ counts,
                      uint32_t* __restrict__ cstart, uint32_t* __restrict__ order, uint32_t* __restrict__ perm,
                      DevState* st) {
  griddep_wait();
  if (st->done) return;
  extern __shared__ uint32_t ob_cnt[];                     // [32 warps][k]
  __shared__ uint32_t part[32];
  __shared__ __align__(16) uint32_t scnt[256];
  __shared__ uint32_t sstart[256];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t steps = (n + 1023u) / 1024u, r0 = (uint32_t)warp * steps * 32u + (uint32_t)lane;
  uint32_t lv[OB_STEPS], rank[OB_STEPS];
#pragma unroll
  for (uint32_t q = 0; q < OB_STEPS; ++q) {
    const uint32_t r = r0 + q * 32u;
    lv[q] = q < steps && r < n ? labels[r] : 0xffffffffu;
  }
  for (uint32_t i = threadIdx.x; i < 32u * k; i += 1024u) ob_cnt[i] = 0u;
  __syncthreads();
  uint32_t* const cnt = ob_cnt + (uint32_t)warp * k;
  bool bad = false;
#pragma unroll
  for (uint32_t q = 0; q < OB_STEPS; ++q) {
    if (q >= steps) break;
    const uint32_t l = lv[q];
    const bool ok = l < k;
    if (!ok && r0 + q * 32u < n) bad = true;
    const unsigned m = __match_any_sync(0xffffffffu, ok ? l : 0xffffffffu);
    const uint32_t before = ok ? cnt[l] : 0u;
    rank[q] = before + (uint32_t)__popc(m & ((1u << lane) - 1u));
    __syncwarp();
    if (ok && (m >> lane) == 1u) cnt[l] = before + (uint32_t)__popc(m);     // the highest lane of the cluster
    __syncwarp();
  }
  if (bad) atomicOr(&st->err, KM_DEVERR_OVERFLOW);
  __syncthreads();
  if (threadIdx.x < 256u) {                                // exclusive over the warps, per cluster
    const uint32_t c = threadIdx.x;
    uint32_t run = 0;
    if (c < k) {
      uint32_t v[32];
#pragma unroll
      for (int w = 0; w < 32; ++w) v[w] = ob_cnt[(uint32_t)w * k + c];
#pragma unroll
      for (int w = 0; w < 32; ++w) { ob_cnt[(uint32_t)w * k + c] = run; run += v[w]; }
      counts[c] = run;
    }
    scnt[c] = run;
  }
  __syncthreads();
  cluster_scan_block(nullptr, k, cstart, order, part, scnt, sstart);
  __syncthreads();
#pragma unroll
  for (uint32_t q = 0; q < OB_STEPS; ++q) {
    if (q >= steps) break;
    const uint32_t l = lv[q];
    if (l < k) perm[sstart[l] + cnt[l] + rank[q]] = r0 + q * 32u;
  }
}

// ---------------------------------------------------------------------------
// (c) Exact centroid update V.X: the cluster's rows are visited in ascending
// index order (the label-sorted permutation) and every column is summed in
// float exactly as the reference's CPU loop (kmeans.cpp:133-137).  Also: the
// squared move per element for the shift test and the objective of this
// iteration's assignment against the centroids that produced it.
//
// One CTA per (cluster, 32-column block), so a cluster's d/32 column chains run
// on as many SMs.  Producer warp p of blk_producers(VEC) fills batches
// p, p + PROD, ... with VEC-column cp.async per lane into a BLK_STAGES-deep ring;
// arrival on the stage's mbarrier fires when its copies land
// (cp.async.mbarrier.arrive.noinc).  VEC is the widest copy that the row starts
// allow (4, 2 or 1 columns: 16, 8 or 4 bytes); the ring and the consumers are the
// same.  Two consumer warps: one holds the ordered chain alone, one the
// objective.
//
// Bounds: the chain of the largest cluster, then HBM.  A dependent FP32 addition
// takes 4.1 cycles and 4.6 with a shared-memory load beside it (5.6 when the loads
// stand in front of the additions), so the chain warp does nothing else; the
// objective warp takes 16-byte loads and packed FP32 pairs, a third of the
// instructions of one load and two operations a row.  Measured: a cluster alone
// 177 -> 322 rows/us (39 -> 263 / 173 for 8- / 4-byte rows, which one warp per 32
// columns gathered and summed before), n = 1M d = 128 k = 256 with 20,473 rows in
// the largest cluster 135 -> 105 us = 5.16 TB/s, n = 300,007 d = 50 k = 37
// 447 -> 72 us.  TMA row gathers (tile::gather4) were slower: 119 rows/us.
//
// Every wait is bounded; on timeout the CTA flags KM_DEVERR_TIMEOUT and drains
// its copies before exiting.  A batch is BLK_ROWS = 128 rows (four groups of 32):
// every batch costs a consumer one wait and one release of fixed latency.
// ---------------------------------------------------------------------------
namespace {
// Producer warps by copy width: narrower copies take two or four times the
// instructions, so six warps issue them.  Measured, one cluster of 100,000 rows:
// 16 bytes 322 rows/us with two, three or six producers (the chain's rate), 8
// bytes 212 with three and 263 with six, 4 bytes 113 and 173.
constexpr int blk_producers(int vec) { return vec == 4 ? 3 : 6; }
constexpr int blk_threads(int vec) { return 32 * (blk_producers(vec) + 2); }
}  // namespace

template <int VEC>
__global__ void __launch_bounds__(blk_threads(VEC))
update_sums_bulk_kernel(const float* __restrict__ X, const uint32_t* __restrict__ perm,
                        const uint32_t* __restrict__ cstart, uint32_t d, uint32_t k,
                        const float* __restrict__ C, float* __restrict__ Cn,
                        float* __restrict__ dsq, double* __restrict__ objpart, DevState* st,
                        const uint32_t* __restrict__ order, uint32_t min_rows) {
  constexpr int PROD = blk_producers(VEC);
  griddep_wait();
  if (st && st->done) return;
  extern __shared__ __align__(128) float ring[];        // [BLK_STAGES][BLK_ROWS][BLK_COLS]
  __shared__ __align__(8) uint64_t full[BLK_STAGES], empty[BLK_STAGES];
  __shared__ int abort_flag;
  const uint32_t nblk = (d + BLK_COLS - 1) / BLK_COLS;
  // with an order, CTAs take the largest clusters first (they are scheduled in
  // index order), so that the longest ordered sums start first
  const uint32_t c = order ? order[blockIdx.x / nblk] : blockIdx.x / nblk;
  const uint32_t j0 = (blockIdx.x % nblk) * BLK_COLS;
  const uint32_t w = min((uint32_t)BLK_COLS, d - j0);   // columns of this block
  const uint32_t s0 = cstart[c], s1 = cstart[c + 1];
  if (s1 - s0 < min_rows) return;                       // update_sums_warp_kernel's
  const uint32_t nb = (s1 - s0 + BLK_ROWS - 1) / BLK_ROWS;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < BLK_STAGES; ++s) { mbar_init(&full[s], 32); mbar_init(&empty[s], objpart ? 2 : 1); }
    abort_flag = 0;
    mbar_fence_init();
  }
  __syncthreads();
  volatile int* ab = &abort_flag;
  auto fail = [&]() {
    abort_flag = 1;
    if (st) atomicOr(&st->err, KM_DEVERR_TIMEOUT);
  };

  const SumsRing R{ring, full, empty, ab};
  if (warp < PROD) {
    if (!sums_produce<VEC, PROD>(R, X + j0, perm + s0, s1 - s0, d, w, 0u, (uint32_t)warp) && lane == 0) fail();
    // Drain: this warp's copies must land before the CTA exits.
    asm volatile("cp.async.wait_all;" ::: "memory");
    return;
  }

  if (warp == PROD) {
    float sum;
    if (!sums_chain(R, s1 - s0, 0u, sum)) { if (lane == 0) fail(); return; }
    if ((uint32_t)lane < w) {
      const uint64_t p = (uint64_t)c * d + j0 + (uint32_t)lane;
      const uint32_t cnt = s1 - s0;
      const float scale = __double2float_rn(1.0 / (double)(cnt > 1 ? cnt : 1));
      const float cn = __fmul_rn(sum, scale);
      Cn[p] = cn;
      if (dsq) {
        const float t = __fsub_rn(cn, C ? C[p] : 0.0f);
        dsq[p] = __fmul_rn(t, t);
      }
    }
  } else if (objpart) {
    // The objective: lane l on columns 4 (l % 8) .. + 3 of every fourth row
    // (rows l / 8, + 4, ...), 16 bytes a load.  Per batch a lane sums its 32
    // rows in FP32, two runs of 16 (the length of a run sets the error of the
    // whole sum), and the runs as an unevaluated sum of FP32 parts (TwoSum; FP64
    // additions are slow on this GPU).  Two parts hold 48 bits; rows that are not
    // 16-byte aligned take three, whose sum holds no less than an FP64 one (n =
    // 300,007 d = 50 k = 37, 10 iterations: 1555 -> 1581 us for the third).
    const uint32_t c4 = ((uint32_t)lane & 7u) * 4u, r0 = (uint32_t)lane >> 3;
    const uint64_t p = (uint64_t)c * d + j0 + c4;
    float cold[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) cold[q] = (C && c4 + q < w) ? C[p + q] : 0.0f;
    const float2 ma = make_float2(-cold[0], -cold[1]), mb = make_float2(-cold[2], -cold[3]);
    // parts h + l (+ g) of columns 0,1 (a) and 2,3 (b)
    float2 ha = make_float2(0.0f, 0.0f), la = ha, ga = ha, hb = ha, lb = ha, gb = ha;
    auto neg = [](float2 v) { return make_float2(-v.x, -v.y); };
    // TwoSum: h <- the rounded h + v; returns the rounding error
    auto two_sum = [&](float2& h, float2 v) {
      const float2 s_ = __fadd2_rn(h, v), bb = __fadd2_rn(s_, neg(h));
      const float2 err = __fadd2_rn(__fadd2_rn(h, neg(__fadd2_rn(s_, neg(bb)))), __fadd2_rn(v, neg(bb)));
      h = s_;
      return err;
    };
    auto sum_add = [&](float2& h, float2& l, float2& g, float2 v) {
      const float2 e = two_sum(h, v);
      if constexpr (VEC == 4) l = __fadd2_rn(l, e);
      else g = __fadd2_rn(g, two_sum(l, e));
    };
    for (uint32_t b = 0; b < nb; ++b) {
      const uint32_t s = b % BLK_STAGES, ph = (b / BLK_STAGES) & 1u;
      const bool ok = mbar_wait_bounded(&full[s], ph, ab, BLK_WAIT_NS, BLK_SUSPEND_NS);
      if (!__all_sync(0xffffffffu, ok)) { if (lane == 0) fail(); return; }
      const uint32_t m = min((uint32_t)BLK_ROWS, s1 - (s0 + b * BLK_ROWS));
      const float4* src = reinterpret_cast<const float4*>(ring + ((size_t)s * BLK_ROWS + r0) * BLK_COLS + c4);
      float2 ea = make_float2(0.0f, 0.0f), eb = ea, fa = ea, fb = ea;
      auto add = [&](const float4 v, float2& ea, float2& eb) {
        const float2 ta = __fadd2_rn(make_float2(v.x, v.y), ma), tb = __fadd2_rn(make_float2(v.z, v.w), mb);
        ea = __ffma2_rn(ta, ta, ea);
        eb = __ffma2_rn(tb, tb, eb);
      };
      if (m == (uint32_t)BLK_ROWS) {
#pragma unroll
        for (int u0 = 0; u0 < BLK_ROWS / 4; u0 += 8) {
          float4 v[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) v[u] = src[(u0 + u) * BLK_COLS];
#pragma unroll
          for (int u = 0; u < 8; ++u) add(v[u], u & 1 ? fa : ea, u & 1 ? fb : eb);
        }
      } else {
        for (uint32_t u = 0; r0 + 4u * u < m; u += 2u) {
          add(src[u * BLK_COLS], ea, eb);
          if (r0 + 4u * u + 4u < m) add(src[(u + 1u) * BLK_COLS], fa, fb);
        }
      }
      sum_add(ha, la, ga, ea);
      sum_add(hb, lb, gb, eb);
      sum_add(ha, la, ga, fa);
      sum_add(hb, lb, gb, fb);
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[s]);
    }
    double o[4] = {(double)ha.x + ((double)la.x + (double)ga.x), (double)ha.y + ((double)la.y + (double)ga.y),
                   (double)hb.x + ((double)lb.x + (double)gb.x), (double)hb.y + ((double)lb.y + (double)gb.y)};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      o[q] += __shfl_xor_sync(0xffffffffu, o[q], 8);
      o[q] += __shfl_xor_sync(0xffffffffu, o[q], 16);
      if (r0 == 0u && c4 + q < w) objpart[p + q] = o[q];
    }
  }
}

// The same for clusters of fewer than max_rows rows: a warp per (cluster, 32 columns), which
// copies its rows 32 at a time into SW_STAGES buffers of its own and adds them, lane =
// column.  Rows past the cluster's end zero-fill (adding +0); the objective in FP32 runs of
// 16 rows, added in FP64.  Bound by latency (four loads one after the other before the
// first addition), so by the warps an SM holds: sixteen, where the ring holds two
// clusters whatever their sizes (launch_update_sums has both sides' times; with the rows in
// registers, a batch ahead, this took two to five times as long).
constexpr int SW_WARPS = 4, SW_STAGES = 3;
constexpr size_t SW_SMEM = sizeof(float) * SW_WARPS * SW_STAGES * 32 * 32;
template <int VEC>
__global__ void __launch_bounds__(32 * SW_WARPS)
update_sums_warp_kernel(const float* __restrict__ X, const uint32_t* __restrict__ perm,
                        const uint32_t* __restrict__ cstart, uint32_t d, uint32_t k, const float* __restrict__ C,
                        float* __restrict__ Cn, float* __restrict__ dsq, double* __restrict__ objpart, DevState* st,
                        uint32_t max_rows) {
  griddep_wait();
  if (st && st->done) return;
  extern __shared__ __align__(128) float ring[];        // [SW_WARPS][SW_STAGES][32 rows][32 columns]
  const uint32_t nblk = (d + BLK_COLS - 1) / BLK_COLS;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t task = (uint64_t)blockIdx.x * SW_WARPS + warp;
  if (task >= (uint64_t)k * nblk) return;
  const uint32_t c = (uint32_t)(task / nblk), j0 = (uint32_t)(task % nblk) * BLK_COLS;
  const uint32_t s0 = cstart[c], cnt = cstart[c + 1] - s0;
  if (cnt >= max_rows) return;
  const bool in = j0 + (uint32_t)lane < d;
  const uint64_t p = (uint64_t)c * d + j0 + (uint32_t)lane;
  const float cold = in && C ? C[p] : 0.0f;
  float* const buf = ring + (size_t)warp * SW_STAGES * 32 * 32;
  constexpr uint32_t LPR = 32 / VEC, RPI = VEC;          // lanes per row, rows per copy instruction
  const uint32_t sub = (uint32_t)lane / LPR, cv = ((uint32_t)lane % LPR) * VEC;
  const bool has_cols = j0 + cv < d;
  const float* const x = X + j0 + cv;
  const uint32_t nb = (cnt + 31u) / 32u;
  auto index = [&](uint32_t b) { return 32u * b + (uint32_t)lane < cnt ? perm[s0 + 32u * b + lane] : 0u; };
  auto issue = [&](uint32_t b, uint32_t idx) {           // (a group of copies every time, empty past the end)
    if (b < nb) {
      float* dst = buf + (b % SW_STAGES) * 32 * 32 + sub * 32 + cv;
#pragma unroll
      for (uint32_t i = 0; i < 32u / RPI; ++i) {
        const uint32_t u = i * RPI + sub, r = __shfl_sync(0xffffffffu, idx, (int)u);
        const bool ok = 32u * b + u < cnt && has_cols;
        cp_async_cols<VEC>(dst + i * RPI * 32, ok ? x + (uint64_t)r * d : X, ok);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float sum = 0.0f;
  double obj = 0.0;
  uint32_t idx = index(0), ahead = index(1);
  issue(0, idx);
  idx = index(2);
  issue(1, ahead);
  for (uint32_t b = 0; b < nb; ++b) {
    ahead = index(b + 3u);
    issue(b + 2u, idx);
    idx = ahead;
    asm volatile("cp.async.wait_group %0;" ::"n"(SW_STAGES - 1) : "memory");
    __syncwarp();
    const float* src = buf + (b % SW_STAGES) * 32 * 32 + lane;
    const uint32_t m = min(32u, cnt - 32u * b);
    float v[32];
#pragma unroll
    for (uint32_t u = 0; u < 32u; ++u) v[u] = src[u * 32];
#pragma unroll
    for (uint32_t u = 0; u < 32u; ++u) sum = __fadd_rn(sum, v[u]);
    if (objpart) {
      float e[2] = {0.0f, 0.0f};
#pragma unroll
      for (uint32_t u = 0; u < 32u; ++u) {
        const float t = u < m ? __fsub_rn(v[u], cold) : 0.0f;
        e[u >> 4] = fmaf(t, t, e[u >> 4]);
      }
      obj += (double)e[0];
      obj += (double)e[1];
    }
    __syncwarp();                                        // the stage is filled again in the next step
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  if (!in) return;
  const float cn = __fmul_rn(sum, __double2float_rn(1.0 / (double)(cnt > 1u ? cnt : 1u)));
  Cn[p] = cn;
  if (dsq) {
    const float t = __fsub_rn(cn, cold);
    dsq[p] = __fmul_rn(t, t);
  }
  if (objpart) objpart[p] = obj;
}

// Opt-in shared memory for the ring; called before any capture.
km_status update_sums_prepare() {
  for (auto kern : {update_sums_bulk_kernel<4>, update_sums_bulk_kernel<2>, update_sums_bulk_kernel<1>})
    KM_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BLK_SMEM));
  return KM_OK;
}

// Rows are copied in the widest pieces whose alignment every row start has
// (row stride d floats from X): 16 bytes, else 8, else 4.  Many clusters of few rows go to
// a warp each, and the ring takes those above: at most n / SUMS_WARP_ROWS of them, which
// order lists first.  The ring takes two clusters' column blocks an SM at a time, of 2 us and
// more each, so it loses as soon as there are more than three waves of them; narrower
// copies cost it more, so that it loses earlier there.  Ring / a warp each: 16-byte rows, n = 160,000 d = 256 k = 20,000 1191 / 191 us, n = 63,500 d = 16 k = 500
// 12 / 17, n = 400,000 d = 64 k = 2000 (200 a cluster) 60 / 65; 4-byte rows, n = 4M d = 7
// k = 20,000 441 / 166, n = 200,000 d = 7 k = 1000 30 / 21, n = 15,000 d = 7 k = 500 16.8 / 10.0, n = 38,100 d = 50
// k = 300 14.6 / 18.2, n = 3000 d = 7 k = 100 12 / 10, n = 6000 d = 50 k = 100 10.1 / 12.2; 8-byte ones, n = 200,000
// d = 50 k = 500 26.9 / 35.5, n = 200,000 d = 50 k = 4000 94 / 30.
km_status launch_update_sums(const float* X, const uint32_t* perm, const uint32_t* cstart, uint64_t n, uint32_t d,
                             uint32_t k, const float* C, float* Cn, float* dsq, double* objpart,
                             DevState* st, cudaStream_t s, const uint32_t* order) {
  const uintptr_t xa = reinterpret_cast<uintptr_t>(X);
  const int vec = (d % 4 == 0 && xa % 16 == 0) ? 4 : (d % 2 == 0 && xa % 8 == 0) ? 2 : 1;
  auto kern = vec == 4 ? update_sums_bulk_kernel<4> : vec == 2 ? update_sums_bulk_kernel<2> : update_sums_bulk_kernel<1>;
  const uint32_t nblk = (d + BLK_COLS - 1) / BLK_COLS;
  const uint64_t blocks = (uint64_t)k * nblk;
  const uint64_t rows = vec == 4 ? (blocks >= 1000u ? 128u : 0u)
                        : blocks >= (vec == 2 ? 2000u : 1000u) ? 1024u
                        : blocks >= 1000u ? 128u : blocks >= 256u ? 64u : 32u;
  const bool few = order && n < k * rows;
  const uint32_t limit = !few ? 0u : vec == 4 ? SUMS_WARP_ROWS : 4u * SUMS_WARP_ROWS;
  if (few) {
    auto small = vec == 4 ? update_sums_warp_kernel<4> : vec == 2 ? update_sums_warp_kernel<2> : update_sums_warp_kernel<1>;
    KM_CUDA_TRY(launch_pdl(small, (unsigned)(((uint64_t)k * nblk + SW_WARPS - 1) / SW_WARPS), 32 * SW_WARPS, SW_SMEM, s, X,
                           perm, cstart, d, k, C, Cn, dsq, objpart, st, limit));
  }
  const uint64_t ctas = (few ? std::min<uint64_t>(k, n / SUMS_WARP_ROWS) : (uint64_t)k) * nblk;
  if (ctas)
    KM_CUDA_TRY(launch_pdl(kern, (unsigned)ctas, blk_threads(vec), BLK_SMEM, s, X, perm, cstart, d, k, C, Cn, dsq, objpart,
                           st, order, limit));
  KM_CUDA_TRY(cudaGetLastError());
  return KM_OK;
}

// One warp per cluster: reference shift test (float sum over j ascending, then
// sqrtf(s) > tol, kmeans.cpp:190-200), FP64 move, FP64 objective of the
// cluster, new ||c||^2 and BF16 copies; then C <- Cn.  The block that finishes
// last (a ticket in DevState) then ends the iteration: deterministic
// reductions over the clusters, the stop decision, counters for the next
// iteration.  Bound by latency and by the FP64 units (two lanes a cycle and SM, so eight
// warps' 40 operations each were 3 us): two warps a block up to 512 clusters (beyond,
// the last block's sums would take longer), maxima of squares with one root at the end.
// d = 64 k = 10 8.4 -> 5.8 us, d = 100 k = 64 11.1 -> 7.8, d = 128 k = 256 9.1 -> 8.1.
__global__ void __launch_bounds__(256)
finalize_kernel(const float* __restrict__ Cn, float* __restrict__ C,
                const float* __restrict__ dsq, const double* __restrict__ objpart,
                const uint32_t* __restrict__ counts, int32_t empty_excl,
                uint32_t d, uint32_t dp, uint32_t k, float tol,
                float* __restrict__ cn2, __nv_bfloat16* __restrict__ Cb,
                __nv_bfloat16* __restrict__ Clo, float* __restrict__ Ct,
                double* __restrict__ move2_c, double* __restrict__ obj_c,
                DevState* st, LoopConsts lc) {
  griddep_wait();
  if (st->done) return;
  __shared__ double s_obj[8];
  __shared__ double s_mv[8];
  __shared__ float s_cm[8];
  __shared__ int is_last;
  const uint32_t c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (c < k) {
    const uint64_t base = (uint64_t)c * d;
    // Reference GPU rule (src/kernels/distances.cu:588-599): an empty cluster's
    // distance is +inf from then on, so it is never chosen again.  Its norm and
    // its column of Ct become +inf; its (zero) centroid row stays finite.
    const bool excl = empty_excl && counts[c] == 0u;
    double nrm = 0.0, mv = 0.0, ob = 0.0;
    float s = 0.0f;   // reference shift test: float sum of dsq over j ascending
    // 128 columns per pass, j = j0 + lane + 32 q: all of the pass's loads are
    // issued before its arithmetic; the ordered float sum takes the terms from
    // the lanes by shuffle (j ascending), the FP64 sums keep each lane's order.
    for (uint32_t j0 = 0; j0 < dp; j0 += 128) {
      float v[4], co[4], dq[4];
      double op[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t j = j0 + (uint32_t)lane + 32u * q;
        const bool in = j < d;
        v[q] = in ? Cn[base + j] : 0.0f;
        co[q] = in ? C[base + j] : 0.0f;
        dq[q] = in ? dsq[base + j] : 0.0f;
        op[q] = in ? objpart[base + j] : 0.0;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t j = j0 + (uint32_t)lane + 32u * q;
        if (j < d) {
          nrm += (double)v[q] * v[q];
          const double t = (double)v[q] - (double)co[q];
          mv += t * t;
          ob += op[q];
          Ct[(uint64_t)j * k + c] = excl ? f_inf() : v[q];
          C[base + j] = v[q];
        }
        if (Cb && j < dp) {
          const __nv_bfloat16 hi = __float2bfloat16_rn(v[q]);
          Cb[(uint64_t)c * dp + j] = hi;
          if (Clo) Clo[(uint64_t)c * dp + j] = __float2bfloat16_rn(v[q] - __bfloat162float(hi));
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t jq = j0 + 32u * q;
        if (jq >= d) break;
#pragma unroll
        for (int l = 0; l < 32; ++l) {
          const float tq = __shfl_sync(0xffffffffu, dq[q], l);
          if (jq + (uint32_t)l < d) s = __fadd_rn(s, tq);
        }
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      nrm += __shfl_xor_sync(0xffffffffu, nrm, o);
      mv += __shfl_xor_sync(0xffffffffu, mv, o);
      ob += __shfl_xor_sync(0xffffffffu, ob, o);
    }
    if (lane == 0) {
      if (sqrtf(s) > tol) st->moved = 1u;
      cn2[c] = excl ? f_inf() : (float)nrm;
      move2_c[c] = mv;
      obj_c[c] = ob;
    }
  }
  // ---- last block: end of iteration ----
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) is_last = (atomicAdd(&st->fin_ticket, 1u) == gridDim.x - 1u) ? 1 : 0;
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  // other blocks' results: read past L1 (this SM may hold stale lines)
  volatile DevState* vs = st;
  double ob = 0.0, mv2 = 0.0;
  float cm = 0.0f;                               // largest squared norm
  for (uint32_t cc = threadIdx.x; cc < k; cc += blockDim.x) {
    ob += __ldcg(obj_c + cc);
    mv2 = fmax(mv2, __ldcg(move2_c + cc));
    const float v = __ldcg(cn2 + cc);
    if (v < f_inf()) cm = fmaxf(cm, v);          // excluded (empty) clusters hold +inf
  }
  for (int o = 16; o > 0; o >>= 1) {
    ob += __shfl_xor_sync(0xffffffffu, ob, o);
    mv2 = fmax(mv2, __shfl_xor_sync(0xffffffffu, mv2, o));
    cm = fmaxf(cm, __shfl_xor_sync(0xffffffffu, cm, o));
  }
  if (lane == 0) { s_obj[threadIdx.x >> 5] = ob; s_mv[threadIdx.x >> 5] = mv2; s_cm[threadIdx.x >> 5] = cm; }
  __syncthreads();
  if (threadIdx.x == 0) {
    const uint32_t it = vs->iter + 1;
    vs->iter = it;
    ob = s_obj[0]; mv2 = s_mv[0]; cm = s_cm[0];
    for (uint32_t w = 1; w < (blockDim.x >> 5); ++w) {
      ob += s_obj[w];
      mv2 = fmax(mv2, s_mv[w]);
      cm = fmaxf(cm, s_cm[w]);
    }
    vs->objective = ob;
    vs->max_move2 = mv2;
    vs->cmax = sqrtf(cm) * 1.000001f;
    const double score = ob - vs->sum_x2;
    vs->score = score;
    bool stop = false;
    if (lc.conv == KM_CONV_SHIFT) {
      if (it > 1 && vs->moved == 0u) { vs->converged_iter = it; stop = true; }
    } else if (lc.conv == KM_CONV_SCORE) {
      if (it < lc.maxiter && it > 1 && fabs(score - vs->last_score) < (double)lc.tol) {
        vs->converged_iter = it; stop = true;
      }
      vs->last_score = score;
    }
    vs->moved = 0u;
    if (it >= lc.maxiter) stop = true;
    if (stop) vs->done = 1u;
    vs->fin_ticket = 0u;
  }
}

}  // namespace km
