// Batched Lloyd k-means: many independent problems of uneven n, d, k, each
// with several seeded restarts, advanced together.
//
// Every restart of every problem is an "instance" and runs the reference CPU
// algorithm to its own end; all instances still running take an iteration in the
// same few launches, whose work items are cut from the instances so that one
// large instance spreads over the whole GPU (one CTA per instance instead left
// the GPU waiting for the largest ones: 64 problems x 4 restarts, n 1024..65536,
// 776 ms, now 83 ms; batches of small instances only keep that form,
// batch_small_kernel):
//   assign   a tile of rows against all centroids of its instance; distances by
//            the CPU formula sum_j fl((x_j - c_j)^2) in column order (exact, no
//            bound or refinement needed), strict '<' over centroids in ascending
//            order (comparisons/CPU_Kmeans/src/kmeans.cpp:86-129);
//   sort     a CTA per instance: stable counting sort of the rows by label;
//   update   a task per (instance, cluster, 32 columns): sum of the cluster's rows
//            in row order, then scale by float(1/(double)max(count,1))
//            (kmeans.cpp:131-155);
//   stop     a CTA per instance: from the second iteration, every centroid moved
//            <= tol (float sqrt of the column-ordered sum of squares,
//            kmeans.cpp:170-200); the CTA that finishes last lists the instances
//            that go on and cuts their work into items.
// Initial centroids are the reference's seeded sample picks, drawn on the host
// (std::mt19937 as the reference does).
#include "km_lloyd.cuh"
#include "km_sums.cuh"

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <random>
#include <type_traits>
#include <vector>

namespace km {

struct BatchInst {
  uint64_t xoff;      // floats: first coordinate of the problem's points
  uint64_t loff;      // uint32: first label (and sorted row) of this instance
  uint64_t coff;      // floats: first centroid value of this instance (k*d)
  uint64_t toff;      // doubles: first objective of 32 rows of this instance
  uint32_t n, d, k;
  uint32_t prob, restart;
};

struct BatchOut {
  uint64_t converged_iter;
  uint64_t iterations;
  double objective;   // FP64 sum of the final assignment's (FP32 CPU-formula) distances
};

// One ordered sum: 32 columns (w of them in use) of one cluster of one instance.
struct BatchTask {
  const float* x;             // first column of the problem's first row
  const uint32_t* perm;       // the cluster's rows, ascending
  float* out;                 // next centroid, same columns
  uint32_t cnt, d, w, vec;    // rows, row stride, columns, columns per copy (4, 2 or 1)
};

// Loop state on the device: the instances still running (act, in descending
// work), the first assign tile of each, the update tasks of this iteration, and
// the counters that hand tiles and tasks out.
struct BatchCtl {
  unsigned long long iter;    // iterations done
  uint32_t nact;
  uint32_t nlong, nshort;     // update tasks of at least BATCH_RING_ROWS rows / of fewer
  uint32_t tile_end[3], next_tile[3];   // assign tiles by group of shapes (batch_group)
  uint32_t next_short, ticket;
  uint32_t epoch;             // of the last iteration whose first assign kernel has waited
  uint32_t err;               // KM_DEVERR_*
};

constexpr uint32_t BATCH_MAX_SMEM_C = 160u * 1024u;   // accepted shapes: d * round_up(k, 32) * 4 bytes at most

namespace {

__device__ __forceinline__ float f_inf_b() { return __int_as_float(0x7f800000); }

// Assign tiles: BA_NT threads as (BA_NT / TX) x TX, each RT rows and CT centroids,
// so TX * CT centroids side by side.  The shapes are 16, 24, 32, 48, 64, 96 and
// 128 centroids wide, so that at most a third of a tile is padding for k > 16
// (k > 128: chunks of 128, or of 96 for k <= 192).
constexpr int BA_NT = 128;
__host__ __device__ constexpr uint32_t batch_cols(uint32_t k) {
  return k <= 16u ? 16u : k <= 24u ? 24u : k <= 32u ? 32u : k <= 48u ? 48u : k <= 64u ? 64u
         : (k <= 96u || (k > 128u && k <= 192u)) ? 96u : 128u;
}
// Shapes are compiled into one kernel per group (two or three shapes each: with
// four the kernel spills), the widest group first.
__host__ __device__ constexpr uint32_t batch_group(uint32_t k) {
  return batch_cols(k) > 64u ? 0u : batch_cols(k) > 32u ? 1u : 2u;
}
__host__ __device__ constexpr uint32_t batch_tile_rows(uint32_t k, uint32_t rt) {
  const uint32_t c = batch_cols(k);
  return rt * (BA_NT / (c <= 32u ? 4u : c <= 64u ? 8u : 16u));
}
__host__ __device__ constexpr uint32_t batch_tiles(uint32_t n, uint32_t k, uint32_t rt) {
  return (n + batch_tile_rows(k, rt) - 1u) / batch_tile_rows(k, rt);
}
// Clusters of at least this many rows are summed by a CTA's ring, smaller ones by
// a warp alone.
constexpr uint32_t BATCH_RING_ROWS = 256;

template <int RT, int TX, int CT>
struct BatchTile {
  static constexpr int ROWS = RT * (BA_NT / TX), COLS = CT * TX;
  static constexpr int KC = TX == 4 && CT == 8 ? 8 : 16;    // coordinates per shared-memory stage
  static constexpr int LDA = ROWS + 4;
  static constexpr int A_FLOATS = KC * LDA, B_FLOATS = KC * COLS * 2, FLOATS = A_FLOATS + B_FLOATS;
  static constexpr int NA = ROWS * KC / (4 * BA_NT);       // float4 loads per thread and stage
  static constexpr int NB = (COLS * KC + 4 * BA_NT - 1) / (4 * BA_NT);
};
template <int RT>
constexpr size_t batch_assign_smem() {
  constexpr int a = BatchTile<RT, 16, 8>::FLOATS, b = BatchTile<RT, 8, 8>::FLOATS, c = BatchTile<RT, 4, 6>::FLOATS;
  static_assert(BatchTile<RT, 4, 8>::FLOATS <= c && BatchTile<RT, 4, 4>::FLOATS <= c, "the widest of its group");
  return 2 * sizeof(float) * (size_t)(a > b ? (a > c ? a : c) : (b > c ? b : c));
}

// One tile.  Bound by the FP32 pipes: three roundings an element (x - c, square,
// add) as the CPU formula has them.  They are done two rows at a time in packed
// FP32 pairs, which take half the issue slots of scalar operations (n = 65536
// d = 128 k = 64: 31.1 T operations/s against 29.5 T scalar, of 33.6 T measured
// for the three in registers alone).  The square is an FMA with -0 (nz, which the
// caller passes so that the compiler cannot see its value): it rounds as the
// product alone, whereas a packed product followed by a packed sum is fused into
// one FMA by the assembler.  The points are staged transposed (pairs of rows
// adjacent), the centroids negated and duplicated (x + (-c) rounds as x - c), both
// a stage ahead in registers.
extern __shared__ __align__(16) float batch_smem[];

// Loads of what an earlier kernel wrote and an acquire has made visible: by the ordinary
// path, which the acquire orders, not the read-only one.
__device__ __forceinline__ float ld_plain(const float* p) {
  float v;
  asm("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float4 ld_plain(const float4* p) {
  float4 v;
  asm("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}

template <int RT, int TX, int CT>
__device__ __forceinline__ void batch_tile(const float* __restrict__ Xp, const float* __restrict__ C, uint32_t n,
                                           uint32_t d, uint32_t k, bool v4, uint32_t m0, uint32_t* __restrict__ lab,
                                           double* __restrict__ objblk, float2 nz) {
  float* const smem = batch_smem;
  using T = BatchTile<RT, TX, CT>;
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  float bv[RT];
  uint32_t bi[RT];
#pragma unroll
  for (int i = 0; i < RT; ++i) { bv[i] = f_inf_b(); bi[i] = 0u; }
  const uint32_t nk = (d + T::KC - 1) / T::KC;
  for (uint32_t c0 = 0; c0 < k; c0 += T::COLS) {
    float2 acc[RT / 2][CT];
#pragma unroll
    for (int i = 0; i < RT / 2; ++i)
#pragma unroll
      for (int j = 0; j < CT; ++j) acc[i][j] = make_float2(0.0f, 0.0f);
    float4 ra[T::NA], rb[T::NB];
    // Four coordinates of a row (of X, or of C): zeros past n / k and past d.
    auto load4 = [&](const float* base, uint32_t row, uint32_t rows, uint32_t col, auto ld) {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (row < rows) {
        const float* p = base + (uint64_t)row * d + col;
        if (v4) {
          if (col < d) v = ld(reinterpret_cast<const float4*>(p));
        } else {
          if (col + 0 < d) v.x = ld(p);
          if (col + 1 < d) v.y = ld(p + 1);
          if (col + 2 < d) v.z = ld(p + 2);
          if (col + 3 < d) v.w = ld(p + 3);
        }
      }
      return v;
    };
    auto ld_x = [](const auto* p) { return __ldg(p); };
    auto ld_c = [](const auto* p) { return ld_plain(p); };
    constexpr int QR = T::KC / 4;                          // float4 per row and stage
    auto gload = [&](uint32_t kc) {
#pragma unroll
      for (int e = 0; e < T::NA; ++e) {
        const uint32_t idx = (uint32_t)(e * BA_NT + tid);
        ra[e] = load4(Xp, m0 + idx / QR, n, kc + 4u * (idx % QR), ld_x);
      }
#pragma unroll
      for (int e = 0; e < T::NB; ++e) {
        const uint32_t idx = (uint32_t)(e * BA_NT + tid);
        if (idx < (uint32_t)(T::COLS * QR)) rb[e] = load4(C, c0 + idx / QR, k, kc + 4u * (idx % QR), ld_c);
      }
    };
    auto sstore = [&](int buf) {
      float* A = smem + buf * T::FLOATS;
      float2* B = reinterpret_cast<float2*>(A + T::A_FLOATS);
#pragma unroll
      for (int e = 0; e < T::NA; ++e) {
        const int idx = e * BA_NT + tid, r = idx / QR, j = 4 * (idx % QR);
        A[(j + 0) * T::LDA + r] = ra[e].x;
        A[(j + 1) * T::LDA + r] = ra[e].y;
        A[(j + 2) * T::LDA + r] = ra[e].z;
        A[(j + 3) * T::LDA + r] = ra[e].w;
      }
#pragma unroll
      for (int e = 0; e < T::NB; ++e) {
        const int idx = e * BA_NT + tid, c = idx / QR, j = 4 * (idx % QR);
        if (idx < T::COLS * QR) {
          B[(j + 0) * T::COLS + c] = make_float2(-rb[e].x, -rb[e].x);
          B[(j + 1) * T::COLS + c] = make_float2(-rb[e].y, -rb[e].y);
          B[(j + 2) * T::COLS + c] = make_float2(-rb[e].z, -rb[e].z);
          B[(j + 3) * T::COLS + c] = make_float2(-rb[e].w, -rb[e].w);
        }
      }
    };
    gload(0);
    sstore(0);
    __syncthreads();
    for (uint32_t kt = 0; kt < nk; ++kt) {
      const float* A = smem + (kt & 1u) * T::FLOATS + ty * RT;
      const float* B = smem + (kt & 1u) * T::FLOATS + T::A_FLOATS + 4 * tx;
      if (kt + 1 < nk) gload((kt + 1) * T::KC);
      const uint32_t left = d - kt * T::KC;                // coordinates of this stage (zeros up to a multiple of 4)
#pragma unroll 1
      for (uint32_t kk = 0; kk < (uint32_t)T::KC && kk < left; kk += 4) {
#pragma unroll 2                    // 4 would spill
        for (int q = 0; q < 4; ++q) {
          const float* a_ = A + (kk + q) * T::LDA;
          const float* b_ = B + (kk + q) * (2 * T::COLS);
          float2 a[RT / 2], b[CT];
#pragma unroll
          for (int i = 0; i < RT / 4; ++i) {
            const float4 v = *reinterpret_cast<const float4*>(a_ + 4 * i);
            a[2 * i] = make_float2(v.x, v.y);
            a[2 * i + 1] = make_float2(v.z, v.w);
          }
#pragma unroll
          for (int j = 0; j < CT / 2; ++j) {
            const float4 v = *reinterpret_cast<const float4*>(b_ + 4 * TX * j);
            b[2 * j] = make_float2(v.x, v.y);
            b[2 * j + 1] = make_float2(v.z, v.w);
          }
#pragma unroll
          for (int i = 0; i < RT / 2; ++i)
#pragma unroll
            for (int j = 0; j < CT; ++j) {
              const float2 t = __fadd2_rn(a[i], b[j]);
              acc[i][j] = __fadd2_rn(acc[i][j], __ffma2_rn(t, t, nz));
            }
        }
      }
      if (kt + 1 < nk) sstore((int)((kt + 1) & 1u));
      __syncthreads();
    }
    // this thread's columns in ascending order: 2 (j/2 TX + tx) + j % 2
#pragma unroll
    for (int j = 0; j < CT; ++j) {
      const uint32_t c = c0 + 2u * (uint32_t)((j >> 1) * TX + tx) + (uint32_t)(j & 1);
      if (c < k) {
#pragma unroll
        for (int i = 0; i < RT / 2; ++i) {
          if (acc[i][j].x < bv[2 * i]) { bv[2 * i] = acc[i][j].x; bi[2 * i] = c; }
          if (acc[i][j].y < bv[2 * i + 1]) { bv[2 * i + 1] = acc[i][j].y; bi[2 * i + 1] = c; }
        }
      }
    }
  }
  // The rows' TX lists: smallest distance, lowest index on ties (a thread whose
  // distances are all +inf holds index 0, as the reference's argmin starts with).
  // Each step also halves the rows that a thread goes on with.
  int row0 = ty * RT;
#pragma unroll
  for (int o = 1, live = RT; o < TX; o <<= 1) {
    const bool up = (tx & o) != 0;
    const int h = live > 1 ? live / 2 : 0;
#pragma unroll
    for (int i = 0; i < (h ? h : 1); ++i) {
      const float sv = h ? (up ? bv[i] : bv[i + h]) : bv[i];
      const uint32_t sx = h ? (up ? bi[i] : bi[i + h]) : bi[i];
      float v = h && up ? bv[i + h] : bv[i];
      uint32_t x = h && up ? bi[i + h] : bi[i];
      const float ov = __shfl_xor_sync(0xffffffffu, sv, o);
      const uint32_t ox = __shfl_xor_sync(0xffffffffu, sx, o);
      if (ov < v || (ov == v && ox < x)) { v = ov; x = ox; }
      bv[i] = v;
      bi[i] = x;
    }
    if (h) { row0 += up ? h : 0; live = h; }
  }
  constexpr int LEFT = RT > TX ? RT / TX : 1;              // rows a thread ends with
  // The objective by blocks of 32 rows, each by one tree over its rows, so that it does
  // not depend on the tile's height.  (The stages are free: the product ends with a barrier.)
  float* const dist = smem;
#pragma unroll
  for (int i = 0; i < LEFT; ++i) {
    const uint32_t row = m0 + (uint32_t)(row0 + i);
    if (tx < RT || RT > TX) {                              // TX > RT: the lanes above hold copies
      dist[row0 + i] = row < n ? bv[i] : 0.0f;
      if (row < n) lab[row] = bi[i];
    }
  }
  __syncthreads();
#pragma unroll
  for (int b = 0; b < T::ROWS / 32; b += BA_NT / 32) {
    const int blk = b + (tid >> 5);
    if (blk >= T::ROWS / 32 || m0 + 32u * (uint32_t)blk >= n) break;
    double o = (double)dist[32 * blk + (tid & 31)];
#pragma unroll
    for (int x = 16; x > 0; x >>= 1) o += __shfl_xor_sync(0xffffffffu, o, x);
    if ((tid & 31) == 0) objblk[blk] = o;
  }
}

// Index of the running instance that owns item t: the last a with first[a] <= t.
__device__ __forceinline__ uint32_t batch_owner(const uint32_t* __restrict__ first, uint32_t nact, uint32_t t) {
  uint32_t lo = 0, hi = nact;
  while (hi - lo > 1u) {
    const uint32_t mid = (lo + hi) / 2u;
    if (__ldcg(first + mid) <= t) lo = mid; else hi = mid;
  }
  return lo;
}

// The tiles of one group.  The groups' kernels follow one another in the stream and may
// overlap.  The first waits for the iteration before and then says so (epoch, a release);
// a later one whose acquire sees that may read what that iteration wrote, and one that
// does not waits for its predecessor.  Each later one waits for its predecessor before it
// ends, so that the next kernel's wait covers all of them.  What the iteration before
// wrote is read by ordinary loads after the acquire, the centroids and tile0 too.
// Against groups one after the other, each with a wait of its own: 21 problems, n 512 to
// 19,142, 3.0 / 3.8 ms, 28 x 3 restarts, n 512 to 12,104, 4.2 / 4.9; 64 x 4, n 1024 to
// 65,536, 82.9 / 79.7.
template <int RT, int GROUP>
__global__ void __launch_bounds__(BA_NT, RT == 8 ? 3 : 4)
batch_assign_kernel(const float* __restrict__ X, const BatchInst* __restrict__ insts, BatchCtl* ctl,
                    const uint32_t* __restrict__ act, const uint32_t* __restrict__ tile0,
                    const float* __restrict__ Call, uint32_t* __restrict__ labels, double* __restrict__ objblk,
                    uint32_t epoch, int first, float neg0) {
  __shared__ uint32_t s_tile;
  if (first) {
    griddep_wait();
    if (blockIdx.x == 0 && threadIdx.x == 0)
      asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(&ctl->epoch), "r"(epoch) : "memory");
  } else {
    if (threadIdx.x == 0) asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(s_tile) : "l"(&ctl->epoch) : "memory");
    __syncthreads();
    if (s_tile != epoch) griddep_wait();
  }
  griddep_launch();
  const uint32_t nact = ctl->nact, begin = GROUP ? ctl->tile_end[GROUP ? GROUP - 1 : 0] : 0u,
                 end = ctl->tile_end[GROUP];
  for (;;) {
    __syncthreads();                       // the tile before is done with s_tile and the stages
    if (threadIdx.x == 0) s_tile = end > begin ? begin + atomicAdd(&ctl->next_tile[GROUP], 1u) : end;
    __syncthreads();
    const uint32_t t = s_tile;
    if (t >= end) break;
    const uint32_t a = batch_owner(tile0, nact, t);
    const BatchInst I = insts[act[a]];
    const uint32_t m0 = (t - tile0[a]) * batch_tile_rows(I.k, RT);
    const float* Xp = X + I.xoff;
    const float* C = Call + I.coff;
    const bool v4 = (I.d % 4u) == 0u && (I.xoff % 4u) == 0u;
    uint32_t* lab = labels + I.loff;
    double* ob = objblk + I.toff + m0 / 32u;
#define KM_BATCH_TILE(TX_, CT_) batch_tile<RT, TX_, CT_>(Xp, C, I.n, I.d, I.k, v4, m0, lab, ob, make_float2(neg0, neg0))
    if constexpr (GROUP == 0) {
      if (batch_cols(I.k) == 96u) KM_BATCH_TILE(16, 6); else KM_BATCH_TILE(16, 8);
    } else if constexpr (GROUP == 1) {
      if (batch_cols(I.k) == 48u) KM_BATCH_TILE(8, 6); else KM_BATCH_TILE(8, 8);
    } else {
      switch (batch_cols(I.k)) {
        case 16: KM_BATCH_TILE(4, 4); break;
        case 24: KM_BATCH_TILE(4, 6); break;
        default: KM_BATCH_TILE(4, 8); break;
      }
    }
#undef KM_BATCH_TILE
  }
  if (!first) griddep_wait();
}

// Stable counting sort of an instance's rows by label: each warp counts and then
// scatters a contiguous run of rows.  Also lists the instance's update tasks.
constexpr int BS_WARPS = 16;
__global__ void __launch_bounds__(32 * BS_WARPS)
batch_sort_kernel(const float* __restrict__ X, const BatchInst* __restrict__ insts, BatchCtl* ctl,
                  const uint32_t* __restrict__ act, const uint32_t* __restrict__ labels,
                  uint32_t* __restrict__ perm_all, float* __restrict__ Cn, BatchTask* __restrict__ longs,
                  BatchTask* __restrict__ shorts) {
  griddep_wait();
  __shared__ uint32_t pos[BS_WARPS][256];
  __shared__ uint32_t part[8];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t nact = ctl->nact;
  for (uint32_t a = blockIdx.x; a < nact; a += gridDim.x) {
    const BatchInst& I = insts[act[a]];
    const uint32_t n = I.n, k = I.k, d = I.d;
    const uint32_t* lab = labels + I.loff;
    uint32_t* perm = perm_all + I.loff;
    for (uint32_t q = tid; q < BS_WARPS * 256u; q += 32 * BS_WARPS) (&pos[0][0])[q] = 0u;
    __syncthreads();
    const uint32_t per = ((n + BS_WARPS - 1) / BS_WARPS + 31u) & ~31u;
    const uint32_t r0 = min(n, (uint32_t)warp * per), r1 = min(n, r0 + per);
    constexpr int U = 8;                                   // labels in flight per lane
    for (uint32_t g = r0; g < r1; g += 32u * U) {
      uint32_t lv[U];
#pragma unroll
      for (int q = 0; q < U; ++q) {
        const uint32_t r = g + 32u * q + lane;
        lv[q] = r < r1 ? lab[r] : 0xffffffffu;
      }
#pragma unroll
      for (int q = 0; q < U; ++q)
        if (lv[q] != 0xffffffffu) atomicAdd(&pos[warp][lv[q]], 1u);
    }
    __syncthreads();
    // thread c: the cluster's count over the warps, then an exclusive scan over
    // the clusters (k <= 256) and over each cluster's warps
    uint32_t cnt = 0;
    if (tid < 256)
      for (int w = 0; w < BS_WARPS; ++w) cnt += pos[w][tid];
    uint32_t inc = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += y;
    }
    if (tid < 256 && lane == 31) part[warp] = inc;
    __syncthreads();
    if (tid < 256) {
      uint32_t base = inc - cnt;
      for (int w = 0; w < warp; ++w) base += part[w];
      // this warp's clusters to the two task lists (their order is free)
      const bool in = (uint32_t)tid < k, ring = in && cnt >= BATCH_RING_ROWS;
      const uint32_t nblk = (d + 31u) / 32u;
      const unsigned ml = __ballot_sync(0xffffffffu, ring), ms = __ballot_sync(0xffffffffu, in && !ring);
      uint32_t bl = 0, bs = 0;
      if (lane == 0) {
        if (ml) bl = atomicAdd(&ctl->nlong, (uint32_t)__popc(ml) * nblk);
        if (ms) bs = atomicAdd(&ctl->nshort, (uint32_t)__popc(ms) * nblk);
      }
      bl = __shfl_sync(0xffffffffu, bl, 0);
      bs = __shfl_sync(0xffffffffu, bs, 0);
      if (in) {
        const uint32_t at = (uint32_t)__popc((ring ? ml : ms) & ((1u << lane) - 1u)) * nblk + (ring ? bl : bs);
        const uint32_t vec = (d % 4u == 0u && I.xoff % 4u == 0u) ? 4u : (d % 2u == 0u && I.xoff % 2u == 0u) ? 2u : 1u;
        BatchTask* out = (ring ? longs : shorts) + at;
        for (uint32_t b = 0; b < nblk; ++b)
          out[b] = BatchTask{X + I.xoff + 32u * b, perm + base, Cn + I.coff + (uint64_t)tid * d + 32u * b, cnt, d,
                             min(32u, d - 32u * b), vec};
      }
      for (int w = 0; w < BS_WARPS; ++w) {
        const uint32_t v = pos[w][tid];
        pos[w][tid] = base;
        base += v;
      }
    }
    __syncthreads();
    for (uint32_t g = r0; g < r1; g += 32u * U) {
      uint32_t lv[U];
#pragma unroll
      for (int q = 0; q < U; ++q) {
        const uint32_t r = g + 32u * q + lane;
        lv[q] = r < r1 ? lab[r] : 0xffffffffu;
      }
#pragma unroll
      for (int q = 0; q < U; ++q) {
        if (g + 32u * q >= r1) break;
        const uint32_t l = lv[q];
        const unsigned m = __match_any_sync(0xffffffffu, l);
        const uint32_t rank = (uint32_t)__popc(m & ((1u << lane) - 1u));
        const bool ok = l != 0xffffffffu;
        const uint32_t base = ok ? pos[warp][l] : 0u;
        __syncwarp();
        if (ok) {
          perm[base + rank] = g + 32u * q + lane;
          if (rank == 0) pos[warp][l] = base + (uint32_t)__popc(m);
        }
        __syncwarp();
      }
    }
    __syncthreads();
  }
}

// A predicated load (0 when !ok) that stays where it is written: plain loads
// were moved down to the additions that use them, one latency each.
__device__ __forceinline__ float ld_global_pinned(const float* p, bool ok) {
  float v;
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\tmov.f32 %0, 0f00000000;\n\t"
               "@q ld.global.nc.f32 %0, [%1];\n\t}"
               : "=f"(v)
               : "l"(p), "r"((uint32_t)ok));
  return v;
}

// Ordered sums.  Warps 0..3 of a CTA walk the long tasks (every gridDim-th) as
// the producers and the chain of a shared-memory ring that runs on from task to
// task (km_sums.cuh); the other warps, and these four once their long tasks are
// done, take short tasks, a warp each, lane = column: 32 rows' loads at a time.
// Rows past the cluster's end add +0, which leaves the sum as it is (it starts at
// +0).  First iteration of the problems above: 0.57 ms for 10 M row segments of up
// to 32 columns, against 4.1 ms with a warp for every task, whose longest chain
// set the time.
constexpr int BU_PROD = 3, BU_WARPS = 8;
__global__ void __launch_bounds__(32 * BU_WARPS, 2)
batch_update_kernel(BatchCtl* ctl, const BatchTask* __restrict__ longs, const BatchTask* __restrict__ shorts) {
  griddep_wait();
  extern __shared__ __align__(128) float ring[];
  __shared__ __align__(8) uint64_t full[BLK_STAGES], empty[BLK_STAGES];
  __shared__ int abort_flag;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t nlong = ctl->nlong, nshort = ctl->nshort;
  if (threadIdx.x == 0) {
    for (int s = 0; s < BLK_STAGES; ++s) { mbar_init(&full[s], 32); mbar_init(&empty[s], 1); }
    abort_flag = 0;
    mbar_fence_init();
  }
  __syncthreads();
  auto write = [&](const BatchTask& t, float sum) {
    if ((uint32_t)lane < t.w) {
      const float scale = (float)(1.0 / (double)(t.cnt > 1u ? t.cnt : 1u));
      t.out[lane] = __fmul_rn(sum, scale);
    }
  };
  if (warp <= BU_PROD) {
    const SumsRing R{ring, full, empty, &abort_flag};
    uint32_t first = 0;
    bool ok = true;
    BatchTask next{};
    if (blockIdx.x < nlong) next = longs[blockIdx.x];
    for (uint32_t e = blockIdx.x; e < nlong && ok; e += gridDim.x) {
      const BatchTask t = next;
      if (e + gridDim.x < nlong) next = longs[e + gridDim.x];
      if (warp < BU_PROD) {
        const uint32_t p = (uint32_t)warp;
        ok = t.vec == 4u   ? sums_produce<4, BU_PROD>(R, t.x, t.perm, t.cnt, t.d, t.w, first, p)
             : t.vec == 2u ? sums_produce<2, BU_PROD>(R, t.x, t.perm, t.cnt, t.d, t.w, first, p)
                           : sums_produce<1, BU_PROD>(R, t.x, t.perm, t.cnt, t.d, t.w, first, p);
      } else {
        float sum;
        ok = sums_chain(R, t.cnt, first, sum);
        if (ok) write(t, sum);
      }
      first += (t.cnt + BLK_ROWS - 1) / BLK_ROWS;
    }
    if (!ok && lane == 0) {
      *(volatile int*)&abort_flag = 1;
      atomicOr(&ctl->err, KM_DEVERR_TIMEOUT);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");   // this warp's copies land before the CTA exits
  }
  for (;;) {
    uint32_t e = 0;
    if (lane == 0) e = nshort ? atomicAdd(&ctl->next_short, 1u) : 0u;
    e = __shfl_sync(0xffffffffu, e, 0);
    if (e >= nshort) break;
    const BatchTask t = shorts[e];
    const float* xc = t.x + lane;
    float sum = 0.0f;
    uint32_t idx = (uint32_t)lane < t.cnt ? __ldg(t.perm + lane) : 0u;
    for (uint32_t g = 0; g < t.cnt; g += 32u) {
      float v[32];
#pragma unroll
      for (int u = 0; u < 32; ++u) {
        const uint32_t r = __shfl_sync(0xffffffffu, idx, u);
        v[u] = ld_global_pinned(xc + (uint64_t)r * t.d, (uint32_t)lane < t.w && g + (uint32_t)u < t.cnt);
      }
      const uint32_t q = g + 32u + (uint32_t)lane;
      idx = q < t.cnt ? __ldg(t.perm + q) : 0u;
#pragma unroll
      for (int u = 0; u < 32; ++u) sum = __fadd_rn(sum, v[u]);
    }
    write(t, sum);
  }
}

// Lists the instances of act[0 .. nact) that are not done (all of them when
// done is null), in order, with the first tile of each; resets the counters.
// One block.
__device__ void batch_list(const BatchInst* __restrict__ insts, BatchCtl* ctl, uint32_t* act, uint32_t* tile0,
                           const uint32_t* done, uint32_t nact, uint32_t rt, uint32_t* sh) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = (int)blockDim.x >> 5;
  uint32_t b0 = 0, b1 = 0;                                 // running totals: instances, tiles
  if (tid < 3) sh[64 + tid] = 0u;                          // last tile of each group + 1
  for (uint32_t g = 0; g < nact; g += blockDim.x) {
    const uint32_t q = g + (uint32_t)tid;
    uint32_t id = 0, f0 = 0, f1 = 0;
    if (q < nact) {
      id = done ? __ldcg(act + q) : q;
      if (!done || __ldcg(done + id) == 0u) {
        const BatchInst& I = insts[id];
        f0 = 1u;
        f1 = batch_tiles(I.n, I.k, rt);
      }
    }
    uint32_t x0 = f0, x1 = f1;                             // inclusive scans over the warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y0 = __shfl_up_sync(0xffffffffu, x0, o), y1 = __shfl_up_sync(0xffffffffu, x1, o);
      if (lane >= o) { x0 += y0; x1 += y1; }
    }
    if (lane == 31) { sh[warp] = x0; sh[32 + warp] = x1; }
    __syncthreads();                                       // every read of this chunk of act is done, too
    uint32_t t0 = 0, t1 = 0, e0 = 0, e1 = 0;
    for (int w = 0; w < nw; ++w) {
      if (w == warp) { e0 = t0; e1 = t1; }
      t0 += sh[w]; t1 += sh[32 + w];
    }
    if (f0) {
      const uint32_t at = b0 + e0 + x0 - 1u;
      act[at] = id;
      tile0[at] = b1 + e1 + x1 - f1;
      atomicMax(&sh[64 + batch_group(insts[id].k)], b1 + e1 + x1);
    }
    b0 += t0; b1 += t1;
    __syncthreads();
  }
  if (tid == 0) {
    ctl->nact = b0;
    for (uint32_t q = 0, e = 0; q < 3u; ++q) {             // an empty group ends where the one before it does
      e = max(e, sh[64 + q]);
      ctl->tile_end[q] = e;
      ctl->next_tile[q] = 0u;
    }
    ctl->nlong = ctl->nshort = ctl->next_short = ctl->ticket = 0u;
  }
}

__global__ void __launch_bounds__(1024)
batch_begin_kernel(const BatchInst* __restrict__ insts, BatchCtl* ctl, uint32_t* act, uint32_t* tile0,
                   uint32_t* done, uint32_t ninst, uint32_t rt) {
  __shared__ uint32_t sh[67];
  for (uint32_t i = threadIdx.x; i < ninst; i += blockDim.x) done[i] = 0u;
  batch_list(insts, ctl, act, tile0, nullptr, ninst, rt, sh);
  if (threadIdx.x == 0) { ctl->iter = 0; ctl->err = 0u; ctl->epoch = 0u; }
}

__global__ void __launch_bounds__(256)
batch_stop_kernel(const BatchInst* __restrict__ insts, BatchCtl* ctl, uint32_t* act, uint32_t* tile0, uint32_t* done,
                  float* __restrict__ Call, const float* __restrict__ Cn_all,
                  const double* __restrict__ objblk, float tol, uint64_t maxiter, uint32_t rt,
                  BatchOut* __restrict__ out) {
  griddep_wait();
  __shared__ int s_moved;
  __shared__ int is_last;
  __shared__ uint32_t sh[67];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t nact = ctl->nact;
  if (nact == 0u) return;
  const uint64_t iter = ctl->iter + 1;
  for (uint32_t a = blockIdx.x; a < nact; a += gridDim.x) {
    const uint32_t id = act[a];
    const BatchInst& I = insts[id];
    const uint32_t d = I.d, k = I.k;
    float* C = Call + I.coff;
    const float* Cn = Cn_all + I.coff;
    if (tid == 0) s_moved = 0;
    __syncthreads();
    if (iter > 1) {
      // a warp per cluster, until one is found that moved
      for (uint32_t c = (uint32_t)warp; c < k && *(volatile int*)&s_moved == 0; c += 8u) {
        float s = 0.0f;                                    // column order
        for (uint32_t j0 = 0; j0 < d; j0 += 32u) {
          const uint32_t j = j0 + (uint32_t)lane;
          float q = 0.0f;
          if (j < d) {
            const float t = __fsub_rn(Cn[(uint64_t)c * d + j], C[(uint64_t)c * d + j]);
            q = __fmul_rn(t, t);
          }
#pragma unroll
          for (int l = 0; l < 32; ++l) s = __fadd_rn(s, __shfl_sync(0xffffffffu, q, l));   // past d: + 0
        }
        if (lane == 0 && sqrtf(s) > tol) s_moved = 1;
        __syncwarp();
      }
    }
    __syncthreads();
    const bool stop = iter > 1 && s_moved == 0;
    for (uint32_t q = tid; q < k * d; q += 256u) C[q] = Cn[q];
    if (stop || iter >= maxiter) {
      if (warp == 0) {
        const uint32_t nt = (I.n + 31u) / 32u;             // blocks of rows (see batch_tile)
        double o = 0.0;
        for (uint32_t t = (uint32_t)lane; t < nt; t += 32u * 8u) {
          double v[8];
#pragma unroll
          for (uint32_t u = 0; u < 8; ++u) v[u] = nt - t > 32u * u ? objblk[I.toff + t + 32u * u] : 0.0;
#pragma unroll
          for (uint32_t u = 0; u < 8; ++u) o += v[u];
        }
        for (int w = 16; w > 0; w >>= 1) o += __shfl_xor_sync(0xffffffffu, o, w);
        if (lane == 0) {
          out[id].converged_iter = stop ? iter : maxiter;
          out[id].iterations = iter;
          out[id].objective = o;
          done[id] = 1u;
        }
      }
    }
    __syncthreads();
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) is_last = (atomicAdd(&ctl->ticket, 1u) == gridDim.x - 1u) ? 1 : 0;
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  batch_list(insts, ctl, act, tile0, done, nact, rt, sh);
  if (tid == 0) ctl->iter = iter;
}

// ---------------------------------------------------------------------------
// Small instances: a CTA takes one instance at a time and runs all of its iterations,
// so that a fit is one launch.  The steps are those above, with the same roundings:
// the centroids live in shared memory (transposed),
// a warp assigns a contiguous run of rows, one row a lane, counts them by label and
// scatters them; a thread adds one (cluster, column) in row order.  Bound by latency:
// five barriers an iteration and the chains of the ordered sums.  (batch_is_small has
// the line to the tiles, and both sides' times.)
// ---------------------------------------------------------------------------
constexpr int SM_NT = 256, SM_WARPS = SM_NT / 32;
// Centroids side by side in a lane's registers (a row is read once for them all), and the
// centroids' padding.
__host__ __device__ constexpr uint32_t small_cg(uint32_t k) { return k <= 8u ? 8u : k <= 16u ? 16u : 32u; }
__host__ __device__ constexpr uint32_t small_kpad(uint32_t k) { return (k + small_cg(k) - 1u) / small_cg(k) * small_cg(k); }

// The nearest centroids of R rows at once (Cs: d x kpad in shared memory).
template <int CG, int R>
__device__ __forceinline__ void small_nearest(const float* const (&x)[R], bool v4, const float* Cs, uint32_t d,
                                              uint32_t k, uint32_t kpad, uint32_t (&bi)[R]) {
  float best[R];
#pragma unroll
  for (int r = 0; r < R; ++r) { best[r] = f_inf_b(); bi[r] = 0u; }
  for (uint32_t c0 = 0; c0 < k; c0 += CG) {
    float acc[R][CG];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int c = 0; c < CG; ++c) acc[r][c] = 0.0f;
    auto add = [&](const float (&xj)[R], uint32_t j) {
#pragma unroll
      for (int q = 0; q < CG / 4; ++q) {
        const float4 v = *reinterpret_cast<const float4*>(Cs + j * kpad + c0 + 4 * q);
        const float cc[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float t = __fsub_rn(xj[r], cc[e]);
            acc[r][4 * q + e] = __fadd_rn(acc[r][4 * q + e], __fmul_rn(t, t));
          }
      }
    };
    if (v4) {                                              // 16-byte loads: d % 4 == 0, rows aligned
      for (uint32_t j = 0; j < d; j += 4u) {
        float4 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = __ldg(reinterpret_cast<const float4*>(x[r] + j));
        float xj[R];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
#pragma unroll
          for (int r = 0; r < R; ++r) xj[r] = e == 0 ? v[r].x : e == 1 ? v[r].y : e == 2 ? v[r].z : v[r].w;
          add(xj, j + (uint32_t)e);
        }
      }
    } else {
#pragma unroll 2
      for (uint32_t j = 0; j < d; ++j) {
        float xj[R];
#pragma unroll
        for (int r = 0; r < R; ++r) xj[r] = __ldg(x[r] + j);
        add(xj, j);
      }
    }
#pragma unroll
    for (int c = 0; c < CG; ++c)
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (c0 + c < k && acc[r][c] < best[r]) { best[r] = acc[r][c]; bi[r] = c0 + c; }
  }
}

constexpr uint32_t BATCH_SMALL_SMEM = 64u * 1024u;   // two copies of the centroids at most
constexpr uint32_t SMALL_WARP_SUMS = 3u * SM_WARPS;

__global__ void __launch_bounds__(SM_NT)
batch_small_kernel(const float* __restrict__ X, const BatchInst* __restrict__ insts, uint32_t ninst, BatchCtl* ctl,
                   const float* __restrict__ C0, float* __restrict__ Call, uint32_t* labels, uint32_t* perm_all,
                   double* objblk, float tol, uint64_t maxiter, BatchOut* __restrict__ out) {
  __shared__ uint32_t pos[SM_WARPS][256];
  __shared__ uint32_t cstart[257], part[SM_WARPS];
  __shared__ uint32_t s_inst;
  __shared__ int s_moved;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (;;) {
    __syncthreads();                                       // the instance before is done with the shared arrays
    if (tid == 0) s_inst = atomicAdd(&ctl->next_short, 1u);
    __syncthreads();
    const uint32_t id = s_inst;
    if (id >= ninst) break;
    const BatchInst I = insts[id];
    const uint32_t n = I.n, d = I.d, k = I.k, kpad = small_kpad(k);
    const float* Xp = X + I.xoff;
    const bool v4 = d % 4u == 0u && I.xoff % 4u == 0u;
    uint32_t* const lab = labels + I.loff;
    uint32_t* const perm = perm_all + I.loff;
    float *Cs = batch_smem, *Cn = batch_smem + d * kpad;
    for (uint32_t q = tid; q < d * kpad; q += SM_NT) {
      const uint32_t j = q / kpad, c = q % kpad;
      Cs[q] = c < k ? C0[I.coff + (uint64_t)c * d + j] : 0.0f;
    }
    const uint32_t per = ((n + SM_WARPS - 1) / SM_WARPS + 31u) & ~31u;
    const uint32_t r0 = min(n, (uint32_t)warp * per), r1 = min(n, r0 + per);
    uint64_t iter = 0;
    bool stop = false;
    while (!stop && iter < maxiter) {
      ++iter;
      for (uint32_t c = lane; c < 256u; c += 32u) pos[warp][c] = 0u;
      __syncthreads();                                     // centroids in place; s_moved has been read
      if (tid == 0) s_moved = 0;
      // assign and count, two rows a lane (one where a warp has no more)
      auto assign = [&](uint32_t g, auto rows) {
        constexpr int R = rows();
        const float* x[R];
        uint32_t bi[R];
#pragma unroll
        for (int r = 0; r < R; ++r) x[r] = Xp + (uint64_t)min(g + 32u * r + (uint32_t)lane, n - 1u) * d;
        if (k <= 8u) small_nearest<8, R>(x, v4, Cs, d, k, kpad, bi);
        else if (k <= 16u) small_nearest<16, R>(x, v4, Cs, d, k, kpad, bi);
        else small_nearest<32, R>(x, v4, Cs, d, k, kpad, bi);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const uint32_t row = g + 32u * r + (uint32_t)lane;
          const unsigned m = __match_any_sync(0xffffffffu, row < r1 ? bi[r] : 0xffffffffu);
          if (row < r1) {
            lab[row] = bi[r];
            if ((m & ((1u << lane) - 1u)) == 0u) pos[warp][bi[r]] += (uint32_t)__popc(m);
          }
          __syncwarp();
        }
      };
      for (uint32_t g = r0; g < r1; g += 64u) {
        if (r1 - g > 32u) assign(g, std::integral_constant<int, 2>{});
        else assign(g, std::integral_constant<int, 1>{});
      }
      __syncthreads();
      // thread c: cluster c's rows over the warps, scanned over the clusters (k <= 256)
      uint32_t cnt = 0;
#pragma unroll
      for (int w = 0; w < SM_WARPS; ++w) cnt += pos[w][tid];
      uint32_t inc = cnt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
      }
      if (lane == 31) part[warp] = inc;
      __syncthreads();
      uint32_t base = inc - cnt;
      for (int w = 0; w < warp; ++w) base += part[w];
      cstart[tid] = base;
      if (tid == 255) cstart[256] = base + cnt;
#pragma unroll
      for (int w = 0; w < SM_WARPS; ++w) {
        const uint32_t v = pos[w][tid];
        pos[w][tid] = base;
        base += v;
      }
      __syncthreads();
      // stable scatter (a lane's own labels, 4 loads in flight)
      for (uint32_t g0 = r0; g0 < r1; g0 += 128u) {
        uint32_t lv[4];
#pragma unroll
        for (uint32_t q = 0; q < 4u; ++q) {
          const uint32_t row = g0 + 32u * q + (uint32_t)lane;
          lv[q] = row < r1 ? lab[row] : 0xffffffffu;
        }
#pragma unroll
        for (uint32_t q = 0; q < 4u; ++q) {
          if (g0 + 32u * q >= r1) break;
          const uint32_t row = g0 + 32u * q + (uint32_t)lane, l = lv[q];
          const unsigned m = __match_any_sync(0xffffffffu, l);
          const uint32_t rank = (uint32_t)__popc(m & ((1u << lane) - 1u));
          const uint32_t at = row < r1 ? pos[warp][l] : 0u;
          __syncwarp();
          if (row < r1) {
            perm[at + rank] = row;
            if (rank == 0u) pos[warp][l] = at + (uint32_t)__popc(m);
          }
          __syncwarp();
        }
      }
      __syncthreads();
      // ordered sums: few of them by a warp each, which loads 32 rows at once and adds
      // them by shuffles, else a thread each
      auto put = [&](uint32_t c, uint32_t j, float sum) {
        const uint32_t count = cstart[c + 1] - cstart[c];
        Cn[j * kpad + c] = __fmul_rn(sum, (float)(1.0 / (double)(count > 1u ? count : 1u)));
      };
      if (k * d <= SMALL_WARP_SUMS && d <= 8u) {
        for (uint32_t q = (uint32_t)warp; q < k * d; q += SM_WARPS) {
          const uint32_t c = q / d, j = q % d, p1 = cstart[c + 1];
          float s = 0.0f, v = 0.0f;
          uint32_t p = cstart[c] + (uint32_t)lane;
          if (p < p1) v = __ldg(Xp + (uint64_t)perm[p] * d + j);
          for (uint32_t p0 = cstart[c]; p0 < p1; p0 += 32u) {
            p += 32u;
            const float w = p < p1 ? __ldg(Xp + (uint64_t)perm[p] * d + j) : 0.0f;
#pragma unroll
            for (int l = 0; l < 32; ++l) s = __fadd_rn(s, __shfl_sync(0xffffffffu, v, l));   // past the end: + 0
            v = w;
          }
          if (lane == 0) put(c, j, s);
        }
      } else {
        for (uint32_t q = tid; q < k * d; q += SM_NT) {
          const uint32_t c = q / d, j = q % d, p1 = cstart[c + 1];
          const float* xj = Xp + j;
          float s = 0.0f;
          uint32_t p = cstart[c];
          for (; p + 8u <= p1; p += 8u) {
            float v[8];
#pragma unroll
            for (uint32_t u = 0; u < 8u; ++u) v[u] = __ldg(xj + (uint64_t)perm[p + u] * d);
#pragma unroll
            for (uint32_t u = 0; u < 8u; ++u) s = __fadd_rn(s, v[u]);
          }
          for (; p < p1; ++p) s = __fadd_rn(s, __ldg(xj + (uint64_t)perm[p] * d));
          put(c, j, s);
        }
      }
      __syncthreads();
      if (iter > 1) {
        for (uint32_t c = tid; c < k; c += SM_NT) {
          float s = 0.0f;                                  // column order
          for (uint32_t j = 0; j < d; ++j) {
            const float t = __fsub_rn(Cn[j * kpad + c], Cs[j * kpad + c]);
            s = __fadd_rn(s, __fmul_rn(t, t));
          }
          if (sqrtf(s) > tol) s_moved = 1;
        }
        __syncthreads();
        stop = s_moved == 0;
      }
      if (stop || iter >= maxiter) {
        // the objective of this assignment, in the order of batch_tile and the stop kernel
        for (uint32_t g = r0; g < r1; g += 32u) {
          const uint32_t row = g + (uint32_t)lane;
          float s = 0.0f;
          if (row < r1) {
            const float* x = Xp + (uint64_t)row * d;
            const uint32_t c = lab[row];
            for (uint32_t j = 0; j < d; ++j) {
              const float t = __fsub_rn(__ldg(x + j), Cs[j * kpad + c]);
              s = __fadd_rn(s, __fmul_rn(t, t));
            }
          }
          double o = (double)s;
#pragma unroll
          for (int x = 16; x > 0; x >>= 1) o += __shfl_xor_sync(0xffffffffu, o, x);
          if (lane == 0) objblk[I.toff + g / 32u] = o;
        }
        for (uint32_t q = tid; q < k * d; q += SM_NT) Call[I.coff + q] = Cn[(q % d) * kpad + q / d];
        __syncthreads();
        if (warp == 0) {
          double o = 0.0;
          for (uint32_t t = (uint32_t)lane; t < (n + 31u) / 32u; t += 32u) o += objblk[I.toff + t];
#pragma unroll
          for (int x = 16; x > 0; x >>= 1) o += __shfl_xor_sync(0xffffffffu, o, x);
          if (lane == 0) out[id] = BatchOut{stop ? iter : maxiter, iter, o};
        }
      }
      float* const t = Cs;
      Cs = Cn;
      Cn = t;
    }
  }
}

// Reference sample picks (kmeans.cpp:22-29, :49-84) on the host copy of X.
bool host_sample_picks(const float* X, uint64_t n, uint32_t d, uint32_t k, int seed, int32_t* picks) {
  std::seed_seq ss{seed};
  std::mt19937 gen(ss);
  std::uniform_int_distribution<int> dist(0, (int)(n - 1));
  uint32_t have = 0;
  uint64_t guard = 0;
  while (have < k) {
    if (++guard > 1000ull * (k + 16) + 100000ull) return false;
    const int p = dist(gen);
    bool found = false;
    for (uint32_t q = 0; q < have && !found; ++q) {
      bool eq = true;
      for (uint32_t j = 0; j < d && eq; ++j) eq = X[(uint64_t)picks[q] * d + j] == X[(uint64_t)p * d + j];
      found = eq;
    }
    if (!found) picks[have++] = p;
  }
  return true;
}

// Whether a CTA an instance wins (every instance has to pass).  An iteration in tiles costs
// four to six launches, 20 to 30 us, whatever it does; a CTA alone has an SM at most.
// Few instances, 20 iterations, CTA / tiles: n 2000 d 8 k 32 0.30 / 0.44 ms, n 4000 d 8 k 32
// 0.55 / 0.56, n 4000 d 1 k 128 0.91 / 0.57, n 30000 d 1 k 2 1.2 / 0.9, n 1000 d 128 k 8
// 0.78 / 0.61.  With instances enough for every SM (the largest no more than an SM's share
// of all rows) the CTAs fill the GPU, and what the tiles win by is reading the points
// fewer times: 152 of n 16000 d 2 k 32 2.5 / 4.1, d 6 k 32 3.8 / 4.8, d 4 k 3 4.1 / 2.0, n
// 4000 d 32 k 8 1.9 / 1.6.  Rows of up to three columns leave most of a tile empty, which
// many centroids make felt: 600 of n 65536 d 3 k 32 44 / 82, 152 of d 2 k 3 17 / 10.
bool batch_is_small(const std::vector<BatchInst>& inst, int num_sms, size_t* smem) {
  uint64_t rows = 0, top = 0;
  for (const BatchInst& I : inst) {
    rows += I.n;
    top = std::max<uint64_t>(top, I.n);
  }
  const bool many = rows >= top * (uint64_t)num_sms;
  *smem = 0;
  for (const BatchInst& I : inst) {
    const uint64_t nd = (uint64_t)I.n * I.d, work = nd * I.k;
    const bool in = many ? (nd <= (1u << 16) && work <= (1u << 23)) ||
                               (I.k >= 32u && (I.d <= 3u || (I.d <= 8u && nd <= (1u << 17))))
                         : nd <= (1u << 15) && work <= 640000u && (uint64_t)I.n * I.k <= (1u << 18) && I.n <= (1u << 13);
    *smem = std::max(*smem, 2 * sizeof(float) * I.d * small_kpad(I.k));
    if (!in || *smem > BATCH_SMALL_SMEM) return false;
  }
  return true;
}

// Tile variants of the assign step: rows per thread and CTAs per SM.
struct BatchVariant {
  int rt, ctas;
};
const BatchVariant kVariants[] = {{8, 3}, {8, 2}, {8, 1}, {4, 4}, {4, 3}, {4, 2}};
constexpr int kDefaultVariant = 0;

}  // namespace
}  // namespace km

using namespace km;

struct km_batch {
  km_batch_params p;
  std::vector<km_batch_problem> probs;
  std::vector<BatchInst> inst;          // LPT order
  int device = 0, num_sms = 0;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  uint32_t groups = 0;                  // groups of assign shapes in use (bit mask)
  bool small = false;                   // every instance is one CTA's work (batch_small_kernel)
  size_t small_smem = 0;
  int small_ctas = 1;                   // of them an SM
  uint64_t x_floats = 0, lab_total = 0, c_total = 0, task_total = 0, t_total = 0;
  float* X = nullptr;
  float* C0 = nullptr;
  float* C = nullptr;                   // current centroids, the result at the end
  float* Cn = nullptr;                  // next centroids
  uint32_t* labels = nullptr;
  uint32_t* perm = nullptr;
  BatchTask* tasks = nullptr;           // long, then short: task_total each
  double* objblk = nullptr;
  BatchInst* dinst = nullptr;
  BatchOut* dout = nullptr;
  BatchCtl* ctl = nullptr;
  uint32_t* lists = nullptr;            // act, tile0, done: one entry per instance each
  BatchCtl* h_ctl = nullptr;            // pinned
  int variant = kDefaultVariant;
  double tune_ms[6] = {0, 0, 0, 0, 0, 0};
  bool ready = false;
  ~km_batch() {
    if (device >= 0) cudaSetDevice(device);
    for (void* q : {(void*)X, (void*)C0, (void*)C, (void*)Cn, (void*)labels, (void*)perm, (void*)tasks,
                    (void*)objblk, (void*)dinst, (void*)dout, (void*)ctl, (void*)lists})
      if (q) cudaFree(q);
    if (h_ctl) cudaFreeHost(h_ctl);
    if (own_stream && stream) cudaStreamDestroy(stream);
  }
};

namespace {

template <typename T>
km_status balloc(T** p, size_t count) {
  if (cudaMalloc(reinterpret_cast<void**>(p), sizeof(T) * std::max<size_t>(count, 1)) != cudaSuccess) {
    (void)cudaGetLastError();
    return KM_ERR_ALLOC;
  }
  return KM_OK;
}

// The launches of one iteration of the running instances.
template <int RT>
km_status enqueue_batch_iteration(km_batch* h, int ctas, const BatchInst* dinst, uint32_t ninst, uint64_t maxiter,
                                  uint32_t epoch) {
  uint32_t *act = h->lists, *tile0 = act + h->inst.size(), *done = tile0 + h->inst.size();
  BatchTask *longs = h->tasks, *shorts = h->tasks + h->task_total;
  const unsigned per_inst = (unsigned)std::min<uint32_t>(ninst, (uint32_t)h->num_sms * 2u);
  int first = 1;
  auto assign = [&](auto kern, int group) -> km_status {
    if (!(h->groups & (1u << group))) return KM_OK;
    KM_CUDA_TRY(launch_pdl(kern, h->num_sms * ctas, BA_NT, batch_assign_smem<RT>(), h->stream, h->X, dinst, h->ctl, act,
                           tile0, h->C, h->labels, h->objblk, epoch, first, -0.0f));
    first = 0;
    return KM_OK;
  };
  KM_TRY(assign(batch_assign_kernel<RT, 0>, 0));
  KM_TRY(assign(batch_assign_kernel<RT, 1>, 1));
  KM_TRY(assign(batch_assign_kernel<RT, 2>, 2));
  KM_CUDA_TRY(launch_pdl(batch_sort_kernel, per_inst, 32 * BS_WARPS, 0, h->stream, h->X, dinst, h->ctl, act, h->labels,
                         h->perm, h->Cn, longs, shorts));
  KM_CUDA_TRY(launch_pdl(batch_update_kernel, h->num_sms * 2, 32 * BU_WARPS, BLK_SMEM, h->stream, h->ctl, longs,
                         shorts));
  KM_CUDA_TRY(launch_pdl(batch_stop_kernel, per_inst, 256, 0, h->stream, dinst, h->ctl, act, tile0, done, h->C, h->Cn,
                         h->objblk, h->p.tol, maxiter, (uint32_t)RT, h->dout));
  return KM_OK;
}

// All iterations of instances [0, ninst) of dinst, a CTA an instance.
km_status enqueue_batch_small(km_batch* h, const BatchInst* dinst, uint32_t ninst, uint64_t maxiter) {
  KM_CUDA_TRY(cudaMemsetAsync(h->ctl, 0, sizeof(BatchCtl), h->stream));
  const unsigned ctas = (unsigned)std::min<uint64_t>(ninst, (uint64_t)h->num_sms * h->small_ctas);
  batch_small_kernel<<<ctas, SM_NT, h->small_smem, h->stream>>>(h->X, dinst, ninst, h->ctl, h->C0, h->C, h->labels,
                                                                h->perm, h->objblk, h->p.tol, maxiter, h->dout);
  KM_CUDA_TRY(cudaGetLastError());
  return KM_OK;
}

// The same by tile variant v, all instances an iteration at a time.
km_status enqueue_batch_tiles(km_batch* h, int v, const BatchInst* dinst, uint32_t ninst, uint64_t maxiter) {
  const BatchVariant& V = kVariants[v];
  const size_t total = h->inst.size();
  KM_CUDA_TRY(cudaMemcpyAsync(h->C, h->C0, sizeof(float) * h->c_total, cudaMemcpyDeviceToDevice, h->stream));
  batch_begin_kernel<<<1, 1024, 0, h->stream>>>(dinst, h->ctl, h->lists, h->lists + total, h->lists + 2 * total,
                                                ninst, (uint32_t)V.rt);
  KM_CUDA_TRY(cudaGetLastError());
  // A few iterations are queued between looks at the device's count of
  // running instances (launches past the end find none and return).
  uint64_t done = 0, step = 2;
  while (done < maxiter) {
    const uint64_t target = std::min<uint64_t>(maxiter, done + step);
    for (; done < target; ++done)
      KM_TRY(V.rt == 8 ? enqueue_batch_iteration<8>(h, V.ctas, dinst, ninst, maxiter, (uint32_t)done + 1u)
                       : enqueue_batch_iteration<4>(h, V.ctas, dinst, ninst, maxiter, (uint32_t)done + 1u));
    if (done >= maxiter) break;
    KM_CUDA_TRY(cudaMemcpyAsync(h->h_ctl, h->ctl, sizeof(BatchCtl), cudaMemcpyDeviceToHost, h->stream));
    KM_CUDA_TRY(cudaStreamSynchronize(h->stream));
    if (h->h_ctl->nact == 0u || h->h_ctl->err) break;
    step = 4;
  }
  return KM_OK;
}

// Runs instances [0, ninst) of dinst to their ends (v: tile variant; SMALL: a CTA an instance).
constexpr int SMALL = -1;
km_status run_batch(km_batch* h, int v, const BatchInst* dinst, uint32_t ninst, uint64_t maxiter,
                    float* ms_out) {
  cudaEvent_t e0, e1;
  KM_CUDA_TRY(cudaEventCreate(&e0));
  if (cudaEventCreate(&e1) != cudaSuccess) { cudaEventDestroy(e0); return KM_ERR_CUDA; }
  auto body = [&]() -> km_status {
    KM_CUDA_TRY(cudaEventRecord(e0, h->stream));
    KM_TRY(v == SMALL ? enqueue_batch_small(h, dinst, ninst, maxiter) : enqueue_batch_tiles(h, v, dinst, ninst, maxiter));
    KM_CUDA_TRY(cudaEventRecord(e1, h->stream));
    KM_CUDA_TRY(cudaMemcpyAsync(h->h_ctl, h->ctl, sizeof(BatchCtl), cudaMemcpyDeviceToHost, h->stream));
    KM_CUDA_TRY(cudaStreamSynchronize(h->stream));
    KM_TRY(status_of_device_error(h->h_ctl->err));
    float ms = 0.f;
    KM_CUDA_TRY(cudaEventElapsedTime(&ms, e0, e1));
    if (ms_out) *ms_out = ms;
    return KM_OK;
  };
  const km_status s = body();
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  return s;
}

}  // namespace

extern "C" {

km_status km_batch_create(const km_batch_params* p, const km_batch_problem* probs, km_batch** out) {
  if (!p || !probs || !out || p->problems == 0 || p->restarts == 0 || p->maxiter == 0 || !(p->tol >= 0.0f))
    return KM_ERR_ARG;
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) { (void)cudaGetLastError(); return KM_ERR_NO_DEVICE; }
  km_batch* h = new (std::nothrow) km_batch();
  if (!h) return KM_ERR_ALLOC;
  h->p = *p;
  h->device = p->device;
  h->probs.assign(probs, probs + p->problems);
  uint64_t xoff = 0;
  for (const km_batch_problem& q : h->probs) {
    if (q.n == 0 || q.d == 0 || q.k == 0 || q.k > q.n || q.k > 256 || q.n >= (1ull << 31)) { delete h; return KM_ERR_ARG; }
    const uint32_t kpad = (q.k + 31) / 32 * 32;
    if ((uint64_t)q.d * kpad * 4 > BATCH_MAX_SMEM_C) { delete h; return KM_ERR_UNSUPPORTED; }
    xoff += q.n * q.d;
  }
  h->x_floats = xoff;
  // instances by group of assign shapes, then in LPT order (n*k*d descending,
  // then problem, restart)
  uint64_t px = 0;
  std::vector<BatchInst> inst;
  for (uint32_t pi = 0; pi < p->problems; ++pi) {
    const km_batch_problem& q = h->probs[pi];
    for (uint32_t r = 0; r < p->restarts; ++r) {
      BatchInst I{};
      I.xoff = px; I.n = (uint32_t)q.n; I.d = q.d; I.k = q.k;
      I.prob = pi; I.restart = r;
      inst.push_back(I);
    }
    px += q.n * q.d;
  }
  std::stable_sort(inst.begin(), inst.end(), [](const BatchInst& a, const BatchInst& b) {
    const uint32_t ga = batch_group(a.k), gb = batch_group(b.k);
    return ga != gb ? ga < gb : (uint64_t)a.n * a.k * a.d > (uint64_t)b.n * b.k * b.d;
  });
  for (const BatchInst& I : inst) h->groups |= 1u << batch_group(I.k);
  uint64_t loff = 0, coff = 0, tasks = 0, toff = 0;
  for (BatchInst& I : inst) {
    I.loff = loff; I.coff = coff; I.toff = toff;
    loff += I.n;
    coff += ((uint64_t)I.k * I.d + 3) / 4 * 4;              // 16-byte aligned centroids
    tasks += (uint64_t)I.k * ((I.d + 31) / 32);
    toff += (I.n + 31) / 32;
  }
  h->lab_total = loff;
  h->c_total = coff;
  h->task_total = tasks;
  h->t_total = toff;
  h->inst = inst;
  km_status s = KM_OK;
  if (cudaSetDevice(h->device) != cudaSuccess) { (void)cudaGetLastError(); delete h; return KM_ERR_CUDA; }
  cudaDeviceGetAttribute(&h->num_sms, cudaDevAttrMultiProcessorCount, h->device);
  h->small = batch_is_small(inst, h->num_sms, &h->small_smem);
  if (p->stream) h->stream = static_cast<cudaStream_t>(p->stream);
  else if (cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) == cudaSuccess) h->own_stream = true;
  else { (void)cudaGetLastError(); delete h; return KM_ERR_CUDA; }
  if (s == KM_OK) s = balloc(&h->X, h->x_floats);
  if (s == KM_OK) s = balloc(&h->C0, h->c_total);
  if (s == KM_OK) s = balloc(&h->C, h->c_total);
  if (s == KM_OK) s = balloc(&h->Cn, h->c_total);
  if (s == KM_OK) s = balloc(&h->labels, h->lab_total);
  if (s == KM_OK) s = balloc(&h->perm, h->lab_total);
  if (s == KM_OK) s = balloc(&h->tasks, 2 * h->task_total);
  if (s == KM_OK) s = balloc(&h->objblk, h->t_total);
  if (s == KM_OK) s = balloc(&h->dinst, inst.size());
  if (s == KM_OK) s = balloc(&h->dout, inst.size());
  if (s == KM_OK) s = balloc(&h->ctl, 1);
  if (s == KM_OK) s = balloc(&h->lists, 3 * inst.size());
  if (s == KM_OK && cudaMallocHost(reinterpret_cast<void**>(&h->h_ctl), sizeof(BatchCtl)) != cudaSuccess)
    s = KM_ERR_ALLOC;
  if (s == KM_OK && cudaMemcpyAsync(h->dinst, inst.data(), sizeof(BatchInst) * inst.size(), cudaMemcpyHostToDevice,
                                    h->stream) != cudaSuccess) s = KM_ERR_CUDA;
  if (s == KM_OK) {
    cudaError_t e = cudaFuncSetAttribute(batch_update_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BLK_SMEM);
    for (auto kern : {batch_assign_kernel<8, 0>, batch_assign_kernel<8, 1>, batch_assign_kernel<8, 2>})
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)batch_assign_smem<8>());
    for (auto kern : {batch_assign_kernel<4, 0>, batch_assign_kernel<4, 1>, batch_assign_kernel<4, 2>})
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)batch_assign_smem<4>());
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(batch_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BATCH_SMALL_SMEM);
    if (e == cudaSuccess && h->small)
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&h->small_ctas, batch_small_kernel, SM_NT, h->small_smem);
    if (e != cudaSuccess || h->small_ctas < 1) s = KM_ERR_CUDA;
  }
  if (s != KM_OK) { (void)cudaGetLastError(); delete h; return s; }
  *out = h;
  return KM_OK;
}

km_status km_batch_set_data(km_batch* h, const float* X_host) {
  if (!h || !X_host) return KM_ERR_ARG;
  KM_CUDA_TRY(cudaSetDevice(h->device));
  for (uint64_t q = 0; q < h->x_floats; ++q)
    if (!std::isfinite(X_host[q])) return KM_ERR_ARG;
  // seeded sample picks of every instance: restart r of problem p uses seed + p*restarts + r
  std::vector<float> C0(h->c_total);
  std::vector<uint64_t> pxoff(h->probs.size());
  uint64_t px = 0;
  for (size_t pi = 0; pi < h->probs.size(); ++pi) { pxoff[pi] = px; px += h->probs[pi].n * h->probs[pi].d; }
  for (const BatchInst& I : h->inst) {
    const float* Xp = X_host + pxoff[I.prob];
    std::vector<int32_t> picks(I.k);
    const int seed = h->p.seed + (int)(I.prob * h->p.restarts + I.restart);
    if (!host_sample_picks(Xp, I.n, I.d, I.k, seed, picks.data())) return KM_ERR_ARG;
    for (uint32_t c = 0; c < I.k; ++c)
      std::memcpy(C0.data() + I.coff + (uint64_t)c * I.d, Xp + (uint64_t)picks[c] * I.d, sizeof(float) * I.d);
  }
  KM_CUDA_TRY(cudaMemcpyAsync(h->X, X_host, sizeof(float) * h->x_floats, cudaMemcpyHostToDevice, h->stream));
  KM_CUDA_TRY(cudaMemcpyAsync(h->C0, C0.data(), sizeof(float) * h->c_total, cudaMemcpyHostToDevice, h->stream));
  KM_CUDA_TRY(cudaStreamSynchronize(h->stream));
  h->ready = true;
  return KM_OK;
}

km_status km_batch_tune(km_batch* h, int32_t* variant_out, double* ms_per_variant) {
  if (!h) return KM_ERR_ARG;
  if (!h->ready) return KM_ERR_STATE;
  KM_CUDA_TRY(cudaSetDevice(h->device));
  // time every variant on an even sample of the instances, two iterations each
  const uint32_t ninst = (uint32_t)h->inst.size();
  const uint32_t want = std::min<uint32_t>(ninst, (uint32_t)h->num_sms * 2);
  std::vector<BatchInst> sample;
  for (uint32_t s = 0; s < want; ++s) sample.push_back(h->inst[(uint64_t)s * ninst / want]);
  BatchInst* ds = nullptr;
  KM_TRY(balloc(&ds, sample.size()));
  km_status st = KM_OK;
  if (cudaMemcpyAsync(ds, sample.data(), sizeof(BatchInst) * sample.size(), cudaMemcpyHostToDevice, h->stream) !=
      cudaSuccess) st = KM_ERR_CUDA;
  int best = -1;
  double bms = 0;
  const int nv = (int)(sizeof(kVariants) / sizeof(kVariants[0]));
  for (int v = 0; v < nv && st == KM_OK; ++v) {
    float ms = 0.f;
    st = run_batch(h, v, ds, (uint32_t)sample.size(), 2, nullptr);      // warm-up
    if (st == KM_OK) st = run_batch(h, v, ds, (uint32_t)sample.size(), 2, &ms);
    h->tune_ms[v] = ms;
    if (ms_per_variant) ms_per_variant[v] = ms;
    if (st == KM_OK && (best < 0 || ms < bms)) { best = v; bms = ms; }
  }
  cudaFree(ds);
  if (st != KM_OK) return st;
  h->variant = best;
  if (variant_out) *variant_out = best;
  return KM_OK;
}

km_status km_batch_fit(km_batch* h, km_batch_result* results, uint32_t* best_labels, float* best_centroids,
                       double* fit_ms) {
  if (!h) return KM_ERR_ARG;
  if (!h->ready) return KM_ERR_STATE;
  KM_CUDA_TRY(cudaSetDevice(h->device));
  float ms = 0.f;
  KM_TRY(run_batch(h, h->small ? SMALL : h->variant, h->dinst, (uint32_t)h->inst.size(), h->p.maxiter, &ms));
  if (fit_ms) *fit_ms = ms;
  std::vector<BatchOut> out(h->inst.size());
  KM_CUDA_TRY(cudaMemcpy(out.data(), h->dout, sizeof(BatchOut) * out.size(), cudaMemcpyDeviceToHost));
  // best restart per problem: lowest objective, then lowest restart
  const uint32_t P = h->p.problems, R = h->p.restarts;
  std::vector<int64_t> best(P, -1);
  for (size_t i = 0; i < h->inst.size(); ++i) {
    const BatchInst& I = h->inst[i];
    if (results) {
      km_batch_result& r = results[(uint64_t)I.prob * R + I.restart];
      r.converged_iter = out[i].converged_iter;
      r.iterations = out[i].iterations;
      r.objective = out[i].objective;
    }
    int64_t& b = best[I.prob];
    if (b < 0 || out[i].objective < out[b].objective ||
        (out[i].objective == out[b].objective && I.restart < h->inst[b].restart))
      b = (int64_t)i;
  }
  uint64_t lo = 0, co = 0;
  for (uint32_t pi = 0; pi < P; ++pi) {
    const BatchInst& I = h->inst[best[pi]];
    if (best_labels)
      KM_CUDA_TRY(cudaMemcpy(best_labels + lo, h->labels + I.loff, sizeof(uint32_t) * I.n, cudaMemcpyDeviceToHost));
    if (best_centroids)
      KM_CUDA_TRY(cudaMemcpy(best_centroids + co, h->C + I.coff, sizeof(float) * I.k * I.d,
                             cudaMemcpyDeviceToHost));
    lo += I.n;
    co += (uint64_t)I.k * I.d;
  }
  return KM_OK;
}

km_status km_batch_instance_labels(km_batch* h, uint32_t problem, uint32_t restart, uint32_t* labels_out,
                                   float* centroids_out) {
  if (!h || problem >= h->p.problems || restart >= h->p.restarts) return KM_ERR_ARG;
  KM_CUDA_TRY(cudaSetDevice(h->device));
  for (const BatchInst& I : h->inst) {
    if (I.prob != problem || I.restart != restart) continue;
    if (labels_out)
      KM_CUDA_TRY(cudaMemcpy(labels_out, h->labels + I.loff, sizeof(uint32_t) * I.n, cudaMemcpyDeviceToHost));
    if (centroids_out)
      KM_CUDA_TRY(cudaMemcpy(centroids_out, h->C + I.coff, sizeof(float) * I.k * I.d, cudaMemcpyDeviceToHost));
    return KM_OK;
  }
  return KM_ERR_ARG;
}

void km_batch_destroy(km_batch* h) { delete h; }

}  // extern "C"
