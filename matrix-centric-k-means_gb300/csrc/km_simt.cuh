// FP32 tile product on the CUDA cores: acc[row][col] = sum over the coordinates in
// ascending order of fma(x, c, acc), for ROWS rows against COLS columns, by NT
// threads as (NT / TX) x TX, each RT rows and CT columns.
//
// Bound by shared memory and the FP32 pipes together: a coordinate costs a thread
// RT * CT products and (RT + CT) * 4 bytes of shared-memory reads, which return 128
// bytes a cycle for the SM whatever they broadcast, against its 128 products: 8 x 8
// needs both all the time, but keeps twelve warps an SM (16 x 8 and 8 x 16 need a
// quarter less, and measured slower with their eight warps).  Two rows go through one
// packed FMA (36 T products/s measured in registers, as scalar, from half the issue
// slots, of which duplicating a column into a pair takes some; scalar FMAs were 10 %
// slower).  The rows are staged transposed (pairs of rows adjacent), the columns
// beside them, both a stage ahead in registers; a coordinate's operands are read
// while the one before is multiplied.
#pragma once

#include "km_internal.cuh"

namespace km {

template <int NT_, int RT_, int TX_, int CT_, int KC_>
struct SimtTile {
  static constexpr int NT = NT_, RT = RT_, TX = TX_, CT = CT_, KC = KC_;
  static constexpr int ROWS = RT * (NT / TX), COLS = CT * TX;
  static constexpr int LDA = ROWS + 4;
  static constexpr int A_FLOATS = KC * LDA, B_FLOATS = KC * COLS, FLOATS = A_FLOATS + B_FLOATS;
  static constexpr size_t SMEM = 2 * sizeof(float) * (size_t)FLOATS;   // two stages
  static constexpr size_t TOT_BYTES = sizeof(float) * (size_t)NT * RT * CT;
  static constexpr int NA = (ROWS * KC + 4 * NT - 1) / (4 * NT);       // float4 loads per thread and stage
  static constexpr int NB = (COLS * KC + 4 * NT - 1) / (4 * NT);
  // Column of this thread's j-th accumulator (ascending in j).
  static __device__ __forceinline__ int col(int tx, int j) {
    return j < 4 * (CT / 4) ? 4 * ((j >> 2) * TX + tx) + (j & 3) : 4 * (CT / 4) * TX + 2 * tx + (j & 1);
  }
};

// Four coordinates of a row (null: zeros; zeros past d).  v4: rows 16-byte aligned
// and d % 4 == 0.
__device__ __forceinline__ float4 simt_load4(const float* row, uint32_t col, uint32_t d, bool v4) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (row) {
    const float* p = row + col;
    if (v4) {
      if (col < d) v = __ldg(reinterpret_cast<const float4*>(p));
    } else {
      if (col + 0 < d) v.x = __ldg(p);
      if (col + 1 < d) v.y = __ldg(p + 1);
      if (col + 2 < d) v.z = __ldg(p + 2);
      if (col + 3 < d) v.w = __ldg(p + 3);
    }
  }
  return v;
}

// The product over all d coordinates.  rowp(r) / colp(c): the tile's row r / column
// c as a pointer to d floats, or null past the end.  Ends with a block barrier.
// RUN > 0: every RUN coordinates start a sum of their own, added in order, so that an
// accumulator's rounding errors are those of a chain of RUN + d / RUN operations
// (simt_chain) instead of d.  The sums so far are kept in shared memory (tot,
// T::TOT_BYTES), which a run of 64 visits for an eighth of the product's own reads.
template <class T, int RUN = 0, class RowP, class ColP>
__device__ __forceinline__ void simt_product(float* smem, uint32_t d, bool v4, RowP rowp, ColP colp,
                                             float2 (&acc)[T::RT / 2][T::CT], float4* tot = nullptr) {
  static_assert(RUN % T::KC == 0 && T::CT % 2 == 0, "whole stages; pairs of accumulators");
  const int tid = threadIdx.x, tx = tid % T::TX, ty = tid / T::TX;
  constexpr int QR = T::KC / 4;                            // float4 per row and stage
  const uint32_t nk = (d + T::KC - 1) / T::KC;
#pragma unroll
  for (int i = 0; i < T::RT / 2; ++i)
#pragma unroll
    for (int j = 0; j < T::CT; ++j) acc[i][j] = make_float2(0.0f, 0.0f);
  static_assert(T::NT % QR == 0, "a thread loads the same coordinates of every row");
  float4 ra[T::NA], rb[T::NB];
  const float *pa[T::NA], *pb[T::NB];                      // this thread's rows and columns (null: zeros)
#pragma unroll
  for (int e = 0; e < T::NA; ++e) {
    const int idx = e * T::NT + tid;
    pa[e] = (T::ROWS * QR % T::NT == 0 || idx < T::ROWS * QR) ? rowp(idx / QR) : nullptr;
  }
#pragma unroll
  for (int e = 0; e < T::NB; ++e) {
    const int idx = e * T::NT + tid;
    pb[e] = (T::COLS * QR % T::NT == 0 || idx < T::COLS * QR) ? colp(idx / QR) : nullptr;
  }
  auto gload = [&](uint32_t kc) {
    const uint32_t c = kc + 4u * (uint32_t)(tid % QR);
#pragma unroll
    for (int e = 0; e < T::NA; ++e) ra[e] = simt_load4(pa[e], c, d, v4);
#pragma unroll
    for (int e = 0; e < T::NB; ++e) rb[e] = simt_load4(pb[e], c, d, v4);
  };
  auto sstore = [&](uint32_t buf) {
    float* A = smem + buf * T::FLOATS;
    float* B = A + T::A_FLOATS;
#pragma unroll
    for (int e = 0; e < T::NA; ++e) {
      const int idx = e * T::NT + tid, r = idx / QR, j = 4 * (idx % QR);
      if (T::ROWS * QR % T::NT == 0 || idx < T::ROWS * QR) {
        A[(j + 0) * T::LDA + r] = ra[e].x;
        A[(j + 1) * T::LDA + r] = ra[e].y;
        A[(j + 2) * T::LDA + r] = ra[e].z;
        A[(j + 3) * T::LDA + r] = ra[e].w;
      }
    }
#pragma unroll
    for (int e = 0; e < T::NB; ++e) {
      const int idx = e * T::NT + tid, c = idx / QR, j = 4 * (idx % QR);
      if (T::COLS * QR % T::NT == 0 || idx < T::COLS * QR) {
        B[(j + 0) * T::COLS + c] = rb[e].x;
        B[(j + 1) * T::COLS + c] = rb[e].y;
        B[(j + 2) * T::COLS + c] = rb[e].z;
        B[(j + 3) * T::COLS + c] = rb[e].w;
      }
    }
  };
  gload(0);
  sstore(0);
  __syncthreads();
  for (uint32_t kt = 0; kt < nk; ++kt) {
    const float* A = smem + (kt & 1u) * T::FLOATS + ty * T::RT;
    const float* B = smem + (kt & 1u) * T::FLOATS + T::A_FLOATS + 4 * tx;
    if (kt + 1 < nk) gload((kt + 1) * T::KC);
    const uint32_t left = d - kt * T::KC;                  // zeros up to a multiple of 4
    float2 a[2][T::RT / 2];
    float b[2][T::CT];
    auto fetch = [&](int f, uint32_t kk) {
      const float* a_ = A + kk * T::LDA;
      const float* b_ = B + kk * T::COLS;
#pragma unroll
      for (int i = 0; i < T::RT / 4; ++i) {
        const float4 v = *reinterpret_cast<const float4*>(a_ + 4 * i);
        a[f][2 * i] = make_float2(v.x, v.y);
        a[f][2 * i + 1] = make_float2(v.z, v.w);
      }
#pragma unroll
      for (int j = 0; j < T::CT / 4; ++j) {
        const float4 v = *reinterpret_cast<const float4*>(b_ + 4 * T::TX * j);
        b[f][4 * j] = v.x; b[f][4 * j + 1] = v.y; b[f][4 * j + 2] = v.z; b[f][4 * j + 3] = v.w;
      }
      if constexpr (T::CT % 4 == 2) {
        const float2 v = *reinterpret_cast<const float2*>(b_ + 4 * (T::CT / 4) * T::TX - 2 * tx);
        b[f][T::CT - 2] = v.x; b[f][T::CT - 1] = v.y;
      }
    };
    auto multiply = [&](int f) {
#pragma unroll
      for (int j = 0; j < T::CT; ++j)
#pragma unroll
        for (int i = 0; i < T::RT / 2; ++i)
          acc[i][j] = __ffma2_rn(a[f][i], make_float2(b[f][j], b[f][j]), acc[i][j]);
    };
    fetch(0, 0);
#pragma unroll 1
    for (uint32_t kk = 0; kk < (uint32_t)T::KC && kk < left; kk += 4) {
      fetch(1, kk + 1);
      multiply(0);
      fetch(0, kk + 2);
      multiply(1);
      fetch(1, kk + 3);
      multiply(0);
      fetch(0, min(kk + 4u, (uint32_t)T::KC - 1u));          // (past the stage: not used)
      multiply(1);
    }
    if (kt + 1 < nk) sstore((kt + 1) & 1u);
    if constexpr (RUN > 0) {                               // (a thread's own slots: no barrier)
      const bool end = kt + 1 == nk;
      if (end ? nk > RUN / T::KC : (kt + 1) % (RUN / T::KC) == 0) {
        const bool first = kt < RUN / T::KC;
#pragma unroll
        for (int i = 0; i < T::RT / 2; ++i)
#pragma unroll
          for (int j = 0; j < T::CT; j += 2) {
            float4* const t = tot + (i * (T::CT / 2) + j / 2) * T::NT + tid;
            float4 v = first ? make_float4(0.0f, 0.0f, 0.0f, 0.0f) : *t;
            v.x = __fadd_rn(v.x, acc[i][j].x); v.y = __fadd_rn(v.y, acc[i][j].y);
            v.z = __fadd_rn(v.z, acc[i][j + 1].x); v.w = __fadd_rn(v.w, acc[i][j + 1].y);
            if (end) {
              acc[i][j] = make_float2(v.x, v.y);
              acc[i][j + 1] = make_float2(v.z, v.w);
            } else {
              *t = v;
              acc[i][j] = acc[i][j + 1] = make_float2(0.0f, 0.0f);
            }
          }
      }
    }
    __syncthreads();
  }
}

}  // namespace km
