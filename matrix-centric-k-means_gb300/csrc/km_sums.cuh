// Ordered column sums over gathered rows: the producer and chain halves of the
// shared-memory ring used by the centroid update (update_sums_bulk_kernel, which
// says what bounds it) and by the batched problems' update.
//
// A task is the rows perm[0 .. cnt) of a matrix with row stride d, w <= 32
// columns from x.  Batches of BLK_ROWS rows are numbered through all tasks of a
// CTA (first = the number of the task's first batch), so that the ring runs on
// from one task to the next: batch B uses stage B % BLK_STAGES for the
// (B / BLK_STAGES)-th time and is filled by producer B % PROD.  BLK_STAGES is a
// multiple of PROD, so a stage is always refilled by the same producer, which
// waits on its phases in order (a parity wait can never alias a later phase).
#pragma once

#include "km_internal.cuh"

namespace km {

constexpr int BLK_ROWS = 128, BLK_GRP = 32, BLK_STAGES = 6, BLK_COLS = 32;
static_assert(BLK_ROWS == 4 * BLK_GRP, "the chain warp alternates two register groups over four groups a batch");
constexpr uint64_t BLK_WAIT_NS = 2000000000ull;
constexpr uint32_t BLK_SUSPEND_NS = 2000;       // try_wait suspend hint
constexpr size_t BLK_SMEM = (size_t)BLK_STAGES * BLK_ROWS * BLK_COLS * sizeof(float);

struct SumsRing {
  float* ring;               // [BLK_STAGES][BLK_ROWS][BLK_COLS]
  uint64_t *full, *empty;    // BLK_STAGES barriers each: 32 arrivals (a producer's lanes), one per consumer
  volatile int* abort;
};

// An ordered shared-memory load (kept beside the arithmetic that follows it).
__device__ __forceinline__ float ld_shared_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}

// VEC columns (4 * VEC bytes, aligned to their size), zero-filled when !ok.
template <int VEC>
__device__ __forceinline__ void cp_async_cols(void* smem, const float* gmem, bool ok) {
  const uint32_t bytes = ok ? 4u * VEC : 0u;
  if constexpr (VEC == 4) {
    cp_async16_zfill(smem, gmem, bytes);
  } else if constexpr (VEC == 2) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_u32(smem)), "l"(gmem), "r"(bytes)
                 : "memory");
  } else {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(smem)), "l"(gmem), "r"(bytes)
                 : "memory");
  }
}

// Producer `p` of PROD: the task's batches that are its own.  Columns past w and
// rows past cnt zero-fill.  Returns false when a wait ran out.
template <int VEC, int PROD>
__device__ __forceinline__ bool sums_produce(const SumsRing& R, const float* __restrict__ x,
                                             const uint32_t* __restrict__ perm, uint32_t cnt, uint32_t d, uint32_t w,
                                             uint32_t first, uint32_t p) {
  static_assert(BLK_STAGES % PROD == 0, "a stage must always belong to the same producer");
  constexpr int P = 2;                       // batches of indices prefetched
  constexpr int G = BLK_ROWS / BLK_GRP;
  constexpr int LPR = BLK_COLS / VEC;        // lanes per row
  constexpr int RPI = 32 / LPR;              // rows per copy instruction
  const int lane = threadIdx.x & 31;
  const uint32_t nb = (cnt + BLK_ROWS - 1) / BLK_ROWS;
  const uint32_t p0 = (p + PROD - first % PROD) % PROD;      // first batch of this producer
  uint32_t pq[P][G];
  auto load_idx = [&](uint32_t (&q)[G], uint32_t b) {        // group g of batch b: rows 32 g + lane
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const uint32_t idx = b * BLK_ROWS + (uint32_t)(g * BLK_GRP) + (uint32_t)lane;
      q[g] = (b < nb && idx < cnt) ? perm[idx] : 0u;
    }
  };
#pragma unroll
  for (int i = 0; i < P; ++i) load_idx(pq[i], p0 + (uint32_t)i * PROD);
  const uint32_t sub = (uint32_t)lane / LPR, cv = ((uint32_t)lane % LPR) * (uint32_t)VEC;
  const bool lane_has_cols = cv < w;
  const float* xl = x + cv;
  // Unrolled by P so that pq[i] is consumed in place, P batches after its load
  // was issued (moving a register whose load is in flight would wait).
  for (uint32_t lb0 = 0; p0 + lb0 * PROD < nb; lb0 += P) {
#pragma unroll
    for (int i = 0; i < P; ++i) {
      const uint32_t b = p0 + (lb0 + (uint32_t)i) * PROD;
      if (b >= nb) break;
      const uint32_t s = (first + b) % BLK_STAGES, ph = ((first + b) / BLK_STAGES) & 1u;
      const bool okw = mbar_wait_bounded(&R.empty[s], ph ^ 1u, R.abort, BLK_WAIT_NS, BLK_SUSPEND_NS);
      if (!__all_sync(0xffffffffu, okw)) return false;
      const uint32_t m = min((uint32_t)BLK_ROWS, cnt - b * BLK_ROWS);
#pragma unroll
      for (int g = 0; g < G; ++g) {
        float* dst = R.ring + ((size_t)s * BLK_ROWS + (size_t)(g * BLK_GRP) + sub) * BLK_COLS + cv;
        // All row indices of the group first: each cp.async is an ordered asm
        // statement, so a shuffle placed between two of them would put its
        // latency on every row.
        uint32_t rr[BLK_GRP / RPI];
#pragma unroll
        for (int ii = 0; ii < BLK_GRP / RPI; ++ii)
          rr[ii] = __shfl_sync(0xffffffffu, pq[i][g], ii * RPI + (int)sub);
#pragma unroll
        for (int ii = 0; ii < BLK_GRP / RPI; ++ii) {
          const uint32_t u = (uint32_t)(g * BLK_GRP + ii * RPI) + sub;
          const bool okr = u < m && lane_has_cols;
          const float* src = okr ? xl + (uint64_t)rr[ii] * d : x;
          cp_async_cols<VEC>(dst + (size_t)ii * RPI * BLK_COLS, src, okr);
        }
      }
      cp_async_mbar_arrive_noinc(&R.full[s]);
      load_idx(pq[i], b + (uint32_t)P * PROD);
    }
  }
  return true;
}

// The ordered chain, lane = column: sum = ((+0 + row 0) + row 1) + ...  A group
// of 32 rows is added while the next one is loaded, one load beside each addition
// (32 loads in a block would hold the warp's issue until the shared-memory queue
// took them all); the next batch's barrier is tested a group ahead of its use.
// Rows past the task's end are zero-filled: adding +0 leaves the sum as it is (a
// sum that starts at +0 is never -0).  Returns false when a wait ran out.
__device__ __forceinline__ bool sums_chain(const SumsRing& R, uint32_t cnt, uint32_t first, float& sum) {
  constexpr uint32_t RB = BLK_COLS * 4u, GB = BLK_GRP * RB, SB = BLK_ROWS * RB;   // bytes of a row, group, stage
  const int lane = threadIdx.x & 31;
  const uint32_t nb = (cnt + BLK_ROWS - 1) / BLK_ROWS;
  float va[BLK_GRP], vb[BLK_GRP];
  sum = 0.0f;
  if (nb == 0u) return true;
  auto step = [&](const float (&v)[BLK_GRP], float (&x)[BLK_GRP], uint32_t src) {
#pragma unroll
    for (int u = 0; u < BLK_GRP; ++u) {
      x[u] = ld_shared_f32(src + (uint32_t)u * RB);
      asm volatile("add.rn.f32 %0, %0, %1;" : "+f"(sum) : "f"(v[u]));
    }
  };
  const uint32_t base = smem_u32(R.ring) + (uint32_t)lane * 4u;
  uint32_t s = first % BLK_STAGES, ph = (first / BLK_STAGES) & 1u;
  bool ok = mbar_wait_bounded(&R.full[s], ph, R.abort, BLK_WAIT_NS, BLK_SUSPEND_NS);
  if (!__all_sync(0xffffffffu, ok)) return false;
#pragma unroll
  for (int u = 0; u < BLK_GRP; ++u) va[u] = ld_shared_f32(base + s * SB + (uint32_t)u * RB);
  for (uint32_t left = nb; left; --left) {
    const uint32_t src = base + s * SB;
    const uint32_t sn = s + 1u == (uint32_t)BLK_STAGES ? 0u : s + 1u, phn = sn ? ph : ph ^ 1u;
    step(va, vb, src + GB);
    step(vb, va, src + 2 * GB);
    ok = left == 1u || mbar_test_wait(&R.full[sn], phn);
    step(va, vb, src + 3 * GB);
    if (!__all_sync(0xffffffffu, ok)) {
      ok = mbar_wait_bounded(&R.full[sn], phn, R.abort, BLK_WAIT_NS, BLK_SUSPEND_NS);
      if (!__all_sync(0xffffffffu, ok)) return false;
    }
    // (after the last batch the next stage holds other rows or none: unused)
    step(vb, va, base + sn * SB);
    __syncwarp();
    if (lane == 0) mbar_arrive(&R.empty[s]);
    s = sn;
    ph = phn;
  }
  return true;
}

}  // namespace km
