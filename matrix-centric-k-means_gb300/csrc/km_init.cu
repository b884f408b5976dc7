// Greedy k-means++ initialisation on the device (the reference's
// init_centroids_plus_plus, src/kmeans.cu:447-769, compiled there behind
// PLUSPLUS): the first centroid is a uniformly drawn point; every further
// round draws s = 2 + ceil(ln k) candidate points with probability
// proportional to their current squared distance to the chosen set
// (raft::random::discrete over min_distances, :585-588), computes for each
// candidate the cost sum_i min(d2_i, ||x_i - x_cand||^2) (:681-693), keeps the
// cheapest (lowest index on equal cost, cub ArgMin :697-715) and updates d2
// with its distances (:721-724).  The reference seeds its generators from
// std::random_device; here the draws come from the caller's seed
// (std::mt19937_64), so the result is reproducible, and every sum has a fixed
// order, so the same seed gives the same centroids on every run.
//
// Two launches a round: distances and costs of the candidates, whose last block
// chooses; the update of d2 and of its chunk sums, whose last block draws the next
// round's candidates.  bsum[b] is the FP64 sum of d2 over the PP_CHUNK rows of
// chunk b, which the sampler walks to find the chunk holding a draw and then scans
// inside the chunk.  Distances are FP32, ||x - c||^2 with partial sums over the
// columns l, l + 32, ... (l = 0..31) added in a fixed tree: bit 4 of l, then bits 3
// to 0, as a 32-lane exchange would add them.
#include "km_lloyd.cuh"

#include <algorithm>
#include <cmath>
#include <random>
#include <vector>

namespace km {

constexpr uint32_t PP_CHUNK = 1024;
constexpr uint32_t PP_MAX_S = 16;
constexpr uint32_t PP_TILE_MAX_D = 256;    // widest rows of the tiled cost kernel: 128 of them fill shared memory
constexpr uint32_t PP_WIDE_ROWS = 256;     // rows of a block of the other

__device__ __forceinline__ uint64_t umin64(uint64_t a, uint64_t b) { return a < b ? a : b; }

// The device state of one seeding.
struct PpState {
  uint32_t ticket;      // blocks done in this launch (the last one resets it)
  int32_t best;         // chosen candidate of the round
};

// True in the block that finishes last; the other blocks' results are then
// visible to reads past L1 (__ldcg).
__device__ __forceinline__ bool pp_last_block(PpState* st, int* flag) {
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) *flag = (atomicAdd(&st->ticket, 1u) == gridDim.x - 1u) ? 1 : 0;
  __syncthreads();
  if (!*flag) return false;
  __threadfence();
  if (threadIdx.x == 0) st->ticket = 0u;
  return true;
}

// Inclusive FP64 scan over the lanes.
__device__ __forceinline__ double pp_scan(double v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  return v;
}

// One warp draws a row ~ d2 / sum(d2) for the uniform u: the chunk holding
// u * sum, then the row inside it, each found by the lanes' runs of consecutive
// values (one scan) and then the values of one run (another).  Rounding at a top
// end takes the last positive value.  Bound by the latency of four loads and four
// scans: the update launch with the draws of 7 candidates at n = 262,144 takes 14
// us (24 us with a scan of every 32 values in turn; 27 us for the draws alone as a
// launch of their own, with the loads between the scans).
__device__ int32_t pp_draw(const float* d2, uint64_t n, const double* bsum, uint32_t nblk, double u) {
  const int lane = threadIdx.x & 31;
  const uint32_t R = (nblk + 31u) / 32u;                       // chunks per lane
  const uint32_t b0 = min(nblk, (uint32_t)lane * R), b1 = min(nblk, b0 + R);
  double own = 0.0;
  for (uint32_t b = b0; b < b1; b += 8) {
    double v[8];
#pragma unroll
    for (int g = 0; g < 8; ++g) v[g] = b + g < b1 ? __ldcg(bsum + b + g) : 0.0;
    own += ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
  }
  double inc = pp_scan(own);
  const double tot = __shfl_sync(0xffffffffu, inc, 31);
  // every point coincides with a chosen one: uniform draw
  if (!(tot > 0.0)) return (int32_t)umin64(n - 1, (uint64_t)(u * (double)n));
  double target = u * tot;
  bool top = false;                                            // rounding at the top end
  unsigned hit = __ballot_sync(0xffffffffu, own > 0.0 && inc > target);
  if (!hit) { hit = 0x80000000u >> __clz(__ballot_sync(0xffffffffu, own > 0.0)); top = true; }
  int L = __ffs(hit) - 1;
  target -= __shfl_sync(0xffffffffu, inc - own, L);
  const uint32_t run0 = (uint32_t)L * R, run1 = min(nblk, run0 + R);
  uint32_t blk = run0;
  double base = 0.0;
  bool found = false;
  for (uint32_t g = run0; g < run1 && !found; g += 32u) {
    const uint32_t b = g + (uint32_t)lane;
    const double v = b < run1 ? __ldcg(bsum + b) : 0.0;
    inc = pp_scan(v);
    const unsigned h = __ballot_sync(0xffffffffu, !top && v > 0.0 && base + inc > target);
    const unsigned pos = __ballot_sync(0xffffffffu, v > 0.0);
    if (h) {
      L = __ffs(h) - 1;
      blk = g + (uint32_t)L;
      target -= __shfl_sync(0xffffffffu, base + inc - v, L);
      found = true;
    } else {
      if (pos) blk = g + 31u - (uint32_t)__clz(pos);
      base += __shfl_sync(0xffffffffu, inc, 31);
    }
  }
  top = !found;
  // row inside the chunk: 32 consecutive rows per lane (float4: a chunk starts
  // 16-byte aligned)
  const uint64_t r0 = (uint64_t)blk * PP_CHUNK, r1 = umin64(n, r0 + PP_CHUNK), l0 = r0 + 32u * (uint32_t)lane;
  double s4[4] = {0.0, 0.0, 0.0, 0.0};
  if (l0 + 32u <= r1) {
    float4 w[8];
#pragma unroll
    for (int g = 0; g < 8; ++g) w[g] = __ldcg(reinterpret_cast<const float4*>(d2 + l0) + g);
#pragma unroll
    for (int g = 0; g < 8; ++g) {
      s4[0] += (double)w[g].x; s4[1] += (double)w[g].y; s4[2] += (double)w[g].z; s4[3] += (double)w[g].w;
    }
  } else {
    for (uint64_t i = l0; i < r1; ++i) s4[0] += (double)__ldcg(d2 + i);
  }
  own = (s4[0] + s4[1]) + (s4[2] + s4[3]);
  inc = pp_scan(own);
  hit = __ballot_sync(0xffffffffu, !top && own > 0.0 && inc > target);
  if (!hit) {
    const unsigned pos = __ballot_sync(0xffffffffu, own > 0.0);
    hit = pos ? 0x80000000u >> __clz(pos) : 1u;
    top = true;
  }
  L = __ffs(hit) - 1;
  target -= __shfl_sync(0xffffffffu, inc - own, L);
  const uint64_t i = r0 + 32u * (uint32_t)L + (uint32_t)lane;
  const double v = i < r1 ? (double)__ldcg(d2 + i) : 0.0;
  inc = pp_scan(v);
  const unsigned h = __ballot_sync(0xffffffffu, !top && v > 0.0 && inc > target);
  const unsigned pos = __ballot_sync(0xffffffffu, v > 0.0);
  const int at = h ? __ffs(h) - 1 : pos ? 31 - __clz(pos) : 0;
  return (int32_t)(r0 + 32u * (uint32_t)L + (uint32_t)at);
}

// The last block's warps draw the s candidates of a round.
__device__ __forceinline__ void pp_draw_all(const float* d2, uint64_t n, const double* bsum, uint32_t nblk,
                                            const double* u, uint32_t s, int32_t* cand) {
  const uint32_t warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (uint32_t j = warp; j < s; j += nw) {
    const int32_t pick = pp_draw(d2, n, bsum, nblk, u[j]);
    if ((threadIdx.x & 31) == 0) cand[j] = pick;
  }
}

// d2_i = ||x_i - x_first||^2; bsum per chunk; draws the first candidates (u
// non-null).
__global__ void __launch_bounds__(256)
pp_first_kernel(const float* __restrict__ X, uint64_t n, uint32_t d, uint64_t first,
                float* d2, double* bsum, PpState* st, const double* __restrict__ u, uint32_t s, int32_t* cand) {
  __shared__ double red[8];
  __shared__ int flag;
  const uint64_t r0 = (uint64_t)blockIdx.x * PP_CHUNK;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float* c = X + first * d;
  double acc = 0.0;
  for (uint32_t t = warp; t < PP_CHUNK; t += 8) {
    const uint64_t i = r0 + t;
    if (i >= n) break;
    const float* x = X + i * d;
    float s = 0.0f;
    for (uint32_t j = lane; j < d; j += 32) {
      const float u = x[j] - c[j];
      s = fmaf(u, u, s);
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) { d2[i] = s; acc += (double)s; }
  }
  if (lane == 0) red[warp] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < 8; ++w) t += red[w];
    bsum[blockIdx.x] = t;
  }
  if (pp_last_block(st, &flag) && u) pp_draw_all(d2, n, bsum, gridDim.x, u, s, cand);
}

// The last block of a cost launch: total cost per candidate over the blocks'
// partial sums, the cheapest (lowest index on ties) becomes centroid number r.
__device__ void pp_choose(const double* cpart, uint32_t nblk, uint32_t s, const int32_t* cand, uint32_t r,
                          int32_t* chosen, PpState* st, double* sh) {
  const uint32_t warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int lane = threadIdx.x & 31;
  for (uint32_t j = warp; j < s; j += nw) {
    double t = 0.0;
    for (uint32_t b0 = 0; b0 < nblk; b0 += 32 * 8) {
      double v[8];
#pragma unroll
      for (int g = 0; g < 8; ++g) {
        const uint32_t b = b0 + 32u * g + lane;
        v[g] = b < nblk ? __ldcg(cpart + (uint64_t)j * nblk + b) : 0.0;
      }
#pragma unroll
      for (int g = 0; g < 8; ++g) t += v[g];
    }
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) sh[j] = t;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t bj = 0;
    for (uint32_t j = 1; j < s; ++j)
      if (sh[j] < sh[bj]) bj = j;
    chosen[r] = cand[bj];
    st->best = (int32_t)bj;
  }
}

// The tree over the partial sums of columns l = V mod 2^K: S distances of one row
// in packed pairs, the row in xs (columns LD floats apart), the candidates negated
// in cs[column][S].
template <int S, int K, int V>
__device__ __forceinline__ void pp_tree(const float* xs, int LD, const float* cs, uint32_t d, float2 (&out)[S / 2]) {
  if constexpr (K == 5) {
#pragma unroll
    for (int c = 0; c < S / 2; ++c) out[c] = make_float2(0.0f, 0.0f);
#pragma unroll 1
    for (uint32_t j = V; j < d; j += 32) {
      const float2 x = make_float2(xs[j * LD], xs[j * LD]);
#pragma unroll
      for (int q = 0; q < S / 4; ++q) {
        const float4 c4 = *reinterpret_cast<const float4*>(cs + j * S + 4 * q);
        const float2 u = __fadd2_rn(x, make_float2(c4.x, c4.y)), w = __fadd2_rn(x, make_float2(c4.z, c4.w));
        out[2 * q] = __ffma2_rn(u, u, out[2 * q]);
        out[2 * q + 1] = __ffma2_rn(w, w, out[2 * q + 1]);
      }
    }
  } else {
    pp_tree<S, K + 1, V>(xs, LD, cs, d, out);
    float2 t[S / 2];
    pp_tree<S, K + 1, V + (1 << K)>(xs, LD, cs, d, t);
#pragma unroll
    for (int c = 0; c < S / 2; ++c) out[c] = __fadd2_rn(out[c], t[c]);
  }
}

// a + b = s + e without a rounding (TwoSum); s is returned.
__device__ __forceinline__ float pp_two_sum(float a, float b, float& e) {
  const float s = __fadd_rn(a, b), bp = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bp)), __fsub_rn(b, bp));
  return s;
}

// h + l + m <- h + l + m + a, an unevaluated sum of three FP32 parts: FP64
// additions are slow on this GPU, and a sum of two parts (48 bits) would hold
// less than FP64's 53.  Only the additions into m, 2^-48 of the sum, round.
__device__ __forceinline__ void pp_sum_add(float& h, float& l, float& m, float a) {
  float e, f;
  h = pp_two_sum(h, a, e);
  l = pp_two_sum(l, e, f);
  m = __fadd_rn(m, f);
}

// D[j][i] = ||x_i - x_cand_j||^2 and the block's costs sum_i min(d2_i, D[j][i]) (three
// FP32 parts, rounded once to FP64), d <= PP_TILE_MAX_D: a thread per row for all candidates, the rows staged
// transposed in shared memory.  Bound by the FP32 pipes (two operations an element
// and candidate, 31 a row and candidate for the tree) and by reading X.  A warp per
// row instead spends most of its instructions exchanging partial sums: n = 262,144
// d = 32, 7 candidates 336 us, now 23 us (46 us with FP64 cost sums in every warp).
template <int S>
__global__ void __launch_bounds__(256)
pp_cost_kernel(const float* __restrict__ X, uint64_t n, uint32_t d, bool v4, const int32_t* cand, uint32_t s,
               const float* __restrict__ d2, float* __restrict__ D, double* cpart, PpState* st, uint32_t r,
               int32_t* chosen) {
  griddep_wait();
  extern __shared__ __align__(16) float pp_smem[];
  __shared__ double tot[S];
  __shared__ int flag;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t rows = blockDim.x, LD = rows + 1u;
  float* cs = pp_smem;                             // [d][S], zeros past s
  float* xs = pp_smem + (size_t)d * S;             // [d][LD]
  for (uint32_t t = tid; t < S * d; t += rows) {
    const uint32_t c = t / d, j = t % d;
    cs[j * S + c] = c < s ? -X[(uint64_t)cand[c] * d + j] : 0.0f;
  }
  const uint64_t r0 = (uint64_t)blockIdx.x * rows;
  const uint32_t nr = (uint32_t)umin64(rows, n - r0);
  const float* xb = X + r0 * d;
  if (v4) {                                        // 16-byte loads: d % 4 == 0 and X 16-byte aligned
    const uint32_t d4 = d / 4u;
    uint32_t rr = (uint32_t)tid / d4, cc = (uint32_t)tid % d4;
    const uint32_t dr = rows / d4, dc = rows % d4;
#pragma unroll 4
    for (uint32_t t = tid; t < nr * d4; t += rows) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(xb) + t);
      float* x = xs + 4u * cc * LD + rr;
      x[0] = v.x; x[LD] = v.y; x[2 * LD] = v.z; x[3 * LD] = v.w;
      rr += dr;
      cc += dc;
      if (cc >= d4) { cc -= d4; ++rr; }
    }
  } else {
    uint32_t rr = (uint32_t)tid / d, cc = (uint32_t)tid % d;
    const uint32_t dr = rows / d, dc = rows % d;
#pragma unroll 8
    for (uint32_t t = tid; t < nr * d; t += rows) {
      xs[cc * LD + rr] = __ldg(xb + t);
      rr += dr;
      cc += dc;
      if (cc >= d) { cc -= d; ++rr; }
    }
  }
  __syncthreads();
  const bool valid = (uint32_t)tid < nr;
  float2 v[S / 2];
  pp_tree<S, 0, 0>(xs + (valid ? tid : 0), (int)LD, cs, d, v);
  const float old = valid ? d2[r0 + tid] : 0.0f;
  __syncthreads();                                 // the staged rows are done with
  float* const mins = xs;                          // [s][rows]
#pragma unroll
  for (int c = 0; c < S; ++c) {
    if ((uint32_t)c >= s) break;
    const float vc = (c & 1) ? v[c / 2].y : v[c / 2].x;
    if (valid) D[(uint64_t)c * n + r0 + tid] = vc;
    mins[c * rows + tid] = valid ? fminf(vc, old) : 0.0f;
  }
  __syncthreads();
  // a warp per candidate: each lane every 32nd row, then the lanes
  for (uint32_t c = (uint32_t)warp; c < s; c += rows / 32u) {
    float h = 0.0f, l = 0.0f, m = 0.0f;
    for (uint32_t t = (uint32_t)lane; t < rows; t += 32u) pp_sum_add(h, l, m, mins[c * rows + t]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ho = __shfl_xor_sync(0xffffffffu, h, o), lo = __shfl_xor_sync(0xffffffffu, l, o);
      const float mo = __shfl_xor_sync(0xffffffffu, m, o);
      pp_sum_add(h, l, m, ho);
      float e;
      l = pp_two_sum(l, lo, e);
      m = __fadd_rn(m, __fadd_rn(mo, e));
    }
    double t = (double)h + ((double)l + (double)m);
    if (__any_sync(0xffffffffu, !isfinite(h))) {     // past the FP32 range: the sum in FP64
      t = 0.0;
      for (uint32_t q = (uint32_t)lane; q < rows; q += 32u) t += (double)mins[c * rows + q];
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    }
    if (lane == 0) cpart[(uint64_t)c * gridDim.x + blockIdx.x] = t;
  }
  if (pp_last_block(st, &flag)) pp_choose(cpart, gridDim.x, s, cand, r, chosen, st, tot);
}

// The same for wider rows: a warp per row, lanes over the columns.  Lane r keeps the
// distances of the r-th of the warp's 32 rows, so that they are stored and summed 32 rows
// at a time (one lane storing each row's alone touches a line per candidate); 256 rows a
// block, so that a few thousand rows reach more than a few SMs.  Seeding, n = 2000 d = 300
// k = 10 6.0 -> 1.9 ms, n = 100,000 d = 512 k = 50 74 -> 22 (1024 rows a block).
__global__ void __launch_bounds__(256)
pp_cost_wide_kernel(const float* __restrict__ X, uint64_t n, uint32_t d, const int32_t* cand,
                    uint32_t s, const float* __restrict__ d2, float* __restrict__ D,
                    double* cpart, PpState* st, uint32_t r, int32_t* chosen) {
  griddep_wait();
  extern __shared__ float cs[];                    // s x d candidate rows
  __shared__ double red[8][PP_MAX_S];
  __shared__ double tot[PP_MAX_S];
  __shared__ int flag;
  for (uint32_t t = threadIdx.x; t < s * d; t += blockDim.x) {
    const uint32_t j = t / d, c = t % d;
    cs[t] = X[(uint64_t)cand[j] * d + c];
  }
  __syncthreads();
  const uint64_t r0 = (uint64_t)blockIdx.x * PP_WIDE_ROWS + 32u * (uint32_t)(threadIdx.x >> 5);   // the warp's rows
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double acc[PP_MAX_S];
#pragma unroll
  for (uint32_t j = 0; j < PP_MAX_S; ++j) acc[j] = 0.0;
  float keep[PP_MAX_S];
#pragma unroll
  for (uint32_t j = 0; j < PP_MAX_S; ++j) keep[j] = 0.0f;
  for (int r = 0; r < 32; ++r) {
    const uint64_t i = r0 + (uint32_t)r;
    if (i >= n) break;
    const float* x = X + i * d;
    float p[PP_MAX_S];
#pragma unroll
    for (uint32_t j = 0; j < PP_MAX_S; ++j) p[j] = 0.0f;
    for (uint32_t c = lane; c < d; c += 32) {
      const float xv = x[c];
#pragma unroll
      for (uint32_t j = 0; j < PP_MAX_S; ++j) {
        if (j < s) {
          const float u = xv - cs[j * d + c];
          p[j] = fmaf(u, u, p[j]);
        }
      }
    }
#pragma unroll
    for (uint32_t j = 0; j < PP_MAX_S; ++j) {
      if (j < s) {
        float v = p[j];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        keep[j] = lane == r ? v : keep[j];
      }
    }
  }
  const uint64_t i = r0 + (uint32_t)lane;
  if (i < n) {
    const float old = d2[i];
#pragma unroll
    for (uint32_t j = 0; j < PP_MAX_S; ++j) {
      if (j < s) {
        D[(uint64_t)j * n + i] = keep[j];
        acc[j] += (double)fminf(keep[j], old);
      }
    }
  }
#pragma unroll
  for (uint32_t j = 0; j < PP_MAX_S; ++j)
    if (j < s)
      for (int o = 16; o > 0; o >>= 1) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
  if (lane == 0) {
#pragma unroll
    for (uint32_t j = 0; j < PP_MAX_S; ++j) red[warp][j] = acc[j];
  }
  __syncthreads();
  if (threadIdx.x < s) {
    double t = 0.0;
    for (int w = 0; w < 8; ++w) t += red[w][threadIdx.x];
    cpart[(uint64_t)threadIdx.x * gridDim.x + blockIdx.x] = t;
  }
  if (pp_last_block(st, &flag)) pp_choose(cpart, gridDim.x, s, cand, r, chosen, st, tot);
}

// d2_i = min(d2_i, D[best][i]); bsum per chunk; draws the next round's candidates
// (u non-null).
__global__ void __launch_bounds__(256)
pp_update_kernel(const float* __restrict__ D, uint64_t n, PpState* st, float* d2, double* bsum,
                 const double* __restrict__ u, uint32_t s, int32_t* cand) {
  griddep_wait();
  __shared__ double red[8];
  __shared__ int flag;
  const uint64_t r0 = (uint64_t)blockIdx.x * PP_CHUNK;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float* Db = D + (uint64_t)st->best * n;
  double acc = 0.0;
  float v[PP_CHUNK / 256];
#pragma unroll
  for (int q = 0; q < (int)PP_CHUNK / 256; ++q) {
    const uint64_t i = r0 + threadIdx.x + 256u * q;
    v[q] = i < n ? fminf(d2[i], Db[i]) : 0.0f;
  }
#pragma unroll
  for (int q = 0; q < (int)PP_CHUNK / 256; ++q) {
    const uint64_t i = r0 + threadIdx.x + 256u * q;
    if (i < n) {
      d2[i] = v[q];
      acc += (double)v[q];
    }
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) red[warp] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < 8; ++w) t += red[w];
    bsum[blockIdx.x] = t;
  }
  if (pp_last_block(st, &flag) && u) pp_draw_all(d2, n, bsum, gridDim.x, u, s, cand);
}

__global__ void pp_gather_kernel(const float* __restrict__ X, uint32_t d, const int32_t* __restrict__ idx,
                                 uint32_t k, float* __restrict__ C) {
  const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (uint64_t)k * d) return;
  const uint32_t r = (uint32_t)(t / d), j = (uint32_t)(t % d);
  C[t] = X[(uint64_t)idx[r] * d + j];
}

namespace {
template <typename T>
struct DevBuf {
  LloydEngine& e;
  Scratch b;
  T* p = nullptr;
  explicit DevBuf(LloydEngine& eng) : e(eng) {}
  ~DevBuf() { scratch_free(b, e.device, e.stream); }
  km_status alloc(size_t count) {
    KM_TRY(scratch_alloc(&b, sizeof(T) * count, e.device, e.stream));
    p = static_cast<T*>(b.p);
    return KM_OK;
  }
};
}  // namespace

km_status plusplus_init(LloydEngine& e, int seed) {
  const uint64_t n = e.n;
  const uint32_t d = e.d, k = e.k;
  const uint32_t s = 2u + (uint32_t)std::ceil(std::log((double)k));
  if (s > PP_MAX_S) return KM_ERR_UNSUPPORTED;
  const size_t smem = (size_t)s * d * sizeof(float);
  if (smem > 200 * 1024) return KM_ERR_UNSUPPORTED;
  const uint32_t nblk = (uint32_t)((n + PP_CHUNK - 1) / PP_CHUNK);
  std::mt19937_64 gen((uint64_t)(int64_t)seed);
  std::uniform_real_distribution<double> uni(0.0, 1.0);
  const uint64_t first = std::uniform_int_distribution<uint64_t>(0, n - 1)(gen);
  std::vector<double> hu((size_t)(k > 1 ? k - 1 : 1) * s);
  for (auto& v : hu) v = uni(gen);
  std::vector<int32_t> hchosen(1, (int32_t)first);

  // Cost tiles: a thread per row, 256 rows a block, 128 where 256 rows of d
  // columns would take most of an SM's shared memory (one block an SM).
  const bool tiled = d <= PP_TILE_MAX_D;
  const uint32_t S = s <= 4u ? 4u : s <= 8u ? 8u : 16u, rows = d <= 128u ? 256u : 128u;
  const uint32_t crows = tiled ? rows : PP_WIDE_ROWS, ncost = (uint32_t)((n + crows - 1) / crows);
  // the rows' minima ([s][rows]) follow the staged rows in the same space
  const size_t cost_smem = tiled ? sizeof(float) * ((size_t)d * S + std::max<size_t>((size_t)d * (rows + 1u), (size_t)s * rows))
                                 : smem;
  const bool v4 = d % 4 == 0 && reinterpret_cast<uintptr_t>(e.X) % 16 == 0;
  auto tile = S == 4u ? pp_cost_kernel<4> : S == 8u ? pp_cost_kernel<8> : pp_cost_kernel<16>;
  DevBuf<float> d2(e), D(e);
  DevBuf<double> bsum(e), cpart(e), u(e);
  DevBuf<int32_t> cand(e), chosen(e);
  DevBuf<PpState> state(e);
  KM_TRY(d2.alloc(n));
  KM_TRY(D.alloc(n * s));
  KM_TRY(bsum.alloc(nblk));
  KM_TRY(cpart.alloc((size_t)ncost * s));
  KM_TRY(u.alloc(hu.size()));
  KM_TRY(cand.alloc(s));
  KM_TRY(chosen.alloc(k));
  KM_TRY(state.alloc(1));
  if (cost_smem > 48 * 1024) {
    if (tiled)
      KM_CUDA_TRY(cudaFuncSetAttribute(tile, cudaFuncAttributeMaxDynamicSharedMemorySize, DYN_SMEM_MAX - 4096));
    else
      KM_CUDA_TRY(cudaFuncSetAttribute(pp_cost_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DYN_SMEM_MAX - 4096));
  }
  cudaStream_t st = e.stream;
  KM_CUDA_TRY(cudaMemsetAsync(state.p, 0, sizeof(PpState), st));
  KM_CUDA_TRY(cudaMemcpyAsync(u.p, hu.data(), sizeof(double) * hu.size(), cudaMemcpyHostToDevice, st));
  KM_CUDA_TRY(cudaMemcpyAsync(chosen.p, hchosen.data(), sizeof(int32_t), cudaMemcpyHostToDevice, st));
  pp_first_kernel<<<nblk, 256, 0, st>>>(e.X, n, d, first, d2.p, bsum.p, state.p, k > 1 ? u.p : nullptr, s, cand.p);
  KM_CUDA_TRY(cudaGetLastError());
  for (uint32_t r = 1; r < k; ++r) {
    if (tiled)
      KM_CUDA_TRY(launch_pdl(tile, ncost, rows, cost_smem, st, e.X, n, d, v4, cand.p, s, d2.p, D.p, cpart.p, state.p,
                             r, chosen.p));
    else
      KM_CUDA_TRY(launch_pdl(pp_cost_wide_kernel, ncost, 256, cost_smem, st, e.X, n, d, cand.p, s, d2.p, D.p, cpart.p,
                             state.p, r, chosen.p));
    KM_CUDA_TRY(launch_pdl(pp_update_kernel, nblk, 256, 0, st, D.p, n, state.p, d2.p, bsum.p,
                           r + 1 < k ? u.p + (size_t)r * s : (const double*)nullptr, s, cand.p));
  }
  pp_gather_kernel<<<(unsigned)(((uint64_t)k * d + 255) / 256), 256, 0, st>>>(e.X, d, chosen.p, k, e.C);
  KM_CUDA_TRY(cudaGetLastError());
  // the host arrays copied from go on return
  KM_CUDA_TRY(cudaStreamSynchronize(st));
  return KM_OK;
}

}  // namespace km
