// Kernel k-means for sm_103a (the reference's current "popcorn" GPU path).
//
//  (a) kernel matrix  K = f(X X^T)  (src/kernels/kernels.cuh:43-118, :568-718):
//      tcgen05 GEMM (BF16 or split-BF16x3 operands, FP32 accumulators in TMEM,
//      TMA-fed) or SIMT FP32 GEMM, with the kernel function applied in the
//      epilogue and K (and diag K) stored once.  The reference stores
//      B = -2 f(.) and runs an n^2 Thrust pass; here f is fused and the -2 is
//      folded into the distance.
//  (c) one iteration (src/kmeans.cu:772-1073, src/kernels/distances.cu:895-1002):
//      E = K V^T streamed over the rows of K once (E[i,c] = sum_{j in c} K_ij,
//      per-lane shared-memory bins, deterministic order), ctilde_c =
//      (1/|c|^2) sum_{i in c} E[i,c] = diag(V K V^T) in FP64 over the
//      label-sorted permutation, then D[i,c] = -2 E[i,c]/|c| + ctilde_c
//      (ctilde_c == 0 -> +inf, distances.cu:588-599), argmin keeping the lowest
//      index from (0, FLT_MAX) (kmeans.cu:923-936), score = sum_i min_c D
//      (kmeans.cu:1054-1061; it leaves out K_ii), stop on |score - last| < tol
//      from iteration 2 when checking (kmeans.cu:1064-1073).
#include "km_lloyd.cuh"
#include "km_simt.cuh"

#include <cudaTypedefs.h>
#include <cmath>
#include <cstring>
#include <cfloat>
#include <new>
#include <type_traits>

namespace km {

__global__ void round_robin_labels_kernel(uint32_t* labels, uint64_t n, uint32_t k);  // km_capi.cu

struct KFn {
  int kind;        // km_kernel_fn
  float gamma, coef, inv2s2;
  int degree;
};

// The kernel functions, the kind fixed at compile time (one small body per
// kernel-matrix instantiation; the epilogues unroll it per column).
template <int KIND>
__device__ __forceinline__ float kfn_apply_k(const KFn& f, float dot, float ni, float nj) {
  if constexpr (KIND == KM_KERNEL_LINEAR) {
    return dot;
  } else if constexpr (KIND == KM_KERNEL_POLY) {
    const float b = fmaf(f.gamma, dot, f.coef);
    if (f.degree == 2) return b * b;          // the loop's 1 * b * b, without the loop
    float r = 1.0f;
#pragma unroll 1
    for (int e = 0; e < f.degree; ++e) r *= b;
    return r;
  } else if constexpr (KIND == KM_KERNEL_SIGMOID) {
    return tanhf(fmaf(f.gamma, dot, f.coef));
  } else {
    const float d2 = fmaxf(ni + nj - 2.0f * dot, 0.0f);
    return expf(-d2 * f.inv2s2);
  }
}

// ||x_i||^2 of the operands the tensor cores see (hi, or hi + lo): the
// Gaussian epilogue's ||x_i||^2 + ||x_j||^2 - 2 x_i.x_j is then the squared
// distance of those operands (K_ii = 1 exactly), instead of mixing FP32 norms
// with a BF16 dot product.
__global__ void kmat_operand_norms_kernel(const __nv_bfloat16* __restrict__ Xb,
                                          const __nv_bfloat16* __restrict__ Xlo, uint64_t n,
                                          uint32_t dp, float* __restrict__ out) {
  const uint64_t r = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (r >= n) return;
  double s = 0.0;
  for (uint32_t j = lane; j < dp; j += 32) {
    float v = __bfloat162float(Xb[r * dp + j]);
    if (Xlo) v += __bfloat162float(Xlo[r * dp + j]);
    s += (double)v * v;
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) out[r] = (float)s;
}

template <bool OUT_BF16>
__device__ __forceinline__ void kstore(void* K, uint64_t idx, float v) {
  if (OUT_BF16) reinterpret_cast<__nv_bfloat16*>(K)[idx] = __float2bfloat16_rn(v);
  else reinterpret_cast<float*>(K)[idx] = v;
}

// ---------------------------------------------------------------------------
// (a) SIMT FP32 kernel matrix, 64 x 128 tiles (km_simt.cuh has the product).
// Builds rows [row0, row_end) of K into K (row stride n, first row = row0); with
// `stop` set it does nothing once the fit has stopped (panels rebuilt per
// iteration).  Symmetry: a build of all rows computes only the blocks of 128 x 128
// on and above the diagonal (two tiles each, column block by column block) and
// stores the ones above it twice, the second time transposed (a product and a
// transposed one multiply and add the same numbers in the same order, so both
// halves are what a full build gives); a panel computes its own rows.
// Bound by the FP32 pipes and the product's shared-memory reads, then by writing K:
// n = 20,000 d = 64 2182 -> 807 us (16 x 16 threads with one buffered stage, scalar
// loads and every tile computed before).
// ---------------------------------------------------------------------------
using KmTile = SimtTile<128, 8, 16, 8, 16>;

template <bool OUT_BF16>
__device__ __forceinline__ void kstore4(void* K, uint64_t idx, const float (&v)[4], bool vec, uint64_t col, uint64_t n) {
  if (vec) {                       // n % 4 == 0 and K aligned: four columns start 16 (8) byte aligned
    if (col >= n) return;
    if (OUT_BF16) {
      const __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
      uint2 u;
      u.x = *reinterpret_cast<const uint32_t*>(&a);
      u.y = *reinterpret_cast<const uint32_t*>(&b);
      *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(K) + idx) = u;
    } else {
      *reinterpret_cast<float4*>(reinterpret_cast<float*>(K) + idx) = make_float4(v[0], v[1], v[2], v[3]);
    }
  } else {
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (col + q < n) kstore<OUT_BF16>(K, idx + q, v[q]);
  }
}

template <bool OUT_BF16, int KIND>
__global__ void __launch_bounds__(128, 3)
kmat_f32_kernel(const float* __restrict__ X, bool v4, const float* __restrict__ xn2, uint64_t n, uint32_t d,
                uint64_t row0, uint64_t row_end, int symmetric, KFn f, void* __restrict__ K, bool vec,
                float* __restrict__ diag, const DevState* stop) {
  using T = KmTile;
  if (stop && stop->done) return;
  extern __shared__ __align__(16) float km_smem[];
  uint64_t m0, c0;
  bool mirror = false;
  if (symmetric) {
    const uint64_t p = blockIdx.x >> 1;                    // pair (bi <= bj), column block bj by column block
    uint64_t bj = (uint64_t)((sqrt(8.0 * (double)p + 1.0) - 1.0) * 0.5);
    while (bj * (bj + 1) / 2 > p) --bj;
    while ((bj + 1) * (bj + 2) / 2 <= p) ++bj;
    const uint64_t bi = p - bj * (bj + 1) / 2;
    m0 = bi * 128 + (blockIdx.x & 1u) * 64;
    c0 = bj * 128;
    mirror = bi < bj;
  } else {
    const uint64_t nb = (n + 127) / 128;
    m0 = row0 + blockIdx.x / nb * 64;
    c0 = blockIdx.x % nb * 128;
  }
  if (m0 >= row_end) return;
  float2 acc[4][8];
  simt_product<T>(
      km_smem, d, v4, [&](int r) { return m0 + (uint64_t)r < row_end ? X + (m0 + (uint64_t)r) * d : (const float*)nullptr; },
      [&](int c) { return c0 + (uint64_t)c < n ? X + (c0 + (uint64_t)c) * d : (const float*)nullptr; }, acc);
  const int tx = threadIdx.x % T::TX, ty = threadIdx.x / T::TX;
  const uint64_t r0 = m0 + (uint64_t)ty * 8;
  float nj[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint64_t c = c0 + (uint64_t)T::col(tx, j);
    nj[j] = (KIND == KM_KERNEL_GAUSSIAN && c < n) ? xn2[c] : 0.0f;
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint64_t row = r0 + i;
    if (row >= row_end) break;
    const float ni = KIND == KM_KERNEL_GAUSSIAN ? xn2[row] : 0.0f;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const uint64_t col = c0 + (uint64_t)T::col(tx, 4 * q);
      float v[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        float& a = (i & 1) ? acc[i / 2][4 * q + e].y : acc[i / 2][4 * q + e].x;
        a = v[e] = kfn_apply_k<KIND>(f, a, ni, nj[4 * q + e]);
        if (diag && col + e == row) diag[row] = v[e];
      }
      kstore4<OUT_BF16>(K, (row - row0) * n + col, v, vec, col, n);
    }
  }
  if (mirror) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint64_t col = c0 + (uint64_t)T::col(tx, j);
      if (col >= n) continue;
#pragma unroll
      for (int h = 0; h < 2; ++h) {                        // four rows of this column
        const float v[4] = {acc[2 * h][j].x, acc[2 * h][j].y, acc[2 * h + 1][j].x, acc[2 * h + 1][j].y};
        kstore4<OUT_BF16>(K, col * n + r0 + 4 * h, v, vec, r0 + 4 * h, n);
      }
    }
  }
}

// ---------------------------------------------------------------------------
// (a) tcgen05 kernel-matrix GEMM.  Persistent CTAs walk 128 x 256 output
// tiles; per K-block the A tile (128 rows) and B tile (256 rows) of the BF16
// copy of X (hi, and lo for X3) come in by TMA into a ring of stages; one
// thread issues the MMAs into a TMEM accumulator (two buffers of 256
// columns); sixteen epilogue warps (two sets of eight, one per buffer; warp w on TMEM
// lanes 32*(w%4) and one half of the columns) read the accumulator 32 columns at a
// time, apply f and store K.  Bound by the stores of K (and, for long rows in the split
// form, the MMAs); with eight warps and a range check at every store the epilogue's
// latency was: n = 24,000 d = 200 Gaussian 966 -> 543 us, n = 65,536 d = 512 polynomial
// 8.28 -> 5.12 ms (split-BF16x3, FP32 K).  Every wait is bounded (2 s) and a timeout raises KM_DEVERR_TIMEOUT after
// draining this CTA's copies and MMAs.  The kernel builds rows
// [prow0, prow_end) of K into K (row stride n, first row = prow0): all of K,
// or one panel of it; with skip_done it does nothing once the fit has stopped.
//
// Symmetry: K is symmetric, so only tiles (row tile mi, column block nj) with
// mi/2 <= nj are computed (the 256-row blocks on or above the diagonal), as
// the reference's SYRK path builds one triangle and mirrors it
// (src/kernels/kernels.cuh:596-649).  A tile strictly above the diagonal
// (mi/2 < nj) also stores its transpose: each warp holds 32 consecutive rows
// in its lanes, so column c of the tile leaves as one contiguous run of row
// c of K.  The tiles come from a list built on the host (kmat_tile_list):
// (mi, nj | direct << 30 | mirror << 31), `direct` when the tile's own rows
// lie in [prow0, prow_end) and `mirror` when its transposed rows do, so a
// panel receives exactly the values the whole matrix holds.  This halves the
// MMA work of a resident build.
// ---------------------------------------------------------------------------
namespace {
constexpr int KM_M = 128, KM_N = 256;
constexpr uint32_t KA_BYTES = KM_M * 128;   // 64-column BF16 K-block of A
constexpr uint32_t KB_BYTES = KM_N * 128;   // 64-column BF16 K-block of B
constexpr uint64_t KWAIT_NS = 2000000000ull;

constexpr uint64_t KM_GROUP = 16;   // row tiles per raster group of the kernel-matrix build


constexpr int KM_EPI_WARPS = 16;
constexpr int KM_THREADS = 32 * (4 + KM_EPI_WARPS);
constexpr uint32_t KM_STG_BYTES = KM_EPI_WARPS * 32u * 16u * 4u;   // epilogue staging tiles, one per epilogue warp

struct KmSmem {
  uint64_t full[8];
  uint64_t empty[8];
  uint64_t tfull[2];
  uint64_t tempty[2];
  uint64_t tdone;
  uint32_t tmem_base;
  int abort;
};
}  // namespace

template <bool X3, bool OUT_BF16, int KIND>
__global__ void __launch_bounds__(KM_THREADS, 1)
kmat_tc_kernel(const __grid_constant__ CUtensorMap tA, const __grid_constant__ CUtensorMap tAlo,
               const __grid_constant__ CUtensorMap tB, const __grid_constant__ CUtensorMap tBlo,
               const float* __restrict__ xn2, uint64_t n, uint64_t prow0, uint64_t prow_end, uint32_t KB,
               uint32_t S, KFn f, void* __restrict__ K, float* __restrict__ diag, int vec, int skip_done,
               DevState* st, const uint32_t* __restrict__ tlist, uint64_t ntiles) {
  if (skip_done && st->done) return;   // uniform over the grid: written by an earlier launch
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~uintptr_t(1023));
  const uint32_t stage_bytes = (KA_BYTES + KB_BYTES) * (X3 ? 2u : 1u);
  float* stg_all = reinterpret_cast<float*>(smem + (size_t)S * stage_bytes);    // [16 warps][32][16]
  KmSmem* ts = reinterpret_cast<KmSmem*>(smem + (size_t)S * stage_bytes + KM_STG_BYTES);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < S; ++s) { mbar_init(&ts->full[s], 1); mbar_init(&ts->empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&ts->tfull[b], 1); mbar_init(&ts->tempty[b], 8); }
    mbar_init(&ts->tdone, 1);
    ts->abort = 0;
    mbar_fence_init();
  }
  if (warp == 2) tmem_alloc(&ts->tmem_base, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = ts->tmem_base;
  volatile int* abort_flag = &ts->abort;
  auto fail = [&](uint32_t where) {
    ts->abort = 1;
    if (atomicOr(&st->err, KM_DEVERR_TIMEOUT) == 0u) st->err_where = 100u + where;
  };
  // tile t -> (mi, nj) from the list (groups of KM_GROUP row tiles, column
  // blocks in the inner loop, so that a group's A tiles stay in L2)
  if (warp == 0) {
    if (lane == 0) {
      uint64_t u = 0;
      bool ok = true;
      for (uint64_t tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
        const uint64_t mi = tlist[2 * tile], nj = tlist[2 * tile + 1] & 0x3fffffffu;
        for (uint32_t kb = 0; kb < KB; ++kb, ++u) {
          const uint32_t s = (uint32_t)(u % S), ph = (uint32_t)((u / S) & 1u);
          if (!mbar_wait_bounded(&ts->empty[s], ph ^ 1u, abort_flag, KWAIT_NS)) { fail(1); ok = false; break; }
          mbar_arrive_expect_tx(&ts->full[s], stage_bytes);
          uint8_t* dst = smem + (size_t)s * stage_bytes;
          tma_load_2d(dst, &tA, (int)(kb * 64), (int)(mi * KM_M), &ts->full[s]);
          tma_load_2d(dst + KA_BYTES, &tB, (int)(kb * 64), (int)(nj * KM_N), &ts->full[s]);
          if (X3) {
            tma_load_2d(dst + KA_BYTES + KB_BYTES, &tAlo, (int)(kb * 64), (int)(mi * KM_M), &ts->full[s]);
            tma_load_2d(dst + 2 * KA_BYTES + KB_BYTES, &tBlo, (int)(kb * 64), (int)(nj * KM_N), &ts->full[s]);
          }
        }
      }
      volatile int no_abort = 0;
      const uint64_t first = u > S ? u - S : 0;
      for (uint64_t v = first; v < u; ++v)
        mbar_wait_bounded(&ts->full[v % S], (uint32_t)((v / S) & 1u), &no_abort, KWAIT_NS);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = idesc_bf16_f32(KM_M, KM_N);
      const uint32_t s0 = smem_u32(smem);
      uint64_t u = 0, t = 0;
      bool ok = true, issued = false;
      for (uint64_t tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x, ++t) {
        const uint32_t buf = (uint32_t)(t & 1u), use = (uint32_t)(t >> 1);
        if (!mbar_wait_bounded(&ts->tempty[buf], (use & 1u) ^ 1u, abort_flag, KWAIT_NS)) { fail(2); ok = false; break; }
        tc_fence_after();
        const uint32_t dt = tmem_base + buf * 256u;
        for (uint32_t kb = 0; kb < KB; ++kb, ++u) {
          const uint32_t s = (uint32_t)(u % S), ph = (uint32_t)((u / S) & 1u);
          if (!mbar_wait_bounded(&ts->full[s], ph, abort_flag, KWAIT_NS)) { fail(3); ok = false; break; }
          tc_fence_after();
          const uint32_t a0 = s0 + s * stage_bytes, b0 = a0 + KA_BYTES;
#pragma unroll
          for (uint32_t kk = 0; kk < 4; ++kk) {
            const uint64_t ad = smem_desc_sw128(a0 + kk * 32u);
            const uint64_t bd = smem_desc_sw128(b0 + kk * 32u);
            tc_mma_bf16(dt, ad, bd, idesc, (kb | kk) != 0u ? 1u : 0u);
            if (X3) {
              const uint64_t adl = smem_desc_sw128(a0 + KA_BYTES + KB_BYTES + kk * 32u);
              const uint64_t bdl = smem_desc_sw128(a0 + 2 * KA_BYTES + KB_BYTES + kk * 32u);
              tc_mma_bf16(dt, ad, bdl, idesc, 1u);
              tc_mma_bf16(dt, adl, bd, idesc, 1u);
            }
          }
          tc_commit(&ts->empty[s]);
          issued = true;
        }
        if (!ok) break;
        tc_commit(&ts->tfull[buf]);
      }
      if (issued) {
        tc_commit(&ts->tdone);
        volatile int no_abort = 0;
        mbar_wait_bounded(&ts->tdone, 0, &no_abort, KWAIT_NS);
      }
    }
  } else if (warp >= 4) {
    // Epilogue: warp (4 + e) on TMEM lanes 32 (warp % 4) of accumulator buffer
    // (e / 4) % 2, columns 128 (e / 8) .. + 127, 32 at a time.
    const int q = warp & 3, set = ((warp - 4) >> 2) & 1, half = (warp - 4) >> 3;
    const uint32_t r = (uint32_t)q * 32u + (uint32_t)lane;
    const uint32_t tbase = tmem_base + (((uint32_t)q * 32u) << 16) + (uint32_t)set * 256u + (uint32_t)half * 128u;
    float* const stg = stg_all + (size_t)(warp - 4) * 32 * 16;
    using KT = std::conditional_t<OUT_BF16, __nv_bfloat16, float>;
    KT* const Kt = reinterpret_cast<KT*>(K);
    uint64_t t = (uint64_t)set;
    for (uint64_t tile = blockIdx.x + (uint64_t)set * gridDim.x; tile < ntiles;
         tile += 2ull * gridDim.x, t += 2) {
      const uint64_t mi = tlist[2 * tile];
      const uint32_t njf = tlist[2 * tile + 1];
      const uint64_t nj = njf & 0x3fffffffu;
      const bool direct = (njf >> 30) & 1u, mirror = (njf >> 31) & 1u;
      const uint64_t row = mi * KM_M + r, row0 = mi * KM_M + (uint64_t)q * 32u;   // this lane's, the warp's first
      const uint64_t c0 = nj * KM_N + (uint64_t)half * 128u;
      const bool row_in = row < n;
      const float ni = (KIND == KM_KERNEL_GAUSSIAN && row_in) ? xn2[row] : 0.0f;
      // whole blocks of the warp inside K (and inside the panel): stores without checks
      const bool fast_d = direct && vec && row0 >= prow0 && row0 + 32 <= prow_end && c0 + 128 <= n;
      const bool fast_m = mirror && row0 + 32 <= n && c0 >= prow0 && c0 + 128 <= prow_end;
      const bool on_diag = diag && direct && mi / 2 == nj && row >= prow0 && row < prow_end;
      const bool okw = mbar_wait_bounded(&ts->tfull[set], (uint32_t)(t >> 1) & 1u, abort_flag, KWAIT_NS);
      if (!__all_sync(0xffffffffu, okw)) { if (lane == 0) fail(4); break; }
      tc_fence_after();
#pragma unroll 1
      for (uint32_t ch = 0; ch < 4; ++ch) {
        const uint64_t cb = c0 + ch * 32u;
        uint32_t acc[32];
        tmem_ld_32x32b_x32(tbase + ch * 32u, acc);
        tmem_ld_wait();
        if (ch == 3) {
          // the accumulator's last columns are in registers: the MMAs of the
          // next tile on this buffer may start while this one is stored
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&ts->tempty[set]);
        }
        float v[32];
#pragma unroll
        for (int c4 = 0; c4 < 8; ++c4) {
          float4 w = make_float4(0.f, 0.f, 0.f, 0.f);      // column norms only matter for the Gaussian kernel
          if (KIND == KM_KERNEL_GAUSSIAN) {
            const uint64_t c = cb + 4 * c4;
            if (c + 3 < n) {
              w = __ldg(reinterpret_cast<const float4*>(xn2 + c));
            } else {
              if (c + 0 < n) w.x = __ldg(xn2 + c);
              if (c + 1 < n) w.y = __ldg(xn2 + c + 1);
              if (c + 2 < n) w.z = __ldg(xn2 + c + 2);
            }
          }
          v[4 * c4 + 0] = kfn_apply_k<KIND>(f, __uint_as_float(acc[4 * c4 + 0]), ni, w.x);
          v[4 * c4 + 1] = kfn_apply_k<KIND>(f, __uint_as_float(acc[4 * c4 + 1]), ni, w.y);
          v[4 * c4 + 2] = kfn_apply_k<KIND>(f, __uint_as_float(acc[4 * c4 + 2]), ni, w.z);
          v[4 * c4 + 3] = kfn_apply_k<KIND>(f, __uint_as_float(acc[4 * c4 + 3]), ni, w.w);
        }
        if (on_diag) {
#pragma unroll
          for (int c = 0; c < 32; ++c)
            if (cb + c == row) diag[row] = v[c];
        }
        // transposed: K[gcol][row]; the warp's lanes write one contiguous run
        if (fast_m) {
          KT* p = Kt + (cb - prow0) * n + row;
#pragma unroll
          for (int c = 0; c < 32; ++c, p += n) kstore<OUT_BF16>(p, 0, v[c]);
        } else if (mirror && row_in) {
#pragma unroll
          for (int c = 0; c < 32; ++c) {
            const uint64_t gcol = cb + c;
            if (gcol >= prow0 && gcol < prow_end) kstore<OUT_BF16>(Kt, (gcol - prow0) * n + row, v[c]);
          }
        }
        if (!direct) continue;
        // Own rows: 16 columns at a time through the warp's staging tile (32 rows x
        // 16 columns, 16-byte chunks XOR-swizzled by row pair), out as row segments:
        // four lanes a row, eight rows a store.
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          __syncwarp();                                    // the previous segment has been read back
#pragma unroll
          for (int c = 0; c < 4; ++c)
            *reinterpret_cast<float4*>(stg + lane * 16 + ((c ^ ((lane >> 1) & 3)) * 4)) =
                make_float4(v[16 * h + 4 * c], v[16 * h + 4 * c + 1], v[16 * h + 4 * c + 2], v[16 * h + 4 * c + 3]);
          __syncwarp();
          const uint32_t r8 = (uint32_t)lane >> 2, c4 = (uint32_t)lane & 3u;
          const uint64_t gcol = cb + 16u * h + 4u * c4;
#pragma unroll
          for (int step = 0; step < 4; ++step) {
            const uint32_t rr = 8u * step + r8;
            const float4 o = *reinterpret_cast<const float4*>(stg + rr * 16 + ((c4 ^ ((rr >> 1) & 3u)) * 4));
            const uint64_t grow = row0 + rr;
            const float ov[4] = {o.x, o.y, o.z, o.w};
            if (fast_d) kstore4<OUT_BF16>(K, (grow - prow0) * n + gcol, ov, true, gcol, n);
            else if (grow >= prow0 && grow < prow_end) kstore4<OUT_BF16>(K, (grow - prow0) * n + gcol, ov, vec, gcol, n);
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 2) tmem_dealloc(tmem_base, 512);
}

// ---------------------------------------------------------------------------
// (c') E = K V^T without K in memory.  The columns of K are taken in
// label-sorted order: the B operand is a copy of the points permuted by the
// stable label sort (perm), so cluster c owns the contiguous columns
// [cstart[c], cstart[c+1]) and E[i,c] is a running sum along row i of
// f(x_i . x_perm(j)), j ascending.  Persistent CTAs take whole 128-row blocks
// of K and sweep its 256-column tiles in order: warp 0 the TMA producer,
// warp 1 the MMA issuer into two TMEM accumulators, warp 2 the TMEM
// allocation, warps 4-7 the epilogue with one row per thread (TMEM lane
// quadrant warp % 4).  Per 64-column chunk the epilogue applies f and, when no
// cluster ends inside the chunk, adds the chunk's pairwise-tree sum to the
// row's running sum; a chunk holding a boundary goes column by column through
// a shared staging tile.  Each E[i,c] is written once, by its row's thread.
// The order of the sum is fixed by the data (deterministic); it is not the
// resident V.K kernel's lane-interleaved order.  Waits are bounded as in
// kmat_tc_kernel.
// ---------------------------------------------------------------------------
namespace {
constexpr uint32_t KF_STG_BYTES = 4u * 64u * 32u * 4u;   // per epilogue warp: 64 columns x 32 rows

struct KfSmem {
  uint64_t full[8];
  uint64_t empty[8];
  uint64_t tfull[2];
  uint64_t tempty[2];
  uint64_t tdone;
  uint32_t tmem_base;
  int abort;
};
}  // namespace

template <bool X3, int KIND>
__global__ void __launch_bounds__(256, 1)
kkm_fused_tc_kernel(const __grid_constant__ CUtensorMap tA, const __grid_constant__ CUtensorMap tAlo,
                    const __grid_constant__ CUtensorMap tB, const __grid_constant__ CUtensorMap tBlo,
                    const float* __restrict__ xn2, const float* __restrict__ xn2p, uint64_t n, uint32_t KB,
                    uint32_t S, KFn f, const uint32_t* __restrict__ cstart, uint32_t k, float* __restrict__ E,
                    DevState* st) {
  if (st->done) return;   // uniform over the grid: written by an earlier launch
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~uintptr_t(1023));
  const uint32_t stage_bytes = (KA_BYTES + KB_BYTES) * (X3 ? 2u : 1u);
  float* stg_all = reinterpret_cast<float*>(smem + (size_t)S * stage_bytes);   // [4 warps][64][32]
  KfSmem* ts = reinterpret_cast<KfSmem*>(smem + (size_t)S * stage_bytes + KF_STG_BYTES);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint64_t mt = (n + KM_M - 1) / KM_M, nt = (n + KM_N - 1) / KM_N;
  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < S; ++s) { mbar_init(&ts->full[s], 1); mbar_init(&ts->empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&ts->tfull[b], 1); mbar_init(&ts->tempty[b], 4); }
    mbar_init(&ts->tdone, 1);
    ts->abort = 0;
    mbar_fence_init();
  }
  if (warp == 2) tmem_alloc(&ts->tmem_base, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = ts->tmem_base;
  volatile int* abort_flag = &ts->abort;
  auto fail = [&](uint32_t where) {
    ts->abort = 1;
    if (atomicOr(&st->err, KM_DEVERR_TIMEOUT) == 0u) st->err_where = 110u + where;
  };
  if (warp == 0) {
    if (lane == 0) {
      uint64_t u = 0;
      bool ok = true;
      for (uint64_t mi = blockIdx.x; mi < mt && ok; mi += gridDim.x) {
        for (uint64_t nj = 0; nj < nt && ok; ++nj) {
          for (uint32_t kb = 0; kb < KB; ++kb, ++u) {
            const uint32_t s = (uint32_t)(u % S), ph = (uint32_t)((u / S) & 1u);
            if (!mbar_wait_bounded(&ts->empty[s], ph ^ 1u, abort_flag, KWAIT_NS)) { fail(1); ok = false; break; }
            mbar_arrive_expect_tx(&ts->full[s], stage_bytes);
            uint8_t* dst = smem + (size_t)s * stage_bytes;
            tma_load_2d(dst, &tA, (int)(kb * 64), (int)(mi * KM_M), &ts->full[s]);
            tma_load_2d(dst + KA_BYTES, &tB, (int)(kb * 64), (int)(nj * KM_N), &ts->full[s]);
            if (X3) {
              tma_load_2d(dst + KA_BYTES + KB_BYTES, &tAlo, (int)(kb * 64), (int)(mi * KM_M), &ts->full[s]);
              tma_load_2d(dst + 2 * KA_BYTES + KB_BYTES, &tBlo, (int)(kb * 64), (int)(nj * KM_N), &ts->full[s]);
            }
          }
        }
      }
      volatile int no_abort = 0;
      const uint64_t first = u > S ? u - S : 0;
      for (uint64_t v = first; v < u; ++v)
        mbar_wait_bounded(&ts->full[v % S], (uint32_t)((v / S) & 1u), &no_abort, KWAIT_NS);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = idesc_bf16_f32(KM_M, KM_N);
      const uint32_t s0 = smem_u32(smem);
      uint64_t u = 0, t = 0;
      bool ok = true, issued = false;
      for (uint64_t mi = blockIdx.x; mi < mt && ok; mi += gridDim.x) {
        for (uint64_t nj = 0; nj < nt && ok; ++nj, ++t) {
          const uint32_t buf = (uint32_t)(t & 1u), use = (uint32_t)(t >> 1);
          if (!mbar_wait_bounded(&ts->tempty[buf], (use & 1u) ^ 1u, abort_flag, KWAIT_NS)) { fail(2); ok = false; break; }
          tc_fence_after();
          const uint32_t dt = tmem_base + buf * 256u;
          for (uint32_t kb = 0; kb < KB; ++kb, ++u) {
            const uint32_t s = (uint32_t)(u % S), ph = (uint32_t)((u / S) & 1u);
            if (!mbar_wait_bounded(&ts->full[s], ph, abort_flag, KWAIT_NS)) { fail(3); ok = false; break; }
            tc_fence_after();
            const uint32_t a0 = s0 + s * stage_bytes, b0 = a0 + KA_BYTES;
#pragma unroll
            for (uint32_t kk = 0; kk < 4; ++kk) {
              const uint64_t ad = smem_desc_sw128(a0 + kk * 32u);
              const uint64_t bd = smem_desc_sw128(b0 + kk * 32u);
              tc_mma_bf16(dt, ad, bd, idesc, (kb | kk) != 0u ? 1u : 0u);
              if (X3) {
                const uint64_t adl = smem_desc_sw128(a0 + KA_BYTES + KB_BYTES + kk * 32u);
                const uint64_t bdl = smem_desc_sw128(a0 + 2 * KA_BYTES + KB_BYTES + kk * 32u);
                tc_mma_bf16(dt, ad, bdl, idesc, 1u);
                tc_mma_bf16(dt, adl, bd, idesc, 1u);
              }
            }
            tc_commit(&ts->empty[s]);
            issued = true;
          }
          if (!ok) break;
          tc_commit(&ts->tfull[buf]);
        }
      }
      if (issued) {
        tc_commit(&ts->tdone);
        volatile int no_abort = 0;
        mbar_wait_bounded(&ts->tdone, 0, &no_abort, KWAIT_NS);
      }
    }
  } else if (warp >= 4) {
    const int q = warp & 3;
    const uint32_t tq = tmem_base + (((uint32_t)q * 32u) << 16);
    float* stg = stg_all + (size_t)q * 64 * 32;
    auto colnorm = [&](uint64_t j) -> float {
      return (KIND == KM_KERNEL_GAUSSIAN) ? __ldg(xn2p + j) : 0.0f;
    };
    uint64_t t = 0;
    bool ok = true;
    for (uint64_t mi = blockIdx.x; mi < mt && ok; mi += gridDim.x) {
      const uint64_t row = mi * KM_M + (uint64_t)q * 32u + (uint64_t)lane;
      const bool valid = row < n;
      const float ni = (KIND == KM_KERNEL_GAUSSIAN && valid) ? xn2[row] : 0.0f;
      float* Er = E + row * k;
      uint32_t cur = 0;                 // cluster of the running sum
      uint64_t nb = cstart[1];          // first column after cluster cur
      float run = 0.0f;
      for (uint64_t nj = 0; nj < nt; ++nj, ++t) {
        const uint32_t buf = (uint32_t)(t & 1u);
        const bool okw = mbar_wait_bounded(&ts->tfull[buf], (uint32_t)(t >> 1) & 1u, abort_flag, KWAIT_NS);
        if (!__all_sync(0xffffffffu, okw)) { if (lane == 0) fail(4); ok = false; break; }
        tc_fence_after();
        for (uint32_t pr = 0; pr < KM_N / 64; ++pr) {
          const uint64_t j0 = nj * KM_N + pr * 64u;
          if (j0 >= n) break;                                   // warp-uniform
          uint32_t acc[64];
          tmem_ld_32x32b_x64(tq + buf * 256u + pr * 64u, acc);
          tmem_ld_wait();
          if (nb >= j0 + 64 && j0 + 64 <= n) {
            float v[64];
#pragma unroll
            for (int c = 0; c < 64; ++c) v[c] = kfn_apply_k<KIND>(f, __uint_as_float(acc[c]), ni, colnorm(j0 + c));
#pragma unroll
            for (int w = 32; w >= 1; w >>= 1)
#pragma unroll
              for (int c = 0; c < w; ++c) v[c] += v[c + w];
            run += v[0];
          } else {
            // a cluster ends inside this chunk (or the points do): column by column
#pragma unroll
            for (int c = 0; c < 64; ++c)
              stg[c * 32 + lane] = (j0 + c < n) ? kfn_apply_k<KIND>(f, __uint_as_float(acc[c]), ni, colnorm(j0 + c))
                                                : 0.0f;
            __syncwarp();
            const uint32_t cols = (uint32_t)((n - j0) < 64 ? (n - j0) : 64);
#pragma unroll 1
            for (uint32_t c = 0; c < cols; ++c) {
              const uint64_t j = j0 + c;
              while (j == nb) {                                 // cluster cur ended before column j
                if (valid) Er[cur] = run;
                run = 0.0f;
                ++cur;
                nb = cstart[cur + 1];
              }
              run += stg[c * 32 + lane];
            }
            __syncwarp();
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ts->tempty[buf]);
      }
      if (!ok) break;
      // the last non-empty cluster, then the empty ones after it
      for (; cur < k; ++cur) {
        if (valid) Er[cur] = run;
        run = 0.0f;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 2) tmem_dealloc(tmem_base, 512);
}

// Label-sorted copies of the tensor-core operands and of their norms: row j of
// a copy is row perm[j] of the original.  One warp per row, 16-byte copies
// (dp is a multiple of 64).
__global__ void kkm_permute_points_kernel(const __nv_bfloat16* __restrict__ Xb,
                                          const __nv_bfloat16* __restrict__ Xlo, const float* __restrict__ xn2,
                                          const uint32_t* __restrict__ perm, uint64_t n, uint32_t dp,
                                          __nv_bfloat16* __restrict__ Xbp, __nv_bfloat16* __restrict__ Xlop,
                                          float* __restrict__ xn2p, const DevState* st) {
  if (st->done) return;
  const uint64_t j = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (j >= n) return;
  const uint64_t src = perm[j];
  const uint32_t w16 = dp / 8;
  const uint4* a = reinterpret_cast<const uint4*>(Xb + src * dp);
  uint4* b = reinterpret_cast<uint4*>(Xbp + j * dp);
  for (uint32_t w = lane; w < w16; w += 32) b[w] = __ldg(a + w);
  if (Xlo) {
    const uint4* al = reinterpret_cast<const uint4*>(Xlo + src * dp);
    uint4* bl = reinterpret_cast<uint4*>(Xlop + j * dp);
    for (uint32_t w = lane; w < w16; w += 32) bl[w] = __ldg(al + w);
  }
  if (lane == 0) xn2p[j] = xn2[src];
}

// ---------------------------------------------------------------------------
// (c) E = K V^T.  One warp per row of K at a time; the labels of all n points
// are bytes (k <= 256), in shared memory when they fit next to the bins
// (GLAB false) or else read from a global byte copy (GLAB true, L2-resident);
// every lane accumulates its columns in ascending order into private bins
// bins[c][lane] (no atomics, fixed order), then a cluster's 32 bins are added in lane
// order.  Rows [row0, row_end) are done; K holds them from row row0 on (the whole
// matrix with row0 = 0, or one panel).  Both label sources give the same sums in the
// same order.
//
// Bound by HBM (K is read once) in FP32, by the bins' round trips through shared memory
// in BF16.  The next batch of loads is in flight while one is summed, and the next
// row's first while a row's bins are reduced; for that the bins pass through registers
// into a layout that both sides reach without bank conflicts (a lane walking its
// cluster's bins in place meets 31 others on the same bank).  Rows of n % 4 != 0 come a
// column a lane, four columns' bins together: one whose label another of the four shares
// takes that one's sum, so that the round trip is paid once for four (with four columns a
// lane and load the selects cost more than they save: 2.59 -> 2.49 ms without).
// An iteration at n = 65,536 k = 64 3.31 -> 2.49 ms (FP32 K, 7 TB/s) and 2.42 -> 2.05 (BF16
// K), n = 20,000 k = 20 414 -> 286 and 320 -> 243 us, n = 40,001 k = 10 2.30 -> 1.67 ms and
// 2.52 -> 1.56.
// ---------------------------------------------------------------------------
namespace {
__device__ __forceinline__ float4 ld_stream4(const float* p, bool ok) {
  float4 v;
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %5, 0;\n\t"
               "mov.f32 %0, 0f00000000;\n\tmov.f32 %1, 0f00000000;\n\tmov.f32 %2, 0f00000000;\n\tmov.f32 %3, 0f00000000;\n\t"
               "@q ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "l"(p), "r"((uint32_t)ok));
  return v;
}
__device__ __forceinline__ uint2 ld_stream4(const __nv_bfloat16* p, bool ok) {
  uint2 v;
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %3, 0;\n\tmov.u32 %0, 0;\n\tmov.u32 %1, 0;\n\t"
               "@q ld.global.nc.L1::no_allocate.v2.u32 {%0, %1}, [%2];\n\t}"
               : "=r"(v.x), "=r"(v.y)
               : "l"(p), "r"((uint32_t)ok));
  return v;
}
__device__ __forceinline__ float4 as_float4(float4 v) { return v; }
__device__ __forceinline__ float4 as_float4(uint2 v) {
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v.y));
  return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ float as_float(float v) { return v; }
__device__ __forceinline__ float as_float(__nv_bfloat16 v) { return __bfloat162float(v); }

// Adds x.x .. x.w in this order to the bins of the four labels in l4 (b: this
// lane's bin of cluster 0, clusters 32 floats apart).
__device__ __forceinline__ void bins_add4(float* b, uint32_t l4, float4 x) {
  const uint32_t l0 = l4 & 255u, l1 = (l4 >> 8) & 255u, l2 = (l4 >> 16) & 255u, l3 = l4 >> 24;
  const float b0 = b[l0 * 32], b1 = b[l1 * 32], b2 = b[l2 * 32], b3 = b[l3 * 32];
  const float r0 = b0 + x.x;
  const float r1 = (l1 == l0 ? r0 : b1) + x.y;
  const float r2 = (l2 == l1 ? r1 : l2 == l0 ? r0 : b2) + x.z;
  const float r3 = (l3 == l2 ? r2 : l3 == l1 ? r1 : l3 == l0 ? r0 : b3) + x.w;
  b[l0 * 32] = r0;      // in order: the last of equal labels stays
  b[l1 * 32] = r1;
  b[l2 * 32] = r2;
  b[l3 * 32] = r3;
}
}  // namespace

template <bool KBF16, bool GLAB>
__global__ void __launch_bounds__(512, 1)
kkm_vk_kernel(const void* __restrict__ K, uint64_t n, uint32_t k, const uint32_t* __restrict__ labels,
              const uint8_t* __restrict__ lab8, uint64_t row0, uint64_t row_end, float* __restrict__ E,
              DevState* st) {
  using T = std::conditional_t<KBF16, __nv_bfloat16, float>;
  using V = std::conditional_t<KBF16, uint2, float4>;
  griddep_wait();
  griddep_launch();
  if (st->done) return;
  extern __shared__ __align__(16) uint8_t kk_smem[];
  const uint8_t* lab = GLAB ? lab8 : kk_smem;                        // n bytes
  float* bins = reinterpret_cast<float*>(kk_smem + (GLAB ? 0ull : ((n + 15) & ~15ull)));  // [warps][k][32]
  if (!GLAB) {
    for (uint64_t i = threadIdx.x; i < n; i += blockDim.x) kk_smem[i] = (uint8_t)labels[i];
    __syncthreads();
  }
  auto lab4 = [&](uint64_t j) -> uint32_t {     // labels j..j+3 (j % 4 == 0)
    return GLAB ? __ldg(reinterpret_cast<const uint32_t*>(lab + j)) : *reinterpret_cast<const uint32_t*>(lab + j);
  };
  auto lab1 = [&](uint64_t j) -> uint32_t { return GLAB ? (uint32_t)__ldg(lab + j) : (uint32_t)lab[j]; };
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* const B = bins + (size_t)warp * k * 32;
  for (uint32_t c = 0; c < k; ++c) B[c * 32 + lane] = 0.0f;
  __syncwarp();
  const uint32_t wpb = blockDim.x >> 5;
  const uint64_t nw = (uint64_t)gridDim.x * wpb;
  // A cluster's bins added in lane order, and cleared: 32 clusters at a time.
  auto reduce = [&](uint64_t row) {
    __syncwarp();
    for (uint32_t c0 = 0; c0 < k; c0 += 32) {
      float* const Bc = B + c0 * 32;
      float r[32];
#pragma unroll
      for (int c = 0; c < 32; ++c) r[c] = c0 + c < k ? Bc[c * 32 + lane] : 0.0f;
      __syncwarp();
#pragma unroll
      for (int c = 0; c < 32; ++c)
        if (c0 + c < k) Bc[c * 32 + (lane ^ c)] = r[c];    // bin l of cluster c at c * 32 + (l ^ c)
      __syncwarp();
      if (c0 + (uint32_t)lane < k) {
        float s = 0.0f;
#pragma unroll
        for (int l = 0; l < 32; ++l) s += Bc[lane * 32 + (l ^ lane)];
        E[row * k + c0 + lane] = s;
      }
      __syncwarp();
#pragma unroll
      for (int c = 0; c < 32; ++c)
        if (c0 + c < k) Bc[c * 32 + lane] = 0.0f;
    }
    __syncwarp();
  };
  const uint64_t first = row0 + (uint64_t)blockIdx.x * wpb + warp;
  // With n % 4 == 0 every row starts 16-byte (FP32) / 8-byte (BF16) aligned: lane l
  // takes columns 4l..4l+3 of each 128-column stride.  Otherwise one column per lane.
  if ((n & 3) == 0) {
    constexpr int U = KBF16 ? 14 : 8;                      // loads per lane and batch
    constexpr uint64_t S = 128ull * U;                     // columns per batch
    const uint64_t j1 = (uint64_t)lane * 4;
    auto load = [&](V (&v)[U], uint64_t row, uint64_t j) {
      const T* p = reinterpret_cast<const T*>(K) + (row - row0) * n + j;
#pragma unroll
      for (int u = 0; u < U; ++u) v[u] = ld_stream4(p + 128 * u, row < row_end && j + 128ull * u < n);
    };
    auto add = [&](const V (&v)[U], uint64_t j) {
      uint32_t l4[U];
#pragma unroll
      for (int u = 0; u < U; ++u) l4[u] = j + 128ull * u < n ? lab4(j + 128ull * u) : 0u;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (j + 128ull * u >= n) break;
        const float4 x = as_float4(v[u]);
        B[(l4[u] & 255u) * 32 + lane] += x.x;
        B[((l4[u] >> 8) & 255u) * 32 + lane] += x.y;
        B[((l4[u] >> 16) & 255u) * 32 + lane] += x.z;
        B[(l4[u] >> 24) * 32 + lane] += x.w;
      }
    };
    V va[U], vb[U];
    load(va, first, j1);
    for (uint64_t row = first; row < row_end; row += nw) {
      for (uint64_t j0 = 0; j0 < n; j0 += 2 * S) {         // batches in pairs; lane 0's column starts the batch
        const bool second = j0 + S < n;
        if (second) load(vb, row, j0 + S + j1);
        add(va, j0 + j1);
        const bool more = j0 + 2 * S < n;
        if (more) load(va, row, j0 + 2 * S + j1);
        else load(va, row + nw, j1);                       // the next row's first batch
        if (second) add(vb, j0 + S + j1);
      }
      reduce(row);
    }
  } else {
    for (uint64_t row = first; row < row_end; row += nw) {
      const T* Kr = reinterpret_cast<const T*>(K) + (row - row0) * n;
      uint64_t j = lane;
      for (; j + 96 < n; j += 128) {                       // columns j, j + 32, j + 64, j + 96 of this lane
        const float4 x = make_float4(as_float(Kr[j]), as_float(Kr[j + 32]), as_float(Kr[j + 64]), as_float(Kr[j + 96]));
        bins_add4(B + lane, lab1(j) | lab1(j + 32) << 8 | lab1(j + 64) << 16 | lab1(j + 96) << 24, x);
      }
      for (; j < n; j += 32) B[lab1(j) * 32 + lane] += as_float(Kr[j]);
      reduce(row);
    }
  }
}

// Sum of one value per thread of a 256-thread block (result in thread 0), fixed order.
__device__ __forceinline__ double block_sum_256(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  return ((red[0] + red[1]) + (red[2] + red[3])) + ((red[4] + red[5]) + (red[6] + red[7]));
}

// ctilde_c = (1/|c|^2) sum_{i in c} E[i, c] in FP64, one block per cluster over its
// rows (label-sorted permutation), fixed reduction order.  Bound by latency (gathered
// loads, FP64 additions of about 40 ns each): four rows in flight per thread.
// n = 20,000 k = 20 17 -> 6 us, n = 65,536 k = 64 30 -> 7 us (a warp per cluster,
// one row after the other, before).
__global__ void __launch_bounds__(256)
kkm_ctilde_kernel(const float* __restrict__ E, uint32_t k, const uint32_t* __restrict__ perm,
                  const uint32_t* __restrict__ cstart, double* __restrict__ ct, DevState* st) {
  griddep_wait();
  griddep_launch();
  if (st->done) return;
  __shared__ double red[8];
  const uint32_t c = blockIdx.x;
  const uint32_t s0 = cstart[c], s1 = cstart[c + 1];
  double s = 0.0;
  for (uint32_t p = s0 + threadIdx.x; p < s1; p += 4u * 256u) {
    float v[4];
#pragma unroll
    for (uint32_t u = 0; u < 4; ++u)
      v[u] = s1 - p > 256u * u ? E[(uint64_t)perm[p + 256u * u] * k + c] : 0.0f;
    s += ((double)v[0] + (double)v[1]) + ((double)v[2] + (double)v[3]);
  }
  s = block_sum_256(s, red);
  if (threadIdx.x == 0) {
    const double cnt = (double)(s1 - s0);
    ct[c] = (s1 > s0) ? s / (cnt * cnt) : 0.0;
  }
}

// D[i,c] = -2 E[i,c]/|c| + ctilde_c (ctilde == 0 -> +inf), argmin from
// (0, FLT_MAX) with strict '<', new label and min; per-block FP64 score partials.
__global__ void __launch_bounds__(256)
kkm_dist_kernel(const float* __restrict__ E, uint64_t n, uint32_t k, const uint32_t* __restrict__ counts,
                const double* __restrict__ ct, uint32_t* __restrict__ newlab,
                double* __restrict__ part, DevState* st) {
  griddep_wait();
  griddep_launch();
  if (st->done) return;
  extern __shared__ float kd_smem[];
  float* inv = kd_smem;            // -2/|c| (0 for empty clusters)
  float* add = kd_smem + k;        // ctilde (+inf where 0)
  for (uint32_t c = threadIdx.x; c < k; c += blockDim.x) {
    const uint32_t cnt = counts[c];
    inv[c] = cnt ? -2.0f / (float)cnt : 0.0f;
    const float cf = (float)ct[c];
    add[c] = (cf == 0.0f) ? __int_as_float(0x7f800000) : cf;
  }
  __syncthreads();
  double acc = 0.0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const float* e = E + i * k;
    float val = FLT_MAX;
    uint32_t key = 0;
    for (uint32_t c = 0; c < k; ++c) {
      const float v = fmaf(inv[c], e[c], add[c]);
      if (v < val) { val = v; key = c; }
    }
    newlab[i] = key;
    acc += (double)val;
  }
  __shared__ double red[8];
  acc = block_sum_256(acc, red);
  if (threadIdx.x == 0) part[blockIdx.x] = acc;
}

// End of iteration: score (fixed-order sum of the block partials) and the stop rule.
// One thread's chain of FP64 additions was 7 us of an iteration at n = 20,000 (79
// partials); by 256 threads and a tree it is hidden in the launch.
__global__ void __launch_bounds__(256) kkm_control_kernel(const double* __restrict__ part, int np, LoopConsts lc,
                                   int check, DevState* st) {
  griddep_wait();
  griddep_launch();
  if (st->done) return;
  __shared__ double red[8];
  double s = 0.0;
  for (int i = threadIdx.x; i < np; i += 256) s += part[i];
  s = block_sum_256(s, red);
  if (threadIdx.x == 0) {
    const uint32_t it = st->iter + 1;
    st->iter = it;
    st->score = s;
    st->objective = s;
    bool stop = false;
    if (it >= lc.maxiter) stop = true;
    else if (check && it > 1 && fabs(s - st->last_score) < (double)lc.tol) { st->converged_iter = it; stop = true; }
    st->last_score = s;
    if (stop) st->done = 1u;
  }
}

// dst8 (optional): the byte copy of the labels that the V.K kernel reads when
// they do not fit shared memory.
__global__ void kkm_copy_labels_kernel(const uint32_t* __restrict__ src, uint32_t* __restrict__ dst,
                                       uint8_t* __restrict__ dst8, uint64_t n, DevState* st) {
  griddep_wait();
  griddep_launch();
  // runs after the control kernel: the labels of the final iteration are
  // copied too (the done flag is set by then), so only stop after copying.
  if (st->iter == 0) return;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    dst[i] = src[i];
    if (dst8) dst8[i] = (uint8_t)src[i];
  }
}

__global__ void kkm_label_bytes_kernel(const uint32_t* __restrict__ src, uint8_t* __restrict__ dst8, uint64_t n) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x)
    dst8[i] = (uint8_t)src[i];
}

}  // namespace km

using namespace km;

struct km_kkm {
  km_kkm_params p;
  LloydEngine eng;          // sort machinery, stream, state (no Lloyd buffers used)
  void* K = nullptr;        // n x n (resident) or panel x n (panels), float or bf16
  float* diag = nullptr;
  uint64_t panel = 0;       // rows of K per panel, 0 when K is resident
  uint8_t* lab8 = nullptr;  // byte labels for the V.K kernel when they do not fit shared memory
  bool glab = false;
  uint64_t kpi = 0;         // kernels launched per iteration
  // fused mode (no K): label-sorted operand copies and the fused kernel's plan
  bool fused = false;
  __nv_bfloat16* Xbp = nullptr;
  __nv_bfloat16* Xlop = nullptr;
  float* xn2p = nullptr;
  CUtensorMap fA{}, fAlo{}, fB{}, fBlo{};
  uint32_t fS = 0;
  size_t fsmem = 0;
  int fgrid = 0;
  float* E = nullptr;       // n x k
  double* ct = nullptr;
  uint32_t* lab = nullptr;  // current labels
  uint32_t* nlab = nullptr; // next labels
  double* part = nullptr;
  int dist_blocks = 0;
  size_t vk_smem = 0;
  uint32_t vk_warps = 8;          // warps per V.K block: as many as the bins leave room for (<= 16)
  bool ready = false;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  int32_t* h_done = nullptr;
  double kbuild_ms = 0.0;   // device time of the last kernel-matrix build
};

namespace km {
namespace {

KFn make_kfn(const km_kkm_params& p) {
  KFn f;
  f.kind = p.kernel_fn;
  f.gamma = p.gamma;
  f.coef = p.coef;
  f.degree = p.degree;
  f.inv2s2 = (p.sigma > 0) ? (float)(1.0 / (2.0 * (double)p.sigma * p.sigma)) : 0.0f;
  return f;
}

km_status kfn_valid(int kind, int degree, float sigma) {
  if (kind < KM_KERNEL_LINEAR || kind > KM_KERNEL_GAUSSIAN) return KM_ERR_ARG;
  if (kind == KM_KERNEL_POLY && (degree < 1 || degree > 16)) return KM_ERR_ARG;
  if (kind == KM_KERNEL_GAUSSIAN && !(sigma > 0)) return KM_ERR_ARG;
  return KM_OK;
}

// Gaussian kernel on the tensor cores: norms of the BF16 operands (see
// kmat_operand_norms_kernel); they overwrite xn2, which the kernel-matrix path
// does not otherwise use.  Once per set of points.
km_status prepare_kmat_norms(LloydEngine& e, uint64_t n, const KFn& f, int precision) {
  if (precision == KM_PREC_FP32 || f.kind != KM_KERNEL_GAUSSIAN) return KM_OK;
  kmat_operand_norms_kernel<<<(unsigned)((n * 32 + 255) / 256), 256, 0, e.stream>>>(
      e.Xb, precision == KM_PREC_BF16X3 ? e.Xlo : nullptr, n, e.dp, e.xn2);
  KM_CUDA_TRY(cudaGetLastError());
  return KM_OK;
}

// Builds rows [row0, row_end) of K (and of diag) from points X (device,
// n x d) on the engine's stream into K (row stride n, first row = row0).  For
// the tensor-core precisions it uses the BF16 copies prepared by the engine
// and the operand norms of prepare_kmat_norms.  skip_done: the launch does
// nothing once the fit has stopped (panels rebuilt inside the iteration).
// Tiles of the symmetric tensor-core build of rows [row0, row_end): row tile
// mi (128 rows) against column block nj (256 columns) for mi / 2 <= nj, in
// groups of KM_GROUP row tiles with the column blocks inside; `direct` when
// the tile's rows meet [row0, row_end), `mirror` (strictly above the
// diagonal blocks) when its transposed rows do.
std::vector<uint32_t> kmat_tile_list(uint64_t n, uint64_t row0, uint64_t row_end) {
  const uint64_t mt = (n + KM_M - 1) / KM_M, nt = (n + KM_N - 1) / KM_N;
  std::vector<uint32_t> t;
  for (uint64_t g = 0; g < mt; g += KM_GROUP)
    for (uint64_t nj = 0; nj < nt; ++nj)
      for (uint64_t mi = g; mi < std::min<uint64_t>(mt, g + KM_GROUP); ++mi) {
        if (mi / 2 > nj) continue;
        const bool direct = mi * KM_M < row_end && mi * KM_M + KM_M > row0;
        const bool mirror = mi / 2 < nj && nj * KM_N < row_end && nj * KM_N + KM_N > row0;
        if (!direct && !mirror) continue;
        t.push_back((uint32_t)mi);
        t.push_back((uint32_t)nj | (direct ? 1u << 30 : 0u) | (mirror ? 1u << 31 : 0u));
      }
  return t;
}

// The device tile list of rows [row0, row_end), built and copied on first use
// (which must not be inside a stream capture: prepare_kmat_lists covers the
// panels of a fit before its graph is captured).
km_status kmat_tiles_dev(LloydEngine& e, uint64_t n, uint64_t row0, uint64_t row_end, const uint32_t** dev,
                         uint64_t* count) {
  for (const auto& l : e.kmat_lists)
    if (l.row0 == row0 && l.row_end == row_end) { *dev = l.dev; *count = l.count; return KM_OK; }
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  KM_CUDA_TRY(cudaStreamIsCapturing(e.stream, &cs));
  if (cs != cudaStreamCaptureStatusNone) return KM_ERR_STATE;
  const std::vector<uint32_t> t = kmat_tile_list(n, row0, row_end);
  KmatTileList l;
  l.row0 = row0;
  l.row_end = row_end;
  l.count = t.size() / 2;
  KM_TRY(e.take(&l.dev, std::max<size_t>(2, t.size())));
  e.kmat_lists.push_back(l);
  // (a copy from pageable memory has left the vector when the call returns)
  KM_CUDA_TRY(cudaMemcpyAsync(l.dev, t.data(), sizeof(uint32_t) * t.size(), cudaMemcpyHostToDevice, e.stream));
  *dev = l.dev;
  *count = l.count;
  return KM_OK;
}

km_status build_kernel_matrix(LloydEngine& e, const float* X, uint64_t n, uint32_t d, const KFn& f,
                              int precision, bool out_bf16, void* K, float* diag, uint64_t row0,
                              uint64_t row_end, bool skip_done) {
  cudaStream_t s = e.stream;
  if (row0 >= row_end || row_end > n) return KM_ERR_ARG;
  const uint64_t rows = row_end - row0;
  if (precision == KM_PREC_FP32) {
    const bool symmetric = rows == n;
    const uint64_t nb = (n + 127) / 128, tiles = symmetric ? nb * (nb + 1) : nb * ((rows + 63) / 64);
    if (tiles > 0x7fffffffull) return KM_ERR_UNSUPPORTED;
    const DevState* stop = skip_done ? e.st : nullptr;
    const bool v4 = d % 4 == 0 && reinterpret_cast<uintptr_t>(X) % 16 == 0;
    const bool vec = n % 4 == 0 && reinterpret_cast<uintptr_t>(K) % 16 == 0;
    auto launch = [&](auto kern) {
      kern<<<(unsigned)tiles, 128, KmTile::SMEM, s>>>(X, v4, e.xn2, n, d, row0, row_end, symmetric ? 1 : 0, f, K, vec, diag,
                                                    stop);
    };
    switch (f.kind) {
      case KM_KERNEL_LINEAR: out_bf16 ? launch(kmat_f32_kernel<true, KM_KERNEL_LINEAR>) : launch(kmat_f32_kernel<false, KM_KERNEL_LINEAR>); break;
      case KM_KERNEL_POLY: out_bf16 ? launch(kmat_f32_kernel<true, KM_KERNEL_POLY>) : launch(kmat_f32_kernel<false, KM_KERNEL_POLY>); break;
      case KM_KERNEL_SIGMOID: out_bf16 ? launch(kmat_f32_kernel<true, KM_KERNEL_SIGMOID>) : launch(kmat_f32_kernel<false, KM_KERNEL_SIGMOID>); break;
      default: out_bf16 ? launch(kmat_f32_kernel<true, KM_KERNEL_GAUSSIAN>) : launch(kmat_f32_kernel<false, KM_KERNEL_GAUSSIAN>); break;
    }
    KM_CUDA_TRY(cudaGetLastError());
    return KM_OK;
  }
  const bool x3 = precision == KM_PREC_BF16X3;
  CUtensorMap tA{}, tAlo{}, tB{}, tBlo{};
  KM_TRY(encode_tmap_bf16(&tA, e.Xb, e.dp, n, 64, KM_M));
  KM_TRY(encode_tmap_bf16(&tB, e.Xb, e.dp, n, 64, KM_N));
  if (x3) {
    KM_TRY(encode_tmap_bf16(&tAlo, e.Xlo, e.dp, n, 64, KM_M));
    KM_TRY(encode_tmap_bf16(&tBlo, e.Xlo, e.dp, n, 64, KM_N));
  } else {
    tAlo = tA;
    tBlo = tB;
  }
  const uint32_t KBn = e.dp / 64;
  const size_t stage = (size_t)(KA_BYTES + KB_BYTES) * (x3 ? 2 : 1);
  const size_t fixed = 1024 + KM_STG_BYTES + sizeof(KmSmem) + 64;
  size_t S = (227 * 1024 - fixed) / stage;
  if (S > 8) S = 8;
  if (S < 2) return KM_ERR_UNSUPPORTED;
  const size_t smem = fixed + S * stage;
  const uint32_t* tl = nullptr;
  uint64_t tiles = 0;
  KM_TRY(kmat_tiles_dev(e, n, row0, row_end, &tl, &tiles));
  const int grid = (int)std::max<uint64_t>(1, std::min<uint64_t>(tiles, (uint64_t)e.num_sms));
  const int vec = (n % 4 == 0) && (reinterpret_cast<uintptr_t>(K) % 16 == 0);
#define KM_LAUNCH_KMAT(X3_, BF_, KIND_)                                                            \
  do {                                                                                             \
    KM_CUDA_TRY(cudaFuncSetAttribute(kmat_tc_kernel<X3_, BF_, KIND_>,                              \
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));     \
    kmat_tc_kernel<X3_, BF_, KIND_><<<grid, KM_THREADS, smem, s>>>(tA, tAlo, tB, tBlo, e.xn2, n, row0,    \
                                                            row_end, KBn, (uint32_t)S, f, K, diag, \
                                                            vec, skip_done ? 1 : 0, e.st, tl, tiles); \
  } while (0)
#define KM_LAUNCH_KIND(X3_, BF_)                                                                   \
  do {                                                                                             \
    switch (f.kind) {                                                                              \
      case KM_KERNEL_LINEAR: KM_LAUNCH_KMAT(X3_, BF_, KM_KERNEL_LINEAR); break;                    \
      case KM_KERNEL_POLY: KM_LAUNCH_KMAT(X3_, BF_, KM_KERNEL_POLY); break;                        \
      case KM_KERNEL_SIGMOID: KM_LAUNCH_KMAT(X3_, BF_, KM_KERNEL_SIGMOID); break;                  \
      default: KM_LAUNCH_KMAT(X3_, BF_, KM_KERNEL_GAUSSIAN); break;                                \
    }                                                                                              \
  } while (0)
  if (x3) { if (out_bf16) KM_LAUNCH_KIND(true, true); else KM_LAUNCH_KIND(true, false); }
  else { if (out_bf16) KM_LAUNCH_KIND(false, true); else KM_LAUNCH_KIND(false, false); }
#undef KM_LAUNCH_KIND
#undef KM_LAUNCH_KMAT
  KM_CUDA_TRY(cudaGetLastError());
  return KM_OK;
}

// Per iteration: V.K (with the K panel builds before each panel's V.K when
// K is not resident), 4 sort kernels, c~, distances/argmin, control, label
// copy; fused: the sort, the operand permutation and the fused kernel
// instead of V.K.
uint64_t kkm_kernels_per_iter(uint64_t n, uint64_t panel, bool fused) {
  if (fused) return 10;
  return panel ? 8 + 2 * ((n + panel - 1) / panel) : 9;
}

template <bool X3, int KIND>
km_status kkm_fused_attr(size_t smem) {
  KM_CUDA_TRY(cudaFuncSetAttribute(kkm_fused_tc_kernel<X3, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)smem));
  return KM_OK;
}

template <bool X3>
km_status kkm_fused_attr_kind(int kind, size_t smem) {
  switch (kind) {
    case KM_KERNEL_LINEAR: return kkm_fused_attr<X3, KM_KERNEL_LINEAR>(smem);
    case KM_KERNEL_POLY: return kkm_fused_attr<X3, KM_KERNEL_POLY>(smem);
    case KM_KERNEL_SIGMOID: return kkm_fused_attr<X3, KM_KERNEL_SIGMOID>(smem);
    default: return kkm_fused_attr<X3, KM_KERNEL_GAUSSIAN>(smem);
  }
}

// Operand copies, tensor maps and launch shape of the fused kernel.
km_status kkm_fused_plan(km_kkm* h) {
  LloydEngine& e = h->eng;
  const uint64_t n = h->p.n;
  const bool x3 = h->p.precision == KM_PREC_BF16X3;
  if (cudaMalloc(&h->Xbp, sizeof(__nv_bfloat16) * n * e.dp) != cudaSuccess ||
      (x3 && cudaMalloc(&h->Xlop, sizeof(__nv_bfloat16) * n * e.dp) != cudaSuccess) ||
      cudaMalloc(&h->xn2p, sizeof(float) * n) != cudaSuccess) {
    (void)cudaGetLastError();
    return KM_ERR_ALLOC;
  }
  KM_TRY(encode_tmap_bf16(&h->fA, e.Xb, e.dp, n, 64, KM_M));
  KM_TRY(encode_tmap_bf16(&h->fB, h->Xbp, e.dp, n, 64, KM_N));
  if (x3) {
    KM_TRY(encode_tmap_bf16(&h->fAlo, e.Xlo, e.dp, n, 64, KM_M));
    KM_TRY(encode_tmap_bf16(&h->fBlo, h->Xlop, e.dp, n, 64, KM_N));
  } else {
    h->fAlo = h->fA;
    h->fBlo = h->fB;
  }
  const size_t stage = (size_t)(KA_BYTES + KB_BYTES) * (x3 ? 2 : 1);
  const size_t fixed = 1024 + KF_STG_BYTES + sizeof(KfSmem) + 64;
  size_t S = (227 * 1024 - fixed) / stage;
  if (S > 8) S = 8;
  if (S < 2) return KM_ERR_UNSUPPORTED;
  h->fS = (uint32_t)S;
  h->fsmem = fixed + S * stage;
  h->fgrid = (int)std::min<uint64_t>((n + KM_M - 1) / KM_M, (uint64_t)e.num_sms);
  if (x3) KM_TRY(kkm_fused_attr_kind<true>(h->p.kernel_fn, h->fsmem));
  else KM_TRY(kkm_fused_attr_kind<false>(h->p.kernel_fn, h->fsmem));
  return KM_OK;
}

km_status kkm_launch_fused(km_kkm* h) {
  LloydEngine& e = h->eng;
  const uint64_t n = h->p.n;
  const bool x3 = h->p.precision == KM_PREC_BF16X3;
  cudaStream_t s = e.stream;
  kkm_permute_points_kernel<<<(unsigned)((n * 32 + 255) / 256), 256, 0, s>>>(
      e.Xb, x3 ? e.Xlo : nullptr, e.xn2, e.perm, n, e.dp, h->Xbp, h->Xlop, h->xn2p, e.st);
  KM_CUDA_TRY(cudaGetLastError());
  const KFn f = make_kfn(h->p);
  const uint32_t KBn = e.dp / 64;
#define KM_LAUNCH_FUSED(X3_, KIND_)                                                                \
  kkm_fused_tc_kernel<X3_, KIND_><<<h->fgrid, 256, h->fsmem, s>>>(h->fA, h->fAlo, h->fB, h->fBlo,  \
                                                                  e.xn2, h->xn2p, n, KBn, h->fS,   \
                                                                  f, e.cstart, h->p.k, h->E, e.st)
#define KM_LAUNCH_FUSED_KIND(X3_)                                                                  \
  do {                                                                                             \
    switch (f.kind) {                                                                              \
      case KM_KERNEL_LINEAR: KM_LAUNCH_FUSED(X3_, KM_KERNEL_LINEAR); break;                        \
      case KM_KERNEL_POLY: KM_LAUNCH_FUSED(X3_, KM_KERNEL_POLY); break;                            \
      case KM_KERNEL_SIGMOID: KM_LAUNCH_FUSED(X3_, KM_KERNEL_SIGMOID); break;                      \
      default: KM_LAUNCH_FUSED(X3_, KM_KERNEL_GAUSSIAN); break;                                    \
    }                                                                                              \
  } while (0)
  if (x3) KM_LAUNCH_FUSED_KIND(true);
  else KM_LAUNCH_FUSED_KIND(false);
#undef KM_LAUNCH_FUSED_KIND
#undef KM_LAUNCH_FUSED
  KM_CUDA_TRY(cudaGetLastError());
  return KM_OK;
}

km_status kkm_launch_vk(km_kkm* h, uint64_t r0, uint64_t r1) {
  LloydEngine& e = h->eng;
  const dim3 grid(e.num_sms), block(h->vk_warps * 32);
  const uint64_t n = h->p.n;
  const uint32_t k = h->p.k;
  cudaStream_t s = e.stream;
  if (h->p.k_bf16) {
    if (h->glab) KM_CUDA_TRY(launch_pdl(kkm_vk_kernel<true, true>, grid, block, h->vk_smem, s, h->K, n, k, h->lab, h->lab8, r0, r1, h->E, e.st));
    else KM_CUDA_TRY(launch_pdl(kkm_vk_kernel<true, false>, grid, block, h->vk_smem, s, h->K, n, k, h->lab, h->lab8, r0, r1, h->E, e.st));
  } else {
    if (h->glab) KM_CUDA_TRY(launch_pdl(kkm_vk_kernel<false, true>, grid, block, h->vk_smem, s, h->K, n, k, h->lab, h->lab8, r0, r1, h->E, e.st));
    else KM_CUDA_TRY(launch_pdl(kkm_vk_kernel<false, false>, grid, block, h->vk_smem, s, h->K, n, k, h->lab, h->lab8, r0, r1, h->E, e.st));
  }
  KM_CUDA_TRY(cudaGetLastError());
  return KM_OK;
}

km_status kkm_enqueue_iteration(km_kkm* h, const LoopConsts& lc) {
  LloydEngine& e = h->eng;
  const uint64_t n = h->p.n;
  const uint32_t k = h->p.k;
  cudaStream_t s = e.stream;
  if (h->fused) {
    // no K: the label sort first (its permutation orders the columns), then
    // the fused K.V^T
    KM_TRY(e.enqueue_sort(h->lab));
    KM_TRY(kkm_launch_fused(h));
  } else if (h->panel) {
    // K is not resident: rebuild it panel by panel, each panel streamed into
    // its rows of E before the next one overwrites it (stream order)
    const KFn f = make_kfn(h->p);
    for (uint64_t r0 = 0; r0 < n; r0 += h->panel) {
      const uint64_t r1 = std::min<uint64_t>(n, r0 + h->panel);
      KM_TRY(build_kernel_matrix(e, e.X, n, h->p.d, f, h->p.precision, h->p.k_bf16 != 0, h->K, nullptr, r0, r1,
                                 true));
      KM_TRY(kkm_launch_vk(h, r0, r1));
    }
  } else {
    KM_TRY(kkm_launch_vk(h, 0, n));
  }
  if (!h->fused) KM_TRY(e.enqueue_sort(h->lab));
  KM_CUDA_TRY(launch_pdl(kkm_ctilde_kernel, k, 256, 0, s, h->E, k, e.perm, e.cstart, h->ct, e.st));
  KM_CUDA_TRY(launch_pdl(kkm_dist_kernel, h->dist_blocks, 256, 2 * k * sizeof(float), s, h->E, n, k, e.counts, h->ct,
                         h->nlab, h->part, e.st));
  KM_CUDA_TRY(launch_pdl(kkm_control_kernel, 1, 256, 0, s, h->part, h->dist_blocks, lc, (int)h->p.check_converged, e.st));
  KM_CUDA_TRY(launch_pdl(kkm_copy_labels_kernel, (unsigned)std::min<uint64_t>((n + 255) / 256, 4096), 256, 0, s, h->nlab,
                         h->lab, h->glab ? h->lab8 : (uint8_t*)nullptr, n, e.st));
  KM_CUDA_TRY(cudaGetLastError());
  return KM_OK;
}

}  // namespace
}  // namespace km

extern "C" {

km_status km_kernel_matrix(const float* X_dev, uint64_t n, uint32_t d, int32_t kernel_fn, float gamma,
                           float coef, int32_t degree, float sigma, int32_t precision, int32_t out_bf16,
                           void* K_dev, float* diag_dev, void* stream) {
  if (!X_dev || !K_dev || n == 0 || d == 0) return KM_ERR_ARG;
  KM_TRY(kfn_valid(kernel_fn, degree, sigma));
  int dev;
  if (cudaGetDevice(&dev) != cudaSuccess) { (void)cudaGetLastError(); return KM_ERR_NO_DEVICE; }
  LloydEngine e;
  KM_TRY(e.init(n, d, 1, precision, dev, stream, EngineUse::KMAT));
  KM_TRY(e.set_points(X_dev, true, false));
  km_kkm_params p{};
  p.kernel_fn = kernel_fn; p.gamma = gamma; p.coef = coef; p.degree = degree; p.sigma = sigma;
  const KFn f = make_kfn(p);
  KM_TRY(prepare_kmat_norms(e, n, f, precision));
  KM_TRY(build_kernel_matrix(e, X_dev, n, d, f, precision, out_bf16 != 0, K_dev, diag_dev, 0, n, false));
  return e.check_device_error();
}

km_status km_kkm_create(const km_kkm_params* p, km_kkm** out) {
  if (!p || !out) return KM_ERR_ARG;
  *out = nullptr;
  if (p->n == 0 || p->d == 0 || p->k == 0 || p->k > p->n || p->maxiter == 0) return KM_ERR_ARG;
  if (p->k > 256) return KM_ERR_UNSUPPORTED;   // byte labels
  if (!(p->tol >= 0.0f)) return KM_ERR_ARG;
  KM_TRY(kfn_valid(p->kernel_fn, p->degree, p->sigma));
  const uint64_t nn = p->n * p->n;
  if (nn / p->n != p->n) return KM_ERR_ARG;
  // V.K: per-warp bins (k x 32 floats), next to the byte labels when those
  // fit beside eight warps' bins, else the labels come from a global byte
  // copy; more warps keep more K rows in flight
  constexpr size_t SMEM = 227 * 1024;
  const size_t lab_bytes = (p->n + 15) & ~15ull, bin_bytes = (size_t)p->k * 32 * sizeof(float);
  const bool glab = lab_bytes + 8 * bin_bytes > SMEM;
  const size_t lb = glab ? 0 : lab_bytes;
  uint32_t vk_warps = glab ? 1 : 8;
  while (vk_warps < 16 && lb + (size_t)(vk_warps + 1) * bin_bytes <= SMEM) ++vk_warps;
  const size_t vk_smem = lb + (size_t)vk_warps * bin_bytes;
  if (vk_smem > SMEM) return KM_ERR_UNSUPPORTED;
  km_kkm* h = new (std::nothrow) km_kkm();
  if (!h) return KM_ERR_ALLOC;
  h->p = *p;
  h->vk_smem = vk_smem;
  h->vk_warps = vk_warps;
  h->glab = glab;
  km_status s = h->eng.init(p->n, p->d, p->k, p->precision, p->device, p->stream, EngineUse::FIT);
  auto fail = [&](km_status st) { km_kkm_destroy(h); return st; };
  if (s != KM_OK) return fail(s);
  h->eng.one_block_sort = false;               // kkm_kernels_per_iter counts the kernels of the general sort
  if (cudaMalloc(&h->diag, sizeof(float) * p->n) != cudaSuccess ||
      cudaMalloc(&h->E, sizeof(float) * p->n * p->k) != cudaSuccess ||
      cudaMalloc(&h->ct, sizeof(double) * p->k) != cudaSuccess ||
      cudaMalloc(&h->lab, sizeof(uint32_t) * p->n) != cudaSuccess ||
      cudaMalloc(&h->nlab, sizeof(uint32_t) * p->n) != cudaSuccess ||
      cudaMalloc(&h->part, sizeof(double) * 1024) != cudaSuccess ||
      (glab && cudaMalloc(&h->lab8, lab_bytes) != cudaSuccess)) {
    (void)cudaGetLastError();
    return fail(KM_ERR_ALLOC);
  }
  // K last: resident (n x n), one panel of rows, or none (fused)
  const size_t bpe = p->k_bf16 ? 2 : 4;
  const bool tensor = p->precision != KM_PREC_FP32;
  uint64_t panel = 0;
  bool fused = false;
  if (p->panel_rows == KM_KKM_FUSED) {
    if (!tensor) return fail(KM_ERR_UNSUPPORTED);
    fused = true;
  } else if (p->panel_rows == KM_KKM_PANEL_AUTO) {
    scratch_trim(h->eng.device);               // what the scratch pool keeps is free for K too
    size_t fr = 0, tot = 0;
    if (cudaMemGetInfo(&fr, &tot) != cudaSuccess) { (void)cudaGetLastError(); return fail(KM_ERR_CUDA); }
    if ((double)nn * bpe > 0.9 * (double)fr) {
      if (tensor) {
        fused = true;
      } else {
        const uint64_t r = (uint64_t)(0.5 * (double)fr / ((double)p->n * bpe)) / 128 * 128;
        panel = std::min<uint64_t>(std::max<uint64_t>(r, 128), p->n);
      }
    }
  } else if (p->panel_rows > 0) {
    panel = std::min<uint64_t>(p->panel_rows, p->n);
  }
  h->panel = panel;
  h->fused = fused;
  h->kpi = kkm_kernels_per_iter(p->n, panel, fused);
  if (fused) {
    s = kkm_fused_plan(h);
    if (s != KM_OK) return fail(s);
  } else {
    const size_t kbytes = (panel ? panel * p->n : nn) * bpe;
    if (cudaMalloc(&h->K, kbytes) != cudaSuccess) { (void)cudaGetLastError(); return fail(KM_ERR_ALLOC); }
  }
  h->dist_blocks = (int)std::min<uint64_t>((p->n + 255) / 256, 1024);
  bool attr_ok = true;
  if (glab) {
    attr_ok = cudaFuncSetAttribute(kkm_vk_kernel<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   DYN_SMEM_MAX) == cudaSuccess &&
              cudaFuncSetAttribute(kkm_vk_kernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   DYN_SMEM_MAX) == cudaSuccess;
  } else {
    attr_ok = cudaFuncSetAttribute(kkm_vk_kernel<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   DYN_SMEM_MAX) == cudaSuccess &&
              cudaFuncSetAttribute(kkm_vk_kernel<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   DYN_SMEM_MAX) == cudaSuccess;
  }
  if (!attr_ok || cudaEventCreate(&h->ev0) != cudaSuccess || cudaEventCreate(&h->ev1) != cudaSuccess ||
      cudaMallocHost(reinterpret_cast<void**>(&h->h_done), sizeof(int32_t)) != cudaSuccess) {
    (void)cudaGetLastError();
    return fail(KM_ERR_CUDA);
  }
  *out = h;
  return KM_OK;
}

km_status km_kkm_set_data(km_kkm* h, const float* X, int on_device) {
  if (!h || !X) return KM_ERR_ARG;
  LloydEngine& e = h->eng;
  KM_TRY(e.set_points(X, on_device != 0, true));
  const KFn f = make_kfn(h->p);
  KM_CUDA_TRY(cudaEventRecord(h->ev0, e.stream));
  KM_TRY(prepare_kmat_norms(e, h->p.n, f, h->p.precision));
  // with panels (or fused), K is built inside every iteration instead; the
  // panels' tile lists are made here, before any iteration is captured
  if (h->panel && h->p.precision != KM_PREC_FP32) {
    for (uint64_t r0 = 0; r0 < h->p.n; r0 += h->panel) {
      const uint32_t* tl = nullptr;
      uint64_t cnt = 0;
      KM_TRY(kmat_tiles_dev(e, h->p.n, r0, std::min<uint64_t>(h->p.n, r0 + h->panel), &tl, &cnt));
    }
  }
  if (!h->panel && !h->fused)
    KM_TRY(build_kernel_matrix(e, e.X, h->p.n, h->p.d, f, h->p.precision, h->p.k_bf16 != 0, h->K, h->diag, 0,
                               h->p.n, false));
  KM_CUDA_TRY(cudaEventRecord(h->ev1, e.stream));
  KM_CUDA_TRY(cudaEventSynchronize(h->ev1));
  float ms = 0.f;
  KM_CUDA_TRY(cudaEventElapsedTime(&ms, h->ev0, h->ev1));
  h->kbuild_ms = ms;
  KM_TRY(e.check_device_error());
  h->ready = true;
  return KM_OK;
}

km_status km_kkm_panel_rows(km_kkm* h, uint64_t* rows) {
  if (!h || !rows) return KM_ERR_ARG;
  *rows = h->fused ? KM_KKM_FUSED : h->panel;
  return KM_OK;
}

km_status km_kkm_build_ms(km_kkm* h, double* ms) {
  if (!h || !ms) return KM_ERR_ARG;
  if (!h->ready) return KM_ERR_STATE;
  *ms = h->kbuild_ms;
  return KM_OK;
}

km_status km_kkm_configure(km_kkm* h, uint64_t maxiter, float tol, int32_t check_converged) {
  if (!h || maxiter == 0 || !(tol >= 0.0f)) return KM_ERR_ARG;
  h->p.maxiter = maxiter;
  h->p.tol = tol;
  h->p.check_converged = check_converged != 0;
  return KM_OK;
}

km_status km_kkm_fit(km_kkm* h, const uint32_t* init_labels, uint32_t* labels_out, km_result* res) {
  if (!h) return KM_ERR_ARG;
  if (!h->ready) return KM_ERR_STATE;
  LloydEngine& e = h->eng;
  KM_CUDA_TRY(cudaSetDevice(e.device));
  KM_TRY(e.reset_state());
  const uint64_t n = h->p.n;
  if (init_labels) {
    for (uint64_t i = 0; i < n; ++i)
      if (init_labels[i] >= h->p.k) return KM_ERR_ARG;
    KM_CUDA_TRY(cudaMemcpyAsync(h->lab, init_labels, sizeof(uint32_t) * n, cudaMemcpyHostToDevice, e.stream));
  } else {
    round_robin_labels_kernel<<<(unsigned)((n + 255) / 256), 256, 0, e.stream>>>(h->lab, n, h->p.k);
    KM_CUDA_TRY(cudaGetLastError());
  }
  if (h->glab) {
    kkm_label_bytes_kernel<<<(unsigned)std::min<uint64_t>((n + 255) / 256, 4096), 256, 0, e.stream>>>(h->lab,
                                                                                                   h->lab8, n);
    KM_CUDA_TRY(cudaGetLastError());
  }
  LoopConsts lc{h->p.maxiter, h->p.tol, h->p.check_converged ? KM_CONV_SCORE : KM_CONV_NONE, 0};
  KM_CUDA_TRY(cudaEventRecord(h->ev0, e.stream));
  uint64_t launched = 0, batch = h->p.check_converged ? 4 : h->p.maxiter;
  while (launched < h->p.maxiter) {
    const uint64_t target = std::min<uint64_t>(h->p.maxiter, launched + batch);
    for (; launched < target; ++launched) KM_TRY(kkm_enqueue_iteration(h, lc));
    if (launched >= h->p.maxiter) break;
    KM_CUDA_TRY(cudaMemcpyAsync(h->h_done, &e.st->done, sizeof(int32_t), cudaMemcpyDeviceToHost, e.stream));
    KM_CUDA_TRY(cudaStreamSynchronize(e.stream));
    if (*h->h_done) break;
    batch = std::min<uint64_t>(batch * 2, 64);
  }
  KM_CUDA_TRY(cudaEventRecord(h->ev1, e.stream));
  KM_TRY(e.check_device_error());
  float ms = 0;
  KM_CUDA_TRY(cudaEventElapsedTime(&ms, h->ev0, h->ev1));
  if (labels_out)
    KM_CUDA_TRY(cudaMemcpyAsync(labels_out, h->lab, sizeof(uint32_t) * n, cudaMemcpyDeviceToHost, e.stream));
  KM_CUDA_TRY(cudaStreamSynchronize(e.stream));
  const DevState& s = *e.h_st;
  if (res) {
    std::memset(res, 0, sizeof(*res));
    res->iterations = s.iter;
    res->converged = s.converged_iter != 0;
    res->converged_iter = s.converged_iter ? s.converged_iter : h->p.maxiter;
    res->objective = s.objective;
    res->score = s.score;
    res->fit_ms = ms;
    res->kernel_launches = launched * h->kpi;
  }
  return KM_OK;
}

void km_kkm_destroy(km_kkm* h) {
  if (!h) return;
  if (h->eng.device >= 0) cudaSetDevice(h->eng.device);
  if (h->K) cudaFree(h->K);
  if (h->diag) cudaFree(h->diag);
  if (h->E) cudaFree(h->E);
  if (h->ct) cudaFree(h->ct);
  if (h->lab) cudaFree(h->lab);
  if (h->nlab) cudaFree(h->nlab);
  if (h->lab8) cudaFree(h->lab8);
  if (h->Xbp) cudaFree(h->Xbp);
  if (h->Xlop) cudaFree(h->Xlop);
  if (h->xn2p) cudaFree(h->xn2p);
  if (h->part) cudaFree(h->part);
  if (h->ev0) cudaEventDestroy(h->ev0);
  if (h->ev1) cudaEventDestroy(h->ev1);
  if (h->h_done) cudaFreeHost(h->h_done);
  delete h;
}

}  // extern "C"
