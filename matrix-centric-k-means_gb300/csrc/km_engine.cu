// Lloyd engine host code: buffers, preparation and the per-iteration launch
// sequence (assign -> refine -> sort -> update -> finalize -> control).
#include "km_lloyd.cuh"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <mutex>
#include <string>

namespace km {

namespace {
thread_local std::string g_last_error;

constexpr int MAX_DEVICES = 64;
std::mutex g_pool_mu;
cudaMemPool_t g_pool[MAX_DEVICES] = {};
bool g_pool_tried[MAX_DEVICES] = {};
std::atomic<uint64_t> g_lent[MAX_DEVICES] = {};   // bytes lent by the device's pool

// The device's pool (null: none), made on the first use.
cudaMemPool_t device_pool(int device) {
  if (device < 0 || device >= MAX_DEVICES) return nullptr;
  std::lock_guard<std::mutex> lk(g_pool_mu);
  if (!g_pool_tried[device]) {
    g_pool_tried[device] = true;
    int ok = 0;
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    uint64_t keep = SCRATCH_KEEP;
    cudaMemPool_t pool = nullptr;
    if (cudaDeviceGetAttribute(&ok, cudaDevAttrMemoryPoolsSupported, device) == cudaSuccess && ok &&
        cudaMemPoolCreate(&pool, &props) == cudaSuccess &&
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) == cudaSuccess)
      g_pool[device] = pool;
    (void)cudaGetLastError();
  }
  return g_pool[device];
}

uint32_t round_up(uint32_t v, uint32_t m) { return (v + m - 1) / m * m; }
}  // namespace

void set_last_error(cudaError_t e, const char* what, const char* file, int line) {
  char buf[512];
  snprintf(buf, sizeof buf, "%s failed: %s (%s:%d)", what, cudaGetErrorString(e), file, line);
  g_last_error = buf;
}

const char* last_error_text() { return g_last_error.c_str(); }

km_status scratch_alloc(Scratch* b, size_t bytes, int device, cudaStream_t s) {
  *b = Scratch{};
  cudaMemPool_t pool = device_pool(device);
  if (pool && g_lent[device].fetch_add(bytes) + bytes > SCRATCH_KEEP) {
    g_lent[device] -= bytes;
    pool = nullptr;
  }
  for (int attempt = 0; attempt < 2; ++attempt) {
    const cudaError_t e = pool ? cudaMallocFromPoolAsync(&b->p, bytes, pool, s) : cudaMalloc(&b->p, bytes);
    if (e == cudaSuccess) {
      b->lent = pool ? bytes : 0;
      return KM_OK;
    }
    set_last_error(e, "scratch allocation", __FILE__, __LINE__);
    (void)cudaGetLastError();
    b->p = nullptr;
    if (e != cudaErrorMemoryAllocation) {
      if (pool) g_lent[device] -= bytes;
      return KM_ERR_CUDA;
    }
    scratch_trim(device);
  }
  if (pool) g_lent[device] -= bytes;
  return KM_ERR_ALLOC;
}

void scratch_free(const Scratch& b, int device, cudaStream_t s) {
  if (!b.p) return;
  if (b.lent) {
    cudaFreeAsync(b.p, s);
    g_lent[device] -= b.lent;
  } else {
    cudaFree(b.p);                           // (waits for the work that uses it)
  }
}

void scratch_trim(int device) {
  if (cudaMemPool_t pool = device_pool(device)) {
    cudaMemPoolTrimTo(pool, 0);
    (void)cudaGetLastError();
  }
}

void scratch_settle(int device, cudaStream_t s) {
  cudaMemPool_t pool = device_pool(device);
  uint64_t held = 0;
  if (pool && cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &held) == cudaSuccess &&
      held > SCRATCH_KEEP && cudaStreamSynchronize(s) == cudaSuccess)
    cudaMemPoolTrimTo(pool, SCRATCH_KEEP);
  (void)cudaGetLastError();
}

km_status LloydEngine::take_bytes(void** p, size_t bytes) {
  *p = nullptr;
  Scratch b;
  if (use != EngineUse::FIT) {
    KM_TRY(scratch_alloc(&b, bytes, device, stream));
  } else {
    cudaError_t e = cudaMalloc(&b.p, bytes);
    if (e == cudaErrorMemoryAllocation) {
      (void)cudaGetLastError();
      scratch_trim(device);
      e = cudaMalloc(&b.p, bytes);
    }
    if (e != cudaSuccess) {
      set_last_error(e, "cudaMalloc", __FILE__, __LINE__);
      (void)cudaGetLastError();
      return KM_ERR_ALLOC;
    }
  }
  owned.push_back(b);
  *p = b.p;
  return KM_OK;
}

// Relative error coefficients of the fast distance path (see TieBound).
TieBound make_tie_bound(int precision, uint32_t d, bool a_exact, uint32_t terms) {
  const double u = std::ldexp(1.0, -24);
  const double ub = std::ldexp(1.0, -8);
  const double uacc = std::ldexp(1.0, -22);  // tensor-core FP32 accumulation, 4 ulp per add
  auto gamma = [](double m, double uu) { return m * uu / (1.0 - m * uu); };
  double eps;
  if (precision == KM_PREC_FP32) {
    eps = gamma((double)(terms ? terms : d), u);
  } else if (precision == KM_PREC_BF16) {
    // |x^ c^ - x c| <= (2ub + ub^2) |x||c| per term (ub only when x^ = x),
    // plus FP32 accumulation of d products
    eps = a_exact ? ub + (1 + ub) * gamma((double)d, uacc)
                  : 2 * ub + ub * ub + (1 + ub) * (1 + ub) * gamma((double)d, uacc);
  } else if (a_exact) {
    // split-2: c = c_hi + c_lo + r, |r| <= ub^2 |c|; 2d exact products accumulated
    eps = ub * ub + (1 + 2 * ub) * gamma(2.0 * d, uacc);
  } else {
    eps = 3.5 * ub * ub + (1 + 5 * ub) * gamma(3.0 * d, uacc);
  }
  TieBound tb;
  tb.A = (float)(2.02 * eps + 2.1 * u);
  tb.B = (float)(2.1 * u);
  tb.g = (float)(gamma((double)d + 2.0, u) * 1.01);
  tb.safety = 1.25f;
  return tb;
}

LloydEngine::~LloydEngine() {
  if (device >= 0) cudaSetDevice(device);
  for (const Scratch& b : owned) scratch_free(b, device, stream);
  if (use != EngineUse::FIT && !owned.empty()) scratch_settle(device, stream);
  if (h_st && h_st != &h_one) cudaFreeHost(h_st);
  if (aux) cudaStreamDestroy(aux);
  if (ev_default) cudaEventDestroy(ev_default);
  if (ev_fork) cudaEventDestroy(ev_fork);
  if (ev_join) cudaEventDestroy(ev_join);
  if (own_stream && stream) cudaStreamDestroy(stream);
}

// A caller without a stream makes and uses its device memory on the default stream, which
// a non-blocking stream does not wait for by itself: its points may still be on their way,
// and memory handed out for the outputs may still be in use.  The default stream in turn
// follows every blocking stream, so their work is waited for too.
km_status LloydEngine::follow_default_stream() {
  if (!own_stream) return KM_OK;
  // While a blocking stream is captured, nothing may be queued on the default stream,
  // by the caller either.
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(cudaStreamLegacy, &cap) != cudaSuccess) {
    (void)cudaGetLastError();
    return KM_OK;
  }
  // Nothing queued there (nor on a blocking stream): nothing to wait for, and the event's
  // 4 us are spared.
  if (cudaStreamQuery(cudaStreamLegacy) == cudaSuccess) return KM_OK;
  (void)cudaGetLastError();
  if (!ev_default) KM_CUDA_TRY(cudaEventCreateWithFlags(&ev_default, cudaEventDisableTiming));
  KM_CUDA_TRY(cudaEventRecord(ev_default, cudaStreamLegacy));
  KM_CUDA_TRY(cudaStreamWaitEvent(stream, ev_default, 0));
  return KM_OK;
}

km_status LloydEngine::init(uint64_t n_, uint32_t d_, uint32_t k_, int precision_, int device_,
                            void* stream_, EngineUse use_) {
  if (n_ == 0 || d_ == 0 || k_ == 0 || k_ > n_) return KM_ERR_ARG;
  if (n_ >= (1ull << 32) - 256) return KM_ERR_ARG;           // labels / perm are 32-bit
  if ((uint64_t)d_ * n_ / d_ != n_) return KM_ERR_ARG;
  if (precision_ < KM_PREC_FP32 || precision_ > KM_PREC_BF16X3) return KM_ERR_ARG;
  n = n_; d = d_; k = k_; precision = precision_; device = device_; use = use_;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) { (void)cudaGetLastError(); return KM_ERR_NO_DEVICE; }
  if (device < 0 || device >= ndev) return KM_ERR_ARG;
  KM_CUDA_TRY(cudaSetDevice(device));
  int major = 0, minor = 0;
  KM_CUDA_TRY(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device));
  KM_CUDA_TRY(cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, device));
  if (major != 10 || minor != 3) return KM_ERR_NO_DEVICE;  // code is built for sm_103a only
  KM_CUDA_TRY(cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, device));
  if (stream_) {
    stream = static_cast<cudaStream_t>(stream_);
  } else {
    KM_CUDA_TRY(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
    own_stream = true;
    if (use != EngineUse::FIT) KM_TRY(follow_default_stream());   // (a handle's device inputs come later)
  }
  dp = round_up(d, 64);
  kp = round_up(std::max<uint32_t>(k, 16), 16);
  if (precision != KM_PREC_FP32) {
    // planned for the widest operands of the precision; SPLIT2 (chosen at
    // set_points when the points turn out to be exact BF16) needs less
    const int plan_mode = precision == KM_PREC_BF16X3 ? TC_SPLIT3 : TC_PLAIN;
    if (kp <= 256) tc = plan_tc(dp, kp, plan_mode, n, num_sms);
    if (!tc.ok) {
      // k > 256, or the centroid operand does not fit shared memory whole
      tc = plan_tc_chunked(dp, k, plan_mode, n, num_sms);
      if (tc.ok) kp = tc.kp;            // centroid operand padded to whole chunks
    }
    if (!tc.ok) return KM_ERR_UNSUPPORTED;
    KM_TRY(tc_set_attributes(tc, plan_mode));
    if (plan_mode == TC_SPLIT3) KM_TRY(tc_set_attributes(tc, TC_SPLIT2));
    tc_mode = plan_mode;
  }
  tb = make_tie_bound(precision, d, false);

  const bool points = use != EngineUse::UPDATE, assigns = use == EngineUse::FIT || use == EngineUse::ASSIGN,
             updates = use == EngineUse::FIT || use == EngineUse::UPDATE;
  if (points) {
    KM_TRY(take(&xn2, n));
    if (use == EngineUse::FIT) {               // sum ||x||^2 (the score) belongs to a fit
      KM_TRY(take(&xn2d, n));
      KM_TRY(take(&red_part, 256));
    }
    if (precision != KM_PREC_FP32) {
      KM_TRY(take(&Xb, (size_t)n * dp));
      if (precision == KM_PREC_BF16X3) KM_TRY(take(&Xlo, (size_t)n * dp));
    }
  }
  if (assigns) {
    if (precision != KM_PREC_FP32) {
      KM_TRY(take(&Cb, (size_t)kp * dp));
      if (precision == KM_PREC_BF16X3) KM_TRY(take(&Clo, (size_t)kp * dp));
    }
    KM_TRY(take(&C, (size_t)k * d));
    KM_TRY(take(&Ct, (size_t)k * d));
    KM_TRY(take(&cn2, (kp + 63) & ~63u));        // padded: +inf up to a multiple of 64
    if (use == EngineUse::FIT) {               // one call writes the caller's arrays
      KM_TRY(take(&labels, n));
      KM_TRY(take(&mindist, n));
    }
    const uint64_t rows = (n + 127) / 128 * 128;     // whole 128-row tiles
    KM_TRY(take(&queue, rows));
    KM_TRY(take(&qfull, rows));
    KM_TRY(take(&qcnt, rows / 32));
    KM_TRY(take(&qfcnt, rows / 32));
    rq = RefineQueues{queue, qfull, qcnt, qfcnt, rows / 32};
    if (precision != KM_PREC_FP32 && tc.chunked) {
      // candidate lists of the chunked distance kernel: up to 256 per row,
      // fewer when the lists would pass 16 GiB
      uint32_t L = 256;
      while (L > 32 && (uint64_t)rows * L * sizeof(uint2) > (16ull << 30)) L -= 32;
      KM_TRY(take(&qwide, rows));
      KM_TRY(take(&qwcnt, rows / 32));
      KM_TRY(take(&wlc, rows));
      KM_TRY(take(&wl, (size_t)rows * L));
      rq.wide = qwide; rq.wcnt = qwcnt; rq.wl = wl; rq.wlc = wlc; rq.L = L;
      KM_TRY(take(&q2, rows));
      KM_TRY(take(&q2full, rows));
      KM_TRY(take(&q2cnt, rows / 32));
      KM_TRY(take(&q2fcnt, rows / 32));
      KM_TRY(take(&fidx, rows));
      KM_TRY(take(&nfull, 1));
      // the FP32 pass's queues; its wide queue and lists take over the first ones'
      rq2 = RefineQueues{q2, q2full, q2cnt, q2fcnt, rows / 32, qwide, qwcnt, wl, wlc, L};
      tb32 = make_tie_bound(KM_PREC_FP32, d, false, f32_gather_terms(d));
    }
    KM_TRY(refine_prepare());
  }
  KM_TRY(take(&st, 1));
  if (use == EngineUse::FIT) KM_CUDA_TRY(cudaMallocHost(reinterpret_cast<void**>(&h_st), sizeof(DevState)));
  else h_st = &h_one;
  std::memset(h_st, 0, sizeof(DevState));
  KM_CUDA_TRY(cudaMemsetAsync(st, 0, sizeof(DevState), stream));
  if (!updates) return KM_OK;

  // Stable-sort geometry: segments of `seg` rows, k x nseg counts.  A segment is one
  // warp's chain of steps, so few rows are sorted in short ones: at most 1024 segments
  // (one group of loads of the scan), and no fewer rows than counts.
  // Scatter at n = 200,000 k = 64 10.5 us with segments of 1024 -> 4.7, n = 1,797 5.3 ->
  // 2.6; up to 2048 segments the scan loses what the scatter gains (6.7 -> 9.1, 4.7 -> 4.8).
  seg = 128;
  while (seg < 1024 && (seg < k || n > (uint64_t)seg * 1024)) seg <<= 1;
  nseg = (uint32_t)((n + seg - 1) / seg);
  while ((uint64_t)k * nseg > (16ull << 20) && seg < (1u << 30)) {
    seg <<= 1;
    nseg = (uint32_t)((n + seg - 1) / seg);
  }
  const size_t per_warp = (size_t)k * 4;
  if (per_warp <= 6144) sort_wpb = 8;
  else sort_wpb = (int)std::max<size_t>(1, (48 * 1024) / per_warp);
  // no more warps a block than spread the segments over one block an SM
  sort_wpb = (int)std::min<uint64_t>(sort_wpb, std::max<uint64_t>(1, (nseg + num_sms - 1) / num_sms));
  sort_smem = per_warp * sort_wpb;
  if (sort_smem > 227 * 1024) return KM_ERR_UNSUPPORTED;
  if (sort_smem > 48 * 1024) {
    KM_CUDA_TRY(cudaFuncSetAttribute(seg_hist_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DYN_SMEM_MAX));
    KM_CUDA_TRY(cudaFuncSetAttribute(seg_scatter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DYN_SMEM_MAX));
  }
  one_block_sort = n <= ONE_BLOCK_ROWS && k <= 256;
  KM_TRY(update_sums_prepare());
  if (use == EngineUse::FIT) {
    KM_TRY(take(&Cn, (size_t)k * d));
    KM_TRY(take(&dsq, (size_t)k * d));
    KM_TRY(take(&objpart, (size_t)k * d));
    KM_TRY(take(&move2_c, k));
    KM_TRY(take(&obj_c, k));
  }
  KM_TRY(take(&seghist, (size_t)k * nseg));
  KM_TRY(take(&counts, k));
  KM_TRY(take(&cstart, (size_t)k + 1));
  KM_TRY(take(&order, k));
  KM_TRY(take(&perm, n));
  return KM_OK;
}

namespace {
// Whether p is memory of this device itself.  A copy takes other GPUs' and managed memory
// as well; a kernel that reads in its place would need access to the other GPU.
bool on_this_device(const void* p, int device) {
  cudaPointerAttributes a;
  const bool ok = cudaPointerGetAttributes(&a, p) == cudaSuccess && a.type == cudaMemoryTypeDevice && a.device == device;
  (void)cudaGetLastError();
  return ok;
}
}  // namespace

km_status LloydEngine::set_points(const float* Xsrc, bool on_device, bool copy) {
  KM_CUDA_TRY(cudaSetDevice(device));
  if (on_device && use == EngineUse::FIT) KM_TRY(follow_default_stream());
  const size_t bytes = sizeof(float) * n * d;
  // A large host source is copied in row chunks alternating between the
  // handle's stream and a second one (two copy engines), and each chunk's
  // preparation (norms, BF16 copies) runs behind its own copy, overlapping
  // the copies of the chunks after it.
  const bool chunked = !on_device && bytes >= (64ull << 20);
  if (copy || !on_device) {
    if (!X_owned) KM_TRY(take(&X_owned, (size_t)n * d));
    X = X_owned;
  } else {
    X = Xsrc;
  }
  refine_v4 = (d % 4 == 0) && (reinterpret_cast<uintptr_t>(X) % 16 == 0);
  KM_CUDA_TRY(cudaMemsetAsync(&st->err, 0, sizeof(uint32_t), stream));
  KM_CUDA_TRY(cudaMemsetAsync(&st->x_not_bf16, 0, sizeof(uint32_t), stream));
  if (chunked) {
    if (!aux) {
      KM_CUDA_TRY(cudaStreamCreateWithFlags(&aux, cudaStreamNonBlocking));
      KM_CUDA_TRY(cudaEventCreateWithFlags(&ev_fork, cudaEventDisableTiming));
      KM_CUDA_TRY(cudaEventCreateWithFlags(&ev_join, cudaEventDisableTiming));
    }
    KM_CUDA_TRY(cudaEventRecord(ev_fork, stream));
    KM_CUDA_TRY(cudaStreamWaitEvent(aux, ev_fork, 0));
    const uint64_t nch = 8, rows = (n + nch - 1) / nch;
    for (uint64_t c = 0; c < nch; ++c) {
      const uint64_t r0 = c * rows, r1 = std::min<uint64_t>(n, r0 + rows);
      if (r0 >= r1) break;
      cudaStream_t sc = (c & 1) ? aux : stream;
      KM_CUDA_TRY(cudaMemcpyAsync(X_owned + r0 * d, Xsrc + r0 * d, sizeof(float) * (r1 - r0) * d,
                                  cudaMemcpyHostToDevice, sc));
      launch_prep_points(X + r0 * d, r1 - r0, d, dp, xn2 + r0, xn2d ? xn2d + r0 : nullptr, nullptr,
                         Xb ? Xb + r0 * dp : nullptr, Xlo ? Xlo + r0 * dp : nullptr, st, num_sms, sc);
    }
    KM_CUDA_TRY(cudaEventRecord(ev_join, aux));
    KM_CUDA_TRY(cudaStreamWaitEvent(stream, ev_join, 0));
  } else {
    // A copy within the device is made by the preparation, which reads the points anyway.
    const bool fused = on_device && copy && on_this_device(Xsrc, device);
    if (!on_device)
      KM_CUDA_TRY(cudaMemcpyAsync(X_owned, Xsrc, bytes, cudaMemcpyHostToDevice, stream));
    else if (copy && !fused)
      KM_CUDA_TRY(cudaMemcpyAsync(X_owned, Xsrc, bytes, cudaMemcpyDeviceToDevice, stream));
    launch_prep_points(fused ? Xsrc : X, n, d, dp, xn2, xn2d, fused ? X_owned : nullptr, Xb, Xlo, st, num_sms, stream);
  }
  KM_CUDA_TRY(cudaGetLastError());
  if (xn2d) {
    reduce_f64_partial_kernel<<<256, 256, 0, stream>>>(xn2d, n, red_part);
    reduce_f64_final_kernel<<<1, 256, 0, stream>>>(red_part, 256, &st->sum_x2);
    KM_CUDA_TRY(cudaGetLastError());
  }
  if (precision != KM_PREC_FP32 && Cb) {
    KM_TRY(encode_tmap_bf16(&tmA, Xb, dp, n, 64, 128));
    const uint32_t bbox = tc.chunked ? tc.NC : kp;    // rows of one B load
    KM_TRY(encode_tmap_bf16(&tmB, Cb, dp, kp, 64, bbox));
    if (precision == KM_PREC_BF16X3) {
      KM_TRY(encode_tmap_bf16(&tmAlo, Xlo, dp, n, 64, 128));
      KM_TRY(encode_tmap_bf16(&tmBlo, Clo, dp, kp, 64, bbox));
    } else {
      tmAlo = tmA;
      tmBlo = tmB;
    }
  }
  KM_TRY(read_state());
  if (h_st->err & KM_DEVERR_NONFINITE) return KM_ERR_ARG;
  a_exact = h_st->x_not_bf16 == 0u;
  tb = make_tie_bound(precision, d, a_exact);
  if (precision == KM_PREC_BF16X3) tc_mode = a_exact ? TC_SPLIT2 : TC_SPLIT3;
  data_ready = true;
  return KM_OK;
}

namespace {
__global__ void bf16_decode_kernel(const uint16_t* __restrict__ src, uint64_t count, float* __restrict__ dst) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count;
       i += (uint64_t)gridDim.x * blockDim.x)
    dst[i] = __uint_as_float((uint32_t)src[i] << 16);
}
}  // namespace

km_status LloydEngine::set_points_bf16(const uint16_t* Xsrc, bool on_device) {
  KM_CUDA_TRY(cudaSetDevice(device));
  if (on_device) KM_TRY(follow_default_stream());
  if (!X_owned) KM_TRY(take(&X_owned, (size_t)n * d));
  const uint64_t count = n * (uint64_t)d;
  const uint16_t* src = Xsrc;
  uint16_t* tmp = nullptr;
  Scratch staging;
  if (!on_device) {
    // host BF16 bits go to a staging buffer (half the bytes of the FP32 copy)
    KM_TRY(scratch_alloc(&staging, sizeof(uint16_t) * count, device, stream));
    tmp = static_cast<uint16_t*>(staging.p);
    KM_CUDA_TRY(cudaMemcpyAsync(tmp, Xsrc, sizeof(uint16_t) * count, cudaMemcpyHostToDevice, stream));
    src = tmp;
  }
  const unsigned blocks = (unsigned)std::min<uint64_t>((count + 255) / 256, (uint64_t)num_sms * 32);
  bf16_decode_kernel<<<blocks, 256, 0, stream>>>(src, count, X_owned);
  cudaError_t le = cudaGetLastError();
  if (tmp) {
    cudaError_t se = cudaStreamSynchronize(stream);
    scratch_free(staging, device, stream);
    KM_CUDA_TRY(le);
    KM_CUDA_TRY(se);
  }
  KM_CUDA_TRY(le);
  return set_points(X_owned, true, false);
}

km_status LloydEngine::reset_state() {
  // Keep sum_x2 (computed at set_points); zero everything else.
  KM_TRY(read_state());
  const double sx = h_st->sum_x2;
  std::memset(h_st, 0, sizeof(DevState));
  h_st->sum_x2 = sx;
  KM_CUDA_TRY(cudaMemcpyAsync(st, h_st, sizeof(DevState), cudaMemcpyHostToDevice, stream));
  KM_CUDA_TRY(cudaStreamSynchronize(stream));
  return KM_OK;
}

km_status LloydEngine::set_centroids_dev(const float* Csrc) {
  if (Csrc != C)
    KM_CUDA_TRY(cudaMemcpyAsync(C, Csrc, sizeof(float) * k * d, cudaMemcpyDeviceToDevice, stream));
  KM_CUDA_TRY(cudaMemsetAsync(&st->cmax, 0, sizeof(float), stream));
  const uint32_t kp64 = (kp + 63) & ~63u;
  const int blocks = (int)((kp64 * 32 + 255) / 256);
  prep_centroids_kernel<<<blocks, 256, 0, stream>>>(C, k, kp, d, dp, cn2, Cb, Clo, Ct, st, kp64);
  KM_CUDA_TRY(cudaGetLastError());
  return KM_OK;
}

km_status LloydEngine::enqueue_distance(float* Dout) {
  if (precision == KM_PREC_FP32) {
    KM_TRY(launch_assign_f32(X, C, cn2, xn2, n, d, k, tb, st, labels, mindist, rq, Dout, stream));
  } else {
    KM_TRY(launch_assign_tc(tc, tc_mode, tmA, tmAlo, tmB, tmBlo, cn2, xn2, n, k,
                            kp, tb, st, labels, mindist, rq, Dout, stream));
  }
  return KM_OK;
}

km_status LloydEngine::enqueue_refine() {
  if (rq.wide)
    return launch_refine_gemm(refine_v4, num_sms, X, C, Ct, cn2, xn2, n, d, k, tb32, st, rq, rq2, fidx,
                              nfull, labels, mindist, stream);
  return launch_refine(refine_v4, num_sms, X, C, Ct, d, k, st, rq, labels, mindist, stream);
}

km_status LloydEngine::enqueue_assign(float* Dout) {
  KM_TRY(enqueue_distance(Dout));
  return enqueue_refine();
}

km_status LloydEngine::enqueue_finalize(const LoopConsts& lc) {
  const unsigned threads = k <= 512 ? 64 : 256;      // (see the kernel)
  KM_CUDA_TRY(launch_pdl(finalize_kernel, (k * 32 + threads - 1) / threads, threads, 0, stream, Cn, C, dsq, objpart, counts,
                         lc.empty, d, dp, k, lc.tol, cn2, Cb, Clo, Ct, move2_c, obj_c, st, lc));
  KM_CUDA_TRY(cudaGetLastError());
  return KM_OK;
}

km_status LloydEngine::enqueue_sort(const uint32_t* lab) {
  if (one_block_sort) {
    KM_CUDA_TRY(launch_pdl(one_block_sort_kernel, 1, 1024, 32 * k * sizeof(uint32_t), stream, lab, (uint32_t)n, k, counts,
                           cstart, order, perm, st));
    KM_CUDA_TRY(cudaGetLastError());
    return KM_OK;
  }
  const unsigned hb = (nseg + sort_wpb - 1) / sort_wpb;
  // programmatic dependent launches: each kernel waits for its predecessor
  // (griddepcontrol.wait) before reading, but is scheduled while it drains
  KM_CUDA_TRY(launch_pdl(seg_hist_kernel, hb, sort_wpb * 32, sort_smem, stream, lab, n, k, seg, nseg, seghist, st));
  // per-cluster segment scans; the last block also scans the cluster counts
  const unsigned st_threads = k <= 256 ? 128 : 512;
  KM_CUDA_TRY(launch_pdl(seg_scan_kernel, (k * 32 + st_threads - 1) / st_threads, st_threads, 0, stream, seghist, k, nseg, counts, st,
                         cstart, order));
  KM_CUDA_TRY(launch_pdl(seg_scatter_kernel, hb, sort_wpb * 32, sort_smem, stream, lab, n, k, seg, nseg, seghist,
                         cstart, perm, st));
  KM_CUDA_TRY(cudaGetLastError());
  return KM_OK;
}

km_status LloydEngine::enqueue_update_step(float tol) {
  (void)tol;
  return launch_update_sums(X, perm, cstart, n, d, k, C, Cn, dsq, objpart, st, stream, order);
}

km_status LloydEngine::enqueue_iteration(const LoopConsts& lc) {
  KM_TRY(enqueue_assign(nullptr));
  KM_TRY(enqueue_sort(labels));
  KM_TRY(enqueue_update_step(lc.tol));
  return enqueue_finalize(lc);
}

km_status LloydEngine::read_state() {
  KM_CUDA_TRY(cudaMemcpyAsync(h_st, st, sizeof(DevState), cudaMemcpyDeviceToHost, stream));
  KM_CUDA_TRY(cudaStreamSynchronize(stream));
  return KM_OK;
}

km_status LloydEngine::check_device_error() {
  KM_TRY(read_state());
  return status_of_device_error(h_st->err);
}

}  // namespace km
