// RMSNorm / LayerNorm forward and backward: one CTA per row (rows of a few
// thousand elements: the row stays in registers between the statistics pass and
// the normalisation pass, so HBM sees exactly one read of x and one write of y),
// fp32 statistics, 128-bit accesses.  Weight gradients are accumulated per CTA
// over a strip of rows and written as [n_strips, cols] fp32 partial sums which
// the caller reduces with the column-sum kernel (deterministic, no atomics).
// Parity: reference torch_musa/csrc/aten/ops/RMSNorm.cpp:113-125,283-306 and
// LayerNorm.cpp:141-147,295-300 (vendor-library calls there).
#include "gemm_common.cuh"   // mbarriers

#include <algorithm>

namespace b200k {
namespace {

constexpr int kMaxRmsStages = 4;

// contiguous bytes from global to shared memory, credited to the barrier (16-byte aligned, a multiple of 16 bytes)
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(gemmdev::smem_u32(dst)), "l"(src), "r"(bytes), "r"(gemmdev::smem_u32(bar))
               : "memory");
}


template <typename T, int THREADS, int VPT>
__global__ void __launch_bounds__(THREADS) rmsnorm_fwd_kernel(T* __restrict__ y, float* __restrict__ rstd_out,
                                                              const T* __restrict__ x, const T* __restrict__ w,
                                                              const T* __restrict__ residual, T* __restrict__ res_out,
                                                              int64_t cols, float eps) {
  constexpr int V = Vec16<T>::N;
  __shared__ float sh[32];
  const int64_t row = blockIdx.x;
  const T* xr = x + row * cols;
  const T* rr = residual ? residual + row * cols : nullptr;
  T* yr = y + row * cols;
  const int nvec = (int)(cols / V);
  Vec16<T> buf[VPT];
  float ss = 0.f;
  int cnt;
  _Pragma("unroll") for (cnt = 0; cnt < VPT; ++cnt) { const int i = threadIdx.x + cnt * THREADS; if (i >= nvec) break;
    Vec16<T> v = ld16_stream(xr + (int64_t)i * V);
    if (rr) {
      Vec16<T> r = ld16_stream(rr + (int64_t)i * V);
#pragma unroll
      for (int k = 0; k < V; ++k) v.v[k] = ToF<T>::from(ToF<T>::to(v.v[k]) + ToF<T>::to(r.v[k]));
      st16(res_out + row * cols + (int64_t)i * V, v);
    }
#pragma unroll
    for (int k = 0; k < V; ++k) {
      float f = ToF<T>::to(v.v[k]);
      ss += f * f;
    }
    if (cnt < VPT) buf[cnt] = v;
  }
  ss = block_sum(ss, sh);
  const float rstd = rsqrtf(ss / (float)cols + eps);
  if (threadIdx.x == 0 && rstd_out) rstd_out[row] = rstd;
  _Pragma("unroll") for (cnt = 0; cnt < VPT; ++cnt) { const int i = threadIdx.x + cnt * THREADS; if (i >= nvec) break;
    Vec16<T> v;
    if (cnt < VPT) v = buf[cnt];
    else v = rr ? ld16(res_out + row * cols + (int64_t)i * V) : ld16(xr + (int64_t)i * V);
    Vec16<T> o;
    if (w) {
      Vec16<T> wv = ld16(w + (int64_t)i * V);
#pragma unroll
      for (int k = 0; k < V; ++k) o.v[k] = ToF<T>::from(ToF<T>::to(v.v[k]) * rstd * ToF<T>::to(wv.v[k]));
    } else {
#pragma unroll
      for (int k = 0; k < V; ++k) o.v[k] = ToF<T>::from(ToF<T>::to(v.v[k]) * rstd);
    }
    st16_stream(yr + (int64_t)i * V, o);
  }
}

// dx = rstd * (dy*w - xhat * mean(dy*w*xhat)) (+ dres), xhat = x*rstd. A CTA walks a strip of rows and keeps
// dw partial sums (dy * xhat) for its columns in registers.  dres is the gradient that reaches the row past the norm (a
// residual stream): adding it here saves a pass over three tensors.
//
// A row's dot product stands between its loads and its stores, so rows come through a ring of `stages` slots in shared
// memory (x, dy, dres of a row each), filled by bulk copies several rows ahead: bound by memory then, not by its latency.
// One barrier per row serves the reduction (its partial sums alternate between two buffers) and says that the slot
// has been read, so thread 0 refills it.  Waits are bounded; a block that gave up leaves as a whole and sets the status.
// 4096 x 4096 bf16 with dres: 60.5 us as two kernels before (44.6 + 15.9), 26.6 now (5.0 TB/s).
struct RmsBwdParams {
  int64_t rows, cols;
  int rows_per_cta, stages;
  int* status;
};

template <typename T, int THREADS, int VPT>
__global__ void __launch_bounds__(THREADS) rmsnorm_bwd_kernel(T* __restrict__ dx, float* __restrict__ dw_partial,
                                                              const T* __restrict__ dy, const T* __restrict__ x,
                                                              const T* __restrict__ w, const float* __restrict__ rstd,
                                                              const T* __restrict__ dres, const RmsBwdParams p) {
  using namespace gemmdev;
  constexpr int V = Vec16<T>::N;
  extern __shared__ __align__(16) uint8_t ring[];
  __shared__ float sh[2][32];
  __shared__ uint64_t full[kMaxRmsStages];
  __shared__ int abort_word;
  volatile int* abort_flag = &abort_word;
  const int64_t cols = p.cols;
  const int nvec = (int)(cols / V);
  const uint32_t row_bytes = (uint32_t)(cols * sizeof(T));
  const int tensors = dres ? 3 : 2;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t r0 = (int64_t)blockIdx.x * p.rows_per_cta;
  const int n = (int)(min(r0 + (int64_t)p.rows_per_cta, p.rows) - r0);
  auto refill = [&](int i) {        // thread 0: row r0 + i into its slot
    uint64_t* bar = &full[i % p.stages];
    uint8_t* slot = ring + (size_t)(i % p.stages) * tensors * row_bytes;
    const int64_t off = (r0 + i) * cols;
    mbar_expect_tx(bar, tensors * row_bytes);
    bulk_copy(slot, x + off, row_bytes, bar);
    bulk_copy(slot + row_bytes, dy + off, row_bytes, bar);
    if (dres) bulk_copy(slot + 2 * (size_t)row_bytes, dres + off, row_bytes, bar);
  };
  if (threadIdx.x == 0) {
    abort_word = 0;
    for (int i = 0; i < p.stages; ++i) mbar_init(&full[i], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    for (int i = 0; i < min(n, p.stages); ++i) refill(i);
  }
  // wide rows (VPT >= 4) are read from their slot a second time and w from the cache: held in registers, they would spill
  constexpr bool HOLD = VPT < 4;
  constexpr int NH = HOLD ? VPT : 1;
  float dwacc[VPT][V];
  Vec16<T> wreg[NH], xb[NH], gb[NH], rb[NH];
  auto load_w = [&](int c) {
    const int i = threadIdx.x + c * THREADS;
#pragma unroll
    for (int k = 0; k < V; ++k) wreg[HOLD ? c : 0].v[k] = ToF<T>::from(1.f);
    if (w && i < nvec) wreg[HOLD ? c : 0] = ld16(w + (int64_t)i * V);
  };
#pragma unroll
  for (int c = 0; c < VPT; ++c) {
#pragma unroll
    for (int k = 0; k < V; ++k) dwacc[c][k] = 0.f;
    if (HOLD) load_w(c);
  }
  __syncthreads();
  float rs_next = n > 0 ? rstd[r0] : 0.f;
  bool ok = true;
  for (int r = 0; r < n; ++r) {
    const float rs = rs_next;
    if (r + 1 < n) rs_next = rstd[r0 + r + 1];
    const uint8_t* slot = ring + (size_t)(r % p.stages) * tensors * row_bytes;
    const T* sx = reinterpret_cast<const T*>(slot);
    const T* sg = reinterpret_cast<const T*>(slot + row_bytes);
    const T* sr = reinterpret_cast<const T*>(slot + 2 * (size_t)row_bytes);
    const bool arrived = mbar_wait(&full[r % p.stages], (uint32_t)((r / p.stages) & 1), abort_flag);
    auto load_row = [&](int c) {
      const int i = threadIdx.x + c * THREADS, d = HOLD ? c : 0;
      xb[d] = ld16(sx + (int64_t)i * V);
      gb[d] = ld16(sg + (int64_t)i * V);
      if (dres) rb[d] = ld16(sr + (int64_t)i * V);
      if (!HOLD) load_w(c);
    };
    float dot = 0.f;
#pragma unroll
    for (int c = 0; c < VPT; ++c) {
      if (threadIdx.x + c * THREADS < nvec) {
        const int d = HOLD ? c : 0;
        load_row(c);
#pragma unroll
        for (int k = 0; k < V; ++k) {
          const float xh = ToF<T>::to(xb[d].v[k]) * rs;
          const float g = ToF<T>::to(gb[d].v[k]);
          dot += g * ToF<T>::to(wreg[d].v[k]) * xh;
          dwacc[c][k] += g * xh;
        }
      }
    }
    dot = warp_sum(dot);
    if (lane == 0) sh[r & 1][wid] = dot;
    ok = __syncthreads_and(arrived);
    if (!ok) break;
    if (HOLD && threadIdx.x == 0 && r + p.stages < n) refill(r + p.stages);
    dot = warp_sum(lane < THREADS / 32 ? sh[r & 1][lane] : 0.f);
    const float m = dot / (float)cols;
#pragma unroll
    for (int c = 0; c < VPT; ++c) {
      const int i = threadIdx.x + c * THREADS;
      if (i < nvec) {
        const int d = HOLD ? c : 0;
        if (!HOLD) load_row(c);
        Vec16<T> o;
#pragma unroll
        for (int k = 0; k < V; ++k) {
          const float xh = ToF<T>::to(xb[d].v[k]) * rs;
          const float g = ToF<T>::to(gb[d].v[k]) * ToF<T>::to(wreg[d].v[k]);
          float v = rs * (g - xh * m);
          if (dres) v += ToF<T>::to(rb[d].v[k]);
          o.v[k] = ToF<T>::from(v);
        }
        st16_stream(dx + (r0 + r) * cols + (int64_t)i * V, o);
      }
    }
    if (!HOLD) {
      __syncthreads();
      if (threadIdx.x == 0 && r + p.stages < n) refill(r + p.stages);
    }
  }
  if (!ok) {       // the copies in flight get a bounded moment to land before the shared memory is released
    if (threadIdx.x == 0) {
      for (int i = 0; i < 200; ++i) __nanosleep(1000);
      if (p.status) atomicExch(p.status, 1);
    }
    __syncthreads();
    return;
  }
  if (dw_partial) {
    float* out = dw_partial + (int64_t)blockIdx.x * cols;
#pragma unroll
    for (int c = 0; c < VPT; ++c) {
      const int i = threadIdx.x + c * THREADS;
      if (i < nvec) {
#pragma unroll
        for (int k = 0; k < V; k += 4)
          *reinterpret_cast<float4*>(out + (int64_t)i * V + k) =
              make_float4(dwacc[c][k], dwacc[c][k + 1], dwacc[c][k + 2], dwacc[c][k + 3]);
      }
    }
  }
}

template <typename T, int THREADS, int VPT>
__global__ void __launch_bounds__(THREADS) layernorm_fwd_kernel(T* __restrict__ y, float* __restrict__ mean_out,
                                                                float* __restrict__ rstd_out, const T* __restrict__ x,
                                                                const T* __restrict__ w, const T* __restrict__ b,
                                                                int64_t cols, float eps) {
  constexpr int V = Vec16<T>::N;
  __shared__ float sh[32];
  const int64_t row = blockIdx.x;
  const T* xr = x + row * cols;
  const int nvec = (int)(cols / V);
  Vec16<T> buf[VPT];
  float s = 0.f;
  int cnt;
  _Pragma("unroll") for (cnt = 0; cnt < VPT; ++cnt) { const int i = threadIdx.x + cnt * THREADS; if (i >= nvec) break;
    buf[cnt] = ld16_stream(xr + (int64_t)i * V);
#pragma unroll
    for (int k = 0; k < V; ++k) s += ToF<T>::to(buf[cnt].v[k]);
  }
  const float mean = block_sum(s, sh) / (float)cols;
  float vs = 0.f;
  _Pragma("unroll") for (cnt = 0; cnt < VPT; ++cnt) { const int i = threadIdx.x + cnt * THREADS; if (i >= nvec) break;
#pragma unroll
    for (int k = 0; k < V; ++k) {
      float d = ToF<T>::to(buf[cnt].v[k]) - mean;
      vs += d * d;
    }
  }
  const float rstd = rsqrtf(block_sum(vs, sh) / (float)cols + eps);
  if (threadIdx.x == 0) {
    if (mean_out) mean_out[row] = mean;
    if (rstd_out) rstd_out[row] = rstd;
  }
  _Pragma("unroll") for (cnt = 0; cnt < VPT; ++cnt) { const int i = threadIdx.x + cnt * THREADS; if (i >= nvec) break;
    Vec16<T> o;
#pragma unroll
    for (int k = 0; k < V; ++k) {
      float v = (ToF<T>::to(buf[cnt].v[k]) - mean) * rstd;
      if (w) v *= ToF<T>::to(w[(int64_t)i * V + k]);
      if (b) v += ToF<T>::to(b[(int64_t)i * V + k]);
      o.v[k] = ToF<T>::from(v);
    }
    st16_stream(y + row * cols + (int64_t)i * V, o);
  }
}

// dx = rstd * (g - mean(g) - xhat * mean(g*xhat)), g = dy*w
template <typename T, int THREADS, int VPT>
__global__ void __launch_bounds__(THREADS) layernorm_bwd_kernel(T* __restrict__ dx, float* __restrict__ dw_partial,
                                                                float* __restrict__ db_partial,
                                                                const T* __restrict__ dy, const T* __restrict__ x,
                                                                const T* __restrict__ w, const float* __restrict__ mean,
                                                                const float* __restrict__ rstd, int64_t rows,
                                                                int64_t cols, int rows_per_cta) {
  constexpr int V = Vec16<T>::N;
  __shared__ float sh[32];
  const int nvec = (int)(cols / V);
  float dwacc[VPT][V], dbacc[VPT][V];
#pragma unroll
  for (int c = 0; c < VPT; ++c)
#pragma unroll
    for (int k = 0; k < V; ++k) { dwacc[c][k] = 0.f; dbacc[c][k] = 0.f; }
  const int64_t r0 = (int64_t)blockIdx.x * rows_per_cta;
  const int64_t r1 = min(r0 + (int64_t)rows_per_cta, rows);
  for (int64_t row = r0; row < r1; ++row) {
    const float mu = mean[row], rs = rstd[row];
    Vec16<T> xb[VPT], gb[VPT];
    float s1 = 0.f, s2 = 0.f;
    int cnt;
    _Pragma("unroll") for (cnt = 0; cnt < VPT; ++cnt) { const int i = threadIdx.x + cnt * THREADS; if (i >= nvec) break;
      xb[cnt] = ld16_stream(x + row * cols + (int64_t)i * V);
      gb[cnt] = ld16_stream(dy + row * cols + (int64_t)i * V);
#pragma unroll
      for (int k = 0; k < V; ++k) {
        float xh = (ToF<T>::to(xb[cnt].v[k]) - mu) * rs;
        float g0 = ToF<T>::to(gb[cnt].v[k]);
        float g = w ? g0 * ToF<T>::to(w[(int64_t)i * V + k]) : g0;
        s1 += g;
        s2 += g * xh;
        dwacc[cnt][k] += g0 * xh;
        dbacc[cnt][k] += g0;
      }
    }
    s1 = block_sum(s1, sh) / (float)cols;
    s2 = block_sum(s2, sh) / (float)cols;
      _Pragma("unroll") for (cnt = 0; cnt < VPT; ++cnt) { const int i = threadIdx.x + cnt * THREADS; if (i >= nvec) break;
      Vec16<T> o;
#pragma unroll
      for (int k = 0; k < V; ++k) {
        float xh = (ToF<T>::to(xb[cnt].v[k]) - mu) * rs;
        float g0 = ToF<T>::to(gb[cnt].v[k]);
        float g = w ? g0 * ToF<T>::to(w[(int64_t)i * V + k]) : g0;
        o.v[k] = ToF<T>::from(rs * (g - s1 - xh * s2));
      }
      st16_stream(dx + row * cols + (int64_t)i * V, o);
    }
  }
  int cnt;
  _Pragma("unroll") for (cnt = 0; cnt < VPT; ++cnt) { const int i = threadIdx.x + cnt * THREADS; if (i >= nvec) break;
#pragma unroll
    for (int k = 0; k < V; ++k) {
      if (dw_partial) dw_partial[(int64_t)blockIdx.x * cols + (int64_t)i * V + k] = dwacc[cnt][k];
      if (db_partial) db_partial[(int64_t)blockIdx.x * cols + (int64_t)i * V + k] = dbacc[cnt][k];
    }
  }
}

// (threads, vectors per thread) for a row of `nvec` 16-byte vectors; rows beyond 512*8 vectors are not covered
#define B200K_ROW_LAUNCH(KERNEL, NVEC, GRID, STREAM, ...)                                        \
  do {                                                                                           \
    /* few threads with several independent 16-byte loads each: more bytes in flight per SM and    \
       more resident CTAs than one vector per thread */                                            \
    if ((NVEC) <= 128) KERNEL<T, 128, 1><<<(GRID), 128, 0, (STREAM)>>>(__VA_ARGS__);             \
    else if ((NVEC) <= 256) KERNEL<T, 128, 2><<<(GRID), 128, 0, (STREAM)>>>(__VA_ARGS__);        \
    else if ((NVEC) <= 512) KERNEL<T, 128, 4><<<(GRID), 128, 0, (STREAM)>>>(__VA_ARGS__);        \
    else if ((NVEC) <= 1024) KERNEL<T, 256, 4><<<(GRID), 256, 0, (STREAM)>>>(__VA_ARGS__);       \
    else if ((NVEC) <= 2048) KERNEL<T, 512, 4><<<(GRID), 512, 0, (STREAM)>>>(__VA_ARGS__);       \
    else KERNEL<T, 512, 8><<<(GRID), 512, 0, (STREAM)>>>(__VA_ARGS__);                           \
  } while (0)

constexpr int64_t kMaxRowVecs = 512 * 8;

// Two CTAs per SM walk strips of rows; each gets half of the shared memory for its ring, or, where a row is so wide that
// not even two slots fit into that half, all of it (one CTA per SM at a time then).  Four slots of 24 KB (4096 bf16 columns
// with dres) already keep 190 KB per SM in flight; more are not used.
template <typename T, int THREADS, int VPT>
int rmsnorm_bwd_go(int nb, cudaStream_t stream, T* dx, float* dwp, const T* dy, const T* x, const T* w, const float* rstd, const T* dres,
                   RmsBwdParams p) {
  constexpr int kHalf = 112 * 1024, kWhole = 224 * 1024;
  const int64_t slot = p.cols * (int64_t)sizeof(T) * (dres ? 3 : 2);
  const int64_t room = slot * 2 <= kHalf ? kHalf : kWhole;
  p.stages = (int)std::min<int64_t>(room / slot, kMaxRmsStages);
  if (p.stages < 1) return (int)cudaErrorNotSupported;
  static OncePerDevice once;
  if (int e = once([&] { return opt_in_smem(rmsnorm_bwd_kernel<T, THREADS, VPT>, kWhole); })) return e;
  rmsnorm_bwd_kernel<T, THREADS, VPT><<<nb, THREADS, p.stages * slot, stream>>>(dx, dwp, dy, x, w, rstd, dres, p);
  B200K_LAUNCH_RET();
}
template <typename T, typename... A>
int rmsnorm_bwd_launch(int64_t nvec, A... args) {
  if (nvec <= 128) return rmsnorm_bwd_go<T, 128, 1>(args...);
  if (nvec <= 256) return rmsnorm_bwd_go<T, 256, 1>(args...);
  if (nvec <= 512) return rmsnorm_bwd_go<T, 256, 2>(args...);
  if (nvec <= 1024) return rmsnorm_bwd_go<T, 512, 2>(args...);
  if (nvec <= 2048) return rmsnorm_bwd_go<T, 512, 4>(args...);
  return rmsnorm_bwd_go<T, 512, 8>(args...);
}

}  // namespace
}  // namespace b200k

using namespace b200k;

extern "C" {

int b200_rmsnorm_bwd_partial_rows(int64_t rows, int64_t cols) {
  (void)cols;
  // ~2 CTAs per SM, each walking a strip of rows
  int64_t ctas = std::min<int64_t>(rows, (int64_t)kSMs * 2);
  if (ctas < 1) ctas = 1;
  int64_t rpc = cdiv(rows, ctas);
  return (int)cdiv(rows, rpc);
}

int b200_rmsnorm_fwd(int dtype, void* y, float* rstd, const void* x, const void* w, const void* residual,
                     void* res_out, int64_t rows, int64_t cols, float eps, cudaStream_t stream) {
  if (rows == 0) return 0;
  B200K_DISPATCH_FLOAT(dtype, T, {
    constexpr int V = Vec16<T>::N;
    int64_t nvec = cols / V;
    if (cols % V != 0 || nvec > kMaxRowVecs || !aligned16((const T*)x) || !aligned16((T*)y) ||
        (w && !aligned16((const T*)w)) || (residual && (!aligned16((const T*)residual) || !aligned16((T*)res_out))))
      return (int)cudaErrorNotSupported;
    B200K_ROW_LAUNCH(rmsnorm_fwd_kernel, nvec, (unsigned)rows, stream, (T*)y, rstd, (const T*)x, (const T*)w,
                     (const T*)residual, (T*)res_out, cols, eps);
    B200K_LAUNCH_RET();
  })
  return (int)cudaErrorNotSupported;
}

int b200_rmsnorm_bwd(int dtype, void* dx, float* dw_partial, int* nblocks_out_host, const void* dy, const void* x,
                     const void* w, const float* rstd, int64_t rows, int64_t cols, cudaStream_t stream) {
  return b200_rmsnorm_residual_bwd(dtype, dx, dw_partial, nblocks_out_host, dy, x, w, rstd, nullptr, rows, cols, stream);
}

int b200_rmsnorm_residual_bwd(int dtype, void* dx, float* dw_partial, int* nblocks_out_host, const void* dy, const void* x,
                              const void* w, const float* rstd, const void* dres, int64_t rows, int64_t cols,
                              cudaStream_t stream) {
  if (rows == 0) return 0;
  int nb = b200_rmsnorm_bwd_partial_rows(rows, cols);
  int rpc = (int)cdiv(rows, nb);
  if (nblocks_out_host) *nblocks_out_host = nb;
  B200K_DISPATCH_FLOAT(dtype, T, {
    constexpr int V = Vec16<T>::N;
    int64_t nvec = cols / V;
    if (cols % V != 0 || nvec > kMaxRowVecs || !aligned16((const T*)x) || !aligned16((const T*)dy) ||
        !aligned16((T*)dx) || (w && !aligned16((const T*)w)) || (dres && !aligned16((const T*)dres)))
      return (int)cudaErrorNotSupported;
    RmsBwdParams p{rows, cols, rpc, 0, gemm_status_word_device()};
    return rmsnorm_bwd_launch<T>(nvec, nb, stream, (T*)dx, dw_partial, (const T*)dy, (const T*)x, (const T*)w, rstd, (const T*)dres, p);
  })
  return (int)cudaErrorNotSupported;
}

int b200_layernorm_fwd(int dtype, void* y, float* mean, float* rstd, const void* x, const void* w, const void* b,
                       int64_t rows, int64_t cols, float eps, cudaStream_t stream) {
  if (rows == 0) return 0;
  B200K_DISPATCH_FLOAT(dtype, T, {
    constexpr int V = Vec16<T>::N;
    int64_t nvec = cols / V;
    if (cols % V != 0 || nvec > kMaxRowVecs || !aligned16((const T*)x) || !aligned16((T*)y))
      return (int)cudaErrorNotSupported;
    B200K_ROW_LAUNCH(layernorm_fwd_kernel, nvec, (unsigned)rows, stream, (T*)y, mean, rstd, (const T*)x, (const T*)w,
                     (const T*)b, cols, eps);
    B200K_LAUNCH_RET();
  })
  return (int)cudaErrorNotSupported;
}

int b200_layernorm_bwd(int dtype, void* dx, float* dw_partial, float* db_partial, const void* dy, const void* x,
                       const void* w, const float* mean, const float* rstd, int64_t rows, int64_t cols,
                       cudaStream_t stream) {
  if (rows == 0) return 0;
  int nb = b200_rmsnorm_bwd_partial_rows(rows, cols);
  int rpc = (int)cdiv(rows, nb);
  B200K_DISPATCH_FLOAT(dtype, T, {
    constexpr int V = Vec16<T>::N;
    int64_t nvec = cols / V;
    if (cols % V != 0 || nvec > kMaxRowVecs || !aligned16((const T*)x) || !aligned16((const T*)dy) ||
        !aligned16((T*)dx))
      return (int)cudaErrorNotSupported;
    B200K_ROW_LAUNCH(layernorm_bwd_kernel, nvec, nb, stream, (T*)dx, dw_partial, db_partial, (const T*)dy, (const T*)x,
                     (const T*)w, mean, rstd, rows, cols, rpc);
    B200K_LAUNCH_RET();
  })
  return (int)cudaErrorNotSupported;
}

}  // extern "C"
