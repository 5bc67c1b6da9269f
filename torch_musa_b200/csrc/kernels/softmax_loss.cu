// Softmax / log-softmax (last dim) and fused cross-entropy, one CTA per row with a
// single-pass online (max, sum-exp) reduction: logits are read once for the
// statistics and once more (L2-resident: a 32000-wide bf16 row is 64 KB) to
// produce the output.  The fused cross-entropy never materialises the
// probabilities: forward keeps (loss, lse) per row, backward regenerates
// softmax from lse and may overwrite the logits in place.
// Parity: reference torch_musa/csrc/aten/ops/SoftMax.cpp:28-36,202-285 (vendor
// softmax), Loss.cpp:547-660 (fused 2-D CE) and
// csrc/extension/FusedCrossEntropyLoss.mu:55,160,293 (vocab-parallel pieces).
#include "common.cuh"

#include <algorithm>

namespace b200k {
namespace {

constexpr int kThreads = 512;

struct MaxSum {
  float m, s;
};
__device__ __forceinline__ MaxSum ms_combine(MaxSum a, MaxSum b) {
  float m = fmaxf(a.m, b.m);
  if (m == -INFINITY) return MaxSum{m, 0.f};
  return MaxSum{m, a.s * __expf(a.m - m) + b.s * __expf(b.m - m)};
}
__device__ __forceinline__ void ms_push(MaxSum& a, float x) {
  if (x > a.m) {
    a.s = a.s * __expf(a.m - x) + 1.f;
    a.m = x;
  } else if (x != -INFINITY) {
    a.s += __expf(x - a.m);
  }
}
__device__ __forceinline__ MaxSum block_ms(MaxSum v, float* shm, float* shs) {
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    MaxSum other{__shfl_xor_sync(0xffffffffu, v.m, o), __shfl_xor_sync(0xffffffffu, v.s, o)};
    v = ms_combine(v, other);
  }
  __syncthreads();
  if (lane == 0) { shm[w] = v.m; shs[w] = v.s; }
  __syncthreads();
  MaxSum r = (lane < nw) ? MaxSum{shm[lane], shs[lane]} : MaxSum{-INFINITY, 0.f};
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    MaxSum other{__shfl_xor_sync(0xffffffffu, r.m, o), __shfl_xor_sync(0xffffffffu, r.s, o)};
    r = ms_combine(r, other);
  }
  return r;
}

__device__ __forceinline__ float exp2f_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// ((x0, x1) - m) * log2(e), two fp32 operations per instruction
__device__ __forceinline__ void log2_ratio(float& d0, float& d1, float x0, float x1, float m) {
  asm("{\n\t.reg .b64 rx, rm, rs, rd;\n\t"
      "mov.b64 rx, {%2, %3};\n\tmov.b64 rm, {%4, %4};\n\tmov.b64 rs, {%5, %5};\n\t"
      "add.rn.f32x2 rd, rx, rm;\n\tmul.rn.f32x2 rd, rd, rs;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(d0), "=f"(d1)
      : "f"(x0), "f"(x1), "f"(-m), "f"(1.4426950408889634f));
}

// N vectors of a row into the running (maximum, sum): the maximum in four chains, one correction of the sum, then the
// exponentials in four chains of additions.  The maximum is subtracted before the scaling by log2(e): rounded on its own,
// the product m * log2(e) would put its error, or for masks near the type's lowest value its overflow, into every term.
template <int N, typename T>
__device__ __forceinline__ void ms_push_vecs(MaxSum& acc, const Vec16<T>* v) {
  constexpr int V = Vec16<T>::N;
  float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
  for (int u = 0; u < N; ++u)
#pragma unroll
    for (int k = 0; k < V; ++k) mx[k & 3] = fmaxf(mx[k & 3], ToF<T>::to(v[u].v[k]));
  const float lm = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
  if (lm > acc.m) { acc.s *= __expf(acc.m - lm); acc.m = lm; }
  if (acc.m == -INFINITY) return;
  float sm[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int u = 0; u < N; ++u)
#pragma unroll
    for (int k = 0; k < V; k += 2) {
      float d0, d1;
      log2_ratio(d0, d1, ToF<T>::to(v[u].v[k]), ToF<T>::to(v[u].v[k + 1]), acc.m);
      sm[k & 3] += exp2f_approx(d0);
      sm[(k & 3) + 1] += exp2f_approx(d1);
    }
  acc.s += (sm[0] + sm[1]) + (sm[2] + sm[3]);
}

// Row statistics with optional 16-byte vector loads (VEC requires cols % V == 0 and an aligned base).
template <typename T, bool VEC>
__device__ __forceinline__ MaxSum row_stats(const T* __restrict__ xr, int64_t cols, float* shm, float* shs) {
  constexpr int V = Vec16<T>::N;
  MaxSum acc{-INFINITY, 0.f};
  if constexpr (VEC) {
    // A group of 16 elements per thread is on its way while the one before it is worked on.  (Groups of 32 16-bit elements took
    // 96 registers, which leaves room for 640 threads on an SM.)
    constexpr int U = 16 / V;
    const int nvec = (int)(cols / V), step = blockDim.x * U;
    Vec16<T> cur[U], nxt[U];
    auto load = [&](Vec16<T>(&v)[U], int i0) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = i0 + u * (int)blockDim.x;
        if (i < nvec) v[u] = ld16(xr + (int64_t)i * V);
      }
    };
    int i0 = threadIdx.x;
    load(cur, i0);
    for (; i0 - (int)threadIdx.x + step <= nvec; i0 += step) {     // whole groups: every thread has U vectors
      load(nxt, i0 + step);
      ms_push_vecs<U>(acc, cur);
#pragma unroll
      for (int u = 0; u < U; ++u) cur[u] = nxt[u];
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i0 + u * (int)blockDim.x < nvec) ms_push_vecs<1>(acc, cur + u);
  } else {
    for (int64_t i = threadIdx.x; i < cols; i += blockDim.x) ms_push(acc, ToF<T>::to(xr[i]));
  }
  return block_ms(acc, shm, shs);
}

template <typename T, bool VEC, bool LOG>
__global__ void __launch_bounds__(kThreads, 2) softmax_fwd_kernel(T* __restrict__ y, const T* __restrict__ x, int64_t cols) {
  constexpr int V = Vec16<T>::N;
  __shared__ float shm[32], shs[32];
  const int64_t row = blockIdx.x;
  const T* xr = x + row * cols;
  T* yr = y + row * cols;
  MaxSum st = row_stats<T, VEC>(xr, cols, shm, shs);
  const float lse = st.m + __logf(st.s);
  const float inv = 1.f / st.s;
  if constexpr (VEC) {
    int64_t nvec = cols / V;
    for (int64_t i = threadIdx.x; i < nvec; i += blockDim.x) {
      Vec16<T> v = ld16(xr + i * V), o;
#pragma unroll
      for (int k = 0; k < V; ++k) {
        float f = ToF<T>::to(v.v[k]);
        o.v[k] = ToF<T>::from(LOG ? f - lse : __expf(f - st.m) * inv);
      }
      st16_stream(yr + i * V, o);
    }
  } else {
    for (int64_t i = threadIdx.x; i < cols; i += blockDim.x) {
      float f = ToF<T>::to(xr[i]);
      yr[i] = ToF<T>::from(LOG ? f - lse : __expf(f - st.m) * inv);
    }
  }
}

// softmax: dx = y * (dy - sum(dy*y)); log-softmax: dx = dy - exp(y) * sum(dy)
template <typename T, bool LOG>
__global__ void __launch_bounds__(kThreads) softmax_bwd_kernel(T* __restrict__ dx, const T* __restrict__ dy,
                                                               const T* __restrict__ y, int64_t cols) {
  __shared__ float sh[32];
  const int64_t row = blockIdx.x;
  const T* gr = dy + row * cols;
  const T* yr = y + row * cols;
  float s = 0.f;
  for (int64_t i = threadIdx.x; i < cols; i += blockDim.x) {
    float g = ToF<T>::to(gr[i]);
    s += LOG ? g : g * ToF<T>::to(yr[i]);
  }
  s = block_sum(s, sh);
  for (int64_t i = threadIdx.x; i < cols; i += blockDim.x) {
    float g = ToF<T>::to(gr[i]), yy = ToF<T>::to(yr[i]);
    dx[row * cols + i] = ToF<T>::from(LOG ? g - __expf(yy) * s : yy * (g - s));
  }
}

template <typename T, bool VEC>
__global__ void __launch_bounds__(kThreads, 2) ce_fwd_kernel(float* __restrict__ loss, float* __restrict__ lse_out,
                                                          const T* __restrict__ logits,
                                                          const int64_t* __restrict__ target, int64_t cols,
                                                          int64_t ignore_index, float smoothing) {
  __shared__ float shm[32], shs[32], sh[32];
  const int64_t row = blockIdx.x;
  const T* xr = logits + row * cols;
  // the target's logit is on its way while the row is read
  int64_t t = 0;
  float xt = 0.f;
  if (threadIdx.x == 0) {
    t = target[row];
    if (t >= 0 && t < cols) xt = ToF<T>::to(xr[t]);
  }
  MaxSum st = row_stats<T, VEC>(xr, cols, shm, shs);
  const float lse = st.m + __logf(st.s);
  float sum_logits = 0.f;
  if (smoothing > 0.f) {
    for (int64_t i = threadIdx.x; i < cols; i += blockDim.x) sum_logits += ToF<T>::to(xr[i]);
    sum_logits = block_sum(sum_logits, sh);
  }
  if (threadIdx.x == 0) {
    lse_out[row] = lse;
    if (t == ignore_index || t < 0 || t >= cols) {
      loss[row] = 0.f;
    } else {
      float nll = lse - xt;
      if (smoothing > 0.f) {
        float smooth = lse - sum_logits / (float)cols;  // mean over classes of -log p
        loss[row] = (1.f - smoothing) * nll + smoothing * smooth;
      } else {
        loss[row] = nll;
      }
    }
  }
}

template <typename T, bool VEC>
__global__ void __launch_bounds__(kThreads) ce_bwd_kernel(T* __restrict__ dlogits, const T* __restrict__ logits,
                                                          const float* __restrict__ lse,
                                                          const int64_t* __restrict__ target,
                                                          const float* __restrict__ grad_loss, int grad_is_scalar,
                                                          float scale, int64_t cols, int64_t ignore_index,
                                                          float smoothing) {
  constexpr int V = Vec16<T>::N;
  const int64_t row = blockIdx.x;
  const int64_t t = target[row];
  const bool ignored = (t == ignore_index || t < 0 || t >= cols);
  const float g = ignored ? 0.f : scale * (grad_loss ? (grad_is_scalar ? grad_loss[0] : grad_loss[row]) : 1.f);
  const float l = lse[row];
  const T* xr = logits + row * cols;
  T* dr = dlogits + row * cols;
  const float on = 1.f - smoothing, off = smoothing / (float)cols;
  if constexpr (VEC) {
    const int64_t nvec = cols / V;
    constexpr int U = 4;   // independent 16-byte loads in flight per thread
    for (int64_t i0 = threadIdx.x; i0 < nvec; i0 += (int64_t)blockDim.x * U) {
      Vec16<T> v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t i = i0 + (int64_t)u * blockDim.x;
        if (i < nvec) v[u] = ld16(xr + i * V);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t i = i0 + (int64_t)u * blockDim.x;
        if (i < nvec) {
          Vec16<T> o;
#pragma unroll
          for (int k = 0; k < V; ++k) {
            const float p = __expf(ToF<T>::to(v[u].v[k]) - l);
            const float y = ((i * V + k) == t ? on : 0.f) + off;
            o.v[k] = ToF<T>::from(g * (p - y));
          }
          st16(dr + i * V, o);
        }
      }
    }
  } else {
    for (int64_t i = threadIdx.x; i < cols; i += blockDim.x) {
      float p = __expf(ToF<T>::to(xr[i]) - l);
      float y = (i == t ? on : 0.f) + off;
      dr[i] = ToF<T>::from(g * (p - y));
    }
  }
}

// One block: the sum of the row losses and the number of targets that count (see b200_cross_entropy_mean).  Launches and the
// gaps between them are what this costs: it stands for seven launches (compare, count, clamp, convert, sum, divide).
__global__ void __launch_bounds__(1024) ce_mean_kernel(float* __restrict__ mean, float* __restrict__ count,
                                                       const float* __restrict__ loss, const int64_t* __restrict__ target,
                                                       int rows, int64_t ignore_index) {
  __shared__ float sh[32];
  float s = 0.f, n = 0.f;      // a block sees at most 65536 rows: the count is exact in fp32
  for (int i = threadIdx.x; i < rows; i += 1024) {
    s += loss[i];
    n += target[i] != ignore_index ? 1.f : 0.f;
  }
  s = block_sum(s, sh);
  n = fmaxf(block_sum(n, sh), 1.f);
  if (threadIdx.x == 0) {
    *mean = s / n;
    *count = n;
  }
}

template <typename T, bool VEC>
__global__ void __launch_bounds__(kThreads, 2) online_stats_kernel(float* __restrict__ stats3,
                                                                const T* __restrict__ logits,
                                                                const int64_t* __restrict__ target, int64_t cols,
                                                                int64_t vocab_start) {
  __shared__ float shm[32], shs[32];
  const int64_t row = blockIdx.x;
  const T* xr = logits + row * cols;
  MaxSum st = row_stats<T, VEC>(xr, cols, shm, shs);
  if (threadIdx.x == 0) {
    int64_t t = target[row] - vocab_start;
    stats3[row * 3 + 0] = st.m;
    stats3[row * 3 + 1] = st.s;
    stats3[row * 3 + 2] = (t >= 0 && t < cols) ? ToF<T>::to(xr[t]) : 0.f;  // summed across shards
  }
}

template <typename T>
__global__ void __launch_bounds__(kThreads) vp_ce_finish_kernel(float* __restrict__ loss, T* __restrict__ logits,
                                                                const float* __restrict__ all_stats, int world,
                                                                const int64_t* __restrict__ target, int64_t rows,
                                                                int64_t cols, int64_t vocab_start,
                                                                int64_t ignore_index) {
  const int64_t row = blockIdx.x;
  // all_stats layout: [world, rows, 3]
  MaxSum g{-INFINITY, 0.f};
  float tl = 0.f;
  for (int r = 0; r < world; ++r) {
    const float* s = all_stats + ((int64_t)r * rows + row) * 3;
    g = ms_combine(g, MaxSum{s[0], s[1]});
    tl += s[2];
  }
  const float lse = g.m + __logf(g.s);
  const int64_t tg = target[row];
  const bool ignored = (tg == ignore_index);
  if (threadIdx.x == 0 && loss) loss[row] = ignored ? 0.f : lse - tl;
  const int64_t t = tg - vocab_start;
  T* xr = logits + row * cols;
  for (int64_t i = threadIdx.x; i < cols; i += blockDim.x) {
    float p = __expf(ToF<T>::to(xr[i]) - lse);
    xr[i] = ToF<T>::from(ignored ? 0.f : (p - (i == t ? 1.f : 0.f)));
  }
}

// ---- threads per row
// Vector loads.  A row's block ends in a reduction and a few dependent scalar operations during which it loads nothing, so many
// small blocks per SM at different points of their rows keep memory busy; with few rows a row has to be spread over more threads
// instead.  From 16 rows per SM on 64 threads are enough for short rows, and for fp32, where a thread's group is twice the bytes.
// Row statistics, 64 / 128 / 256 / 512 threads: 4096 x 32000 bf16 58 / 55 / 62 / 75 us, fp32 85 / 86 / 84 / 94, x 50304 fp32 124 /
// 129 / 125 / 134, x 8192 bf16 18 / 20 / 27 / 42; 1184 x 32000 bf16 24 / 19 / 21 / 24; 600 x 32000 22 / 14.3 / 15.4 / 15.5; 32 x
// 32000 12 / 7.4 / 5.2 / 4.6.  (4096 x 32000 bf16 took 89 us with 512 threads and one chain of maxima and sums.)
inline int vec_threads(int64_t rows, int64_t cols, int elem) {
  const bool small = elem == 4 || cols * elem < 24 * 1024;
  int t = rows >= kSMs * 16 && small ? 64 : rows >= kSMs * 4 ? 128 : rows >= kSMs * 2 ? 256 : kThreads;
  while (t > 32 && (int64_t)t * 4 >= cols) t /= 2;
  return t;
}
// Element by element (ragged or misaligned rows) a thread is a chain of dependent exponentials: the time is the number of waves
// of blocks times what one block takes, a fixed part worth about six elements and its share of the row.  1184 x 50257 at 128 /
// 256 / 512 threads: 209 / 110 / 115 us; 4096 x 50257: 413 / 417 / 388; 4096 x 4001: 43 / 46 / 52.
inline int scalar_threads(int64_t rows, int64_t cols) {
  int best = kThreads;
  double best_cost = 1e300;
  for (int t = kThreads; t >= 64; t /= 2) {
    const double cost = (double)cdiv(rows * t, (int64_t)kSMs * 2048) * (6.0 + (double)cols / t);
    if (cost <= best_cost) { best = t; best_cost = cost; }
  }
  return best;
}
inline int stats_threads(bool vec, int64_t rows, int64_t cols, int elem) {
  return vec ? vec_threads(rows, cols, elem) : scalar_threads(rows, cols);
}
// The second pass of a softmax reads its row again: with a thread per 256 bytes the rows in flight (1024 threads per SM) are 38 MB
// and come from L2.  4096 x 32000 at 128 / 256 / 512 threads: bf16 135 / 115 / 131 us, fp32 248 / 220 / 178.
inline int softmax_threads(bool vec, int64_t rows, int64_t cols, int elem) {
  int t = stats_threads(vec, rows, cols, elem);
  if (!vec || rows >= kSMs * 4)
    while (t < kThreads && (int64_t)t * 256 < cols * elem) t *= 2;
  return t;
}
// The loss's gradient streams in and out; rows of 112 KB and more keep whole blocks.  4096 x 32000 at 128 / 256 / 512 threads:
// bf16 91 / 93 / 104 us, fp32 172 / 164 / 162; 1184 x 50257 fp32 110 / 97 / 94.
inline int ce_bwd_threads(bool vec, int64_t rows, int64_t cols, int elem) {
  if (cols * elem >= 112 * 1024) return kThreads;
  if (!vec) return std::max(128, scalar_threads(rows, cols));
  return rows >= kSMs * 8 ? 128 : rows >= kSMs * 4 ? 256 : kThreads;
}

}  // namespace
}  // namespace b200k

using namespace b200k;

extern "C" {

int b200_softmax_fwd(int dtype, void* y, const void* x, int64_t rows, int64_t cols, int log_softmax,
                     cudaStream_t stream) {
  if (rows == 0 || cols == 0) return 0;
  B200K_DISPATCH_FLOAT(dtype, T, {
    bool vec = cols % Vec16<T>::N == 0 && aligned16((const T*)x) && aligned16((T*)y);
    dim3 grid((unsigned)rows);
    const int threads = softmax_threads(vec, rows, cols, (int)sizeof(T));
    if (vec) {
      if (log_softmax) softmax_fwd_kernel<T, true, true><<<grid, threads, 0, stream>>>((T*)y, (const T*)x, cols);
      else softmax_fwd_kernel<T, true, false><<<grid, threads, 0, stream>>>((T*)y, (const T*)x, cols);
    } else {
      if (log_softmax) softmax_fwd_kernel<T, false, true><<<grid, threads, 0, stream>>>((T*)y, (const T*)x, cols);
      else softmax_fwd_kernel<T, false, false><<<grid, threads, 0, stream>>>((T*)y, (const T*)x, cols);
    }
    B200K_LAUNCH_RET();
  })
  return (int)cudaErrorNotSupported;
}

int b200_softmax_bwd(int dtype, void* dx, const void* dy, const void* y, int64_t rows, int64_t cols, int log_softmax,
                     cudaStream_t stream) {
  if (rows == 0 || cols == 0) return 0;
  B200K_DISPATCH_FLOAT(dtype, T, {
    dim3 grid((unsigned)rows);
    if (log_softmax) softmax_bwd_kernel<T, true><<<grid, kThreads, 0, stream>>>((T*)dx, (const T*)dy, (const T*)y, cols);
    else softmax_bwd_kernel<T, false><<<grid, kThreads, 0, stream>>>((T*)dx, (const T*)dy, (const T*)y, cols);
    B200K_LAUNCH_RET();
  })
  return (int)cudaErrorNotSupported;
}

int b200_cross_entropy_fwd(int dtype, float* loss, float* lse, const void* logits, const int64_t* target, int64_t rows,
                           int64_t cols, int64_t ignore_index, float label_smoothing, cudaStream_t stream) {
  if (rows == 0) return 0;
  B200K_DISPATCH_FLOAT(dtype, T, {
    bool vec = cols % Vec16<T>::N == 0 && aligned16((const T*)logits);
    dim3 grid((unsigned)rows);
    const int threads = stats_threads(vec, rows, cols, (int)sizeof(T));
    if (vec) ce_fwd_kernel<T, true><<<grid, threads, 0, stream>>>(loss, lse, (const T*)logits, target, cols, ignore_index, label_smoothing);
    else ce_fwd_kernel<T, false><<<grid, threads, 0, stream>>>(loss, lse, (const T*)logits, target, cols, ignore_index, label_smoothing);
    B200K_LAUNCH_RET();
  })
  return (int)cudaErrorNotSupported;
}

int b200_cross_entropy_mean(float* mean, float* count, const float* loss, const int64_t* target, int64_t rows,
                            int64_t ignore_index, cudaStream_t stream) {
  if (rows <= 0 || rows > 65536) return (int)cudaErrorNotSupported;
  ce_mean_kernel<<<1, 1024, 0, stream>>>(mean, count, loss, target, (int)rows, ignore_index);
  B200K_LAUNCH_RET();
}

int b200_cross_entropy_bwd(int dtype, void* dlogits, const void* logits, const float* lse, const int64_t* target,
                           const float* grad_loss, int grad_is_scalar, float scale, int64_t rows, int64_t cols,
                           int64_t ignore_index, float label_smoothing, cudaStream_t stream) {
  if (rows == 0) return 0;
  B200K_DISPATCH_FLOAT(dtype, T, {
    bool vec = cols % Vec16<T>::N == 0 && aligned16((const T*)logits) && aligned16((T*)dlogits);
    dim3 grid((unsigned)rows);
    const int threads = ce_bwd_threads(vec, rows, cols, (int)sizeof(T));
    if (vec) ce_bwd_kernel<T, true><<<grid, threads, 0, stream>>>((T*)dlogits, (const T*)logits, lse, target, grad_loss, grad_is_scalar, scale, cols, ignore_index, label_smoothing);
    else ce_bwd_kernel<T, false><<<grid, threads, 0, stream>>>((T*)dlogits, (const T*)logits, lse, target, grad_loss, grad_is_scalar, scale, cols, ignore_index, label_smoothing);
    B200K_LAUNCH_RET();
  })
  return (int)cudaErrorNotSupported;
}

int b200_online_softmax_stats(int dtype, float* stats3, const void* logits, const int64_t* target, int64_t rows,
                              int64_t cols, int64_t vocab_start, cudaStream_t stream) {
  if (rows == 0) return 0;
  B200K_DISPATCH_FLOAT(dtype, T, {
    bool vec = cols % Vec16<T>::N == 0 && aligned16((const T*)logits);
    dim3 grid((unsigned)rows);
    const int threads = stats_threads(vec, rows, cols, (int)sizeof(T));
    if (vec) online_stats_kernel<T, true><<<grid, threads, 0, stream>>>(stats3, (const T*)logits, target, cols, vocab_start);
    else online_stats_kernel<T, false><<<grid, threads, 0, stream>>>(stats3, (const T*)logits, target, cols, vocab_start);
    B200K_LAUNCH_RET();
  })
  return (int)cudaErrorNotSupported;
}

int b200_vocab_parallel_ce_finish(int dtype, float* loss, void* logits_inout, const float* all_stats, int world,
                                  const int64_t* target, int64_t rows, int64_t cols, int64_t vocab_start,
                                  int64_t ignore_index, cudaStream_t stream) {
  if (rows == 0) return 0;
  B200K_DISPATCH_FLOAT(dtype, T, {
    vp_ce_finish_kernel<T><<<(unsigned)rows, kThreads, 0, stream>>>(loss, (T*)logits_inout, all_stats, world, target, rows, cols, vocab_start, ignore_index);
    B200K_LAUNCH_RET();
  })
  return (int)cudaErrorNotSupported;
}

}  // extern "C"
