// bf16 / fp16 GEMM for few rows (decode steps, small batches) on tcgen05:
//
//   D[M,N] (+)= alpha * A[M,K] * B[N,K]^T (+ bias) (act),   M <= 64, both operands K-major
//
// Such a product is the streaming of B: 2 N K bytes for 2 M N K operations.  The general kernel makes M its 128-row
// operand (padding for the most part) and B a 256-wide one, which leaves 16 to 144 CTAs on 148 SMs and sends split-K
// partial products through global memory and a second kernel.  Here the operands change places: 128 rows of B are the M128
// operand and the rows of A, padded to 16 / 32 / 64, the N operand, so a stage of the ring is 16 KB of B and 2 to 8 KB of A.
// K is cut over the CTAs of a cluster until about two CTAs per SM stream B together (each has half of an SM's shared memory
// as its ring, 190 KB per SM in flight): while the CTAs are no more than two per SM they all are resident, share the memory's
// bandwidth and end together, so an uneven number per SM does not matter.  From 130 tiles of B on K stays whole, with 130 to 148
// tiles there is less than one CTA per SM (n = 16512 27.1 us, 16640 28.9, still ahead of the general kernel's 34), and past 296
// tiles a second wave begins (n = 37888 53.0 us, 38016 64.0 against 74.0).  The cluster adds its partial sums over distributed
// shared memory in rank order (the result does not depend on timing), each CTA a share of the rows of A.
// What bounds it: memory, and for small products the launch, the ring's first fill and the epilogue (about 5 us).  Streams of
// products with weights out of L2, K = 4096, M = 32, general kernel with split-K -> this one: n = 12288 27.8 -> 22.2 us (4.5
// TB/s), 22016 37.7 -> 34.8 (5.2), 32000 47.7 -> 45.5 (5.8), 6144 18.5 -> 14.4, 512 9.9 -> 7.0.
// Waits are bounded as in the dense kernel; every thread takes part in both cluster barriers whatever happened before.
//
// Parity: the reference sends mm/addmm to a closed vendor library (reference torch_musa/csrc/aten/ops/Matmul.cpp:293-335).
#include "gemm_common.cuh"

#include <algorithm>

namespace b200k {
namespace {
using namespace gemmdev;

constexpr int BN = 128;               // rows of B per tile: the M extent of the instruction
constexpr int BK = 64;
constexpr int kThreads = 192;         // TMA, MMA, 4 epilogue warps
constexpr int kMaxSplit = 8;          // portable cluster size

template <int MP>
struct Cfg {
  static constexpr int kBTile = BN * BK * 2;          // 16 KB
  static constexpr int kATile = MP * BK * 2;          // 2 / 4 / 8 KB
  static constexpr int kStage = kBTile + kATile;
  static constexpr int kStages = 104 * 1024 / kStage;  // 5 / 5 / 4: two CTAs per SM
  static constexpr uint32_t kTmemCols = MP < 32 ? 32 : MP;
  static constexpr int kSmem = kStages * kStage + 1024 /*alignment*/ + 256 /*barriers*/;
  static_assert(MP * BN * 4 <= kStages * kStage, "the partial sums reuse the ring");
};

struct SkinnyParams {
  int m, n, k;
  int64_t ldd;
  const void* bias;
  int bias_f32, act, accumulate;
  float alpha;
  uint32_t idesc;
  int* status;
  int splits;
};

__device__ __forceinline__ float4 ld_cluster_f32x4(uint32_t addr, uint32_t rank) {
  uint32_t remote;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(remote)
               : "memory");
  return v;
}

template <typename OutT, int MP>
__global__ void __launch_bounds__(kThreads, 2)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, OutT* __restrict__ d,
                   const SkinnyParams p) {
  using C = Cfg<MP>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kStages * C::kStage);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + C::kStages;
  uint64_t* tfull_bar = bars + 2 * C::kStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tfull_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* part = reinterpret_cast<float*>(smem);       // [MP][BN], after the last product has read the ring

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)(blockIdx.x % p.splits), n0 = (int)(blockIdx.x / p.splits) * BN;
  const int k_blocks = (p.k + BK - 1) / BK;
  const int kb0 = (int)((long long)k_blocks * rank / p.splits), kb1 = (int)((long long)k_blocks * (rank + 1) / p.splits);

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < C::kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(tfull_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    prefetch_tmap(&tmap_a);
    prefetch_tmap(&tmap_b);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, C::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag)) break;
        mbar_expect_tx(&full_bar[stage], C::kStage);
        uint8_t* sb = smem + stage * C::kStage;
        tma_load_3d(sb, &tmap_b, &full_bar[stage], kb * BK, n0, 0);
        tma_load_3d(sb + C::kBTile, &tmap_a, &full_bar[stage], kb * BK, 0, 0);
        if (++stage == C::kStages) { stage = 0; phase ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    const bool issuer = elect_one();
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!mbar_wait_warp(&full_bar[stage], phase, abort_flag)) { ok = false; break; }
      tc_fence_after();
      if (issuer) {
        const uint32_t sb = smem_u32(smem + stage * C::kStage), sa = sb + C::kBTile;
#pragma unroll
        for (int kk = 0; kk < BK / 16; ++kk)
          umma_f16(tmem_base, make_desc(sb + kk * 32, 16, 1024), make_desc(sa + kk * 32, 16, 1024), p.idesc,
                   (kb > kb0 || kk != 0) ? 1u : 0u);
        umma_commit(&empty_bar[stage]);
      }
      if (++stage == C::kStages) { stage = 0; phase ^= 1; }
    }
    if (ok && issuer) umma_commit(tfull_bar);
    __syncwarp();
  }

  // ---- epilogue.  Warps 2..5: lane = row of B = column of D, TMEM column = row of D; through shared memory, so that a row of
  // D is then added up (over the cluster) and written by one warp, four neighbouring columns per lane
  if (warp >= 2 && mbar_wait_warp(tfull_bar, 0, abort_flag)) {
    tc_fence_after();
    const int q = warp & 3, r = q * 32 + lane;
#pragma unroll
    for (int c = 0; c < MP / 16; ++c) {
      uint32_t raw[16];
      tmem_ld16(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(c * 16), raw);
      tmem_ld_wait();
#pragma unroll
      for (int e = 0; e < 16; ++e) part[(c * 16 + e) * BN + r] = __uint_as_float(raw[e]);
    }
  }
  if (p.splits > 1) {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  } else {
    __syncthreads();
  }
  const int col = n0 + lane * 4;
  const bool vec = sizeof(OutT) == 2 && p.ldd % 4 == 0 && (reinterpret_cast<uintptr_t>(d) & 7) == 0 && col + 4 <= p.n;
  if (!*abort_flag && col < p.n) {
    const uint32_t base = smem_u32(part) + (uint32_t)lane * 16;
    for (int m = rank + p.splits * warp; m < p.m; m += p.splits * (kThreads / 32)) {
      float4 t;
      if (p.splits > 1) {
        float4 v[kMaxSplit];
#pragma unroll
        for (int s = 0; s < kMaxSplit; ++s)
          if (s < p.splits) v[s] = ld_cluster_f32x4(base + (uint32_t)(m * BN * 4), s);
        t = v[0];
#pragma unroll
        for (int s = 1; s < kMaxSplit; ++s)
          if (s < p.splits) { t.x += v[s].x; t.y += v[s].y; t.z += v[s].z; t.w += v[s].w; }
      } else {
        t = *reinterpret_cast<const float4*>(part + m * BN + lane * 4);
      }
      float f[4] = {t.x * p.alpha, t.y * p.alpha, t.z * p.alpha, t.w * p.alpha};
      OutT* o = d + (int64_t)m * p.ldd + col;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (p.bias && col + e < p.n)
          f[e] += p.bias_f32 ? reinterpret_cast<const float*>(p.bias)[col + e]
                             : ToF<OutT>::to(reinterpret_cast<const OutT*>(p.bias)[col + e]);
        if (p.act) f[e] = apply_act(f[e], p.act);
        if (p.accumulate && col + e < p.n) f[e] += ToF<OutT>::to(o[e]);
      }
      if (vec) {
        OutT h[4] = {ToF<OutT>::from(f[0]), ToF<OutT>::from(f[1]), ToF<OutT>::from(f[2]), ToF<OutT>::from(f[3])};
        *reinterpret_cast<uint2*>(o) = *reinterpret_cast<const uint2*>(h);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (col + e < p.n) o[e] = ToF<OutT>::from(f[e]);
      }
    }
  }
  if (p.splits > 1) {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");   // a peer may still read this CTA's sums
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::kTmemCols);
  }
  settle_abort(abort_flag, p.status);
}

template <typename OutT, int MP>
int go(const b200_gemm_desc_t* g, void* d, const void* a, const void* b, int splits, cudaStream_t stream) {
  using C = Cfg<MP>;
  CUtensorMap ma, mb;
  if (!gemm_make_map(&ma, a, g->in_dtype, (uint64_t)g->k, (uint64_t)g->m, 1, (uint64_t)g->lda * 2, 0, BK, MP) ||
      !gemm_make_map(&mb, b, g->in_dtype, (uint64_t)g->k, (uint64_t)g->n, 1, (uint64_t)g->ldb * 2, 0, BK, BN))
    return (int)cudaErrorNotSupported;
  const uint32_t fmt = g->in_dtype == B200_BF16 ? 1u : 0u;
  SkinnyParams p{};
  p.m = g->m; p.n = g->n; p.k = g->k;
  p.ldd = g->ldd;
  p.bias = g->bias;
  p.bias_f32 = g->bias_dtype == B200_F32;
  p.act = g->act;
  p.accumulate = g->accumulate;
  p.alpha = g->alpha;
  p.idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(MP >> 3) << 17) | ((uint32_t)(BN >> 4) << 24);
  p.status = gemm_status_word_device();
  p.splits = splits;
  auto kern = gemm_skinny_kernel<OutT, MP>;
  static OncePerDevice once;
  if (int e = once([&] { return opt_in_smem(kern, C::kSmem); })) return e;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(((g->n + BN - 1) / BN) * splits));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = C::kSmem;
  cfg.stream = stream;
  cudaLaunchAttribute cluster{};
  cluster.id = cudaLaunchAttributeClusterDimension;
  cluster.val.clusterDim.x = (unsigned)splits;
  cluster.val.clusterDim.y = cluster.val.clusterDim.z = 1;
  cfg.attrs = &cluster;
  cfg.numAttrs = splits > 1 ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, ma, mb, (OutT*)d, (const SkinnyParams)p);
  if (e != cudaSuccess) return (int)e;
  B200K_LAUNCH_RET();
}

template <typename OutT>
int by_rows(const b200_gemm_desc_t* g, void* d, const void* a, const void* b, int splits, cudaStream_t stream) {
  if (g->m <= 16) return go<OutT, 16>(g, d, a, b, splits, stream);
  if (g->m <= 32) return go<OutT, 32>(g, d, a, b, splits, stream);
  return go<OutT, 64>(g, d, a, b, splits, stream);
}

}  // namespace

// The line: up to 64 rows (N operand of the instruction) and K long enough to pay for the ring's first fill and the epilogue,
// which grows with the rows, is not overlapped with another tile and in a second wave is paid twice.  General kernel -> this
// one: 64 x 64 x 256 5.1 -> 6.7 us, x 768 7.5 -> 8.0; 64 x 12288 x 512 9.9 -> 10.6, x 768 11.4 -> 11.0; 64 x 28672 x 1024 15.9 ->
// 16.3, x 3072 34.6 -> 34.4; 64 x 38016 x 2048 39.2 -> 40.1, x 3072 55.9 -> 55.3; 48 x 38016 x 1024 22.2 -> 23.3; 32 x 38016 x
// 512 13.7 -> 15.0, x 1024 22.9 -> 22.0; up to 16 rows never slower from K = 256 on (128: 6.6 -> 7.7).  Few columns with a very
// long K stay with the general kernel, whose split-K is not limited to the eight CTAs of a cluster.
bool gemm_skinny_fits(const b200_gemm_desc_t* g) {
  if (g->m > 64 || std::max(g->batch, 1) != 1 || !g->a_kmajor || !g->b_kmajor || g->in_dtype == B200_F32 || g->n < 64) return false;
  const int tiles = (g->n + BN - 1) / BN, sms = gemm_sm_count();
  const bool waves = tiles > 2 * sms;
  int k_min = 256;
  if (tiles == 1) k_min = g->m > 48 ? 1024 : g->m > 32 ? 768 : g->m > 16 ? 512 : 256;
  else if (g->m > 48) k_min = waves ? 3072 : tiles > sms ? 2048 : tiles > sms / 2 ? 768 : 512;
  else if (g->m > 32) k_min = waves ? 2048 : tiles > sms / 2 ? 768 : 256;
  else if (g->m > 16) k_min = waves ? 1024 : 256;
  return g->k >= k_min && (g->n >= 2048 || g->k <= 8192);
}

int gemm_launch_skinny(const b200_gemm_desc_t* g, void* d, const void* a, const void* b, cudaStream_t stream) {
  // as many CTAs per tile as keep all of them resident (two per SM) with at least four K blocks each
  const int tiles = (g->n + BN - 1) / BN, k_blocks = (g->k + BK - 1) / BK;
  // (a power of two, with some room: clusters do not straddle the chip's partitions, so 288 CTAs in threes were two waves)
  int splits = 1;
  while (splits < kMaxSplit && tiles * splits * 2 <= gemm_sm_count() * 7 / 4 && k_blocks >= splits * 8) splits *= 2;
  switch (g->out_dtype) {
    case B200_BF16: return by_rows<__nv_bfloat16>(g, d, a, b, splits, stream);
    case B200_F16: return by_rows<__half>(g, d, a, b, splits, stream);
    case B200_F32: return by_rows<float>(g, d, a, b, splits, stream);
    default: return (int)cudaErrorNotSupported;
  }
}

}  // namespace b200k
