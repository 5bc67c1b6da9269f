// Flash-attention forward on the 5th-generation tensor cores (head_dim 128, bf16 / fp16, optional causal mask,
// grouped-query heads): two query tiles per CTA in ping-pong, scores and the output accumulators in TMEM, K / V through
// a TMA ring, every mbarrier wait bounded (status word as for the GEMMs).  The kernel comment below has the pipeline.
//
// Parity: the reference calls a closed vendor flash kernel (reference torch_musa/csrc/aten/ops/attention/mudnn/SDP.cpp:470-673).
#include "attention_common.cuh"

#include <algorithm>
#include <type_traits>

namespace b200k {
namespace {
using namespace gemmdev;
using namespace attndev;

constexpr int AQ = 128, AK = 128, AD = 128;          // query rows per tile, keys per block, head dim
constexpr int kTile = 128 * 128 * 2;                  // 32 KB: any of Q, K, V
constexpr int kRing = 5;                              // K / V tiles in flight
constexpr int kAttnSmem = 2 * kTile /*Q0,Q1*/ + kRing * kTile + 1024 + 256;
constexpr int kAttnThreads = 384;                     // 2 softmax warpgroups; one with the TMA warp and the MMA warp
constexpr int kSoftmaxRegs = 216, kOtherRegs = 72;    // after the split: a row of scores stays in registers
constexpr int kLaunchRegs = (2 * kSoftmaxRegs + kOtherRegs + 2) / 3;   // what the launch has to bring for that split
constexpr uint32_t kAttnTmemCols = 512;               // S0, S1, O0, O1
constexpr int kFirstPart = 64;                        // keys of a block whose P is released before the rest is computed
constexpr float kRescaleThreshold = 8.f;              // log2 domain: P stays below 2^8

struct AttnParams {
  int B, H, Hkv, Sq, Sk;
  int causal;
  float scale_log2;           // softmax scale * log2(e)
  int64_t o_sb, o_sh, o_ss;   // output strides in elements (last dim contiguous)
  float* lse;                 // [B, H, Sq]; packed sequences: [H, total_q]
  int q_blocks, q_pairs;
  // packed variable-length sequences (NULL: dense batch): sequence b holds rows [cu_q[b], cu_q[b + 1]) of the packed
  // q / out [total_q, H, 128] and rows [cu_k[b], cu_k[b + 1]) of k / v; Sq / Sk are then the longest lengths
  const int* cu_q;
  const int* cu_k;
  int total_q;
  int* status;
};

// One CTA owns two adjacent 128-row query tiles of one (batch, head).  Per block of 128 keys and per tile t:
//   S_t = Q_t K^T     tcgen05.mma M128 N128 K16 x 8 into TMEM (operands in 128B-swizzled shared memory);
//   softmax           warpgroup t, one query row per thread: the row of S comes into registers once, P = exp2(S * scale - m)
//                     goes back as 16-bit pairs into TMEM over the columns of S, the block maximum is found on the side;
//   O_t += P_t V      tcgen05.mma with A = P from TMEM, accumulating in TMEM over all key blocks.
// P never touches shared memory: the M128 N128 products with both operands there already take all of its 128 bytes per
// clock, and writing P there, fencing the async proxy and reading it back stood in the middle of the chain S -> softmax ->
// P V.  One barrier per tile says "all products of this tile so far are done" (S of block j and, before it, P V of block
// j - 1), so the softmax may overwrite S with P and rescale O without another wait.  What bounds the kernel now is that
// chain: per block of 128 keys an SM spends 3900 clocks on both tiles, the starts and ends of its CTAs included; the tensor core
// is busy for 2050 of them (its counter: 50 %) and the special-function units, which the two warpgroups share, for 2050 too (52 %):
// the softmax of a tile, its products and the hand-over follow one another, and two tiles are not enough to fill the gaps of
// both.  Measured at 32 heads x 4096 x 128 bf16, before -> after: causal 174 -> 139 us (990 TFLOP/s), full 300 -> 255 us;
// 32 heads x 16384 causal 1790 us (1230 TFLOP/s).  Tried and not kept: a quarter to a half of the exponentials as polynomials
// on the FMA pipe (+2 to +10 % time), two warpgroups per tile (+11 %), S in halves of 64 keys issued ahead (+12 %: an N64
// product is bound by reading A from shared memory).
// The exponent's reference maximum m is only raised when the running maximum has grown by more than 2^8 ("lazy"
// rescaling): then the warpgroup multiplies its rows of O in TMEM (tcgen05.ld / st) before it releases P.  That is rare
// after the first blocks, so O normally never leaves TMEM until the epilogue.
// The MMA warp alternates between the tiles (P V and next S of tile 0, then of tile 1), so one tile's softmax runs while
// the tensor core works for the other; K and V tiles stream through a five-slot TMA ring.
template <typename T>
__global__ void __launch_bounds__(kAttnThreads, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                const __grid_constant__ CUtensorMap tmap_v, T* __restrict__ out, const AttnParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* sQ = smem;                          // [2][kTile]
  uint8_t* sR = smem + 2 * kTile;              // [kRing][kTile]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (2 + kRing) * kTile);
  uint64_t* q_full = bars;                     // [2]
  uint64_t* r_full = bars + 2;                 // [kRing]
  uint64_t* r_empty = bars + 2 + kRing;        // [kRing]  tcgen05.commit
  uint64_t* mma_done = bars + 2 + 2 * kRing;   // [2]      tcgen05.commit: P V of block j - 1 and S of block j
  uint64_t* p_ready = mma_done + 2;            // [2][2]   four softmax warps: first / second part of P of block j is in TMEM
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(p_ready + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // heavy (late) query tiles first, across all (batch, head) instances
  const int n_bh = p.B * p.H;
  const int qp = p.q_pairs - 1 - (int)(blockIdx.x / n_bh);
  const int bh = (int)(blockIdx.x % n_bh);
  const int b = bh / p.H, h = bh - b * p.H;
  const int hk = h / (p.H / p.Hkv);
  // this instance's sequence: lengths, first packed rows and the batch coordinate of the tensor maps.  Rows past a
  // packed sequence's end belong to the next sequence: they are loaded, masked by index and never stored.
  int Sq = p.Sq, Sk = p.Sk, qoff = 0, koff = 0, bt = b;
  if (p.cu_q) {
    qoff = p.cu_q[b];
    Sq = p.cu_q[b + 1] - qoff;
    koff = p.cu_k[b];
    Sk = p.cu_k[b + 1] - koff;
    bt = 0;
  }
  int nb[2];
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const int q0 = (2 * qp + t) * AQ;
    int k_end = Sk;
    if (p.causal) k_end = min(Sk, q0 + AQ);
    nb[t] = q0 < Sq ? (k_end + AK - 1) / AK : 0;
  }
  const int nbmax = max(nb[0], nb[1]);

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int t = 0; t < 2; ++t) {
      mbar_init(&q_full[t], 1);
      mbar_init(&mma_done[t], 1);
      mbar_init(&p_ready[2 * t], 4);
      mbar_init(&p_ready[2 * t + 1], 4);
    }
    for (int s = 0; s < kRing; ++s) {
      mbar_init(&r_full[s], 1);
      mbar_init(&r_empty[s], 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    prefetch_tmap(&tmap_q);
    prefetch_tmap(&tmap_k);
    prefetch_tmap(&tmap_v);
  }
  if (warp == 9) {
    tmem_alloc(tmem_slot, kAttnTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp >= 8) {
    regs_dec<kOtherRegs>();
    if (warp == 8) {
      // ------------------------------------------------------------ TMA producer
      if (lane == 0) {
        for (int t = 0; t < 2; ++t) {
          if (nb[t] == 0) continue;
          const int q0 = (2 * qp + t) * AQ;
          mbar_expect_tx(&q_full[t], kTile);
          tma_load_4d(sQ + t * kTile, &tmap_q, &q_full[t], 0, qoff + q0, h, bt);                 // d 0..63
          tma_load_4d(sQ + t * kTile + kTile / 2, &tmap_q, &q_full[t], 64, qoff + q0, h, bt);    // d 64..127
        }
        for (int n = 0; n < 2 * nbmax; ++n) {
          const int st = n % kRing;
          if (!mbar_wait(&r_empty[st], (uint32_t)(((n / kRing) & 1) ^ 1), abort_flag)) break;
          mbar_expect_tx(&r_full[st], kTile);
          const int k0 = (n >> 1) * AK;
          const CUtensorMap* map = (n & 1) ? &tmap_v : &tmap_k;   // V is read as an MN-major B operand: same boxes
          tma_load_4d(sR + st * kTile, map, &r_full[st], 0, koff + k0, hk, bt);
          tma_load_4d(sR + st * kTile + kTile / 2, map, &r_full[st], 64, koff + k0, hk, bt);
        }
      }
      __syncwarp();
    } else if (warp == 9) {
      // ------------------------------------------------------------ MMA issuer (the whole warp waits, one lane issues)
      // instruction descriptors: fp32 accumulate, bf16/fp16 operands, M128 N128; S: both K-major; PV: B MN-major
      constexpr uint32_t fmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
      constexpr uint32_t idesc_s = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(128 >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
      constexpr uint32_t idesc_o = idesc_s | (1u << 16);
      const bool leader = elect_one();
      const uint64_t q_desc = make_desc(smem_u32(sQ), 16, 1024);             // K-major tiles; + (bytes >> 4) for an offset
      const uint64_t k_desc = make_desc(smem_u32(sR), 16, 1024);
      const uint64_t v_desc = make_desc(smem_u32(sR), kTile / 2, 1024);      // MN-major
      auto wait = [&](uint64_t* bar, uint32_t parity) { return mbar_wait_warp(bar, parity, abort_flag); };
      auto ring_wait = [&](int n) { return wait(&r_full[n % kRing], (uint32_t)((n / kRing) & 1)); };
      auto issue_s = [&](int t, int n) {     // S_t = Q_t K^T with K in ring item n
        const uint64_t qa = q_desc + (uint32_t)(t * (kTile >> 4)), ka = k_desc + (uint32_t)((n % kRing) * (kTile >> 4));
  #pragma unroll
        for (int kk = 0; kk < AD / 16; ++kk) {
          const uint32_t off = ((uint32_t)(kk >> 2) * (kTile / 2) + (uint32_t)(kk & 3) * 32) >> 4;   // 64-column atom, 32 B per k16
          umma_f16(tmem_base + (uint32_t)(t * 128), qa + off, ka + off, idesc_s, kk != 0 ? 1u : 0u);
        }
      };
      auto issue_pv = [&](int t, int n, bool first, int kk0, int kk1) {   // O_t (+)= P_t V with V in ring item n
        const uint32_t pa = tmem_base + (uint32_t)(t * 128);
        const uint64_t va = v_desc + (uint32_t)((n % kRing) * (kTile >> 4));
  #pragma unroll
        for (int kk = kk0; kk < kk1; ++kk)
          // A = P in TMEM, 8 columns per 16 keys; B = V (MN-major): 16 key rows = 2048 B, next 64-wide d box 16 KB on
          umma_f16_ts(tmem_base + 256u + (uint32_t)(t * 128), pa + (uint32_t)(kk * 8), va + (uint32_t)(kk * (2048 >> 4)), idesc_o,
                      (first && kk == 0) ? 0u : 1u);
      };
      bool ok = true;
      for (int t = 0; t < 2 && ok; ++t)
        if (nb[t] > 0) ok = wait(&q_full[t], 0);
      if (ok && nbmax > 0) ok = ring_wait(0);
      if (ok && nbmax > 0) {
        tc_fence_after();
        if (leader) {
          for (int t = 0; t < 2; ++t)
            if (nb[t] > 0) {
              issue_s(t, 0);
              umma_commit(&mma_done[t]);
            }
          umma_commit(&r_empty[0]);
        }
      }
      for (int j = 0; j < nbmax && ok; ++j) {
        const int nv = 2 * j + 1, nk = 2 * j + 2;
        if (!ring_wait(nv)) { ok = false; break; }
        if (j + 1 < nbmax && !ring_wait(nk)) { ok = false; break; }
        for (int t = 0; t < 2; ++t) {
          if (j >= nb[t]) continue;
          if (!wait(&p_ready[2 * t], (uint32_t)(j & 1))) { ok = false; break; }
          tc_fence_after();
          if (leader) issue_pv(t, nv, j == 0, 0, kFirstPart / 16);
          if (!wait(&p_ready[2 * t + 1], (uint32_t)(j & 1))) { ok = false; break; }
          tc_fence_after();
          if (leader) {
            issue_pv(t, nv, false, kFirstPart / 16, AK / 16);
            if (j + 1 < nb[t]) issue_s(t, nk);     // over P of block j: the tensor core works in issue order
            umma_commit(&mma_done[t]);
          }
        }
        if (!ok) break;
        if (leader) {
          umma_commit(&r_empty[nv % kRing]);
          if (j + 1 < nbmax) umma_commit(&r_empty[nk % kRing]);
        }
      }
      __syncwarp();
    }
  } else {
    regs_inc<kSoftmaxRegs>();
    // ------------------------------------------------------------ softmax warpgroup t (warps 4t .. 4t+3)
    const int t = warp >> 2;
    const int qw = warp & 3;                 // TMEM lane quarter of this warp
    const int r = qw * 32 + lane;            // query row inside the tile = TMEM lane
    const int qi = (2 * qp + t) * AQ + r;
    const uint32_t lane_base = ((uint32_t)(qw * 32) << 16);
    const uint32_t s_addr = tmem_base + lane_base + (uint32_t)(t * 128);
    const uint32_t o_addr = tmem_base + lane_base + 256u + (uint32_t)(t * 128);
    float m_ref = -INFINITY;                 // maximum the exponents refer to (raised lazily)
    float l_run = 0.f;
    bool ok = true;
    const int n_blocks = nb[t];
    // warp-uniform wait: the warp-collective TMEM accesses and votes below need all 32 lanes to take the same path
    auto wait_all = [&](uint64_t* bar, uint32_t parity) {
      const bool w = mbar_wait(bar, parity, abort_flag);
      return __all_sync(0xffffffffu, w);
    };
    for (int j = 0; j < n_blocks; ++j) {
      if (!wait_all(&mma_done[t], (uint32_t)(j & 1))) { ok = false; break; }
      tc_fence_after();
      const int k0 = j * AK;
      // the row's visible keys: [0, lim)
      int lim = Sk - k0;
      if (p.causal) lim = min(lim, qi - k0 + 1);
      lim = max(0, min(lim, AK));
      const bool full = __all_sync(0xffffffffu, lim == AK);
      // the whole row of scores in registers
      uint32_t raw[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld32(s_addr + (uint32_t)(c * 32), raw[c]);
      tmem_ld_wait();
      // P = exp2(S * scale - m) as bf16 / fp16 pairs over the first 64 columns of S; packed fp32 arithmetic, one
      // special-function instruction per exponential, one conversion per pair.  Two instantiations: with the mask test
      // inside one, every element pays a compare and a select.
      float l0, l1;
      uint32_t pk[4][16];
      auto chunk_p = [&](auto masked, int c, float neg_m) {
#pragma unroll
        for (int e = 0; e < 32; e += 2) {
          float x0, x1;
          fma2(x0, x1, __uint_as_float(raw[c][e]), __uint_as_float(raw[c][e + 1]), p.scale_log2, neg_m);
          float p0 = ex2_approx(x0), p1 = ex2_approx(x1);
          if constexpr (decltype(masked)::value) {
            if (c * 32 + e >= lim) p0 = 0.f;
            if (c * 32 + e + 1 >= lim) p1 = 0.f;
          }
          add2(l0, l1, p0, p1);
          pk[c][e >> 1] = pack2<T>(p0, p1);
        }
      };
      auto block = [&](auto masked) {
        // The first part is computed against the reference maximum as it stands, while the block's own maximum is found
        // beside it (four chains of three-input maxima under the special-function unit's shadow): m is raised in the first
        // block and hardly ever after it, and only then is the first part computed again.
        l0 = l1 = 0.f;
        const float m_old = m_ref == -INFINITY ? 0.f : m_ref;
#pragma unroll
        for (int c = 0; c < kFirstPart / 32; ++c) chunk_p(masked, c, -m_old);
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int e = 0; e < 32; e += 2) {
            float a = __uint_as_float(raw[c][e]), b2 = __uint_as_float(raw[c][e + 1]);
            if constexpr (decltype(masked)::value) {
              if (c * 32 + e >= lim) a = -INFINITY;
              if (c * 32 + e + 1 >= lim) b2 = -INFINITY;
            }
            mx[(e >> 1) & 3] = max3(mx[(e >> 1) & 3], a, b2);
          }
        const float m_blk = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
        const float m_new = fmaxf(m_ref, m_blk * p.scale_log2);
        const bool raise = m_new - m_ref > kRescaleThreshold;      // also true for the first finite maximum
        if (__any_sync(0xffffffffu, raise)) {
          const float alpha = raise ? exp2f(m_ref - m_new) : 1.f;   // 0 when m_ref = -inf
          if (j > 0) {
#pragma unroll
            for (int c = 0; c < AD / 16; ++c) {
              uint32_t o16[16];
              tmem_ld16(o_addr + (uint32_t)(c * 16), o16);
              tmem_ld_wait();
#pragma unroll
              for (int e = 0; e < 16; ++e) o16[e] = __float_as_uint(__uint_as_float(o16[e]) * alpha);
              tmem_st16(o_addr + (uint32_t)(c * 16), o16);
            }
          }
          if (raise) {
            l_run *= alpha;
            m_ref = m_new;
          }
          l0 = l1 = 0.f;
          const float m_use = m_ref == -INFINITY ? 0.f : m_ref;     // row without any visible key so far
#pragma unroll
          for (int c = 0; c < kFirstPart / 32; ++c) chunk_p(masked, c, -m_use);
        }
#pragma unroll
        for (int c = 0; c < kFirstPart / 32; ++c) tmem_st16(s_addr + (uint32_t)(c * 16), pk[c]);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_ready[2 * t]);
        const float m_use = m_ref == -INFINITY ? 0.f : m_ref;
#pragma unroll
        for (int c = kFirstPart / 32; c < 4; ++c) {
          chunk_p(masked, c, -m_use);
          tmem_st16(s_addr + (uint32_t)(c * 16), pk[c]);
        }
      };
      if (full) block(std::false_type{});
      else block(std::true_type{});
      l_run += l0 + l1;
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_ready[2 * t + 1]);
    }
    if (ok && n_blocks > 0) ok = wait_all(&mma_done[t], (uint32_t)(n_blocks & 1));
    if (ok && n_blocks > 0) {
      tc_fence_after();
      const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
      T* orow = out + (int64_t)bt * p.o_sb + (int64_t)h * p.o_sh + (int64_t)(qoff + qi) * p.o_ss;
#pragma unroll
      for (int c = 0; c < AD / 32; ++c) {
        uint32_t raw[32];
        tmem_ld32(o_addr + (uint32_t)(c * 32), raw);
        tmem_ld_wait();
        if (qi < Sq) {
#pragma unroll
          for (int g8 = 0; g8 < 4; ++g8) {
            Vec16<T> v;
#pragma unroll
            for (int e = 0; e < 8; ++e) v.v[e] = ToF<T>::from(__uint_as_float(raw[g8 * 8 + e]) * inv);
            st16(orow + c * 32 + g8 * 8, v);
          }
        }
      }
      if (qi < Sq && p.lse)
        p.lse[p.cu_q ? (int64_t)h * p.total_q + qoff + qi : ((int64_t)b * p.H + h) * p.Sq + qi] = l_run > 0.f ? (m_ref + log2f(l_run)) * 0.6931471805599453f : -INFINITY;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kAttnTmemCols);
  }
  settle_abort(abort_flag, p.status);
}

template <typename K>
int fwd_setup(K kern) {
  cudaFuncAttributes at;
  cudaError_t e = cudaFuncGetAttributes(&at, kern);
  if (e != cudaSuccess) return (int)e;
  if (at.numRegs < kLaunchRegs) return (int)cudaErrorNotSupported;   // the register split would wait for ever
  return opt_in_smem(kern, kAttnSmem);
}

}  // namespace
}  // namespace b200k

using namespace b200k;

extern "C" int b200_flash_attn_fwd(const b200_attn_t* a, void* out, float* lse, const void* q, const void* k,
                                   const void* v, cudaStream_t stream) {
  if (a->head_dim != AD || (a->dtype != B200_BF16 && a->dtype != B200_F16) || a->B <= 0 || a->H <= 0 || a->Hkv <= 0 ||
      a->H % a->Hkv != 0 || a->Sq <= 0 || a->Sk <= 0)
    return (int)cudaErrorNotSupported;
  auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  auto st_ok = [](int64_t s) { return s % 8 == 0; };
  if (!al(q) || !al(k) || !al(v) || !al(out) || !st_ok(a->q_sb) || !st_ok(a->q_sh) || !st_ok(a->q_ss) || !st_ok(a->k_sb) ||
      !st_ok(a->k_sh) || !st_ok(a->k_ss) || !st_ok(a->v_sb) || !st_ok(a->v_sh) || !st_ok(a->v_ss) || !st_ok(a->o_sb) ||
      !st_ok(a->o_sh) || !st_ok(a->o_ss))
    return (int)cudaErrorNotSupported;
  // a broadcast (zero) stride cannot be a tensor-map stride
  if ((a->B > 1 && !a->cu_seqlens_q && (a->q_sb == 0 || a->k_sb == 0 || a->v_sb == 0)) || (a->H > 1 && a->q_sh == 0) ||
      (a->Hkv > 1 && (a->k_sh == 0 || a->v_sh == 0)) || a->q_ss == 0 || a->k_ss == 0 || a->v_ss == 0)
    return (int)cudaErrorNotSupported;
  const int bf16 = a->dtype == B200_BF16;
  CUtensorMap mq, mk, mv;
  auto nz = [](int64_t s, int64_t fallback) { return s ? s : fallback; };
  const bool packed = a->cu_seqlens_q != nullptr;
  if (packed) {
    if (!a->cu_seqlens_k || a->total_q <= 0 || a->total_k <= 0) return (int)cudaErrorNotSupported;
    // one "batch" of total rows: the kernel adds each sequence's first row to its tile coordinates
    if (!make_attn_map(&mq, q, bf16, 1, a->H, a->total_q, (int64_t)a->total_q * a->q_ss, nz(a->q_sh, 8), a->q_ss) ||
        !make_attn_map(&mk, k, bf16, 1, a->Hkv, a->total_k, (int64_t)a->total_k * a->k_ss, nz(a->k_sh, 8), a->k_ss) ||
        !make_attn_map(&mv, v, bf16, 1, a->Hkv, a->total_k, (int64_t)a->total_k * a->v_ss, nz(a->v_sh, 8), a->v_ss))
      return (int)cudaErrorNotSupported;
  } else if (!make_attn_map(&mq, q, bf16, a->B, a->H, a->Sq, nz(a->q_sb, 8), nz(a->q_sh, 8), a->q_ss) ||
             !make_attn_map(&mk, k, bf16, a->B, a->Hkv, a->Sk, nz(a->k_sb, 8), nz(a->k_sh, 8), a->k_ss) ||
             !make_attn_map(&mv, v, bf16, a->B, a->Hkv, a->Sk, nz(a->v_sb, 8), nz(a->v_sh, 8), a->v_ss))
    return (int)cudaErrorNotSupported;
  AttnParams p{};
  p.B = a->B; p.H = a->H; p.Hkv = a->Hkv; p.Sq = a->Sq; p.Sk = a->Sk;
  p.causal = a->causal;
  p.scale_log2 = a->scale * 1.4426950408889634f;
  p.o_sb = a->o_sb; p.o_sh = a->o_sh; p.o_ss = a->o_ss;
  p.lse = lse;
  p.cu_q = a->cu_seqlens_q;
  p.cu_k = a->cu_seqlens_k;
  p.total_q = a->total_q;
  p.q_blocks = (a->Sq + AQ - 1) / AQ;
  p.q_pairs = (p.q_blocks + 1) / 2;
  p.status = gemm_status_word_device();
  const long long grid = (long long)a->B * a->H * p.q_pairs;
  if (grid > 2147483647ll) return (int)cudaErrorNotSupported;
  if (bf16) {
    static OncePerDevice once;
    if (int e = once([] { return fwd_setup(attn_fwd_kernel<__nv_bfloat16>); })) return e;
    attn_fwd_kernel<__nv_bfloat16><<<(unsigned)grid, kAttnThreads, kAttnSmem, stream>>>(mq, mk, mv, (__nv_bfloat16*)out, p);
  } else {
    static OncePerDevice once;
    if (int e = once([] { return fwd_setup(attn_fwd_kernel<__half>); })) return e;
    attn_fwd_kernel<__half><<<(unsigned)grid, kAttnThreads, kAttnSmem, stream>>>(mq, mk, mv, (__half*)out, p);
  }
  B200K_LAUNCH_RET();
}
