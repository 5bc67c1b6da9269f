// Flash-attention backward on the 5th-generation tensor cores (head_dim 128, bf16 / fp16, optional causal mask,
// grouped-query heads).
//
// One CTA owns one block of 128 keys of one (batch, kv head); K and V stay resident in shared memory, dK and dV
// accumulate in TMEM over every query block (and every query head of the group) that sees the keys.  Everything is
// computed transposed, keys along the 128 TMEM lanes, so that one thread owns one key row:
//   S^T  = K Q^T          tcgen05.mma, both operands K-major                         -> TMEM columns [0, 128)
//   dP^T = V dO^T         the same shape                                             -> TMEM columns [128, 256)
//   P^T  = exp2(S^T * scale - lse[q])     two warpgroups, half of the query columns each; 16-bit pairs into TMEM over S^T
//   dV  += P^T dO         A = P^T from TMEM, B = dO read MN-major                    -> TMEM columns [256, 384)
//   dS^T = P^T * (dP^T - delta[q]) * scale   the same warpgroups; 16-bit into shared memory in the layout of an A operand
//   dQ   = dS K           A = dS^T read MN-major, B = K read MN-major, fresh         -> TMEM columns [128, 256) again
//   dK  += dS^T Q         A = dS^T, B = Q read MN-major                              -> TMEM columns [384, 512)
// A third warpgroup takes dQ of every (query block, key block) pair out of TMEM, stages it as fp32 in two 16 KB boxes of
// its own and adds it to an fp32 buffer in global memory by TMA reductions (cp.reduce.async.bulk.tensor ... add); the
// caller converts that buffer afterwards.  delta = rowsum(dO * O) comes from a small kernel that also zeroes the buffer.
//
// What runs beside what, per pair: S^T of the next pair is issued right after dV, so its exponentials run while the tensor
// core does dQ and dK; dQ leaves TMEM into registers while dK runs, which frees its columns for the next dP^T; the staging
// and the reductions have the whole next pair's time.  The loop that remains is dS -> dQ -> (dQ out of TMEM, under dK) ->
// next dP^T -> next dS.  P^T in TMEM instead of shared memory pays for the separate staging boxes.  Q streams through two
// slots, dO through one (it is free after dV), lse and delta through a two-slot ring filled by a warp of its own; every wait
// is bounded.
// What bounds it now is shared memory: per pair an SM spends 5060 clocks, the starts and ends of its CTAs included; the products
// read 2300 wavefronts of 128 bytes (288 KB) and the threads' loads and stores (dS^T, the staged dQ, lse and delta) take 2840
// more, 1290 of them without the conflicts, while the tensor core is busy for 2560 (counters at 32 heads x 4096 x 128).  bf16,
// before -> after: causal 672 -> 351 us (980 TFLOP/s), full 1310 -> 640.  Registers: 96 for the warps that issue keep their
// descriptors out of local memory, whose traffic goes through the same shared-memory path (with 56: +9 %).
// Tried and not kept: starting each block of keys at another query block (+10 %).
//
// Parity: the reference calls a closed vendor flash backward (reference torch_musa/csrc/aten/ops/attention/mudnn/SDP.cpp:678-845).
#include "attention_common.cuh"

#include <algorithm>
#include <type_traits>

namespace b200k {
namespace {
using namespace gemmdev;
using namespace attndev;

constexpr int BQ = 128, BK = 128, BD = 128;
constexpr int kTile = 128 * 128 * 2;
constexpr int kStage = 128 * 32 * 4;                  // 16 KB: 32 fp32 columns of dQ
constexpr int kBwdSlack = 768;                        // for the alignment of the tiles to 1024 bytes (checked by the kernel)
constexpr int kBwdSmem = 2 * kTile /*K, V*/ + 2 * kTile /*Q*/ + kTile /*dO*/ + kTile /*dS^T*/ + 2 * kStage /*dQ*/ +
                         2 * 2 * 128 * 4 /*lse, delta*/ + 256 /*barriers*/ + kBwdSlack;
static_assert(kBwdSmem <= 232448, "exceeds the 227 KB of shared memory a CTA can have");
constexpr int kBwdThreads = 512;                      // 2 compute warpgroups, dQ warpgroup, TMA / MMA / lse-delta warps
constexpr int kComputeRegs = 136, kDqRegs = 144, kOtherRegs = 96;    // register split (sum: what 128 per thread brings)
constexpr int kLaunchRegs = (2 * kComputeRegs + kDqRegs + kOtherRegs + 3) / 4;
constexpr uint32_t kBwdTmemCols = 512;

struct BwdParams {
  int B, H, Hkv, Sq, Sk;
  int causal;
  float scale, scale_log2;
  const float* lse;       // [B, H, Sq] natural log
  const float* delta;     // [B, H, Sq]
  float* dq;              // [B, H, Sq, 128] fp32
  int64_t dk_sb, dk_sh, dk_ss, dv_sb, dv_sh, dv_ss;
  int kv_blocks, q_blocks;
  int* status;
  // packed variable-length sequences (NULL: dense batch), as in the forward kernel; lse / delta are then [H, total_q]
  // and dq [H, total_q, 128]
  const int* cu_q;
  const int* cu_k;
  int total_q;
};

// adds a [128 rows x 32 floats] box of shared memory (128B-swizzled) into global memory at (x, y) of the tensor map
__device__ __forceinline__ void tma_reduce_add_2d(const CUtensorMap* map, const void* smem_src, int x, int y) {
  asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"(map), "r"(smem_u32(smem_src)), "r"(x), "r"(y)
               : "memory");
}

template <typename T>
__global__ void __launch_bounds__(kBwdThreads, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_do,
                const __grid_constant__ CUtensorMap tmap_dq, T* __restrict__ dk, T* __restrict__ dv, const BwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  if (smem - smem_raw > kBwdSlack) {        // cannot happen while the kernel has no static shared memory
    if (threadIdx.x == 0 && p.status) atomicExch(p.status, 1);
    return;
  }
  uint8_t* sK = smem;
  uint8_t* sV = smem + kTile;
  uint8_t* sQ = smem + 2 * kTile;                    // [2][kTile]
  uint8_t* sdO = smem + 4 * kTile;
  uint8_t* sS = smem + 5 * kTile;                    // dS^T [keys x queries]
  uint8_t* sStage = smem + 6 * kTile;                // [2][kStage] fp32 dQ
  float* s_lse = reinterpret_cast<float*>(smem + 6 * kTile + 2 * kStage);   // [2][128]
  float* s_dlt = s_lse + 2 * 128;                                             // [2][128]
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_dlt + 2 * 128);
  uint64_t* kv_full = bars;                  // 1
  uint64_t* q_full = bars + 1;               // [2]
  uint64_t* q_empty = bars + 3;              // [2]  tcgen05.commit after dK
  uint64_t* do_full = bars + 5;              // 1
  uint64_t* do_empty = bars + 6;             // tcgen05.commit after dV
  uint64_t* s_full = bars + 7;               // tcgen05.commit: S^T
  uint64_t* dp_full = bars + 8;              // tcgen05.commit: dP^T (and with it everything issued before)
  uint64_t* p_ready = bars + 9;              // 8 warps: P^T in TMEM
  uint64_t* ds_ready = bars + 10;            // 8 warps: dS^T in shared memory, dP^T read
  uint64_t* dq_full = bars + 11;             // tcgen05.commit: dQ
  uint64_t* dq_drained = bars + 12;          // 4 warps: dQ is in registers
  uint64_t* all_done = bars + 13;            // tcgen05.commit: dV, dK complete
  uint64_t* ld_full = bars + 14;             // [2]  lse and delta of a query block are there
  uint64_t* ld_empty = bars + 16;            // [2]  8 warps
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 18);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // all (batch, head) instances of the earliest key block first: under a causal mask it meets the most query blocks
  const int n_bh = p.B * p.Hkv;
  const int kb = (int)(blockIdx.x / n_bh);
  const int bh = (int)(blockIdx.x % n_bh);
  const int b = bh / p.Hkv, hk = bh - b * p.Hkv;
  const int G = p.H / p.Hkv;
  const int k0 = kb * BK;
  // this instance's sequence (see the forward kernel): rows past a packed sequence's end are loaded, masked by index
  // (their probabilities and score gradients are exact zeros) and never stored
  int Sq = p.Sq, Sk = p.Sk, qoff = 0, koff = 0, bt = b, q_blocks = p.q_blocks;
  if (p.cu_q) {
    qoff = p.cu_q[b];
    Sq = p.cu_q[b + 1] - qoff;
    koff = p.cu_k[b];
    Sk = p.cu_k[b + 1] - koff;
    bt = 0;
    q_blocks = (Sq + BQ - 1) / BQ;
  }
  const int i0 = p.causal ? min(q_blocks, k0 / BQ) : 0;   // first query block that sees these keys
  const int n_i = k0 < Sk ? q_blocks - i0 : 0;            // a key block past the sequence's end has nothing to do
  const int n_it = n_i * G;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    mbar_init(kv_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 1);
      mbar_init(&ld_full[i], 1);
      mbar_init(&ld_empty[i], 8);
    }
    mbar_init(do_full, 1);
    mbar_init(do_empty, 1);
    mbar_init(s_full, 1);
    mbar_init(dp_full, 1);
    mbar_init(p_ready, 8);
    mbar_init(ds_ready, 8);
    mbar_init(dq_full, 1);
    mbar_init(dq_drained, 4);
    mbar_init(all_done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    prefetch_tmap(&tmap_q);
    prefetch_tmap(&tmap_k);
    prefetch_tmap(&tmap_v);
    prefetch_tmap(&tmap_do);
    prefetch_tmap(&tmap_dq);
  }
  if (warp == 13) {
    tmem_alloc(tmem_slot, kBwdTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  constexpr uint32_t kColS = 0, kColDP = 128, kColDV = 256, kColDK = 384;

  if (warp >= 12) {
    regs_dec<kOtherRegs>();
    if (warp == 12) {
      // ------------------------------------------------------------ TMA producer
      if (lane == 0 && n_it > 0) {
        mbar_expect_tx(kv_full, 2 * kTile);
        tma_load_4d(sK, &tmap_k, kv_full, 0, koff + k0, hk, bt);
        tma_load_4d(sK + kTile / 2, &tmap_k, kv_full, 64, koff + k0, hk, bt);
        tma_load_4d(sV, &tmap_v, kv_full, 0, koff + k0, hk, bt);
        tma_load_4d(sV + kTile / 2, &tmap_v, kv_full, 64, koff + k0, hk, bt);
        int h = hk * G, i = 0;
        for (int it = 0; it < n_it; ++it) {
          const int q0 = (i0 + i) * BQ, st = it & 1;
          if (!mbar_wait(&q_empty[st], (uint32_t)(((it >> 1) & 1) ^ 1), abort_flag)) break;
          mbar_expect_tx(&q_full[st], kTile);
          tma_load_4d(sQ + st * kTile, &tmap_q, &q_full[st], 0, qoff + q0, h, bt);
          tma_load_4d(sQ + st * kTile + kTile / 2, &tmap_q, &q_full[st], 64, qoff + q0, h, bt);
          if (!mbar_wait(do_empty, (uint32_t)((it & 1) ^ 1), abort_flag)) break;
          mbar_expect_tx(do_full, kTile);
          tma_load_4d(sdO, &tmap_do, do_full, 0, qoff + q0, h, bt);
          tma_load_4d(sdO + kTile / 2, &tmap_do, do_full, 64, qoff + q0, h, bt);
          if (++i == n_i) { i = 0; ++h; }
        }
      }
      __syncwarp();
    } else if (warp == 13) {
      // ------------------------------------------------------------ MMA issuer (the whole warp waits, one lane issues)
      constexpr uint32_t fmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
      constexpr uint32_t idesc_kk = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(128 >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
      constexpr uint32_t idesc_kmn = idesc_kk | (1u << 16);                 // B read MN-major
      constexpr uint32_t idesc_mnmn = idesc_kk | (1u << 15) | (1u << 16);   // A and B read MN-major
      const bool issuer = elect_one();
      auto wait = [&](uint64_t* bar, int n) { return mbar_wait_warp(bar, (uint32_t)(n & 1), abort_flag); };
      auto kdesc = [&](const uint8_t* tile) { return make_desc(smem_u32(tile), 16, 1024); };            // read K-major
      auto mndesc = [&](const uint8_t* tile) { return make_desc(smem_u32(tile), kTile / 2, 1024); };    // read MN-major
      const uint64_t dK_k = kdesc(sK), dV_k = kdesc(sV), dO_k = kdesc(sdO), dQ_k = kdesc(sQ), dS_k = kdesc(sS);
      const uint64_t dK_mn = mndesc(sK), dO_mn = mndesc(sdO), dQ_mn = mndesc(sQ), dS_mn = mndesc(sS);
      auto koff16 = [](int kk) { return (uint32_t)(((kk >> 2) * (kTile / 2) + (kk & 3) * 32) >> 4); };   // K-major: two 64-column atoms
      auto mnoff16 = [](int kk) { return (uint32_t)((kk * 2048) >> 4); };                                // MN-major: 16 rows of 128 bytes
      bool ok = n_it > 0 && wait(kv_full, 0) && wait(&q_full[0], 0);
      if (ok) {
        tc_fence_after();
        if (issuer) {
#pragma unroll
          for (int kk = 0; kk < 8; ++kk) umma_f16(tmem_base + kColS, dK_k + koff16(kk), dQ_k + koff16(kk), idesc_kk, kk != 0 ? 1u : 0u);
          umma_commit(s_full);
        }
      }
      for (int it = 0; it < n_it && ok; ++it) {
        const uint32_t tq = (uint32_t)((it & 1) * (kTile >> 4)), tq_next = (uint32_t)(((it + 1) & 1) * (kTile >> 4));
        if (!wait(do_full, it)) { ok = false; break; }
        if (it > 0 && !wait(dq_drained, it - 1)) { ok = false; break; }
        tc_fence_after();
        if (issuer) {
#pragma unroll
          for (int kk = 0; kk < 8; ++kk) umma_f16(tmem_base + kColDP, dV_k + koff16(kk), dO_k + koff16(kk), idesc_kk, kk != 0 ? 1u : 0u);
          umma_commit(dp_full);                        // dP^T = V dO^T
        }
        if (!wait(p_ready, it)) { ok = false; break; }
        tc_fence_after();
        if (issuer) {
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)               // dV += P^T dO; P^T of 64 queries over the left of its half of S^T
            umma_f16_ts(tmem_base + kColDV, tmem_base + kColS + (uint32_t)((kk >> 2) * 64 + (kk & 3) * 8), dO_mn + mnoff16(kk),
                        idesc_kmn, (it == 0 && kk == 0) ? 0u : 1u);
          umma_commit(do_empty);
        }
        if (it + 1 < n_it) {
          if (!wait(&q_full[(it + 1) & 1], (it + 1) >> 1)) { ok = false; break; }
          tc_fence_after();
          if (issuer) {
#pragma unroll
            for (int kk = 0; kk < 8; ++kk)             // S^T of the next pair, over P^T of this one
              umma_f16(tmem_base + kColS, dK_k + koff16(kk), dQ_k + tq_next + koff16(kk), idesc_kk, kk != 0 ? 1u : 0u);
            umma_commit(s_full);
          }
        }
        if (!wait(ds_ready, it)) { ok = false; break; }
        tc_fence_after();
        if (issuer) {
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)               // dQ = dS K over the consumed dP^T
            umma_f16(tmem_base + kColDP, dS_mn + mnoff16(kk), dK_mn + mnoff16(kk), idesc_mnmn, kk != 0 ? 1u : 0u);
          umma_commit(dq_full);
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)               // dK += dS^T Q
            umma_f16(tmem_base + kColDK, dS_k + koff16(kk), dQ_mn + tq + mnoff16(kk), idesc_kmn, (it == 0 && kk == 0) ? 0u : 1u);
          umma_commit(&q_empty[it & 1]);
          if (it + 1 == n_it) umma_commit(all_done);
        }
      }
      __syncwarp();
    } else if (warp == 14) {
      // ------------------------------------------------------------ lse (log2 domain, negated: an addend of the exponent) and
      // delta (times the softmax scale, negated) of every query block; an lse of -inf switches a row off
      // (read one block ahead, all eight loads in flight at once)
      int h = hk * G, i = 0;
      float l[4], d[4];
      auto fetch = [&]() {
        const int64_t base = p.cu_q ? (int64_t)h * p.total_q + qoff : ((int64_t)b * p.H + h) * p.Sq;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int qi = (i0 + i) * BQ + e * 32 + lane;
          l[e] = qi < Sq ? __ldg(p.lse + base + qi) : -INFINITY;
          d[e] = qi < Sq ? __ldg(p.delta + base + qi) : 0.f;
        }
      };
      if (n_it > 0) fetch();
      for (int it = 0; it < n_it; ++it) {
        const int st = it & 1;
        if (!mbar_wait_warp(&ld_empty[st], (uint32_t)(((it >> 1) & 1) ^ 1), abort_flag)) break;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          s_lse[st * 128 + e * 32 + lane] = l[e] > -INFINITY ? -l[e] * 1.4426950408889634f : -INFINITY;
          s_dlt[st * 128 + e * 32 + lane] = -d[e] * p.scale;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&ld_full[st]);
        if (++i == n_i) { i = 0; ++h; }
        if (it + 1 < n_it) fetch();
      }
    }
  } else if (warp >= 8) {
    regs_inc<kDqRegs>();
    // ------------------------------------------------------------ dQ warpgroup: TMEM -> registers -> shared memory -> global
    const int qw = warp & 3;
    const int r = qw * 32 + lane;                 // query row inside the block = TMEM lane
    const uint32_t addr = tmem_base + ((uint32_t)(qw * 32) << 16) + kColDP;
    int h = hk * G, i = 0;
    for (int it = 0; it < n_it; ++it) {
      const int q0 = (i0 + i) * BQ;
      bool ok = mbar_wait_warp(dq_full, (uint32_t)(it & 1), abort_flag);
      tc_fence_after();
      uint32_t raw[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld32(addr + (uint32_t)(c * 32), raw[c]);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(dq_drained);
      const int row0 = p.cu_q ? (int)((int64_t)h * p.total_q + qoff + q0) : (int)(((int64_t)b * p.H + h) * p.Sq + q0);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        // the reduction that read this box two chunks ago has finished with it
        if (threadIdx.x == 8 * 32) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
        if (!named_bar_and(1, 128, ok)) { ok = false; break; }     // one answer for the four warps
        uint8_t* box = sStage + (c & 1) * kStage + (size_t)r * 128;
#pragma unroll
        for (int ch = 0; ch < 8; ++ch)
          *reinterpret_cast<uint4*>(box + (size_t)((ch ^ (r & 7)) * 16)) =
              make_uint4(raw[c][ch * 4], raw[c][ch * 4 + 1], raw[c][ch * 4 + 2], raw[c][ch * 4 + 3]);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        named_bar_sync(1, 128);
        if (threadIdx.x == 8 * 32) {
          tma_reduce_add_2d(&tmap_dq, sStage + (c & 1) * kStage, c * 32, row0);
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
      }
      if (!ok) break;
      if (++i == n_i) { i = 0; ++h; }
    }
    // every reduction must have completed before the CTA exits
    if (threadIdx.x == 8 * 32) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  } else {
    regs_inc<kComputeRegs>();
    // ------------------------------------------------------------ two compute warpgroups (warps 0-3, 4-7)
    const int wg = warp >> 2;
    const int qw = warp & 3;
    const int r = qw * 32 + lane;                 // key row inside the block = TMEM lane
    const int kj = k0 + r;
    const uint32_t lane_base = ((uint32_t)(qw * 32) << 16);
    const uint32_t s_addr = tmem_base + lane_base + kColS + (uint32_t)(wg * 64);
    const uint32_t dp_addr = tmem_base + lane_base + kColDP + (uint32_t)(wg * 64);
    uint8_t* srow = sS + (size_t)wg * (kTile / 2) + (size_t)r * 128;   // this warpgroup's 64 query columns = atom `wg`
    const bool key_off = kj >= Sk;
    const bool block_off = k0 + BK > Sk;
    bool ok = true;
    auto wait_all = [&](uint64_t* bar, uint32_t parity) { return mbar_wait_warp(bar, parity, abort_flag); };
    int i = 0;
    for (int it = 0; it < n_it; ++it) {
      const uint32_t par = (uint32_t)(it & 1);
      const int st = it & 1, q0 = (i0 + i) * BQ;
      const float4* nlse4 = reinterpret_cast<const float4*>(s_lse + st * 128 + wg * 64);
      const float4* ndlt4 = reinterpret_cast<const float4*>(s_dlt + st * 128 + wg * 64);
      // only then can a query be older than a key of this block, or a key be past the end
      const bool masked = (p.causal && q0 < k0 + BK) || block_off;
      if (!wait_all(&ld_full[st], (uint32_t)((it >> 1) & 1)) || !wait_all(s_full, par)) { ok = false; break; }
      tc_fence_after();
      float pf[64];
      auto probs = [&](auto mask) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t raw[32], pk[16];
          tmem_ld32(s_addr + (uint32_t)(c * 32), raw);
          tmem_ld_wait();
#pragma unroll
          for (int e4 = 0; e4 < 8; ++e4) {
            const float4 nl = nlse4[c * 8 + e4];
            const float nls[4] = {nl.x, nl.y, nl.z, nl.w};
#pragma unroll
            for (int e2 = 0; e2 < 4; e2 += 2) {
              const int e = e4 * 4 + e2, cc = c * 32 + e;
              float x0, x1;
              fma2v(x0, x1, __uint_as_float(raw[e]), __uint_as_float(raw[e + 1]), p.scale_log2, nls[e2], nls[e2 + 1]);
              float p0 = ex2_approx(x0), p1 = ex2_approx(x1);
              if constexpr (decltype(mask)::value) {
                const int qi = q0 + wg * 64 + cc;
                if (key_off || (p.causal && qi < kj)) p0 = 0.f;
                if (key_off || (p.causal && qi + 1 < kj)) p1 = 0.f;
              }
              pf[cc] = p0;
              pf[cc + 1] = p1;
              pk[e >> 1] = pack2<T>(p0, p1);
            }
          }
          tmem_st16(s_addr + (uint32_t)(c * 16), pk);   // over columns of S^T that this thread has read
        }
      };
      if (masked) probs(std::true_type{});
      else probs(std::false_type{});
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_ready);
      // dP^T; its commit also says that the products which read the previous dS^T have completed
      if (!wait_all(dp_full, par)) { ok = false; break; }
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t raw[32], pk[16];
        tmem_ld32(dp_addr + (uint32_t)(c * 32), raw);
        tmem_ld_wait();
#pragma unroll
        for (int e4 = 0; e4 < 8; ++e4) {
          const float4 nd = ndlt4[c * 8 + e4];
          const float nds[4] = {nd.x, nd.y, nd.z, nd.w};
#pragma unroll
          for (int e2 = 0; e2 < 4; e2 += 2) {
            const int e = e4 * 4 + e2, cc = c * 32 + e;
            float t0, t1, d0, d1;
            fma2v(t0, t1, __uint_as_float(raw[e]), __uint_as_float(raw[e + 1]), p.scale, nds[e2], nds[e2 + 1]);
            mul2(d0, d1, pf[cc], pf[cc + 1], t0, t1);
            pk[e >> 1] = pack2<T>(d0, d1);
          }
        }
#pragma unroll
        for (int g8 = 0; g8 < 4; ++g8) {
          const int ch = c * 4 + g8;
          *reinterpret_cast<uint4*>(srow + (size_t)((ch ^ (r & 7)) * 16)) =
              make_uint4(pk[g8 * 4], pk[g8 * 4 + 1], pk[g8 * 4 + 2], pk[g8 * 4 + 3]);
        }
      }
      tc_fence_before();
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(ds_ready);
        mbar_arrive(&ld_empty[st]);
      }
      if (++i == n_i) i = 0;
    }
    if (ok && n_it > 0) ok = wait_all(all_done, 0);
    // ---- dK, dV of this key block
    if (ok) {
      tc_fence_after();
      const bool row_ok = kj < Sk;
      T* dk_row = dk + (int64_t)bt * p.dk_sb + (int64_t)hk * p.dk_sh + (int64_t)(koff + kj) * p.dk_ss + wg * 64;
      T* dv_row = dv + (int64_t)bt * p.dv_sb + (int64_t)hk * p.dv_sh + (int64_t)(koff + kj) * p.dv_ss + wg * 64;
#pragma unroll
      for (int which = 0; which < 2; ++which) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t raw[32];
          if (n_it > 0) {
            tmem_ld32(tmem_base + lane_base + (which ? kColDK : kColDV) + (uint32_t)(wg * 64 + c * 32), raw);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int e = 0; e < 32; ++e) raw[e] = 0u;
          }
          if (row_ok) {
            T* dst = (which ? dk_row : dv_row) + c * 32;
#pragma unroll
            for (int g8 = 0; g8 < 4; ++g8) {
              Vec16<T> v;
#pragma unroll
              for (int e = 0; e < 8; ++e) v.v[e] = ToF<T>::from(__uint_as_float(raw[g8 * 8 + e]));
              st16(dst + g8 * 8, v);
            }
          }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 13) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kBwdTmemCols);
  }
  settle_abort(abort_flag, p.status);
}

bool make_dq_map(CUtensorMap* out, float* ptr, int64_t rows) {
  static EncodeTiledFn enc = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess) {
      (void)cudaGetLastError();
      return (EncodeTiledFn) nullptr;
    }
    return (EncodeTiledFn)p;
  }();
  if (!enc || rows <= 0) return false;
  cuuint64_t dims[2] = {128, (cuuint64_t)rows};
  cuuint64_t strides[1] = {128 * sizeof(float)};
  cuuint32_t box[2] = {32, 128};
  cuuint32_t estr[2] = {1, 1};
  return enc(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, ptr, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// delta[b, h, q] = sum_d O[b, h, q, d] * dO[b, h, q, d], and the row of the fp32 dQ buffer is zeroed on the way.  Sixteen
// lanes per row with 16-byte accesses, 64 consecutive rows of one (batch, head) per block, four rows in flight per lane:
// bound by memory (2 x 256 bytes in, 512 out per row).  32 x 4096 rows: 24 us, against 30 (8-byte loads, a row per warp,
// 64-bit divisions for its place) + 11 for the memset it replaces.
constexpr int kDeltaRows = 64;
template <typename T>
__global__ void __launch_bounds__(256) attn_delta_kernel(const T* __restrict__ o, const T* __restrict__ d_o, float* __restrict__ delta,
                                                         float* __restrict__ dq, int H, int Sq, int row_blocks, int64_t o_sb,
                                                         int64_t o_sh, int64_t o_ss, int64_t g_sb, int64_t g_sh, int64_t g_ss) {
  const int bh = (int)(blockIdx.x / row_blocks);
  const int b = bh / H, h = bh - b * H;
  const int q0 = (int)(blockIdx.x - (unsigned)bh * row_blocks) * kDeltaRows + (threadIdx.x >> 4);
  const int l16 = threadIdx.x & 15;
  const T* po = o + b * o_sb + h * o_sh + l16 * 8;
  const T* pg = d_o + b * g_sb + h * g_sh + l16 * 8;
  Vec16<T> av[4], gv[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int q = q0 + i * 16;
    if (q < Sq) {
      av[i] = ld16(po + q * o_ss);
      gv[i] = ld16(pg + q * g_ss);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int q = q0 + i * 16;
    float s = 0.f;
    if (q < Sq) {
#pragma unroll
      for (int e = 0; e < 8; ++e) s += ToF<T>::to(av[i].v[e]) * ToF<T>::to(gv[i].v[e]);
    }
#pragma unroll
    for (int w = 8; w > 0; w >>= 1) s += __shfl_xor_sync(0xffffffffu, s, w);
    if (q < Sq) {
      const int64_t row = (int64_t)bh * Sq + q;
      if (l16 == 0) delta[row] = s;
      float4* z = reinterpret_cast<float4*>(dq + row * BD);
      z[l16] = make_float4(0.f, 0.f, 0.f, 0.f);
      z[l16 + 16] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
}

template <typename K>
int bwd_setup(K kern) {
  cudaFuncAttributes at;
  cudaError_t e = cudaFuncGetAttributes(&at, kern);
  if (e != cudaSuccess) return (int)e;
  if (at.numRegs < kLaunchRegs) return (int)cudaErrorNotSupported;   // the register split would wait for ever
  return opt_in_smem(kern, kBwdSmem);
}

}  // namespace
}  // namespace b200k

using namespace b200k;

extern "C" int b200_flash_attn_bwd(const b200_attn_t* a, float* dq_accum, void* dk, void* dv, float* delta, const void* q,
                                   const void* k, const void* v, const void* o, const void* d_o, const float* lse,
                                   const int64_t* extra_strides, cudaStream_t stream) {
  // extra_strides: do_sb, do_sh, do_ss, dk_sb, dk_sh, dk_ss, dv_sb, dv_sh, dv_ss (elements)
  if (a->head_dim != BD || (a->dtype != B200_BF16 && a->dtype != B200_F16) || a->B <= 0 || a->H <= 0 || a->Hkv <= 0 ||
      a->H % a->Hkv != 0 || a->Sq <= 0 || a->Sk <= 0)
    return (int)cudaErrorNotSupported;
  auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  const int64_t* x = extra_strides;
  const int64_t strides[] = {a->q_sb, a->q_sh, a->q_ss, a->k_sb, a->k_sh, a->k_ss, a->v_sb, a->v_sh, a->v_ss,
                             a->o_sb, a->o_sh, a->o_ss, x[0], x[1], x[2], x[3], x[4], x[5], x[6], x[7], x[8]};
  for (int64_t s : strides)
    if (s % 8 != 0) return (int)cudaErrorNotSupported;
  if (!al(q) || !al(k) || !al(v) || !al(o) || !al(d_o) || !al(dk) || !al(dv) || !al(dq_accum)) return (int)cudaErrorNotSupported;
  const bool packed = a->cu_seqlens_q != nullptr;
  if (packed && (!a->cu_seqlens_k || a->total_q <= 0 || a->total_k <= 0)) return (int)cudaErrorNotSupported;
  if ((a->B > 1 && !packed && (a->q_sb == 0 || a->k_sb == 0 || a->v_sb == 0 || x[0] == 0)) ||
      (a->H > 1 && (a->q_sh == 0 || x[1] == 0)) || (a->Hkv > 1 && (a->k_sh == 0 || a->v_sh == 0)) || a->q_ss == 0 ||
      a->k_ss == 0 || a->v_ss == 0 || x[2] == 0)
    return (int)cudaErrorNotSupported;
  const int bf16 = a->dtype == B200_BF16;
  CUtensorMap mq, mk, mv, mdo;
  auto nz = [](int64_t s, int64_t fallback) { return s ? s : fallback; };
  if (packed) {
    // one "batch" of total rows: the kernel adds each sequence's first row to its tile coordinates
    if (!make_attn_map(&mq, q, bf16, 1, a->H, a->total_q, (int64_t)a->total_q * a->q_ss, nz(a->q_sh, 8), a->q_ss) ||
        !make_attn_map(&mk, k, bf16, 1, a->Hkv, a->total_k, (int64_t)a->total_k * a->k_ss, nz(a->k_sh, 8), a->k_ss) ||
        !make_attn_map(&mv, v, bf16, 1, a->Hkv, a->total_k, (int64_t)a->total_k * a->v_ss, nz(a->v_sh, 8), a->v_ss) ||
        !make_attn_map(&mdo, d_o, bf16, 1, a->H, a->total_q, (int64_t)a->total_q * x[2], nz(x[1], 8), x[2]))
      return (int)cudaErrorNotSupported;
  } else if (!make_attn_map(&mq, q, bf16, a->B, a->H, a->Sq, nz(a->q_sb, 8), nz(a->q_sh, 8), a->q_ss) ||
             !make_attn_map(&mk, k, bf16, a->B, a->Hkv, a->Sk, nz(a->k_sb, 8), nz(a->k_sh, 8), a->k_ss) ||
             !make_attn_map(&mv, v, bf16, a->B, a->Hkv, a->Sk, nz(a->v_sb, 8), nz(a->v_sh, 8), a->v_ss) ||
             !make_attn_map(&mdo, d_o, bf16, a->B, a->H, a->Sq, nz(x[0], 8), nz(x[1], 8), x[2]))
    return (int)cudaErrorNotSupported;
  // dq_accum as a [B * H * Sq, 128] ([H * total_q, 128] when packed) fp32 matrix; one box = 32 columns of 128 rows
  const long long rows = packed ? (long long)a->H * a->total_q : (long long)a->B * a->H * a->Sq;
  const int dB = packed ? 1 : a->B, dS = packed ? a->total_q : a->Sq;     // the row-dot kernel's view of o and d_o
  CUtensorMap mdq;
  if (!make_dq_map(&mdq, dq_accum, rows)) return (int)cudaErrorNotSupported;
  BwdParams p{};
  p.B = a->B; p.H = a->H; p.Hkv = a->Hkv; p.Sq = a->Sq; p.Sk = a->Sk;
  p.causal = a->causal;
  p.scale = a->scale;
  p.scale_log2 = a->scale * 1.4426950408889634f;
  p.lse = lse;
  p.delta = delta;
  p.dq = dq_accum;
  p.dk_sb = x[3]; p.dk_sh = x[4]; p.dk_ss = x[5];
  p.dv_sb = x[6]; p.dv_sh = x[7]; p.dv_ss = x[8];
  p.kv_blocks = (a->Sk + BK - 1) / BK;
  p.q_blocks = (a->Sq + BQ - 1) / BQ;
  p.status = gemm_status_word_device();
  p.cu_q = a->cu_seqlens_q;
  p.cu_k = a->cu_seqlens_k;
  p.total_q = a->total_q;
  const long long grid = (long long)a->B * a->Hkv * p.kv_blocks;
  if (grid > 2147483647ll || rows / 8 + 1 > 2147483647ll) return (int)cudaErrorNotSupported;
  const int row_blocks = (dS + kDeltaRows - 1) / kDeltaRows;
  const unsigned delta_grid = (unsigned)((long long)dB * a->H * row_blocks);
  if (bf16) {
    static OncePerDevice once;
    if (int e = once([] { return bwd_setup(attn_bwd_kernel<__nv_bfloat16>); })) return e;
    attn_delta_kernel<__nv_bfloat16><<<delta_grid, 256, 0, stream>>>((const __nv_bfloat16*)o, (const __nv_bfloat16*)d_o, delta, dq_accum,
                                                                     a->H, dS, row_blocks, a->o_sb, a->o_sh, a->o_ss, x[0], x[1], x[2]);
    attn_bwd_kernel<__nv_bfloat16><<<(unsigned)grid, kBwdThreads, kBwdSmem, stream>>>(mq, mk, mv, mdo, mdq, (__nv_bfloat16*)dk,
                                                                                     (__nv_bfloat16*)dv, p);
  } else {
    static OncePerDevice once;
    if (int e = once([] { return bwd_setup(attn_bwd_kernel<__half>); })) return e;
    attn_delta_kernel<__half><<<delta_grid, 256, 0, stream>>>((const __half*)o, (const __half*)d_o, delta, dq_accum, a->H, dS, row_blocks,
                                                              a->o_sb, a->o_sh, a->o_ss, x[0], x[1], x[2]);
    attn_bwd_kernel<__half><<<(unsigned)grid, kBwdThreads, kBwdSmem, stream>>>(mq, mk, mv, mdo, mdq, (__half*)dk, (__half*)dv, p);
  }
  note_launch(2);
  return (int)cudaGetLastError();
}
