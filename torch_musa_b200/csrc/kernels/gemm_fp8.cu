// Block-scaled fp8 (e4m3 / e5m2) GEMM on the 5th-generation tensor cores.
//
//   D[M,N] = sum over 128-wide K blocks kb of  sa[m, kb] * sb[n / 128, kb] * (A[m, kb] . B[n, kb])   (* ra[m] * rb[n]) (+ bias)
//
// A [M,K] and B [N,K] are fp8, K contiguous.  Persistent CTAs walk 128 x FN output tiles (FN = 256, or 128 where that
// gives more of them to few rows).  One warp feeds a ring of 128-byte-wide A and B tiles with TMA (128-byte swizzle); one issues
// tcgen05.mma kind::f8f6f4 (M128, K32, four per K block) into one of two TMEM accumulators, a fresh accumulation per K block;
// two warpgroups promote: each takes half of the columns of the finished block product from TMEM, multiplies it by the
// block's two scale factors and adds it to fp32 accumulators in registers (a thread owns one row of its half), while the tensor
// core works on the next block in the other accumulator.  The epilogue applies optional per-row / per-column factors (row-wise
// and tensor-wise scaling are the special case of block factors 1) and the bias, and stores bf16 / fp16 / fp32; the ring fills
// for the next tile meanwhile.
// What bounds it: the promotion.  At FN = 256 an SM spends 1560 clocks on a K block, the epilogues included, of which the tensor
// core is busy for 512 (its counter: 33 %) and shared memory for 768 (48 KB in, 48 KB read); the multiply-adds and TMEM reads of
// the promotion take 512 issue clocks per scheduler, with only two warps there to hide the latency of the reads.  4096 x 14336 x
// 4096: 545 us with one promotion warpgroup, FN = 128, no persistence and row-wise 16-byte stores; 361 now (1330 TFLOP/s; with
// parts left out: products alone 290, promotion alone 306), of which the staged epilogue is worth 20; 4096 x 11008 x 14336 1099
// -> 811 (1595 TFLOP/s).  Four promotion warpgroups were slower (626 us), a TMEM read per 32 columns too (372).
// Every mbarrier wait is bounded.
//
// Parity: the reference forwards _scaled_mm to its vendor library (reference torch_musa/csrc/aten/ops/Matmul.cpp:670-681).
#include "attention_common.cuh"   // packed fp32 arithmetic, register split

#include <cuda_fp8.h>

#include <algorithm>

namespace b200k {
namespace {
using namespace gemmdev;
using attndev::fma2v;
using attndev::regs_dec;
using attndev::regs_inc;

constexpr int FM = 128, FK = 128;                // FK fp8 elements = 128 bytes = one swizzle row
constexpr int kF8Threads = 384;                  // two promotion warpgroups; one with the TMA warp and the MMA warp
constexpr int kPromoteRegs = 208, kOtherRegs = 88;
constexpr int kLaunchRegs = (2 * kPromoteRegs + kOtherRegs + 2) / 3;   // what the launch has to bring for that split
constexpr int kF8Out = 8 * 32 * 128;             // staging of the output: 32 rows x 128 bytes per promotion warp

template <int FN>
struct F8Cfg {
  static constexpr int kATile = FM * FK, kBTile = FN * FK, kStage = kATile + kBTile;
  static constexpr int kStages = FN == 256 ? 4 : 6;                     // 192 KB
  static constexpr int kSmem = kStages * kStage + kF8Out + 1024 + 256;
  static constexpr uint32_t kTmemCols = 2 * FN;                         // two accumulators
};

struct F8Params {
  int m, n, k;
  int64_t ldd;
  const float* sa; int64_t sa_sm, sa_sk;         // block scales of A: sa[m * sa_sm + kb * sa_sk]   (NULL: 1)
  const float* sb; int64_t sb_sn, sb_sk;         // block scales of B: sb[(n / 128) * sb_sn + kb * sb_sk] (NULL: 1)
  const float* ra; int64_t ra_s;                 // final per-row factor ra[m * ra_s] (NULL: 1; ra_s 0: one scalar)
  const float* rb; int64_t rb_s;                 // final per-column factor rb[n * rb_s]
  const void* bias; int bias_f32;
  uint32_t idesc;
  int* status;
  int tiles_m, tiles_n, group_m;
};

__device__ __forceinline__ void umma_f8(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

template <typename OutT, int FN>
__global__ void __launch_bounds__(kF8Threads, 1)
gemm_fp8_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                OutT* __restrict__ d, const F8Params p) {
  using C = F8Cfg<FN>;
  constexpr int HN = FN / 2;                  // columns of one promotion warpgroup
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::kStages * C::kStage + kF8Out);
  uint64_t* full_bar = bars;                  // [stages]
  uint64_t* empty_bar = bars + C::kStages;    // [stages]
  uint64_t* tfull_bar = bars + 2 * C::kStages;// [2]
  uint64_t* tempty_bar = tfull_bar + 2;       // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int k_blocks = (p.k + FK - 1) / FK;
  const int total_tiles = p.tiles_m * p.tiles_n;

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < C::kStages; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int s = 0; s < 2; ++s) { mbar_init(&tfull_bar[s], 1); mbar_init(&tempty_bar[s], 8); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    prefetch_tmap(&tmap_a);
    prefetch_tmap(&tmap_b);
  }
  if (warp == 9) {
    tmem_alloc(tmem_slot, C::kTmemCols);
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
        int stage = 0;
        uint32_t phase = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
          int mt, nt;
          decode_tile(tile, p.tiles_m, p.tiles_n, p.group_m, mt, nt);
          for (int kb = 0; kb < k_blocks; ++kb) {
            if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag)) { ok = false; break; }
            mbar_expect_tx(&full_bar[stage], C::kStage);
            uint8_t* sa = smem + stage * C::kStage;
            tma_load_3d(sa, &tmap_a, &full_bar[stage], kb * FK, mt * FM, 0);
#pragma unroll
            for (int q = 0; q < FN / 128; ++q)
              tma_load_3d(sa + C::kATile + q * 128 * FK, &tmap_b, &full_bar[stage], kb * FK, nt * FN + q * 128, 0);
            if (++stage == C::kStages) { stage = 0; phase ^= 1; }
          }
        }
      }
      __syncwarp();
    } else if (warp == 9) {
      // ------------------------------------------------------------ MMA issuer (the whole warp waits, one lane issues)
      const bool issuer = elect_one();
      int stage = 0;
      uint32_t phase = 0;
      uint32_t g = 0;                        // K blocks issued so far: accumulator g & 1
      bool ok = true;
      for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
        for (int kb = 0; kb < k_blocks; ++kb, ++g) {
          const uint32_t slot = g & 1;
          // the promotion warps must have drained this accumulator (two blocks ago)
          if (!mbar_wait_warp(&tempty_bar[slot], ((g >> 1) & 1) ^ 1, abort_flag)) { ok = false; break; }
          if (!mbar_wait_warp(&full_bar[stage], phase, abort_flag)) { ok = false; break; }
          tc_fence_after();
          if (issuer) {
            const uint32_t sa = smem_u32(smem + stage * C::kStage), sb = sa + C::kATile;
            const uint32_t tmem_d = tmem_base + slot * FN;
#pragma unroll
            for (int kk = 0; kk < FK / 32; ++kk)
              umma_f8(tmem_d, make_desc(sa + kk * 32, 16, 1024), make_desc(sb + kk * 32, 16, 1024), p.idesc, kk != 0 ? 1u : 0u);
            umma_commit(&empty_bar[stage]);
            umma_commit(&tfull_bar[slot]);
          }
          if (++stage == C::kStages) { stage = 0; phase ^= 1; }
        }
      }
      __syncwarp();
    }
  } else {
    regs_inc<kPromoteRegs>();
    // ------------------------------------------------------------ promotion + epilogue: rows by lane, half of the columns
    const int q = warp & 3, half = warp >> 2;
    uint8_t* stage_out = smem + C::kStages * C::kStage + warp * (32 * 128);
    const bool vec_ok = (p.ldd % (16 / (int)sizeof(OutT)) == 0) && ((reinterpret_cast<uintptr_t>(d) & 15) == 0);
    uint32_t g = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
      int mt, nt;
      decode_tile(tile, p.tiles_m, p.tiles_n, p.group_m, mt, nt);
      const int row = mt * FM + q * 32 + lane, n0 = nt * FN + half * HN;
      const float* sa_row = p.sa ? p.sa + (int64_t)min(row, p.m - 1) * p.sa_sm : nullptr;
      const float* sb_blk = p.sb ? p.sb + (int64_t)(min(n0, p.n - 1) / 128) * p.sb_sn : nullptr;
      auto factor = [&](int kb) {
        if (kb >= k_blocks) return 0.f;
        return (sa_row ? __ldg(sa_row + (int64_t)kb * p.sa_sk) : 1.f) * (sb_blk ? __ldg(sb_blk + (int64_t)kb * p.sb_sk) : 1.f);
      };
      float acc[HN];
#pragma unroll
      for (int c = 0; c < HN; ++c) acc[c] = 0.f;
      float f0 = factor(0), f1 = factor(1);     // the scales come two blocks ahead
      for (int kb = 0; kb < k_blocks; ++kb, ++g) {
        const uint32_t slot = g & 1;
        const float f = f0;
        f0 = f1;
        f1 = factor(kb + 2);
        if (!mbar_wait_warp(&tfull_bar[slot], (g >> 1) & 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + slot * FN + (uint32_t)(half * HN);
#pragma unroll
        for (int c = 0; c < HN / 64; ++c) {
          uint32_t raw[2][32];
          tmem_ld32(taddr + (uint32_t)(c * 64), raw[0]);
          tmem_ld32(taddr + (uint32_t)(c * 64 + 32), raw[1]);
          tmem_ld_wait();
          if (c + 1 == HN / 64) {
            tc_fence_before();               // everything has been read: the next product may go there
            __syncwarp();
            if (lane == 0) mbar_arrive(&tempty_bar[slot]);
          }
#pragma unroll
          for (int e = 0; e < 64; e += 2)
            fma2v(acc[c * 64 + e], acc[c * 64 + e + 1], __uint_as_float(raw[e >> 5][e & 31]), __uint_as_float(raw[e >> 5][(e & 31) + 1]),
                  f, acc[c * 64 + e], acc[c * 64 + e + 1]);
        }
      }
      if (!ok) break;
      // epilogue: 128 bytes of every row at a time through the warp's own staging (16-byte chunks swizzled over the banks), so
      // that a store instruction writes 4 rows x 128 bytes and not 32 x 16
      const float fr = p.ra && row < p.m ? p.ra[(int64_t)row * p.ra_s] : 1.f;
      constexpr int CW = 128 / (int)sizeof(OutT), CE = 16 / (int)sizeof(OutT);     // columns per step, per 16 bytes
#pragma unroll
      for (int c = 0; c < HN / CW; ++c) {
        const int col0 = n0 + c * CW;
        if (col0 >= p.n) break;
#pragma unroll
        for (int ch = 0; ch < 8; ++ch) {
          Vec16<OutT> o;
#pragma unroll
          for (int e = 0; e < CE; ++e) {
            const int col = col0 + ch * CE + e;
            float x = acc[c * CW + ch * CE + e] * fr;
            if (p.rb && col < p.n) x *= p.rb[(int64_t)col * p.rb_s];
            if (p.bias && col < p.n)
              x += p.bias_f32 ? reinterpret_cast<const float*>(p.bias)[col] : ToF<OutT>::to(reinterpret_cast<const OutT*>(p.bias)[col]);
            o.v[e] = ToF<OutT>::from(x);
          }
          *reinterpret_cast<Vec16<OutT>*>(stage_out + lane * 128 + ((ch ^ (lane & 7)) * 16)) = o;
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int r = i * 4 + (lane >> 3), ch = lane & 7, m = mt * FM + q * 32 + r, col = col0 + ch * CE;
          const Vec16<OutT> o = *reinterpret_cast<const Vec16<OutT>*>(stage_out + r * 128 + ((ch ^ (r & 7)) * 16));
          if (m < p.m) {
            OutT* dst = d + (int64_t)m * p.ldd + col;
            if (vec_ok && col + CE <= p.n) st16(dst, o);
            else {
#pragma unroll
              for (int e = 0; e < CE; ++e)
                if (col + e < p.n) dst[e] = o.v[e];
            }
          }
        }
        __syncwarp();
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    tc_fence_after();
    tmem_dealloc(tmem_base, C::kTmemCols);
  }
  settle_abort(abort_flag, p.status);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

bool make_u8_map(CUtensorMap* out, const void* ptr, uint64_t k, uint64_t rows, uint64_t ld_bytes) {
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
  if (!enc) return false;
  cuuint64_t dims[3] = {k, rows, 1};
  cuuint64_t strides[2] = {ld_bytes, ld_bytes * rows};
  cuuint32_t box[3] = {FK, 128, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  return enc(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(ptr), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <typename OutT, int FN>
int launch_fp8(const b200_fp8_gemm_t* g, void* d, const void* a, const void* b, cudaStream_t stream) {
  CUtensorMap ma, mb;
  if (!make_u8_map(&ma, a, (uint64_t)g->k, (uint64_t)g->m, (uint64_t)g->lda) ||
      !make_u8_map(&mb, b, (uint64_t)g->k, (uint64_t)g->n, (uint64_t)g->ldb))
    return (int)cudaErrorNotSupported;
  F8Params p{};
  p.m = g->m; p.n = g->n; p.k = g->k;
  p.ldd = g->ldd;
  p.sa = g->block_scale_a; p.sa_sm = g->bsa_stride_m; p.sa_sk = g->bsa_stride_kb;
  p.sb = g->block_scale_b; p.sb_sn = g->bsb_stride_nb; p.sb_sk = g->bsb_stride_kb;
  p.ra = g->row_scale; p.ra_s = g->row_scale_stride;
  p.rb = g->col_scale; p.rb_s = g->col_scale_stride;
  p.bias = g->bias; p.bias_f32 = g->bias_dtype == B200_F32;
  // kind::f8f6f4 instruction descriptor: fp32 accumulate, operand formats (0 = e4m3, 1 = e5m2), K-major, N>>3, M>>4
  const uint32_t fa = g->a_e5m2 ? 1u : 0u, fb = g->b_e5m2 ? 1u : 0u;
  p.idesc = (1u << 4) | (fa << 7) | (fb << 10) | ((uint32_t)(FN >> 3) << 17) | ((uint32_t)(FM >> 4) << 24);
  p.status = gemm_status_word_device();
  p.tiles_m = (g->m + FM - 1) / FM;
  p.tiles_n = (g->n + FN - 1) / FN;
  p.group_m = gemm_group_m(FM, g->m, g->k / 2);     // one byte per element
  using C = F8Cfg<FN>;
  auto kern = gemm_fp8_kernel<OutT, FN>;
  static OncePerDevice once;
  const int setup = once([&] {
    cudaFuncAttributes at;
    cudaError_t e = cudaFuncGetAttributes(&at, kern);
    if (e != cudaSuccess) return (int)e;
    if (at.numRegs < kLaunchRegs) return (int)cudaErrorNotSupported;   // the register split would wait for ever
    return opt_in_smem(kern, C::kSmem);
  });
  if (setup != 0) return setup;
  const int grid = std::min(p.tiles_m * p.tiles_n, gemm_sm_count());
  kern<<<grid, kF8Threads, C::kSmem, stream>>>(ma, mb, (OutT*)d, p);
  B200K_LAUNCH_RET();
}

// Which tile: waves over the SMs times the time of a tile.  A 128 x 256 tile takes 1.6 to 1.7 times as long as a 128 x 128 one
// (4096 x 14336 x 4096: 356 us in 13 waves, the narrow tile 418 in 25; 3072 x 11008 x 4096: 196 in 7, 238 in 14), so it wins as
// soon as the SMs have enough tiles of it: 1 wave against 2 21 / 24 us (640 x 4096 x 2048), 3 against 5 86 / 88 (2560 x 4096 x 4096), 4
// against 7 112 / 119; 2 against 3 goes to the narrow one, 59 / 55 (1536 x 4096 x 4096), and 1 against 1 30 / 20.
template <typename OutT>
int launch_fp8_any(const b200_fp8_gemm_t* g, void* d, const void* a, const void* b, cudaStream_t stream) {
  const long long sms = gemm_sm_count(), tm = (g->m + FM - 1) / FM;
  const long long wide = (tm * ((g->n + 255) / 256) + sms - 1) / sms, narrow = (tm * ((g->n + 127) / 128) + sms - 1) / sms;
  if (wide * 16 <= narrow * 10) return launch_fp8<OutT, 256>(g, d, a, b, stream);
  return launch_fp8<OutT, 128>(g, d, a, b, stream);
}

// ---- 1 x 128 block quantisation of activations
// One CTA per row, 16 bytes per lane (16 lanes per block of 16-bit elements), four loads in flight per lane.  Bound by memory.
// 4096 x 4096 bf16: 24.7 us with a warp per block, 8-byte loads and a 64-bit division per block; 18.2 now.
template <typename T>
__global__ void __launch_bounds__(256) quant_rows_kernel(const T* __restrict__ x, uint8_t* __restrict__ q, float* __restrict__ scales,
                                                         int k, int64_t ldx, int e5m2) {
  constexpr int V = Vec16<T>::N, LPB = 128 / V, U = 4;      // elements per load, lanes per block, loads in flight
  const int64_t row = blockIdx.x;
  const T* src = x + row * ldx;
  uint8_t* dst = q + row * (int64_t)k;
  float* sc = scales + row * (k / 128);
  const int nvec = k / V;                                    // a multiple of LPB: lanes of a block are valid together
  const float fmax = e5m2 ? 57344.f : 448.f;
  for (int i0 = threadIdx.x; i0 - (int)threadIdx.x < nvec; i0 += 256 * U) {
    Vec16<T> v[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i0 + u * 256 < nvec) v[u] = ld16_stream(src + (int64_t)(i0 + u * 256) * V);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * 256;
      float amax = 0.f;
      if (i < nvec) {
#pragma unroll
        for (int e = 0; e < V; ++e) amax = fmaxf(amax, fabsf(ToF<T>::to(v[u].v[e])));
      }
#pragma unroll
      for (int w = LPB / 2; w > 0; w >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, w));
      if (i < nvec) {
        const float scale = amax > 0.f ? amax / fmax : 1.f;
        const float inv = 1.f / scale;
        uint32_t packed[V / 4];
#pragma unroll
        for (int w = 0; w < V / 4; ++w) {
          packed[w] = 0;
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float y = fminf(fmaxf(ToF<T>::to(v[u].v[w * 4 + e]) * inv, -fmax), fmax);
            packed[w] |= (uint32_t)__nv_cvt_float_to_fp8(y, __NV_SATFINITE, e5m2 ? __NV_E5M2 : __NV_E4M3) << (8 * e);
          }
        }
        if constexpr (V == 8) *reinterpret_cast<uint2*>(dst + (int64_t)i * V) = make_uint2(packed[0], packed[1]);
        else *reinterpret_cast<uint32_t*>(dst + (int64_t)i * V) = packed[0];
        if ((threadIdx.x & (LPB - 1)) == 0) sc[i / LPB] = scale;
      }
    }
  }
}

// any alignment: one warp per 128-element block
template <typename T>
__global__ void quant_1x128_kernel(const T* __restrict__ x, uint8_t* __restrict__ q, float* __restrict__ scales,
                                   int64_t rows, int k, int64_t ldx, int e5m2) {
  const int kblocks = k / 128;
  const int64_t nblk = rows * kblocks;
  const int lane = threadIdx.x & 31;
  const float fmax = e5m2 ? 57344.f : 448.f;
  for (int64_t b = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); b < nblk; b += (int64_t)gridDim.x * (blockDim.x >> 5)) {
    const int64_t r = b / kblocks;
    const int kb = (int)(b - r * kblocks);
    const T* src = x + r * ldx + kb * 128 + lane * 4;
    float v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = ToF<T>::to(src[i]);
    float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
    amax = warp_max(amax);
    const float scale = amax > 0.f ? amax / fmax : 1.f;
    const float inv = 1.f / scale;
    uint32_t packed = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float y = fminf(fmaxf(v[i] * inv, -fmax), fmax);
      const __nv_fp8_storage_t f8 = __nv_cvt_float_to_fp8(y, __NV_SATFINITE, e5m2 ? __NV_E5M2 : __NV_E4M3);
      packed |= (uint32_t)f8 << (8 * i);
    }
    *reinterpret_cast<uint32_t*>(q + r * (int64_t)k + kb * 128 + lane * 4) = packed;
    if (lane == 0) scales[r * kblocks + kb] = scale;
  }
}

}  // namespace
}  // namespace b200k

using namespace b200k;

extern "C" {

int b200_gemm_fp8(const b200_fp8_gemm_t* g, void* d, const void* a, const void* b, cudaStream_t stream) {
  if (g->m <= 0 || g->n <= 0) return 0;
  auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  if (g->k <= 0 || g->k % 16 != 0 || g->lda % 16 != 0 || g->ldb % 16 != 0 || !al(a) || !al(b)) return (int)cudaErrorNotSupported;
  if ((g->block_scale_a || g->block_scale_b) && g->k % 128 != 0) return (int)cudaErrorNotSupported;
  switch (g->out_dtype) {
    case B200_BF16: return launch_fp8_any<__nv_bfloat16>(g, d, a, b, stream);
    case B200_F16: return launch_fp8_any<__half>(g, d, a, b, stream);
    case B200_F32: return launch_fp8_any<float>(g, d, a, b, stream);
    default: return (int)cudaErrorNotSupported;
  }
}

int b200_quantize_fp8_1x128(int dtype, const void* x, void* q, float* scales, int64_t rows, int k, int64_t ldx, int e5m2,
                            cudaStream_t stream) {
  if (rows == 0 || k == 0) return 0;
  if (k % 128 != 0 || ldx % 4 != 0 || (reinterpret_cast<uintptr_t>(q) & 3)) return (int)cudaErrorNotSupported;
  const int64_t nblk = rows * (k / 128);
  const int grid = (int)std::min<int64_t>((nblk + 7) / 8, (int64_t)kSMs * 16);
  // A CTA per row pays with enough rows to fill the SMs, and with rows wide enough that every thread has two vectors: with few
  // rows a warp per block spreads them better.  16 x 14336 bf16: 4.0 us a row per CTA, 2.1 a warp per block; 300 x 14336: 6.6 and
  // 7.9; 600 x 2048: 4.1 and 3.4; fp32 300 x 14336: 9.1 and 7.9, 600 x 14336: 12.0 and 13.8.
  const bool wide = dtype == B200_F32 ? rows >= 512 && k >= 2048 : rows >= 256 && k >= 4096;
  if (wide && (reinterpret_cast<uintptr_t>(x) & 15) == 0 && ldx * (dtype == B200_F32 ? 4 : 2) % 16 == 0 &&
      (reinterpret_cast<uintptr_t>(q) & 7) == 0 && rows <= 2147483647ll) {
    B200K_DISPATCH_FLOAT(dtype, T, (quant_rows_kernel<T><<<(unsigned)rows, 256, 0, stream>>>((const T*)x, (uint8_t*)q, scales, k, ldx, e5m2)));
    B200K_LAUNCH_RET();
  }
  B200K_DISPATCH_FLOAT(dtype, T, (quant_1x128_kernel<T><<<grid, 256, 0, stream>>>((const T*)x, (uint8_t*)q, scales, rows, k, ldx, e5m2)));
  B200K_LAUNCH_RET();
}

}  // extern "C"
