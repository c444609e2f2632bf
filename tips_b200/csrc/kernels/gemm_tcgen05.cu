// bf16 GEMM on the 5th-generation tensor cores: C[M,N] = act(A[M,K] * B[N,K]^T + bias).
//
// Both operands are K-major (row-major A and row-major B = "TN"), which is the
// layout of a linear layer's forward pass (activations [M,K], weight [N,K]).
// Pipeline inside one CTA (192 threads):
//   warp 0      TMA producer: cp.async.bulk.tensor.2d (no multicast) brings a
//               128 x 64 tile of A and a BN x 64 tile of B per stage into
//               128-byte-swizzled shared memory, signalling an mbarrier
//   warp 1      MMA issuer: one elected thread issues tcgen05.mma (kind::f16,
//               M=128, N=BN, K=16) four times per stage with shared-memory
//               descriptors, accumulating in TMEM; tcgen05.commit releases the
//               stage back to the producer and finally signals the epilogue
//   warps 2-5   epilogue: tcgen05.ld the fp32 accumulator rows out of TMEM, add
//               the bias, apply the activation, convert to bf16 and store
// Every mbarrier wait is bounded; on a timeout the kernel sets an error word,
// frees its TMEM and returns.
//
// The reference contains no GEMM (its only math is an elementwise loop,
// tips/core/common/vec.h:194-216); this kernel serves the CTR model's MLP and
// the BERT-shaped encoder's linear layers.
#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <map>
#include <mutex>
#include <tuple>

#include "kernels/common.cuh"
#include "kernels/tcgen05.cuh"
#include "kernels/tips_kernels.h"

namespace tipsk {
namespace {

struct GemmParams {
  __nv_bfloat16* c;
  __nv_bfloat16* pre;          // optional: pre-activation output
  const __nv_bfloat16* bias;   // optional, [N]
  int32_t* error;              // device error word
  int m, n, k;
  int ldc;
  int act;                     // 0 none, 1 relu, 2 gelu
  int tma_store;               // 1: the output goes through shared memory and the TMA store unit
  int accumulate;              // 1 (TMA store path only): add to what C holds, with a reduce-add store
  int bias_vec;                // 1: bias is 16-byte aligned, so eight values can be read with one load
  float* partial;              // pair kernel, K split over several tiles: [splits][m][n] fp32 partial products
  int splits;
};

// Eight consecutive bias values as floats (zeros without a bias): one 16-byte load when the bias is 16-byte aligned
// and the eight columns exist, scalar loads at a ragged edge.
__device__ __forceinline__ void LoadBias8(const GemmParams& p, int col, float (&bv)[8]) {
#pragma unroll
  for (int j = 0; j < 8; ++j) bv[j] = 0.f;
  if (p.bias == nullptr) return;
  if (p.bias_vec && col + 8 <= p.n) {
    const uint4 q = *reinterpret_cast<const uint4*>(p.bias + col);
    const __nv_bfloat16* b = reinterpret_cast<const __nv_bfloat16*>(&q);
#pragma unroll
    for (int j = 0; j < 8; ++j) bv[j] = __bfloat162float(b[j]);
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (col + j < p.n) bv[j] = __bfloat162float(p.bias[col + j]);
  }
}

// The activation of a value that is rounded to bf16 next, and of a pair of them.
__device__ __forceinline__ float2 GemmAct2(float x, float y, int act) {
  if (act == 1) return make_float2(fmaxf(x, 0.f), fmaxf(y, 0.f));
  if (act == 2) return SplitF2(Gelu2(MakeF2(x, y)));
  return make_float2(x, y);
}
__device__ __forceinline__ float GemmAct(float x, int act) { return GemmAct2(x, x, act).x; }

// Hands a staged 64-column box to the TMA store unit: a plain store, or a bf16 reduce-add into global memory.
__device__ __forceinline__ void TmaStoreOrAdd2D(const CUtensorMap* tmap, int x, int y, const void* smem_src, int add) {
  if (add) {
    asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%1, %2}], [%3];" ::"l"(
                     reinterpret_cast<uint64_t>(tmap)),
                 "r"(x), "r"(y), "r"(SmemAddr(smem_src))
                 : "memory");
  } else {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(
                     reinterpret_cast<uint64_t>(tmap)),
                 "r"(x), "r"(y), "r"(SmemAddr(smem_src))
                 : "memory");
  }
}

template <int BN>
struct GemmCfg {
  // Up to 128 columns: three stages (<= 97 KB) so that two CTAs fit on an SM and one CTA's epilogue
  // overlaps the other's main loop; 256 columns: one CTA per SM with four stages.
  static constexpr int kStages     = BN >= 256 ? 4 : 3;
  static constexpr int kABytes     = kBM * kBK * 2;
  static constexpr int kBBytes     = BN * kBK * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kTmemCols   = BN < 32 ? 32 : BN;
  static constexpr int kSmemBytes  = kStages * kStageBytes + 1024 /*alignment slack*/ + 256 /*barriers*/;
};

// kBMn: B is given as [K, N] row-major (the contraction runs over its rows), loaded as BN/64 boxes of
// [64 x 64] and read by the MMA as an MN-major operand; used for dx = dy * W without transposing W.
template <int BN, bool kBMn = false>
__global__ void __launch_bounds__(kGemmThreads, 1)
GemmTnKernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
             const __grid_constant__ CUtensorMap tmap_c, const __grid_constant__ CUtensorMap tmap_pre, GemmParams p) {
  using Cfg = GemmCfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar  = reinterpret_cast<uint64_t*>(smem + Cfg::kStages * Cfg::kStageBytes);
  uint64_t* empty_bar = full_bar + Cfg::kStages;
  uint64_t* tmem_full = empty_bar + Cfg::kStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_full + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int m0   = blockIdx.y * kBM;
  const int n0   = blockIdx.x * BN;
  const int num_k = (p.k + kBK - 1) / kBK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::kStages; ++s) {
      MbarInit(&full_bar[s], 1);
      MbarInit(&empty_bar[s], 1);
    }
    MbarInit(tmem_full, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(SmemAddr(tmem_slot)),
                 "r"(static_cast<uint32_t>(Cfg::kTmemCols))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  TcFenceBefore();
  __syncthreads();
  TcFenceAfter();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(tmem_slot);

  if (warp == 0) {
    if (ElectOne()) {
      for (int kt = 0; kt < num_k; ++kt) {
        const int s = kt % Cfg::kStages;
        const uint32_t parity = ((kt / Cfg::kStages) & 1) ^ 1;
        if (!MbarWait(&empty_bar[s], parity)) {
          atomicExch(p.error, 1);
          break;
        }
        uint8_t* a_dst = smem + s * Cfg::kStageBytes;
        uint8_t* b_dst = a_dst + Cfg::kABytes;
        MbarExpectTx(&full_bar[s], Cfg::kStageBytes);
        TmaLoad2D(a_dst, &tmap_a, kt * kBK, m0, &full_bar[s]);
        if (kBMn) {
#pragma unroll
          for (int j = 0; j < BN / 64; ++j) TmaLoad2D(b_dst + j * 8192, &tmap_b, n0 + j * 64, kt * kBK, &full_bar[s]);
        } else {
          TmaLoad2D(b_dst, &tmap_b, kt * kBK, n0, &full_bar[s]);
        }
      }
    }
  } else if (warp == 1) {
    {  // the whole warp walks the loop, one lane issues
      constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (kBMn ? (1u << 16) : 0u) |
                                 (static_cast<uint32_t>(BN >> 3) << 17) | (static_cast<uint32_t>(kBM >> 4) << 24);
      bool ok = true;
      for (int kt = 0; kt < num_k && ok; ++kt) {
        const int s = kt % Cfg::kStages;
        const uint32_t parity = (kt / Cfg::kStages) & 1;
        if (!MbarWaitWarp(&full_bar[s], parity)) {
          if (lane == 0) atomicExch(p.error, 2);
          ok = false;
          break;
        }
        TcFenceAfter();
        const uint32_t a_addr = SmemAddr(smem + s * Cfg::kStageBytes);
        const uint32_t b_addr = a_addr + Cfg::kABytes;
        const uint64_t adesc  = SmemDescSw128(a_addr);
        const uint64_t bdesc  = kBMn ? SmemDescMnSw128(b_addr, 8192) : SmemDescSw128(b_addr);
        if (ElectOne()) {
#pragma unroll
          for (int k = 0; k < kBK / 16; ++k) {
            // advancing 16 elements (32 bytes) along K inside the swizzle row = +2 in the address field;
            // for the MN-major B sixteen K rows = 2048 bytes = +128
            UmmaBf16(tmem_base, adesc + 2 * k, bdesc + (kBMn ? 128 : 2) * k, idesc, (kt > 0 || k > 0) ? 1u : 0u);
          }
          UmmaCommit(&empty_bar[s]);
        }
      }
      if (ElectOne()) UmmaCommit(tmem_full);  // arrives when every MMA issued so far has completed
    }
  } else {
    const int q = warp & 3;  // TMEM lane quarter this warp may access
    const bool ok = MbarWait(tmem_full, 0);
    if (!ok && lane == 0) atomicExch(p.error, 3);
    TcFenceAfter();
    const int row = m0 + q * 32 + lane;
    if (p.tma_store) {
      if (ok) {
      // Coalesced path: convert in registers, stage the tile in shared memory in the 128-byte-swizzled
      // layout of the output tensor map (the pipeline stages are free once every MMA has completed),
      // then one thread hands 64-column boxes to the TMA store unit.  Rows / columns beyond M / N are
      // clipped by the TMA unit.
      const int r = q * 32 + lane;  // row inside the tile
#pragma unroll 1
      for (int c = 0; c < BN / 32; ++c) {
        uint32_t acc[32];
        TmemLoad32(tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(c * 32), acc);
        const int col0 = n0 + c * 32;
        uint8_t* box   = smem + (c >> 1) * (kBM * 128);
        uint8_t* pbox  = box + (BN / 64) * (kBM * 128);  // the second output's boxes follow
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          alignas(16) __nv_bfloat16 o[8];
          alignas(16) __nv_bfloat16 pr[8];
          float bv[8];
          LoadBias8(p, col0 + g * 8, bv);
#pragma unroll
          for (int j = 0; j < 8; j += 2) {
            const float x = __uint_as_float(acc[g * 8 + j]) + bv[j], y = __uint_as_float(acc[g * 8 + j + 1]) + bv[j + 1];
            const float2 z = GemmAct2(x, y, p.act);
            *reinterpret_cast<__nv_bfloat162*>(&pr[j]) = __floats2bfloat162_rn(x, y);
            *reinterpret_cast<__nv_bfloat162*>(&o[j])  = __floats2bfloat162_rn(z.x, z.y);
          }
          const int off = r * 128 + ((((c & 1) * 4 + g) ^ (r & 7)) << 4);  // 16-byte chunk inside the swizzled row
          *reinterpret_cast<uint4*>(box + off) = *reinterpret_cast<uint4*>(o);
          if (p.pre) *reinterpret_cast<uint4*>(pbox + off) = *reinterpret_cast<uint4*>(pr);
        }
      }
      }
      // every epilogue warp reaches this barrier, whether or not its wait succeeded
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("bar.sync 1, 128;" ::: "memory");  // the four epilogue warps
      if (ok && warp == 2 && lane == 0) {
#pragma unroll 1
        for (int b = 0; b < BN / 64; ++b) {
          if (n0 + b * 64 < p.n) {
            TmaStoreOrAdd2D(&tmap_c, n0 + b * 64, m0, smem + b * (kBM * 128), p.accumulate);
            if (p.pre) TmaStoreOrAdd2D(&tmap_pre, n0 + b * 64, m0, smem + (BN / 64 + b) * (kBM * 128), 0);
          }
        }
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
      }
    } else if (ok) {
#pragma unroll 1
      for (int c = 0; c < BN / 32 + (BN % 32 ? 1 : 0); ++c) {
        uint32_t r[32];
        if (BN >= 32 || c == 0) {
          TmemLoad32(tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(c * 32), r);
        }
        const int col0 = n0 + c * 32;
        if (row < p.m && col0 < p.n) {
          float v[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            v[j] = __uint_as_float(r[j]);
            if (p.bias && col0 + j < p.n) v[j] += __bfloat162float(p.bias[col0 + j]);
          }
          __nv_bfloat16* crow = p.c + static_cast<int64_t>(row) * p.ldc + col0;
          __nv_bfloat16* prow = p.pre ? p.pre + static_cast<int64_t>(row) * p.ldc + col0 : nullptr;
          const bool vec_ok = (p.ldc % 8 == 0) && (col0 + 32 <= p.n) && (BN >= 32);
          if (vec_ok) {
#pragma unroll
            for (int g = 0; g < 4; ++g) {
              alignas(16) __nv_bfloat16 o[8];
              if (prow) {
                alignas(16) __nv_bfloat16 pr[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) pr[j] = __float2bfloat16_rn(v[g * 8 + j]);
                *reinterpret_cast<uint4*>(prow + g * 8) = *reinterpret_cast<uint4*>(pr);
              }
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                float x = v[g * 8 + j];
                o[j] = __float2bfloat16_rn(GemmAct(x, p.act));
              }
              *reinterpret_cast<uint4*>(crow + g * 8) = *reinterpret_cast<uint4*>(o);
            }
          } else {
            for (int j = 0; j < 32 && col0 + j < p.n && j < BN; ++j) {
              float x = v[j];
              if (prow) prow[j] = __float2bfloat16_rn(x);
              crow[j] = __float2bfloat16_rn(GemmAct(x, p.act));
            }
          }
        }
      }
    }
  }
  TcFenceBefore();
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(static_cast<uint32_t>(Cfg::kTmemCols))
                 : "memory");
  }
}

// ---------------------------------------------------------------- persistent variant
// One CTA per SM walks over the output tiles (tile = blockIdx.x + i * gridDim.x, N fastest).  The
// accumulator is double-buffered in TMEM, so the epilogue of tile i (TMEM -> registers -> swizzled
// shared memory -> TMA store) overlaps the TMA loads and MMAs of tile i+1.  Used when there are more
// tiles than SMs and the output qualifies for the TMA store path.
template <int BN>
struct PersistCfg {
  static constexpr int kStages     = 5;
  static constexpr int kABytes     = kBM * kBK * 2;
  static constexpr int kBBytes     = BN * kBK * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kStagingBytes = kBM * BN * 2;
  static constexpr int kTmemCols   = 2 * BN;  // two accumulators
  static constexpr int kSmemBytes  = kStages * kStageBytes + kStagingBytes + 1024 + 256;
};

template <int BN, bool kBMn = false>
__global__ void __launch_bounds__(kGemmThreads, 1)
GemmTnPersistentKernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                       const __grid_constant__ CUtensorMap tmap_c, GemmParams p) {
  using Cfg = PersistCfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem    = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* staging = smem + Cfg::kStages * Cfg::kStageBytes;
  uint64_t* full_bar   = reinterpret_cast<uint64_t*>(staging + Cfg::kStagingBytes);
  uint64_t* empty_bar  = full_bar + Cfg::kStages;
  uint64_t* tmem_full  = empty_bar + Cfg::kStages;  // [2]
  uint64_t* tmem_empty = tmem_full + 2;             // [2]
  uint32_t* tmem_slot  = reinterpret_cast<uint32_t*>(tmem_empty + 2);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int num_k   = (p.k + kBK - 1) / kBK;
  const int tiles_n = (p.n + BN - 1) / BN;
  const int tiles_m = (p.m + kBM - 1) / kBM;
  const int num_tiles = tiles_m * tiles_n;

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::kStages; ++s) {
      MbarInit(&full_bar[s], 1);
      MbarInit(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      MbarInit(&tmem_full[b], 1);
      MbarInit(&tmem_empty[b], 4);  // one arrival per epilogue warp
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(SmemAddr(tmem_slot)),
                 "r"(static_cast<uint32_t>(Cfg::kTmemCols))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  TcFenceBefore();
  __syncthreads();
  TcFenceAfter();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(tmem_slot);

  if (warp == 0) {
    if (ElectOne()) {
      uint32_t it = 0;  // running k-stage counter over all tiles
      bool ok = true;
      for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
        const int m0 = (tile / tiles_n) * kBM, n0 = (tile % tiles_n) * BN;
        for (int kt = 0; kt < num_k; ++kt, ++it) {
          const int s = it % Cfg::kStages;
          if (!MbarWait(&empty_bar[s], ((it / Cfg::kStages) & 1) ^ 1)) {
            atomicExch(p.error, 1);
            ok = false;
            break;
          }
          uint8_t* a_dst = smem + s * Cfg::kStageBytes;
          MbarExpectTx(&full_bar[s], Cfg::kStageBytes);
          TmaLoad2D(a_dst, &tmap_a, kt * kBK, m0, &full_bar[s]);
          if (kBMn) {
#pragma unroll
            for (int j = 0; j < BN / 64; ++j)
              TmaLoad2D(a_dst + Cfg::kABytes + j * 8192, &tmap_b, n0 + j * 64, kt * kBK, &full_bar[s]);
          } else {
            TmaLoad2D(a_dst + Cfg::kABytes, &tmap_b, kt * kBK, n0, &full_bar[s]);
          }
        }
      }
    }
  } else if (warp == 1) {
    {  // the whole warp walks the loop, one lane issues
      constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (kBMn ? (1u << 16) : 0u) |
                                 (static_cast<uint32_t>(BN >> 3) << 17) | (static_cast<uint32_t>(kBM >> 4) << 24);
      uint32_t it = 0;
      int local = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x, ++local) {
        const int buf = local & 1;
        if (!MbarWaitWarp(&tmem_empty[buf], ((local >> 1) & 1) ^ 1)) {  // the epilogue has drained this accumulator
          if (lane == 0) atomicExch(p.error, 4);
          break;
        }
        TcFenceAfter();
        const uint32_t tmem_d = tmem_base + static_cast<uint32_t>(buf * BN);
        for (int kt = 0; kt < num_k; ++kt, ++it) {
          const int s = it % Cfg::kStages;
          if (!MbarWaitWarp(&full_bar[s], (it / Cfg::kStages) & 1)) {
            if (lane == 0) atomicExch(p.error, 2);
            ok = false;
            break;
          }
          TcFenceAfter();
          const uint32_t a_addr = SmemAddr(smem + s * Cfg::kStageBytes);
          const uint64_t adesc  = SmemDescSw128(a_addr);
          const uint64_t bdesc  = kBMn ? SmemDescMnSw128(a_addr + Cfg::kABytes, 8192) : SmemDescSw128(a_addr + Cfg::kABytes);
          if (ElectOne()) {
#pragma unroll
            for (int k = 0; k < kBK / 16; ++k)
              UmmaBf16(tmem_d, adesc + 2 * k, bdesc + (kBMn ? 128 : 2) * k, idesc, (kt > 0 || k > 0) ? 1u : 0u);
            UmmaCommit(&empty_bar[s]);
          }
        }
        if (ok && ElectOne()) UmmaCommit(&tmem_full[buf]);
      }
    }
  } else {
    const int q = warp & 3;
    const int r = q * 32 + lane;
    int local = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x, ++local) {
      const int m0 = (tile / tiles_n) * kBM, n0 = (tile % tiles_n) * BN;
      const int buf = local & 1;
      if (ok && !MbarWait(&tmem_full[buf], (local >> 1) & 1)) {
        if (lane == 0) atomicExch(p.error, 3);
        ok = false;
      }
      TcFenceAfter();
      if (ok) {
#pragma unroll 1
        for (int c = 0; c < BN / 32; ++c) {
          uint32_t acc[32];
          TmemLoad32(tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(buf * BN + c * 32), acc);
          const int col0 = n0 + c * 32;
          uint8_t* box   = staging + (c >> 1) * (kBM * 128);
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            alignas(16) __nv_bfloat16 o[8];
#pragma unroll
            float bv[8];
            LoadBias8(p, col0 + g * 8, bv);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              float x = __uint_as_float(acc[g * 8 + j]) + bv[j];
              o[j] = __float2bfloat16_rn(GemmAct(x, p.act));
            }
            const int chunk = (c & 1) * 4 + g;
            *reinterpret_cast<uint4*>(box + r * 128 + ((chunk ^ (r & 7)) << 4)) = *reinterpret_cast<uint4*>(o);
          }
        }
        // this warp is done with the accumulator: hand it back to the MMA warp
        TcFenceBefore();
        __syncwarp();
        if (lane == 0) MbarArrive(&tmem_empty[buf]);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (warp == 2 && lane == 0) {
        if (ok) {
#pragma unroll 1
          for (int b = 0; b < BN / 64; ++b) {
            if (n0 + b * 64 < p.n) {
              TmaStoreOrAdd2D(&tmap_c, n0 + b * 64, m0, staging + b * (kBM * 128), p.accumulate);
            }
          }
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // staging may be overwritten afterwards
      }
      asm volatile("bar.sync 1, 128;" ::: "memory");
    }
  }
  TcFenceBefore();
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(static_cast<uint32_t>(Cfg::kTmemCols))
                 : "memory");
  }
}

// ---------------------------------------------------------------- CTA pairs, 256 x 256 tiles
// A pair of CTAs computes a 256 x 256 tile: per K block each SM takes 128 rows of A and 128 columns of B from L2
// (32 KB) for 512 tensor-core clocks, 64 bytes per clock, where a single CTA's 128 x 256 tile needs 96; and the
// accumulators take 256 TMEM columns per CTA, so two tiles fit and the epilogue of one overlaps the MMAs of the next.
// Eight epilogue warps: the GELU of 128 x 256 values per CTA costs about as many issue slots as the 8192 clocks of MMAs of
// a K = 1024 tile, so it needs two warps per scheduler, and two values per instruction (with erff, one at a time, the
// same product took 183 us).  A second output
// (the value before the activation, which the backward pass of GELU reads) leaves through the same staging boxes.
// Bound by the tensor cores.  Measured against the single-CTA kernels it took over from (us, M x N x K): 16384 x 4096 x
// 1024 with bias 100 : 114 (1377 TFLOP/s), the same with GELU and the second output 139 : 307 (159 with two staging boxes), 1232 x 30528 x 1024 71 : 105;
// A and B MN-major (a weight gradient) 4096 x 1024 x 16384 92 : 114, 30528 x 1024 x 1232 57 : 128.
template <bool kPre>
struct PairCfgOf {
  static constexpr int kBN            = 256;
  static constexpr int kStages        = kPre ? 4 : 5;
  static constexpr int kABytes        = kBM * kBK * 2;
  static constexpr int kBBytes        = (kBN / 2) * kBK * 2;
  static constexpr int kStageBytes    = kABytes + kBBytes;      // 32 KB per CTA
  static constexpr int kBoxBytes      = kBM * 128;              // 128 rows x 64 columns
  static constexpr int kGroupBoxes    = kPre ? 3 : 2;           // staging boxes of an epilogue group, used in turn
  static constexpr int kStagingBytes  = 2 * kGroupBoxes * kBoxBytes;
  static constexpr int kTmemCols      = 512;
  static constexpr int kThreads       = 320;                    // TMA warp, MMA warp, eight epilogue warps
  static constexpr int kSmemBytes     = kStages * kStageBytes + kStagingBytes + 1024 + 256;
};

using PairCfg = PairCfgOf<false>;

// What the epilogue of the pair kernel writes: the bf16 result, also the value before the activation, or fp32 partials.
constexpr int kOutPlain = 0, kOutPre = 1, kOutPartial = 2;

__host__ __device__ __forceinline__ int SplitBegin(int k_blocks, int split, int splits) {
  return static_cast<int>(static_cast<int64_t>(k_blocks) * split / splits);
}

template <bool kAMn, bool kBMn, int kOut>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PairCfg::kThreads, 1)
GemmPairKernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
               const __grid_constant__ CUtensorMap tmap_c, const __grid_constant__ CUtensorMap tmap_pre, GemmParams p) {
  constexpr bool kPre = kOut == kOutPre, kSplit = kOut == kOutPartial;
  using Cfg = PairCfgOf<kPre>;
  constexpr int BN = Cfg::kBN;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem    = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* staging = smem + Cfg::kStages * Cfg::kStageBytes;
  uint64_t* full_bar   = reinterpret_cast<uint64_t*>(staging + Cfg::kStagingBytes);  // the leader's copy is used
  uint64_t* empty_bar  = full_bar + Cfg::kStages;   // each CTA's own
  uint64_t* tmem_full  = empty_bar + Cfg::kStages;  // [2], each CTA's own
  uint64_t* tmem_empty = tmem_full + 2;             // [2], the leader's copy is used
  uint32_t* tmem_slot  = reinterpret_cast<uint32_t*>(tmem_empty + 2);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int cta  = static_cast<int>(ClusterCtaRank());
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int all_k   = (p.k + kBK - 1) / kBK;
  const int tiles_n = (p.n + BN - 1) / BN;
  const int tiles_m = (p.m + 2 * kBM - 1) / (2 * kBM);
  const int plane     = tiles_m * tiles_n;
  const int num_tiles = kSplit ? plane * p.splits : plane;  // a tile of split s covers its share of the K blocks

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::kStages; ++s) {
      MbarInit(&full_bar[s], 1);
      MbarInit(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      MbarInit(&tmem_full[b], 1);
      MbarInit(&tmem_empty[b], 16);  // eight epilogue warps of each CTA
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(SmemAddr(tmem_slot)),
                 "r"(static_cast<uint32_t>(Cfg::kTmemCols))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  TcFenceBefore();
  __syncthreads();
  ClusterSync();  // both CTAs' barriers exist before any remote arrival
  TcFenceAfter();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(tmem_slot);

  if (warp == 0) {
    if (ElectOne()) {
      uint32_t it = 0;
      bool ok = true;
      for (int tile = pair; tile < num_tiles && ok; tile += pairs) {
        const int mn = kSplit ? tile % plane : tile, sp = kSplit ? tile / plane : 0;
        const int k_lo = kSplit ? SplitBegin(all_k, sp, p.splits) : 0;
        const int k_hi = kSplit ? SplitBegin(all_k, sp + 1, p.splits) : all_k;
        const int m0 = (mn / tiles_n) * 2 * kBM + cta * kBM, n0 = (mn % tiles_n) * BN + cta * (BN / 2);
        for (int kt = k_lo; kt < k_hi; ++kt, ++it) {
          const int s = it % Cfg::kStages;
          if (!MbarWait(&empty_bar[s], ((it / Cfg::kStages) & 1) ^ 1)) {
            atomicExch(p.error, 1);
            ok = false;
            break;
          }
          uint8_t* a_dst = smem + s * Cfg::kStageBytes;
          uint8_t* b_dst = a_dst + Cfg::kABytes;
          if (cta == 0) MbarExpectTx(&full_bar[s], 2 * Cfg::kStageBytes);  // both CTAs' bytes
          if (kAMn) {
            TmaLoad2DPair(a_dst, &tmap_a, m0, kt * kBK, &full_bar[s]);
            TmaLoad2DPair(a_dst + 8192, &tmap_a, m0 + 64, kt * kBK, &full_bar[s]);
          } else {
            TmaLoad2DPair(a_dst, &tmap_a, kt * kBK, m0, &full_bar[s]);
          }
          if (kBMn) {
            TmaLoad2DPair(b_dst, &tmap_b, n0, kt * kBK, &full_bar[s]);
            TmaLoad2DPair(b_dst + 8192, &tmap_b, n0 + 64, kt * kBK, &full_bar[s]);
          } else {
            TmaLoad2DPair(b_dst, &tmap_b, kt * kBK, n0, &full_bar[s]);
          }
        }
      }
      // The leader's commits arrive on this CTA's barriers: wait for the last of every stage before leaving.
      for (uint32_t i = it > Cfg::kStages ? it - Cfg::kStages : 0; i < it && ok; ++i)
        if (!MbarWait(&empty_bar[i % Cfg::kStages], (i / Cfg::kStages) & 1)) {
          atomicExch(p.error, 1);
          ok = false;
        }
    }
  } else if (warp == 1) {
    if (cta == 0) {  // the whole warp walks the loop, one lane issues
      constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (kAMn ? (1u << 15) : 0u) | (kBMn ? (1u << 16) : 0u) |
                                 (static_cast<uint32_t>(BN >> 3) << 17) | (static_cast<uint32_t>((2 * kBM) >> 4) << 24);
      uint32_t it = 0;
      int local = 0;
      bool ok = true;
      for (int tile = pair; tile < num_tiles && ok; tile += pairs, ++local) {
        const int buf = local & 1;
        if (!MbarWaitWarp(&tmem_empty[buf], ((local >> 1) & 1) ^ 1)) {
          if (lane == 0) atomicExch(p.error, 4);
          break;
        }
        TcFenceAfter();
        const uint32_t tmem_d = tmem_base + static_cast<uint32_t>(buf * BN);
        const int sp    = kSplit ? tile / plane : 0;
        const int num_k = kSplit ? SplitBegin(all_k, sp + 1, p.splits) - SplitBegin(all_k, sp, p.splits) : all_k;
        for (int kt = 0; kt < num_k; ++kt, ++it) {
          const int s = it % Cfg::kStages;
          if (!MbarWaitWarp(&full_bar[s], (it / Cfg::kStages) & 1)) {
            if (lane == 0) atomicExch(p.error, 2);
            ok = false;
            break;
          }
          TcFenceAfter();
          const uint32_t a_addr = SmemAddr(smem + s * Cfg::kStageBytes);
          const uint64_t adesc  = kAMn ? SmemDescMnSw128(a_addr, 8192) : SmemDescSw128(a_addr);
          const uint64_t bdesc  = kBMn ? SmemDescMnSw128(a_addr + Cfg::kABytes, 8192) : SmemDescSw128(a_addr + Cfg::kABytes);
          if (ElectOne()) {
#pragma unroll
            for (int k = 0; k < kBK / 16; ++k)
              UmmaBf16Pair(tmem_d, adesc + (kAMn ? 128 : 2) * k, bdesc + (kBMn ? 128 : 2) * k, idesc,
                           (kt > 0 || k > 0) ? 1u : 0u);
            UmmaCommitPair(&empty_bar[s]);
          }
        }
        if (ok && ElectOne()) UmmaCommitPair(&tmem_full[buf]);
      }
    }
  } else {
    // Two groups of four warps: group g drains columns [128 g, 128 g + 128) as two boxes of 64.
    const int q = warp & 3;                // TMEM lane quarter
    const int g = (warp - 2) >> 2;
    const int r = q * 32 + lane;           // row of this CTA's half tile
    const bool issuer = (warp == 2 || warp == 6) && lane == 0;
    uint8_t* boxes = staging + g * Cfg::kGroupBoxes * Cfg::kBoxBytes;
    int slot = 0;  // next staging box
    int local = 0;
    bool ok = true;
    for (int tile = pair; tile < num_tiles; tile += pairs, ++local) {
      const int mn = kSplit ? tile % plane : tile;
      const int m0 = (mn / tiles_n) * 2 * kBM + cta * kBM, n0 = (mn % tiles_n) * BN + g * (BN / 2);
      const int buf = local & 1;
      if (ok && !MbarWait(&tmem_full[buf], (local >> 1) & 1)) {
        if (lane == 0) atomicExch(p.error, 3);
        ok = false;
      }
      TcFenceAfter();
      const uint32_t tsrc = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(buf * BN + g * (BN / 2));
      uint32_t acc[2][32];
      if (ok) TmemLoad32Async(tsrc, acc[0]);
      if constexpr (kSplit) {  // fp32 partial rows, straight from the registers: 128 bytes per lane and chunk
        float* row = p.partial + (static_cast<int64_t>(tile / plane) * p.m + m0 + r) * p.n;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if (!ok) continue;
          TmemLoadWait(acc[c & 1]);
          if (c + 1 < 4) TmemLoad32Async(tsrc + static_cast<uint32_t>((c + 1) * 32), acc[(c + 1) & 1]);
          const int col0 = n0 + c * 32;
          if (m0 + r < p.m) {
#pragma unroll
            for (int u = 0; u < 8; ++u)  // n is a multiple of 8, so a vector is inside or outside as a whole
              if (col0 + u * 4 < p.n)
                *reinterpret_cast<uint4*>(row + col0 + u * 4) = make_uint4(acc[c & 1][u * 4], acc[c & 1][u * 4 + 1],
                                                                           acc[c & 1][u * 4 + 2], acc[c & 1][u * 4 + 3]);
          }
        }
        if (ok) {
          TcFenceBefore();
          __syncwarp();
          if (lane == 0) MbarArriveLeader(&tmem_empty[buf]);
        }
        continue;
      }
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        uint8_t* box = boxes + slot * Cfg::kBoxBytes;
        slot = slot + 1 == Cfg::kGroupBoxes ? 0 : slot + 1;
        uint8_t* pbox = boxes + slot * Cfg::kBoxBytes;
        if (kPre) slot = slot + 1 == Cfg::kGroupBoxes ? 0 : slot + 1;
        // every store is a group of its own, and all but the newest have been read: two boxes of the three, one of the two
        if (issuer) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
        NamedBarSync(1 + g, 128);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int c = 2 * b + half;
          if (ok) {
            const int col0 = n0 + c * 32;
            TmemLoadWait(acc[c & 1]);
            if (c + 1 < 4) TmemLoad32Async(tsrc + static_cast<uint32_t>((c + 1) * 32), acc[(c + 1) & 1]);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              float bv[8];
              LoadBias8(p, col0 + u * 8, bv);
              alignas(16) __nv_bfloat16 o[8];
              alignas(16) __nv_bfloat16 pr[8];
#pragma unroll
              for (int j = 0; j < 8; j += 2) {
                const float x = __uint_as_float(acc[c & 1][u * 8 + j]) + bv[j];
                const float y = __uint_as_float(acc[c & 1][u * 8 + j + 1]) + bv[j + 1];
                const float2 z = GemmAct2(x, y, p.act);
                if (kPre) *reinterpret_cast<__nv_bfloat162*>(&pr[j]) = __floats2bfloat162_rn(x, y);
                *reinterpret_cast<__nv_bfloat162*>(&o[j]) = __floats2bfloat162_rn(z.x, z.y);
              }
              const int off = r * 128 + (((half * 4 + u) ^ (r & 7)) << 4);
              *reinterpret_cast<uint4*>(box + off) = *reinterpret_cast<uint4*>(o);
              if (kPre) *reinterpret_cast<uint4*>(pbox + off) = *reinterpret_cast<uint4*>(pr);
            }
          }
        }
        if (b == 1 && ok) {  // this warp's share of the accumulator is drained
          TcFenceBefore();
          __syncwarp();
          if (lane == 0) MbarArriveLeader(&tmem_empty[buf]);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        NamedBarSync(1 + g, 128);
        if (issuer) {
          if (ok && n0 + b * 64 < p.n && m0 < p.m) {
            TmaStoreOrAdd2D(&tmap_c, n0 + b * 64, m0, box, p.accumulate);
            if (kPre) {
              asm volatile("cp.async.bulk.commit_group;" ::: "memory");
              TmaStoreOrAdd2D(&tmap_pre, n0 + b * 64, m0, pbox, 0);
            }
          }
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
      }
    }
    if (!kSplit && issuer) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  TcFenceBefore();
  __syncthreads();
  ClusterSync();  // no CTA leaves while its peer may still signal its barriers or use its TMEM
  TcFenceAfter();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(static_cast<uint32_t>(Cfg::kTmemCols))
                 : "memory");
  }
}

// Sum of the partial products in the order of the splits, then bias and activation as in the other epilogues: four
// columns per thread, so that a warp reads 512 contiguous bytes of each share and small outputs still fill the SMs.  With
// `accumulate` the sum is added to what C holds.
__global__ void __launch_bounds__(256)
GemmSplitSumKernel(GemmParams p) {
  const int vecs      = p.n / 4;
  const int64_t total = static_cast<int64_t>(p.m) * vecs, plane = static_cast<int64_t>(p.m) * p.n;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x; i < total; i += static_cast<int64_t>(gridDim.x) * 256) {
    const int64_t row = i / vecs;
    const int col     = static_cast<int>(i - row * vecs) * 4;
    const float* src  = p.partial + row * p.n + col;
    float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int s = 0; s < p.splits; ++s) {
      const float4 a = *reinterpret_cast<const float4*>(src + s * plane);
      v[0] += a.x; v[1] += a.y; v[2] += a.z; v[3] += a.w;
    }
    __nv_bfloat16* dst = p.c + row * p.ldc + col;
    alignas(8) __nv_bfloat16 o[4], pr[4];
    if (p.accumulate) *reinterpret_cast<uint2*>(o) = *reinterpret_cast<const uint2*>(dst);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float x = v[j] + (p.bias ? __bfloat162float(p.bias[col + j]) : 0.f);
      pr[j] = __float2bfloat16_rn(x);
      x     = GemmAct(x, p.act);
      o[j]  = __float2bfloat16_rn(p.accumulate ? __bfloat162float(o[j]) + x : x);
    }
    if (p.pre) *reinterpret_cast<uint2*>(p.pre + row * p.ldc + col) = *reinterpret_cast<const uint2*>(pr);
    *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(o);
  }
}

// ------------------------------------------------------------------ host side

// Row-major [rows, cols] bf16 matrix with leading dimension ld (elements); box = 64 x box_rows, 128B swizzle.
int MakeTmap(CUtensorMap* out, const void* base, int64_t rows, int64_t cols, int64_t ld, int box_rows) {
  EncodeFn enc = GetEncodeFn();
  if (!enc) return SetError(-7, "cuTensorMapEncodeTiled is not available from the driver");
  if (reinterpret_cast<uintptr_t>(base) % 16 != 0) return SetError(-2, "gemm: operand base must be 16-byte aligned");
  if ((ld * 2) % 16 != 0) return SetError(-2, "gemm: operand row stride must be a multiple of 16 bytes");
  cuuint64_t dims[2]    = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * 2};
  cuuint32_t box[2]     = {static_cast<cuuint32_t>(kBK), static_cast<cuuint32_t>(box_rows)};
  cuuint32_t estr[2]    = {1, 1};
  CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return SetError(-7, "cuTensorMapEncodeTiled failed with code " + std::to_string((int)r));
  return 0;
}

int32_t* GemmErrorWord() {
  static int32_t* word = nullptr;
  if (!word) {
    if (cudaMalloc(reinterpret_cast<void**>(&word), sizeof(int32_t)) != cudaSuccess) return nullptr;
    cudaMemset(word, 0, sizeof(int32_t));
  }
  return word;
}

template <int BN, bool kBMn = false>
int LaunchGemm(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const CUtensorMap& tp,
               const GemmParams& p, cudaStream_t s) {
  using Cfg = GemmCfg<BN>;
  static bool configured = false;
  if (!configured) {
    TIPSK_CUDA(cudaFuncSetAttribute(GemmTnKernel<BN, kBMn>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes));
    TIPSK_CUDA(cudaFuncSetAttribute(GemmTnKernel<BN, kBMn>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                    cudaSharedmemCarveoutMaxShared));
    configured = true;
  }
  dim3 grid((p.n + BN - 1) / BN, (p.m + kBM - 1) / kBM);
  GemmTnKernel<BN, kBMn><<<grid, kGemmThreads, Cfg::kSmemBytes, s>>>(ta, tb, tc, tp, p);
  TIPSK_LAUNCH_CHECK();
  return 0;
}

template <int BN, bool kBMn = false>
int LaunchGemmPersistent(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const GemmParams& p,
                         cudaStream_t s) {
  using Cfg = PersistCfg<BN>;
  static bool configured = false;
  if (!configured) {
    TIPSK_CUDA(cudaFuncSetAttribute(GemmTnPersistentKernel<BN, kBMn>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    Cfg::kSmemBytes));
    configured = true;
  }
  const int tiles = ((p.n + BN - 1) / BN) * ((p.m + kBM - 1) / kBM);
  const int grid  = tiles < NumSMs() ? tiles : NumSMs();
  GemmTnPersistentKernel<BN, kBMn><<<grid, kGemmThreads, Cfg::kSmemBytes, s>>>(ta, tb, tc, p);
  TIPSK_LAUNCH_CHECK();
  return 0;
}

// Pairs of SMs that can run a cluster of the pair kernel at the same time (an odd SM of a GPC stays without a partner).
template <bool kAMn, bool kBMn, int kOut>
int LaunchPair(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const CUtensorMap& tp,
               const GemmParams& p, cudaStream_t s) {
  using Cfg = PairCfgOf<kOut == kOutPre>;
  static std::atomic<int> resident{0};
  int pairs = resident.load(std::memory_order_acquire);
  if (pairs == 0) {
    TIPSK_CUDA(cudaFuncSetAttribute(GemmPairKernel<kAMn, kBMn, kOut>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim          = dim3(NumSMs() & ~1);
    cfg.blockDim         = dim3(Cfg::kThreads);
    cfg.dynamicSmemBytes = Cfg::kSmemBytes;
    cudaLaunchAttribute at{};
    at.id               = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = 2;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs    = &at;
    cfg.numAttrs = 1;
    TIPSK_CUDA(cudaOccupancyMaxActiveClusters(&pairs, GemmPairKernel<kAMn, kBMn, kOut>, &cfg));
    TIPSK_REQUIRE(pairs > 0, "gemm: no CTA pair fits on this device");
    resident.store(pairs, std::memory_order_release);
  }
  const int64_t tiles = static_cast<int64_t>(CeilDiv(p.n, Cfg::kBN)) * CeilDiv(p.m, 2 * kBM) * (kOut == kOutPartial ? p.splits : 1);
  const int grid = 2 * static_cast<int>(tiles < pairs ? tiles : pairs);
  GemmPairKernel<kAMn, kBMn, kOut><<<grid, Cfg::kThreads, Cfg::kSmemBytes, s>>>(ta, tb, tc, tp, p);
  TIPSK_LAUNCH_CHECK();
  return 0;
}

// Both halves of a product whose K is split: the partial products, then their sum.
template <bool kAMn, bool kBMn>
int LaunchPairSplit(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p, cudaStream_t s) {
  int rc = LaunchPair<kAMn, kBMn, kOutPartial>(ta, tb, ta, ta, p, s);
  if (rc) return rc;
  const int64_t vecs = static_cast<int64_t>(p.m) * (p.n / 4);
  const int64_t grid = std::min<int64_t>((vecs + 255) / 256, NumSMs() * 8);
  GemmSplitSumKernel<<<static_cast<int>(grid), 256, 0, s>>>(p);
  TIPSK_LAUNCH_CHECK();
  return 0;
}

// Whether the CTA-pair kernel should take the problem: from about 1.25 tiles per pair of SMs on.  Measured against the
// single-CTA kernels (us, M x N x K): 192 tiles 4096 x 3072 x 1024 32 : 45, 128 tiles 8192 x 1024 x 1024 27 : 32, 96
// tiles 2048 x 3072 x 1024 26 : 31; below, a pair's single 256 x 256 tile and its exposed epilogue take longer than
// two small CTAs per SM: 64 tiles 4096 x 1024 x 1024 21 : 17, 8192 x 512 x 1728 25 : 21.
// Where N ends inside a tile, 128-column tiles cover it more closely.  They stay ahead while all of them are resident at once,
// two per SM (12000 x 384 x 1024 12.7 : 17.1, 12000 x 264 x 264 9.8 : 12.3; with more 14000 x 384 x 1024 20.7 : 17.5), and
// with a short K, where the epilogues are most of the time, up to three per SM (16384 x 320 x 128 11.7 : 13.2, 8192 x 640 x
// 64 10.8 : 13.4, 6000 x 1032 x 256 13.7 : 14.6; with more 12000 x 640 x 64 17.5 : 13.7).
bool PreferPair(int m, int n, int k) {
  const int64_t tiles = static_cast<int64_t>(CeilDiv(m, 2 * kBM)) * CeilDiv(n, PairCfg::kBN);
  if (n <= 128 || tiles * 4 < (NumSMs() / 2) * 5) return false;
  const bool ragged   = static_cast<int64_t>(m) * n * 10 < tiles * 2 * kBM * PairCfg::kBN * 9;
  const int64_t small = static_cast<int64_t>(CeilDiv(m, kBM)) * CeilDiv(n, 128);
  return !ragged || small > NumSMs() * (k <= 256 ? 3 : 2);
}

}  // namespace
}  // namespace tipsk

using namespace tipsk;

extern "C" {

/* 1 when tipsk_gemm_bf16 accepts the problem (alignment of the leading dimensions). */
int tipsk_gemm_supported(int m, int n, int k, int lda, int ldb) {
  return (m > 0 && n > 0 && k > 0 && lda % 8 == 0 && ldb % 8 == 0) ? 1 : 0;
}

/* C[m,n] = act(A[m,k] * B[n,k]^T + bias); bf16 in, fp32 accumulate in TMEM, bf16 out.
 * lda/ldb/ldc are leading dimensions in elements; `pre` (optional) receives the value before the activation. */
int tipsk_gemm_bf16(const void* a, const void* b, void* c, const void* bias, void* pre, int m, int n, int k, int lda,
                    int ldb, int ldc, int act, void* stream) {
  TIPSK_REQUIRE(tipsk_gemm_supported(m, n, k, lda, ldb), "gemm: lda and ldb must be multiples of 8 elements");
  int bn = 128;
  if (n <= 16) bn = 16;
  else if (n <= 32) bn = 32;
  else if (n <= 64) bn = 64;
  else if (n % 256 == 0 && (static_cast<int64_t>(m) / kBM) * (n / 256) >= NumSMs()) bn = 256;
  GemmParams p{};
  p.c     = static_cast<__nv_bfloat16*>(c);
  p.pre   = static_cast<__nv_bfloat16*>(pre);
  p.bias  = static_cast<const __nv_bfloat16*>(bias);
  p.error = GemmErrorWord();
  TIPSK_REQUIRE(p.error != nullptr, "gemm: cannot allocate the error word");
  p.m = m; p.n = n; p.k = k; p.ldc = ldc; p.act = act; p.accumulate = 0;
  p.bias_vec = (bias != nullptr && reinterpret_cast<uintptr_t>(bias) % 16 == 0) ? 1 : 0;
  // The coalesced store path needs 64-column boxes and 16-byte aligned, 16-byte strided outputs.
  p.tma_store = (bn >= 64 && ldc % 8 == 0 && reinterpret_cast<uintptr_t>(c) % 16 == 0 &&
                 reinterpret_cast<uintptr_t>(pre) % 16 == 0) ? 1 : 0;
  const bool pair = p.tma_store && PreferPair(m, n, k);
  CUtensorMap ta, tb;
  int rc = MakeTmap(&ta, a, m, k, lda, kBM);
  if (rc) return rc;
  rc = MakeTmap(&tb, b, n, k, ldb, pair ? PairCfg::kBN / 2 : bn);
  if (rc) return rc;
  CUtensorMap tc = ta, tp = ta;
  if (p.tma_store) {
    rc = MakeTmap(&tc, c, m, n, ldc, kBM);
    if (rc) return rc;
    if (pre) rc = MakeTmap(&tp, pre, m, n, ldc, kBM);
    if (rc) return rc;
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (pair)
    return pre ? LaunchPair<false, false, kOutPre>(ta, tb, tc, tp, p, s) : LaunchPair<false, false, kOutPlain>(ta, tb, tc, tp, p, s);
  // More tiles than SMs and a TMA-storable output: the persistent kernel overlaps epilogue and main loop.
  if (p.tma_store && pre == nullptr && bn == 128) {
    const int64_t tiles = static_cast<int64_t>((n + bn - 1) / bn) * ((m + kBM - 1) / kBM);
    // Measured on B200: the overlap pays when the epilogue is a visible share of a tile (K <= 2048) and
    // there are enough tiles to fill several waves; otherwise two independent CTAs per SM do better.
    if (tiles >= 3 * NumSMs() && k <= 2048) {
      return LaunchGemmPersistent<128>(ta, tb, tc, p, s);
    }
  }
  switch (bn) {
    case 16: return LaunchGemm<16>(ta, tb, tc, tp, p, s);
    case 32: return LaunchGemm<32>(ta, tb, tc, tp, p, s);
    case 64: return LaunchGemm<64>(ta, tb, tc, tp, p, s);
    case 256: return LaunchGemm<256>(ta, tb, tc, tp, p, s);
    default: return LaunchGemm<128>(ta, tb, tc, tp, p, s);
  }
}

/* C[m,n] = A[m,k] * B[k,n]: B row-major with the contraction over its rows (no transposed copy is made; the MMA
 * reads it as an MN-major operand).  Serves dx = dy * W of a linear layer with W stored [out, in].  n >= 64.
 * With `accumulate` the product is added (in bf16, by reduce-add stores) to what C already holds. */
int tipsk_gemm_bf16_nn(const void* a, const void* b, void* c, int m, int n, int k, int lda, int ldb, int ldc,
                       int accumulate, void* stream) {
  TIPSK_REQUIRE(m > 0 && n >= 64 && k > 0 && lda % 8 == 0 && ldb % 8 == 0 && ldc % 8 == 0,
                "gemm_nn: leading dimensions must be multiples of 8 elements and n >= 64");
  TIPSK_REQUIRE(reinterpret_cast<uintptr_t>(c) % 16 == 0, "gemm_nn: output must be 16-byte aligned");
  int bn = 128;
  if (n <= 64) bn = 64;
  else if (n % 256 == 0 && (static_cast<int64_t>(m) / kBM) * (n / 256) >= NumSMs()) bn = 256;
  CUtensorMap ta, tb, tc;
  int rc = MakeTmap(&ta, a, m, k, lda, kBM);
  if (rc) return rc;
  rc = MakeTmap(&tb, b, k, n, ldb, kBK);  // boxes of 64 contraction rows x 64 columns
  if (rc) return rc;
  rc = MakeTmap(&tc, c, m, n, ldc, kBM);
  if (rc) return rc;
  GemmParams p{};
  p.c = static_cast<__nv_bfloat16*>(c);
  p.pre = nullptr;
  p.bias = nullptr;
  p.error = GemmErrorWord();
  TIPSK_REQUIRE(p.error != nullptr, "gemm: cannot allocate the error word");
  p.m = m; p.n = n; p.k = k; p.ldc = ldc; p.act = 0; p.tma_store = 1; p.accumulate = accumulate ? 1 : 0;
  p.bias_vec = 0;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (PreferPair(m, n, k)) return LaunchPair<false, true, kOutPlain>(ta, tb, tc, tc, p, s);
  if (bn == 128) {
    const int64_t tiles = static_cast<int64_t>((n + bn - 1) / bn) * ((m + kBM - 1) / kBM);
    if (tiles >= 3 * NumSMs() && k <= 2048) {
      return LaunchGemmPersistent<128, true>(ta, tb, tc, p, s);
    }
  }
  switch (bn) {
    case 64: return LaunchGemm<64, true>(ta, tb, tc, tc, p, s);
    case 256: return LaunchGemm<256, true>(ta, tb, tc, tc, p, s);
    default: return LaunchGemm<128, true>(ta, tb, tc, tc, p, s);
  }
}

/* Whether the pair kernel is the one to run a product of this kind (the kinds of tipsk_gemm_bf16_split). */
int tipsk_gemm_prefers_pair(int kind, int m, int n, int k) {
  if (m < 64 || n < 64 || n % 8 != 0 || k <= 0) return 0;
  if (kind != 2) return PreferPair(m, n, k) ? 1 : 0;
  // Weight gradients: the alternative is the convolution's kernel, which spreads K over all SMs with 128-row tiles as narrow as
  // 64 columns, adds fp32 sums into a cleared buffer and is followed by a cast.  Measured, pair : convolution kernel in us
  // (M x N x K).
  const int64_t tiles  = static_cast<int64_t>(CeilDiv(m, 2 * kBM)) * CeilDiv(n, PairCfg::kBN);
  const int64_t splits = tipsk_gemm_splits(m, n, k), pairs = NumSMs() / 2;
  // Outputs that leave half of their 256 x 256 tiles empty waste the pair's MMAs: 64 x 64 x 401408 44 : 23, 256 x 64 x 200704
  // 37 : 30, 192 x 320 x 32768 24 : 18.  But columns that fill whole tiles suit the alternative's widest tile no better, and
  // its sums cost more, up to middling K: 64 x 256 x 12544 14 : 18, 64 x 512 x 16384 16 : 19, 64 x 256 x 200704 39 : 35.
  const bool few_k = k <= 256 && m >= 128 && n % 128 == 0;  // 192 x 128 x 256 7.3 : 7.8
  if (!few_k && !(n >= PairCfg::kBN && 2 * static_cast<int64_t>(m) * n >= tiles * 2 * kBM * PairCfg::kBN) &&
      !(n % PairCfg::kBN == 0 && k <= 32768))
    return 0;
  // Very long K amortises the alternative's costs: 256 x 256 x 131072 47 : 44 (74 partial tiles to add), 2304 x 768 x 131072
  // 359 : 333 (27 tiles in two shares leave 20 of 74 pairs idle); with the pairs busy 768 x 768 x 131072 122 : 131.
  if (k > 65536 && (tiles < 2 || tiles * splits * 5 < pairs * 4)) return 0;
  // Few tiles walk an unsplit K on few SMs, 5 us plus 0.35 us per 64 rows: 512 x 256 x 1000 11.0 : 10.6, 256 x 512 x 256 7.6 : 10,
  // 384 x 1024 x 1000 11 : 18, 512 x 1728 x 2048 16 : 18.
  return (k <= 256 || (tiles >= 4 && k <= 1024) || tiles >= 12 || splits > 1) ? 1 : 0;
}

/* Number of K splits with which tipsk_gemm_bf16_split should run the product (1: use the unsplit entry points). */
int tipsk_gemm_splits(int m, int n, int k) {
  if (m <= 0 || n < 64 || n % 8 != 0 || k <= 0) return 1;
  const int64_t tiles = static_cast<int64_t>(CeilDiv(m, 2 * kBM)) * CeilDiv(n, PairCfg::kBN);
  const int64_t pairs = NumSMs() / 2, blocks = CeilDiv(k, kBK);
  if (2 * tiles > pairs) return 1;
  const int64_t s = std::min<int64_t>(pairs / tiles, blocks / 8);  // at least eight K blocks per share
  // A second launch and the partial products cost about 8 us: from K = 4096 on the shorter chain is worth them (us, split
  // against not: 1024 x 1024 x 4096 25 : 28, 512 x 1024 x 4096 23 : 28, 1024 x 1024 x 30528 63 : 150; 2048 x 1024 x 4096
  // with two shares 31 : 31, 1024 x 1024 x 2048 23 : 20).
  if (k < 4096 || (k < 8192 && s < 4)) return 1;
  return s < 2 ? 1 : static_cast<int>(s);
}

/* The three products of a linear layer with the contraction split over `splits` shares (few output tiles, long K):
 *   kind 0  C[m,n] = act(A[m,k] * B[n,k]^T + bias), `pre` as in tipsk_gemm_bf16
 *   kind 1  C[m,n] = A[m,k] * B[k,n], with `accumulate` added to C
 *   kind 2  C[m,n] = A[k,m]^T * B[k,n]
 * `partial`: fp32 workspace of splits * m * n elements.  n a multiple of 8, 16-byte aligned rows throughout. */
int tipsk_gemm_bf16_split(int kind, const void* a, const void* b, void* c, const void* bias, void* pre, float* partial,
                          int splits, int m, int n, int k, int lda, int ldb, int ldc, int act, int accumulate,
                          void* stream) {
  TIPSK_REQUIRE(kind >= 0 && kind <= 2 && m > 0 && n >= 64 && n % 8 == 0 && k > 0, "gemm_split: unsupported shape");
  TIPSK_REQUIRE(lda % 8 == 0 && ldb % 8 == 0 && ldc % 8 == 0, "gemm_split: leading dimensions must be multiples of 8");
  TIPSK_REQUIRE(partial != nullptr && splits >= 1 && splits <= CeilDiv(k, kBK), "gemm_split: workspace or split count");
  TIPSK_REQUIRE(reinterpret_cast<uintptr_t>(c) % 16 == 0 && reinterpret_cast<uintptr_t>(pre) % 16 == 0 &&
                    reinterpret_cast<uintptr_t>(partial) % 16 == 0,
                "gemm_split: outputs must be 16-byte aligned");
  CUtensorMap ta, tb;
  int rc = kind == 2 ? MakeTmap(&ta, a, k, m, lda, kBK) : MakeTmap(&ta, a, m, k, lda, kBM);
  if (rc) return rc;
  rc = kind == 0 ? MakeTmap(&tb, b, n, k, ldb, PairCfg::kBN / 2) : MakeTmap(&tb, b, k, n, ldb, kBK);
  if (rc) return rc;
  GemmParams p{};
  p.c     = static_cast<__nv_bfloat16*>(c);
  p.pre   = static_cast<__nv_bfloat16*>(pre);
  p.bias  = static_cast<const __nv_bfloat16*>(bias);
  p.error = GemmErrorWord();
  TIPSK_REQUIRE(p.error != nullptr, "gemm: cannot allocate the error word");
  p.m = m; p.n = n; p.k = k; p.ldc = ldc; p.act = act; p.accumulate = accumulate ? 1 : 0;
  p.bias_vec = (bias != nullptr && reinterpret_cast<uintptr_t>(bias) % 16 == 0) ? 1 : 0;
  p.partial  = partial;
  p.splits   = splits;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (kind == 0) return LaunchPairSplit<false, false>(ta, tb, p, s);
  if (kind == 1) return LaunchPairSplit<false, true>(ta, tb, p, s);
  return LaunchPairSplit<true, true>(ta, tb, p, s);
}

/* C[m,n] = A[k,m]^T * B[k,n], both operands row-major with the contraction over their rows (MN-major for the MMA, no
 * transposed copies): the weight gradient dW = dz^T x of a linear layer, written in bf16 once.  m, n >= 64. */
int tipsk_gemm_bf16_tt(const void* a, const void* b, void* c, int m, int n, int k, int lda, int ldb, int ldc,
                       void* stream) {
  TIPSK_REQUIRE(m >= 64 && n >= 64 && k > 0 && lda % 8 == 0 && ldb % 8 == 0 && ldc % 8 == 0,
                "gemm_tt: leading dimensions must be multiples of 8 elements, m and n >= 64");
  TIPSK_REQUIRE(reinterpret_cast<uintptr_t>(c) % 16 == 0, "gemm_tt: output must be 16-byte aligned");
  CUtensorMap ta, tb, tc;
  int rc = MakeTmap(&ta, a, k, m, lda, kBK);  // boxes of 64 contraction rows x 64 columns
  if (rc) return rc;
  rc = MakeTmap(&tb, b, k, n, ldb, kBK);
  if (rc) return rc;
  rc = MakeTmap(&tc, c, m, n, ldc, kBM);
  if (rc) return rc;
  GemmParams p{};
  p.c = static_cast<__nv_bfloat16*>(c);
  p.error = GemmErrorWord();
  TIPSK_REQUIRE(p.error != nullptr, "gemm: cannot allocate the error word");
  p.m = m; p.n = n; p.k = k; p.ldc = ldc; p.tma_store = 1;
  return LaunchPair<true, true, kOutPlain>(ta, tb, tc, tc, p, static_cast<cudaStream_t>(stream));
}

/* Reads and clears the GEMM error word (0 ok; 1/2/3 = producer / MMA / epilogue wait ran out). Synchronises. */
int tipsk_gemm_status(void) {
  int32_t* w = GemmErrorWord();
  if (!w) return -7;
  int32_t v = 0;
  if (cudaMemcpy(&v, w, sizeof(v), cudaMemcpyDeviceToHost) != cudaSuccess) return -7;
  if (v) cudaMemset(w, 0, sizeof(v));
  return v;
}

}  // extern "C"
