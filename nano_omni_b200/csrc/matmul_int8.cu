// INT8 and BF16 GEMMs with a fused epilogue for sm_100a: the projections on either side of attention and
// their LoRA side products.
//
// Replaces the reference program matmul_int8 (src/nano_omni/kernels/matmul/matmul_int8.py:53-160, arithmetic of its
// ref_program :209-240):
//   acc[m, n]  = sum_k input[m, k] * weight[n, k]                  (int8 x int8 -> int32)
//   value      = ((float(acc) * weight_scale[n]) * input_scale[m]) [+ bias[n]] [+ residual[m, n]]
//   value      = silu(value) if use_silu;  value *= multiply[m, n] if given;  output[m, n] = bf16(value)
// input int8 [M, K], weight int8 [N, K] (both K-major), output / residual / multiply bf16 [M, N], bias bf16 [N],
// weight_scale f32 [N, 1], input_scale f32 [M].
// The BF16 form replaces matmul_bf16 (src/nano_omni/kernels/matmul/matmul_bf16.py:29-160, ref_program :183-207):
// bf16 operands, fp32 accumulation, value = acc * output_scale, then the same bias / residual / SiLU / multiply.
//
// Organisation.  Persistent PAIRS of CTAs (clusters of two) walk output tiles of 256 x BN, N fastest, so that the pairs
// in flight share A panels in L2.  `tcgen05.mma.cta_group::2` multiplies a tile on both SMs at once: CTA r holds rows
// 128 r .. of A and rows BN/2 r .. of B in its shared memory and gets rows 128 r .. of the accumulator in its TMEM.  A
// stage of 128 bytes of K is thus 16 + BN/16 KiB per SM and 2 BN cycles of tensor work; one CTA per tile (128 x 256)
// needed 48 KiB for 512 cycles, more than the 64 bytes per cycle that an SM reads from L2, and waited for its loads.
//   warp 0    TMA producer (each CTA its own halves; all copies report to the leader CTA's barrier), 5-stage ring,
//             128-byte swizzle, no multicast
//   warp 1    of the leader issues kind::i8 MMAs of 256 x BN x 32 (kind::f16, 256 x BN x 16 for bf16: the same 32 bytes
//             of K) into one of two 256-column accumulators; its commits release the stage in both CTAs
//   warps 2-9 drain the other accumulator, a row per thread and 32 columns per step, the epilogue in the ref_program's
//             order with separately rounded fp32 operations.  The residual arrives by TMA two steps ahead and the
//             result leaves by TMA, both through the warp's own staging tiles of 32 x 32: a thread per row touches 32
//             different lines per instruction, and that bounded the products with a short K (LoRA updates).
// These kernels by themselves: int8 15104 x 5376 x 7168 395 -> 347 us (2 N M K at the measured rate: 354), the rank-64 pair
// beside it 175 -> 144 us, bf16 512 x 7168 x 5376 42 -> 36 us (launched back to back; timed call by call 41.5 us).
// Low-rank adapters (the ADAPTED form) are multiplied inside: sum_r compressed[m, r] * expansion[n, r], one more chunk of
// K per 64 of the rank.  bf16: behind the main operands' chunks, into the same accumulator.  int8: the epilogue warps first
// turn the int32 accumulator into scaled fp32 in place, and kind::f16 MMAs add to that, behind the first chunks of the next
// tile so that the tensor pipe does not wait for them.  As GEMMs of their own the updates are bound by the output they read
// and write: the whole operator of 15104 x 5376 x 7168 int8 with a rank-64 pair and a residual took 678 us, with the pair
// inside it takes 614, at an error against 64 bits that is 13 to 27 % lower (one rounding to bf16 for two).
// BN is 64 .. 256, chosen per shape by tile_width().  Every wait is bounded.
#include <cuda.h>

#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "fa_common.cuh"
#include "tensor_map.cuh"
#include "../../include/nano_omni_b200.h"

namespace nob200 {
namespace {

constexpr int kBM = 256, kBK = 128;  // rows of a tile (both CTAs); bytes along K: 128 int8 or 64 bf16 elements
constexpr int kMaxBN = 256, kMinBN = 64;
constexpr int kStages = 5;
constexpr int kABytes = kBM / 2 * kBK, kBBytes = kMaxBN / 2 * kBK;  // per CTA
constexpr int kThreads = 320;  // producer, issuer, eight epilogue warps (two per TMEM lane quarter)
constexpr int kEpilogueWarps = 8;
constexpr int kStep = 32;         // columns per epilogue step
constexpr int kStagingTiles = 4;  // per epilogue warp: [32 rows][64 bytes], 64-byte swizzle
constexpr int kStagingBytes = 32 * kStep * 2;
constexpr uint32_t kTmemCols = 512;
constexpr int kMaxAdapters = 2;
// int8 form: the adapters of a tile are multiplied behind this many chunks of the next one, when the epilogue warps have
// long turned the tile's accumulator into fp32 (about three chunks) and long before they must have drained it
constexpr int kAdapterDelay = 8;

struct __align__(1024) GemmShared {
  uint8_t a[kStages][kABytes];
  uint8_t b[kStages][kBBytes];
  uint8_t staging[kEpilogueWarps][kStagingTiles][kStagingBytes];
  uint64_t full[kStages];  // the leader's; counts the bytes of both CTAs
  uint64_t empty[kStages];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];  // the leader's; sixteen warps arrive
  uint64_t acc_scaled[2];    // int8 with adapters, the leader's: the accumulator holds scaled fp32; sixteen warps arrive
  uint64_t adapter_full[2];  // and the adapters' products
  uint64_t residual_full[kEpilogueWarps][kStagingTiles];
  uint32_t tmem_base;
  uint32_t abort;
};

struct GemmParams {
  const float* weight_scale;
  const float* input_scale;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* residual;
  const __nv_bfloat16* multiply;
  __nv_bfloat16* output;
  int m, n, k, use_silu;  // k in bytes of a row
  int bn;                 // columns of a tile, a multiple of 32
  float output_scale;     // bf16 form only
  int adapter_chunks[kMaxAdapters];  // ADAPTED form: chunks of 64 columns of each adapter's rank
  uint32_t* status;
};

// Operands of the adapters' products, bf16: the compressed activations [M, rank] and the expansion [N, rank].
struct AdapterMaps {
  CUtensorMap compressed[kMaxAdapters], expansion[kMaxAdapters];
};

__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

// ---- CTA pairs
__device__ __forceinline__ uint32_t pair_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void pair_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// address of the leader CTA's copy of a shared-memory object
__device__ __forceinline__ uint32_t leader_address(const void* p) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(smem_u32(p)));
  return r;
}
__device__ __forceinline__ void leader_arrive(uint32_t leader_bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(leader_bar) : "memory");
}
// a copy into this CTA's shared memory that reports to a barrier of either CTA of the pair
__device__ __forceinline__ void tma_load_pair(void* dst, const void* tmap, uint32_t bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(dst)),
      "l"(tmap), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
__device__ __forceinline__ void tma_store_3d(const void* tmap, const void* src, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(tmap),
               "r"(smem_u32(src)), "r"(c0), "r"(c1), "r"(c2)
               : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
// until at most PENDING of this thread's latest stores still read their source
template <int PENDING>
__device__ __forceinline__ void tma_store_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(PENDING) : "memory");
}
// the commit arrives at the barrier of the same offset in both CTAs
__device__ __forceinline__ void commit_pair(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          smem_u32(bar)),
      "h"(static_cast<uint16_t>(3))
      : "memory");
}
// D[tmem of both] (+)= A * B over 128 bytes of K: four MMAs, 32 bytes apart in both operands
template <bool BF16>
__device__ __forceinline__ void mma_pair_chunk(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
#define NOB_MMA4(KIND)                                                                    \
  asm volatile(                                                                           \
      "{\n\t.reg .pred p0, p1;\n\t"                                                       \
      "setp.ne.b32 p0, %2, 0;\n\tsetp.eq.b32 p1, 0, 0;\n\t"                               \
      "tcgen05.mma.cta_group::2.kind::" KIND " [%0], %3, %7, %1, p0;\n\t"                 \
      "tcgen05.mma.cta_group::2.kind::" KIND " [%0], %4, %8, %1, p1;\n\t"                 \
      "tcgen05.mma.cta_group::2.kind::" KIND " [%0], %5, %9, %1, p1;\n\t"                 \
      "tcgen05.mma.cta_group::2.kind::" KIND " [%0], %6, %10, %1, p1;\n\t}" ::"r"(d),     \
      "r"(idesc), "r"(accumulate), "l"(a), "l"(a + 2), "l"(a + 4), "l"(a + 6), "l"(b), "l"(b + 2), "l"(b + 4), \
      "l"(b + 6)                                                                          \
      : "memory")
  if constexpr (BF16) {
    NOB_MMA4("f16");
  } else {
    NOB_MMA4("i8");
  }
#undef NOB_MMA4
}

template <bool BF16, bool ADAPTED>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
matmul_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
              const __grid_constant__ CUtensorMap map_residual, const __grid_constant__ CUtensorMap map_output,
              const __grid_constant__ AdapterMaps maps, const GemmParams P) {
  extern __shared__ uint8_t smem_raw[];
  GemmShared& S = *reinterpret_cast<GemmShared*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = static_cast<int>(pair_rank());
  volatile uint32_t* abort_flag = &S.abort;
  uint32_t* status = P.status;
  const int bn = P.bn;
  const int m_tiles = (P.m + kBM - 1) / kBM, n_tiles = (P.n + bn - 1) / bn;
  const int num_tiles = m_tiles * n_tiles;
  const int first_tile = blockIdx.x >> 1, tile_stride = gridDim.x >> 1;
  const int k_chunks = (P.k + kBK - 1) / kBK;
  const int adapter_at = min(kAdapterDelay, k_chunks - 1);  // chunk of a tile ahead of which the tile before is completed

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&S.full[s], 1);
      mbar_init(&S.empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&S.acc_full[b], 1);
      mbar_init(&S.acc_empty[b], 2 * kEpilogueWarps);
      mbar_init(&S.acc_scaled[b], 2 * kEpilogueWarps);
      mbar_init(&S.adapter_full[b], 1);
    }
    for (int w = 0; w < kEpilogueWarps; ++w)
      for (int i = 0; i < kStagingTiles; ++i) mbar_init(&S.residual_full[w][i], 1);
    S.abort = 0;
    mbar_fence_init();
  }
  if (warp == 0) {
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&S.tmem_base)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  __syncwarp();
  pair_sync();  // the peer's barriers exist before anything reports to them
  tc_fence_after();
  const uint32_t tmem = S.tmem_base;
  // Launched as a programmatic dependent: everything above happens while the kernel before it drains.  All CTAs are
  // resident at once, so the next kernel may be brought up from here on.
  pdl_wait();
  pdl_release();

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (lane == 0) {
      tma_prefetch_desc(&map_a);
      tma_prefetch_desc(&map_b);
      const uint32_t stage_bytes = static_cast<uint32_t>(kABytes + bn / 2 * kBK);
      int issued = 0;
      bool ok = true;
      auto load = [&](const CUtensorMap* a, const CUtensorMap* b, int column, int m0, int n0) {
        const int st = issued % kStages;
        if (issued >= kStages) {
          ok = mbar_wait(&S.empty[st], ((issued / kStages) - 1) & 1, abort_flag, status, kWaitTimeoutRing);
          if (!ok) return;
        }
        // the phase cannot complete before the leader's arrival, so the follower's bytes may come first
        if (rank == 0) mbar_expect_tx(&S.full[st], 2 * stage_bytes);
        const uint32_t bar = leader_address(&S.full[st]);
        tma_load_pair(S.a[st], a, bar, column, m0, 0);
        tma_load_pair(S.b[st], b, bar, column, n0, 0);
        ++issued;
      };
      auto load_adapters = [&](int tile) {
        const int m0 = (tile / n_tiles) * kBM + rank * (kBM / 2), n0 = (tile % n_tiles) * bn + rank * (bn / 2);
        for (int i = 0; i < kMaxAdapters; ++i)
          for (int c = 0; ok && c < P.adapter_chunks[i]; ++c)
            load(&maps.compressed[i], &maps.expansion[i], c * (kBK / 2), m0, n0);
      };
      for (int tile = first_tile; ok && tile < num_tiles; tile += tile_stride) {
        const int m0 = (tile / n_tiles) * kBM + rank * (kBM / 2), n0 = (tile % n_tiles) * bn + rank * (bn / 2);
        for (int kc = 0; ok && kc < k_chunks; ++kc) {
          if (ADAPTED && !BF16 && kc == adapter_at && tile != first_tile) load_adapters(tile - tile_stride);
          constexpr int kElementsPerChunk = BF16 ? kBK / 2 : kBK;
          if (ok) load(&map_a, &map_b, kc * kElementsPerChunk, m0, n0);
        }
        if (ADAPTED && (BF16 || tile + tile_stride >= num_tiles)) load_adapters(tile);
      }
      // the last commits have reported here before this CTA's barriers go away
      for (int i = issued > kStages ? issued - kStages : 0; ok && i < issued; ++i)
        ok = mbar_wait(&S.empty[i % kStages], (i / kStages) & 1, abort_flag, status, kWaitTimeoutRing);
    }
  } else if (warp == 1) {
    // ------------------------------------------ tcgen05 issuer, the leader's: warp-uniform flow, one elected lane
    if (rank == 0) {
      const uint32_t idesc = BF16 ? umma_idesc(kDF32, kFmtBF16, kFmtBF16, 0, 0, kBM, bn)
                                  : umma_idesc(kDS32, kFmtS8, kFmtS8, 0, 0, kBM, bn);
      const uint64_t desc = umma_smem_desc(0, 16, 1024, kSwizzle128B);
      const uint64_t a0 = desc + (smem_u32(S.a[0]) >> 4), b0 = desc + (smem_u32(S.b[0]) >> 4);
      int taken = 0, round = 0;
      bool ok = true;
      // the next stage of the ring, into accumulator `d`
      auto multiply = [&](auto bf16_tag, uint32_t d, uint32_t instruction, bool accumulate, uint64_t* then) {
        const int st = taken % kStages;
        ok = warp_rest(&S.full[st], (taken / kStages) & 1, abort_flag, status, kWaitTimeoutLoad);
        if (!ok) return;
        tc_fence_after();
        if (elect_one()) {
          mma_pair_chunk<decltype(bf16_tag)::value>(d, a0 + st * (kABytes >> 4), b0 + st * (kBBytes >> 4), instruction,
                                                    accumulate ? 1u : 0u);
          commit_pair(&S.empty[st]);
          if (then) commit_pair(then);
        }
        __syncwarp();
        ++taken;
      };
      const int adapter_chunks = ADAPTED ? P.adapter_chunks[0] + P.adapter_chunks[1] : 0;
      // int8: the adapters of the tile of round `r`, on top of its scaled fp32 accumulator
      auto adapters = [&](int r) {
        const int buf = r & 1;
        ok = warp_rest(&S.acc_scaled[buf], (r >> 1) & 1, abort_flag, status, kWaitTimeoutSoftmax);
        if (!ok) return;
        tc_fence_after();
        for (int c = 0; ok && c < adapter_chunks; ++c)
          multiply(std::true_type{}, tmem + buf * kMaxBN, umma_idesc(kDF32, kFmtBF16, kFmtBF16, 0, 0, kBM, bn), true,
                   c + 1 == adapter_chunks ? &S.adapter_full[buf] : nullptr);
      };
      for (int tile = first_tile; ok && tile < num_tiles; tile += tile_stride, ++round) {
        const int buf = round & 1;
        if (round >= 2) {  // both CTAs' epilogues must have drained this accumulator (its (round / 2)-th use)
          ok = warp_rest(&S.acc_empty[buf], ((round >> 1) - 1) & 1, abort_flag, status, kWaitTimeoutSoftmax);
          if (!ok) break;
          tc_fence_after();
        }
        const uint32_t d = tmem + buf * kMaxBN;
        const int chunks = k_chunks + (BF16 ? adapter_chunks : 0);
        for (int kc = 0; ok && kc < chunks; ++kc) {
          if (ADAPTED && !BF16 && kc == adapter_at && round > 0) adapters(round - 1);
          if (ok) multiply(std::bool_constant<BF16>{}, d, idesc, kc > 0, kc + 1 == chunks ? &S.acc_full[buf] : nullptr);
        }
        if (ADAPTED && !BF16 && ok && tile + tile_stride >= num_tiles) adapters(round);
      }
    }
  } else {
    // ------------------------------------------------------------- epilogue warps
    const int quarter = warp & 3;        // TMEM lanes [32 quarter, 32 quarter + 32)
    const int group = (warp - 2) >> 2;   // steps group, group + 2, ... of a tile
    const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
    uint8_t(*staging)[kStagingBytes] = S.staging[warp - 2];
    uint64_t* residual_full = S.residual_full[warp - 2];
    const int steps = bn / kStep;
    const int row_in_tile = rank * (kBM / 2) + quarter * 32;  // of the warp's first row
    int used = 0;  // steps that lie inside the output: number `used` works in staging tile used % kStagingTiles
    // residual tiles requested so far, and the step the next request looks at
    int requested = 0, next_tile = first_tile, next_c = group;
    auto request = [&]() {
      while (next_tile < num_tiles) {
        const int row0 = (next_tile / n_tiles) * kBM + row_in_tile, col0 = (next_tile % n_tiles) * bn + next_c * kStep;
        next_c += 2;
        if (next_c >= steps) next_c = group, next_tile += tile_stride;
        if (row0 < P.m && col0 < P.n) {
          if (lane == 0) {
            const int tile = requested % kStagingTiles;
            tma_store_wait_read<1>();  // the store that last left this staging tile is at least two stores back
            mbar_expect_tx(&residual_full[tile], kStagingBytes);
            tma_load_3d(staging[tile], &map_residual, &residual_full[tile], col0, row0, 0);
          }
          ++requested;
          return;
        }
      }
    };
    if (P.residual) {
      request();
      request();
    }
    int round = 0;
    bool ok = true;
    for (int tile = first_tile; ok && tile < num_tiles; tile += tile_stride, ++round) {
      const int buf = round & 1;
      const int row0 = (tile / n_tiles) * kBM + row_in_tile, n0 = (tile % n_tiles) * bn;
      const int row = row0 + lane;
      const bool live = row < P.m;
      const float in_scale = (!BF16 && live) ? P.input_scale[row] : 0.f;
      const size_t row_offset = static_cast<size_t>(live ? row : 0) * P.n;
      ok = warp_rest(&S.acc_full[buf], (round >> 1) & 1, abort_flag, status, kWaitTimeoutMma);
      if (!ok) break;
      tc_fence_after();
      if constexpr (ADAPTED && !BF16) {
        // the products of the main operands to scaled fp32, in place, and the adapters' on top of them
#pragma unroll 1
        for (int c = group; c < steps; c += 2) {
          const int col0 = n0 + kStep * c;
          const uint32_t addr = tmem + lane_base + buf * kMaxBN + kStep * c;
          uint32_t acc[kStep];
          tmem_ld32(addr, acc);
          tc_wait_ld();
#pragma unroll
          for (int i = 0; i < kStep; i += 4) {
            const float4 ws = col0 + i < P.n ? *reinterpret_cast<const float4*>(P.weight_scale + col0 + i)
                                             : make_float4(0.f, 0.f, 0.f, 0.f);
            const float w[4] = {ws.x, ws.y, ws.z, ws.w};
#pragma unroll
            for (int k = 0; k < 4; ++k)
              acc[i + k] = __float_as_uint(__fmul_rn(__fmul_rn(static_cast<float>(static_cast<int>(acc[i + k])), w[k]), in_scale));
          }
          tmem_st32(addr, acc);
        }
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) leader_arrive(leader_address(&S.acc_scaled[buf]));
        ok = warp_rest(&S.adapter_full[buf], (round >> 1) & 1, abort_flag, status, kWaitTimeoutMma);
        if (!ok) break;
        tc_fence_after();
      }
#pragma unroll 1
      for (int c = group; c < steps; c += 2) {
        const int col0 = n0 + kStep * c;
        const bool inside = row0 < P.m && col0 < P.n;  // warp-uniform
        uint8_t* mine = staging[used % kStagingTiles] + lane * 64;
        auto piece = [&](int g) { return reinterpret_cast<uint4*>(mine + ((g ^ ((lane >> 1) & 3)) << 4)); };
        if (inside) {
          if (P.residual) {
            request();
            ok = warp_rest(&residual_full[used % kStagingTiles], (used / kStagingTiles) & 1, abort_flag, status,
                           kWaitTimeoutLoad);
          } else {
            if (lane == 0) tma_store_wait_read<kStagingTiles - 1>();
            __syncwarp();
          }
        }
        uint32_t acc[kStep];
        __syncwarp();
        tmem_ld32(tmem + lane_base + buf * kMaxBN + kStep * c, acc);
        tc_wait_ld();
        if (c + 2 >= steps) {
          // the accumulator is in registers: the issuer may start the tile after next on it
          tc_fence_before();
          __syncwarp();
          if (lane == 0) leader_arrive(leader_address(&S.acc_empty[buf]));
        }
        if (!ok) break;
        if (!inside) continue;
#pragma unroll
        for (int g = 0; g < 4; ++g) {  // 8 columns = 16 bytes of bf16 at a time
          const int col = col0 + 8 * g;
          if (col < P.n) {
            float v[8];
            if constexpr (ADAPTED) {
#pragma unroll
              for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(acc[8 * g + i]);
            } else if constexpr (BF16) {
#pragma unroll
              for (int i = 0; i < 8; ++i) v[i] = __fmul_rn(__uint_as_float(acc[8 * g + i]), P.output_scale);
            } else {
              const float4 w0 = *reinterpret_cast<const float4*>(P.weight_scale + col);
              const float4 w1 = *reinterpret_cast<const float4*>(P.weight_scale + col + 4);
              const float ws[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
              for (int i = 0; i < 8; ++i)
                v[i] = __fmul_rn(__fmul_rn(static_cast<float>(static_cast<int>(acc[8 * g + i])), ws[i]), in_scale);
            }
            if (P.bias) {
              const uint4 raw = *reinterpret_cast<const uint4*>(P.bias + col);
              const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                v[2 * i] = __fadd_rn(v[2 * i], bf16_lo(w[i]));
                v[2 * i + 1] = __fadd_rn(v[2 * i + 1], bf16_hi(w[i]));
              }
            }
            if (P.residual) {
              const uint4 raw = *piece(g);
              const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                v[2 * i] = __fadd_rn(v[2 * i], bf16_lo(w[i]));
                v[2 * i + 1] = __fadd_rn(v[2 * i + 1], bf16_hi(w[i]));
              }
            }
            if (P.use_silu) {
#pragma unroll
              for (int i = 0; i < 8; ++i) v[i] = __fdividef(v[i], 1.0f + __expf(-v[i]));
            }
            if (P.multiply) {
              const uint4 raw = live ? *reinterpret_cast<const uint4*>(P.multiply + row_offset + col) : make_uint4(0, 0, 0, 0);
              const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                v[2 * i] = __fmul_rn(v[2 * i], bf16_lo(w[i]));
                v[2 * i + 1] = __fmul_rn(v[2 * i + 1], bf16_hi(w[i]));
              }
            }
            uint32_t o[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const __nv_bfloat162 pair = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
              o[i] = *reinterpret_cast<const uint32_t*>(&pair);
            }
            *piece(g) = make_uint4(o[0], o[1], o[2], o[3]);
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) tma_store_3d(&map_output, staging[used % kStagingTiles], col0, row0, 0);  // clips past the edges
        ++used;
      }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }

  if (*abort_flag) {  // gave up: let the copies in flight land before the pair exits (a microsecond; one millisecond)
    for (const uint64_t start = global_timer_ns(); global_timer_ns() - start < 1000000ull;) {
    }
  }
  tc_fence_before();
  __syncthreads();
  __syncwarp();
  pair_sync();  // nothing of the pair reads or reports to this CTA's shared memory any more
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
}

}  // namespace
}  // namespace nob200

namespace nob200 {
namespace {

// Columns of a tile: the width whose waves over the pairs cost least.  A chunk of K takes 2 BN cycles of tensor work or,
// below 256 columns, the load of its 16 KiB + BN/2 x 128 bytes per SM at 64 bytes per cycle; a tile's start and end
// count as some chunks' worth.  Wide tiles win on long calls; a call of one short wave is spread over more pairs.
// All seven widths timed on twelve shapes (int8 and bf16, 256 to 15104 rows, rank-64 products among them): the rule takes
// the fastest in each (operators of the time of that comparison, 512 x 7168 x 5376 bf16: 44.2 us at 224, 97.3 at 64, 46.1 at
// 256; 1000 x 5376 x 7168 int8: 52.2 at 160, 58.4 at 256), with any constant from 0 to 4000 in place of the 1000 cycles.
int tile_width(int m, int n, int k_chunks, int pairs) {
  const long long m_tiles = (m + kBM - 1) / kBM;
  int best = kMaxBN;
  long long best_cost = 0;
  for (int bn = kMaxBN; bn >= kMinBN; bn -= 32) {
    const long long tiles = m_tiles * ((n + bn - 1) / bn);
    const long long waves = (tiles + pairs - 1) / pairs;
    const long long cost = waves * (static_cast<long long>(k_chunks) * (2 * bn > 256 + bn ? 2 * bn : 256 + bn) + 1000);
    if (bn == kMaxBN || cost < best_cost) best = bn, best_cost = cost;
  }
  return best;
}

// Pairs of CTAs of this kernel that the device holds at once, asked once per device and form of the kernel (both forms
// have the same function type, so the form itself is the parameter).
template <bool BF16, bool ADAPTED>
int resident_pairs(size_t smem, int device) {
  auto kernel = matmul_kernel<BF16, ADAPTED>;
  static std::atomic<int> known[64];
  if (device >= 0 && device < 64) {
    const int pairs = known[device].load(std::memory_order_relaxed);
    if (pairs > 0) return pairs;
  }
  int sms = 148, pairs = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  cudaLaunchAttribute attribute = {};
  attribute.id = cudaLaunchAttributeClusterDimension;
  attribute.val.clusterDim.x = 2, attribute.val.clusterDim.y = 1, attribute.val.clusterDim.z = 1;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(sms & ~1), config.blockDim = dim3(kThreads), config.dynamicSmemBytes = smem;
  config.attrs = &attribute, config.numAttrs = 1;
  if (cudaOccupancyMaxActiveClusters(&pairs, kernel, &config) != cudaSuccess || pairs <= 0) {
    (void)cudaGetLastError();
    pairs = sms / 2;
  }
  if (device >= 0 && device < 64) known[device].store(pairs, std::memory_order_relaxed);
  return pairs;
}

struct Adapters {  // rank 0: there is none
  const void* compressed[kMaxAdapters] = {};
  const void* expansion[kMaxAdapters] = {};
  int ranks[kMaxAdapters] = {};
};

int check_adapters(const char* name, const Adapters& adapters) {
  NOB_REQUIRE(adapters.ranks[0] > 0, "%s: rank %d of the first adapter", name, adapters.ranks[0]);
  for (int i = 0; i < kMaxAdapters; ++i) {
    NOB_REQUIRE(adapters.ranks[i] >= 0 && adapters.ranks[i] % 64 == 0, "%s: rank %d of adapter %d is no multiple of 64", name,
                adapters.ranks[i], i);
    NOB_REQUIRE(adapters.ranks[i] == 0 || (adapters.compressed[i] && adapters.expansion[i]), "%s: NULL tensor of adapter %d",
                name, i);
  }
  return kOk;
}

template <bool BF16, bool ADAPTED>
int launch_matmul(const char* name, int num_tokens, const void* input, const void* weight, int n, int k,
                  GemmParams params, void* stream, const Adapters& adapters = Adapters()) {
  const int element = BF16 ? 2 : 1;
  params.m = num_tokens;
  params.n = n;
  params.k = k * element;
  params.status = status_word_device_ptr();
  if (!params.status) return fail(kCudaError, "%s: no current CUDA device", name);

  auto kernel = matmul_kernel<BF16, ADAPTED>;
  const size_t smem = sizeof(GemmShared) + 1024;
  cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (err != cudaSuccess)
    return fail(kCudaError, "%s: cannot reserve %zu B of shared memory: %s", name, smem, cudaGetErrorString(err));
  int device = 0;
  cudaGetDevice(&device);
  const int pairs = resident_pairs<BF16, ADAPTED>(smem, device);
  params.bn = tile_width(num_tokens, n, (params.k + kBK - 1) / kBK, pairs);

  CUtensorMap ma, mb, mr, mo;
  const CUtensorMapDataType dtype = BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8;
  const uint64_t pitch = static_cast<uint64_t>(k) * element, out_pitch = static_cast<uint64_t>(n) * 2;
  int rc;
  if ((rc = make_tensor_map_3d(&ma, dtype, input, k, num_tokens, 1, pitch, pitch * num_tokens, kBK / element, kBM / 2, 1)))
    return rc;
  if ((rc = make_tensor_map_3d(&mb, dtype, weight, k, n, 1, pitch, pitch * n, kBK / element, params.bn / 2, 1))) return rc;
  auto wide = [&](CUtensorMap* map, const void* base) {
    return make_tensor_map_3d(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, base, n, num_tokens, 1, out_pitch,
                              out_pitch * num_tokens, kStep, 32, 1, CU_TENSOR_MAP_SWIZZLE_64B);
  };
  if ((rc = wide(&mo, params.output))) return rc;
  mr = mo;
  if (params.residual && (rc = wide(&mr, params.residual))) return rc;

  AdapterMaps maps = {};
  for (int i = 0; i < kMaxAdapters && adapters.ranks[i]; ++i) {
    const uint64_t rank = adapters.ranks[i];
    params.adapter_chunks[i] = adapters.ranks[i] / 64;
    if ((rc = make_tensor_map_3d(&maps.compressed[i], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, adapters.compressed[i], rank,
                                 num_tokens, 1, rank * 2, rank * 2 * num_tokens, 64, kBM / 2, 1)))
      return rc;
    if ((rc = make_tensor_map_3d(&maps.expansion[i], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, adapters.expansion[i], rank, n, 1,
                                 rank * 2, rank * 2 * n, 64, params.bn / 2, 1)))
      return rc;
  }

  const long long tiles = static_cast<long long>((num_tokens + kBM - 1) / kBM) * ((n + params.bn - 1) / params.bn);
  const int grid = 2 * static_cast<int>(tiles < pairs ? tiles : pairs);
  return launch_pdl(name, kernel, grid, kThreads, smem, stream, ma, mb, mr, mo, maps, params);
}

}  // namespace
}  // namespace nob200

namespace nob200 {
namespace {
int matmul_int8(const char* name, int num_tokens, const void* input, const void* weight, const void* bias,
                const void* residual, const void* multiply, void* output, const void* weight_scale, const void* input_scale,
                int n, int k, int use_silu, const Adapters* adapters, void* stream) {
  NOB_REQUIRE(num_tokens > 0 && n > 0 && k > 0, "%s: sizes must be positive", name);
  NOB_REQUIRE(input && weight && output && weight_scale && input_scale, "%s: NULL tensor", name);
  NOB_REQUIRE(k % 16 == 0, "%s: k (%d) must be a multiple of 16 (row pitch of the TMA tiles)", name, k);
  NOB_REQUIRE(n % 8 == 0, "%s: n (%d) must be a multiple of 8 (16-byte rows of the bf16 epilogue)", name, n);
  GemmParams params = {};
  params.weight_scale = static_cast<const float*>(weight_scale);
  params.input_scale = static_cast<const float*>(input_scale);
  params.bias = static_cast<const __nv_bfloat16*>(bias);
  params.residual = static_cast<const __nv_bfloat16*>(residual);
  params.multiply = static_cast<const __nv_bfloat16*>(multiply);
  params.output = static_cast<__nv_bfloat16*>(output);
  params.use_silu = use_silu != 0;
  if (!adapters) return launch_matmul<false, false>(name, num_tokens, input, weight, n, k, params, stream);
  if (const int rc = check_adapters(name, *adapters)) return rc;
  return launch_matmul<false, true>(name, num_tokens, input, weight, n, k, params, stream, *adapters);
}

int matmul_bf16(const char* name, int num_tokens, const void* input, const void* weight, const void* bias,
                const void* residual, const void* multiply, void* output, float output_scale, int n, int k, int use_silu,
                const Adapters* adapters, void* stream) {
  NOB_REQUIRE(num_tokens > 0 && n > 0 && k > 0, "%s: sizes must be positive", name);
  NOB_REQUIRE(input && weight && output, "%s: NULL tensor", name);
  NOB_REQUIRE(k % 8 == 0, "%s: k (%d) must be a multiple of 8 (row pitch of the TMA tiles)", name, k);
  NOB_REQUIRE(n % 8 == 0, "%s: n (%d) must be a multiple of 8 (16-byte rows of the bf16 epilogue)", name, n);
  GemmParams params = {};
  params.bias = static_cast<const __nv_bfloat16*>(bias);
  params.residual = static_cast<const __nv_bfloat16*>(residual);
  params.multiply = static_cast<const __nv_bfloat16*>(multiply);
  params.output = static_cast<__nv_bfloat16*>(output);
  params.output_scale = output_scale;
  params.use_silu = use_silu != 0;
  if (!adapters) return launch_matmul<true, false>(name, num_tokens, input, weight, n, k, params, stream);
  if (const int rc = check_adapters(name, *adapters)) return rc;
  return launch_matmul<true, true>(name, num_tokens, input, weight, n, k, params, stream, *adapters);
}
}  // namespace
}  // namespace nob200

extern "C" int nob200_matmul_int8(int num_tokens, const void* input, const void* weight, const void* bias,
                                  const void* residual, const void* multiply, void* output, const void* weight_scale,
                                  const void* input_scale, int n, int k, int use_silu, void* stream) {
  return nob200::matmul_int8("matmul_int8", num_tokens, input, weight, bias, residual, multiply, output, weight_scale,
                             input_scale, n, k, use_silu, nullptr, stream);
}

extern "C" int nob200_matmul_int8_adapters(int num_tokens, const void* input, const void* weight, const void* bias,
                                           const void* residual, const void* multiply, void* output,
                                           const void* weight_scale, const void* input_scale, int n, int k, int use_silu,
                                           const void* compressed0, const void* expansion0, int rank0,
                                           const void* compressed1, const void* expansion1, int rank1, void* stream) {
  const nob200::Adapters adapters{{compressed0, compressed1}, {expansion0, expansion1}, {rank0, rank1}};
  return nob200::matmul_int8("matmul_int8_adapters", num_tokens, input, weight, bias, residual, multiply, output,
                             weight_scale, input_scale, n, k, use_silu, &adapters, stream);
}

extern "C" int nob200_matmul_bf16(int num_tokens, const void* input, const void* weight, const void* bias,
                                  const void* residual, const void* multiply, void* output, float output_scale, int n,
                                  int k, int use_silu, void* stream) {
  return nob200::matmul_bf16("matmul_bf16", num_tokens, input, weight, bias, residual, multiply, output, output_scale, n, k,
                             use_silu, nullptr, stream);
}

extern "C" int nob200_matmul_bf16_adapters(int num_tokens, const void* input, const void* weight, const void* bias,
                                           const void* residual, const void* multiply, void* output, int n, int k,
                                           int use_silu, const void* compressed0, const void* expansion0, int rank0,
                                           const void* compressed1, const void* expansion1, int rank1, void* stream) {
  const nob200::Adapters adapters{{compressed0, compressed1}, {expansion0, expansion1}, {rank0, rank1}};
  return nob200::matmul_bf16("matmul_bf16_adapters", num_tokens, input, weight, bias, residual, multiply, output, 1.0f, n, k,
                             use_silu, &adapters, stream);
}
