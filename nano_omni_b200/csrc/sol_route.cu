// Routing of the "sol" block-sparse attention: block pooling, centroid statistics and the
// selection mask.  CUDA-core kernels (HBM-bound pooling; the router's pooled GEMM is small).
//
// Reference programs replaced:
//   sol_pool / sol_int8_fp8_pool / sol_nvfp4_pool   src/nano_omni/kernels/attention/sol/pool.py:29-62,
//       int8_fp8/sol_pool.py:25-58, nvfp4/sol_pool.py:34-67
//   sol_stats                                        src/nano_omni/kernels/attention/sol/stats.py:28-67
//   sol_nvfp4_select                                 src/nano_omni/kernels/attention/nvfp4/sol_select.py:42-120
//
// Masks are compared bit for bit with a CPU restatement, so every reduction has a fixed order:
// sums over the tokens of a block and over blocks are sequential fp32 additions in index order;
// dot products over the 128 channels are sequential acc = acc + a*b with product and sum each
// rounded to fp32 (__fmul_rn / __fadd_rn keep the compiler from fusing them); divisions and
// square roots are IEEE.
#include "common.cuh"
#include "../../include/nano_omni_b200.h"

namespace nob200 {
namespace {

constexpr float kSqrt128 = 11.313708498984761f;

// ---------------------------------------------------------------- pooling
// One CTA of 64 threads per (block, head); thread c2 owns channels 2*c2, 2*c2+1 and walks
// the block's tokens in order (4-byte loads, 256 B per token row across the CTA).
__global__ void __launch_bounds__(64)
sol_pool_kernel(const __nv_bfloat16* key, const __nv_bfloat16* value,
                const float* key_mean, __nv_bfloat16* out, int num_tokens, int heads,
                int block, int num_blocks) {
  pdl_wait();
  pdl_release();
  const int b = blockIdx.x, head = blockIdx.y, c = threadIdx.x * 2;
  const int begin = b * block, end = min(begin + block, num_tokens);
  const size_t row_stride = static_cast<size_t>(heads) * 128;
  const __nv_bfloat16* kp = key + static_cast<size_t>(begin) * row_stride + head * 128 + c;
  const __nv_bfloat16* vp = value + static_cast<size_t>(begin) * row_stride + head * 128 + c;
  float k0 = 0.f, k1 = 0.f, v0 = 0.f, v1 = 0.f;
#pragma unroll 8
  for (int t = begin; t < end; ++t, kp += row_stride, vp += row_stride) {
    const uint32_t kr = *reinterpret_cast<const uint32_t*>(kp);
    const uint32_t vr = *reinterpret_cast<const uint32_t*>(vp);
    k0 = __fadd_rn(k0, __uint_as_float(kr << 16));
    k1 = __fadd_rn(k1, __uint_as_float(kr & 0xffff0000u));
    v0 = __fadd_rn(v0, __uint_as_float(vr << 16));
    v1 = __fadd_rn(v1, __uint_as_float(vr & 0xffff0000u));
  }
  const float len = static_cast<float>(end - begin);
  const float m0 = __fdiv_rn(k0, len), m1 = __fdiv_rn(k1, len);
  const size_t plane = static_cast<size_t>(heads) * num_blocks * 128;
  const size_t at = (static_cast<size_t>(head) * num_blocks + b) * 128 + c;
  auto store = [&](size_t offset, float a, float bb) {
    *reinterpret_cast<__nv_bfloat162*>(out + offset) = __floats2bfloat162_rn(a, bb);
  };
  store(at, m0, m1);
  if (key_mean) {
    store(plane + at, __fsub_rn(m0, key_mean[head * 128 + c]), __fsub_rn(m1, key_mean[head * 128 + c + 1]));
    store(2 * plane + at, v0, v1);
  } else {
    store(plane + at, v0, v1);
  }
}

// Eight consecutive bf16 of a row as one 16-byte load where the tensor is 16-byte aligned, else one by one.  The choice
// is a template parameter: a branch around each load would keep a thread's loads from being in flight together.
template <bool ALIGNED>
__device__ __forceinline__ uint4 load8(const __nv_bfloat16* p) {
  if constexpr (ALIGNED) return *reinterpret_cast<const uint4*>(p);
  const uint16_t* h = reinterpret_cast<const uint16_t*>(p);
  auto two = [&](int i) { return static_cast<uint32_t>(h[i]) | (static_cast<uint32_t>(h[i + 1]) << 16); };
  return make_uint4(two(0), two(2), two(4), two(6));
}

// ------------------------------------------------------------- statistics
// One CTA per (head, 32 channels).  The sums over blocks are one chain of additions per channel, so all that can be
// done in parallel is the loading: 256 threads bring 512 blocks at a time into shared memory and the first warp runs
// the chains from there.  With the loads inside the chain the kernel waited for memory at every few blocks: 24 heads x
// 1024 blocks 50 us, this form 12 us.
constexpr int kStatsBlocks = 512, kStatsChannels = 32;

template <bool ALIGNED>
__global__ void __launch_bounds__(256)
sol_stats_kernel(const __nv_bfloat16* pooled, float* out, int num_blocks) {
  pdl_wait();
  pdl_release();
  __shared__ uint4 staged[kStatsBlocks][kStatsChannels / 8];
  const int head = blockIdx.x, c0 = blockIdx.y * kStatsChannels, lane = threadIdx.x;
  const __nv_bfloat16* p = pooled + static_cast<size_t>(head) * num_blocks * 128 + c0;
  float sum = -0.f, sq = -0.f;  // -0 + x = x for every x: the chains start with their first element
  for (int b0 = 0; b0 < num_blocks; b0 += kStatsBlocks) {
    const int count = min(kStatsBlocks, num_blocks - b0);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kStatsBlocks * kStatsChannels / 8 / 256; ++i) {
      const int at = threadIdx.x + 256 * i, b = at >> 2, g = at & 3;
      if (b < count) staged[b][g] = load8<ALIGNED>(p + static_cast<size_t>(b0 + b) * 128 + 8 * g);
    }
    __syncthreads();
    if (lane < kStatsChannels) {
      const __nv_bfloat16* column = reinterpret_cast<const __nv_bfloat16*>(staged) + lane;
#pragma unroll 16
      for (int b = 0; b < count; ++b) {
        const float x = __bfloat162float(column[b * kStatsChannels]);
        sum = __fadd_rn(sum, x);
        sq = __fadd_rn(sq, __fmul_rn(x, x));
      }
    }
  }
  if (lane < kStatsChannels) {
    const float n = static_cast<float>(num_blocks);
    const float mean = __fdiv_rn(sum, n);
    const float second = __fdiv_rn(sq, n);
    out[(head * 2 + 0) * 128 + c0 + lane] = mean;
    out[(head * 2 + 1) * 128 + c0 + lane] = fmaxf(__fsub_rn(second, __fmul_rn(mean, mean)), 0.f);
  }
}

// ----------------------------------------------------------------- router
// One CTA of four warps per (4 * ROWS query blocks, head).  Phase 1: the block means of Q (sequential over tokens, 16
// bytes = 8 channels per load) and their thresholds.  Phase 2: scores against 128 key blocks at a time, as a
// register-tiled product: a lane owns ROWS query blocks x 4 key blocks, and every score is the canonical chain
// acc = q[0] * k[0]; acc = acc + q[d] * k[d], d = 1..127, product and sum rounded separately (packed mul and add, two
// key blocks per instruction).  The chains leave the FMA pipe as the bound (2 * blocks^2 * heads * 128 lane operations),
// and the tile keeps shared memory below it: per channel a lane reads 16 bytes of K and, broadcast, 8 bytes per query
// block (its mean, twice) for 4 * ROWS products.  K arrives in chunks of 32 channels, converted and transposed on the
// way, the next chunk's loads in flight during the present one.  One chain pair per thread with both operands read
// from shared memory at every step, the earlier form, took 1482 us at 1024 blocks x 24 heads and 704 us at 950 x 14;
// this one 444 and 183 us.
constexpr int kSelectThreads = 128;
constexpr int kKbTile = 128;
constexpr int kDChunk = 32;

template <int ROWS>
struct SelectShared {
  float2 qdup[128][4 * ROWS];     // [channel][query block]: the mean, twice
  float kc[2][kDChunk][kKbTile];  // [channel][key block]
  float thr[4 * ROWS];
};

__device__ __forceinline__ uint64_t mul_pair(uint64_t x, uint64_t y) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y));
  return r;
}
__device__ __forceinline__ uint64_t add_pair(uint64_t x, uint64_t y) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y));
  return r;
}

template <int ROWS, bool ALIGNED>
__global__ void __launch_bounds__(kSelectThreads, 3)  // shared memory holds three; registers for 16 loads in flight
sol_select_kernel(const __nv_bfloat16* query, const __nv_bfloat16* pooled_key,
                  const float* stats, uint8_t* mask, float* scores,
                  int num_tokens, int heads, int block, int num_blocks, int num_protected, float tau) {
  pdl_wait();
  pdl_release();
  constexpr int kQb = 4 * ROWS;
  extern __shared__ __align__(16) uint8_t select_smem[];
  SelectShared<ROWS>& S = *reinterpret_cast<SelectShared<ROWS>*>(select_smem);
  const int head = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int qb0 = blockIdx.x * kQb;
  const size_t row_stride = static_cast<size_t>(heads) * 128;

  // K chunk `it`: channels 32 * (it % 4) .. of key blocks 128 * (it / 4) ..; thread r fetches key block r of the tile
  const int chunks = ((num_blocks + kKbTile - 1) / kKbTile) * (128 / kDChunk);
  uint4 next[4];
  auto fetch = [&](int it) {
    const int kb = (it / (128 / kDChunk)) * kKbTile + threadIdx.x;
    const __nv_bfloat16* p =
        pooled_key + (static_cast<size_t>(head) * num_blocks + kb) * 128 + (it % (128 / kDChunk)) * kDChunk;
#pragma unroll
    for (int i = 0; i < 4; ++i) next[i] = kb < num_blocks ? load8<ALIGNED>(p + 8 * i) : make_uint4(0, 0, 0, 0);
  };
  auto place = [&](int buffer) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t w[4] = {next[i].x, next[i].y, next[i].z, next[i].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        S.kc[buffer][8 * i + 2 * j][threadIdx.x] = __uint_as_float(w[j] << 16);
        S.kc[buffer][8 * i + 2 * j + 1][threadIdx.x] = __uint_as_float(w[j] & 0xffff0000u);
      }
    }
  };
  fetch(0);

  // phase 1a: block means of Q; a thread owns 8 channels of one query block per pass
#pragma unroll 1
  for (int qi = threadIdx.x >> 4; qi < kQb; qi += kSelectThreads / 16) {
    const int c = (threadIdx.x & 15) * 8, qb = qb0 + qi;
    float acc[8] = {};
    if (qb < num_blocks) {
      const int begin = qb * block, end = min(begin + block, num_tokens);
      const __nv_bfloat16* p = query + static_cast<size_t>(begin) * row_stride + head * 128 + c;
#pragma unroll 16
      for (int t = begin; t < end; ++t, p += row_stride) {
        const uint4 raw = load8<ALIGNED>(p);
        const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[2 * j] = __fadd_rn(acc[2 * j], __uint_as_float(w[j] << 16));
          acc[2 * j + 1] = __fadd_rn(acc[2 * j + 1], __uint_as_float(w[j] & 0xffff0000u));
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] = __fdiv_rn(acc[j], static_cast<float>(end - begin));
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) S.qdup[c + j][qi] = make_float2(acc[j], acc[j]);
  }
  place(0);
  __syncthreads();
  // phase 1b: thresholds (one thread per query block)
  if (mask && threadIdx.x < kQb) {
    const float* mu = stats + (head * 2 + 0) * 128;
    const float* var = stats + (head * 2 + 1) * 128;
    float m = -0.f, v = -0.f;
#pragma unroll 16
    for (int d = 0; d < 128; ++d) {
      const float q = S.qdup[d][threadIdx.x].x;
      m = __fadd_rn(m, __fmul_rn(q, mu[d]));
      v = __fadd_rn(v, __fmul_rn(__fmul_rn(q, q), var[d]));
    }
    const float mean = __fdiv_rn(m, kSqrt128);
    const float variance = __fdiv_rn(v, 128.0f);
    const float deviation = __fsqrt_rn(__fadd_rn(fmaxf(variance, 0.f), 1e-6f));
    S.thr[threadIdx.x] = __fadd_rn(mean, __fmul_rn(tau, deviation));
  }
  __syncthreads();
  // phase 2
  constexpr uint64_t kNegativeZeros = 0x8000000080000000ull;  // -0 + x = x: the chains start with their first product
  uint64_t acc[ROWS][2];
#pragma unroll
  for (int r = 0; r < ROWS; ++r) acc[r][0] = acc[r][1] = kNegativeZeros;
#pragma unroll 1
  for (int it = 0; it < chunks; ++it) {
    if (it + 1 < chunks) fetch(it + 1);
    const int d0 = (it % (128 / kDChunk)) * kDChunk;
    const float(*kc)[kKbTile] = S.kc[it & 1];
#pragma unroll 4
    for (int d = 0; d < kDChunk; ++d) {
      const ulonglong2 k = *reinterpret_cast<const ulonglong2*>(&kc[d][4 * lane]);
      uint64_t q[ROWS];
#pragma unroll
      for (int r = 0; r < ROWS; r += 2) {
        const ulonglong2 two = *reinterpret_cast<const ulonglong2*>(&S.qdup[d0 + d][warp * ROWS + r]);
        q[r] = two.x;
        q[r + 1] = two.y;
      }
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        acc[r][0] = add_pair(acc[r][0], mul_pair(q[r], k.x));
        acc[r][1] = add_pair(acc[r][1], mul_pair(q[r], k.y));
      }
    }
    if (d0 + kDChunk == 128) {  // the scores of this tile of key blocks are complete
      const int kb = (it / (128 / kDChunk)) * kKbTile + 4 * lane;
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        const int qi = warp * ROWS + r, qb = qb0 + qi;
        float score[4];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          score[2 * j] = __fdiv_rn(__uint_as_float(static_cast<uint32_t>(acc[r][j])), kSqrt128);
          score[2 * j + 1] = __fdiv_rn(__uint_as_float(static_cast<uint32_t>(acc[r][j] >> 32)), kSqrt128);
          acc[r][j] = kNegativeZeros;
        }
        if (qb < num_blocks && kb < num_blocks) {
          const size_t at = (static_cast<size_t>(qb) * heads + head) * num_blocks + kb;
          const int count = min(4, num_blocks - kb);
          if (scores) {
            if (count == 4 && (reinterpret_cast<uintptr_t>(scores + at) & 15) == 0) {
              *reinterpret_cast<float4*>(scores + at) = make_float4(score[0], score[1], score[2], score[3]);
            } else {
#pragma unroll
              for (int j = 0; j < 4; ++j)
                if (j < count) scores[at + j] = score[j];
            }
          }
          if (mask) {
            uint32_t bits = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const int delta = qb - (kb + j);
              const bool keep = kb + j < num_protected || score[j] > S.thr[qi] || (delta >= -1 && delta <= 1);
              bits |= (keep ? 1u : 0u) << (8 * j);
            }
            if (count == 4 && (reinterpret_cast<uintptr_t>(mask + at) & 3) == 0) {
              *reinterpret_cast<uint32_t*>(mask + at) = bits;
            } else {
#pragma unroll
              for (int j = 0; j < 4; ++j)
                if (j < count) mask[at + j] = static_cast<uint8_t>(bits >> (8 * j));
            }
          }
        }
      }
    }
    if (it + 1 < chunks) place((it + 1) & 1);  // its last readers passed the barrier of the previous chunk
    __syncthreads();
  }
}

// ------------------------------------------------------------------ top-k
// One warp per (query block, head): keep the k highest scores among the unprotected key blocks (ties: lower block index
// first) plus every protected block.  Only the set is asked for, not its order, so the warp holds the row in registers
// as order-preserving integers and finds the k-th largest bit by bit (count the elements at or above a candidate; done
// early when a candidate separates exactly k).  Sorting the row in shared memory, the earlier form, took 1205 us for
// 24576 rows of 1024; this one 230 us.
constexpr int kTopkMax = 2048;
constexpr int kTopkWarps = 4;

template <int PER_LANE>
__global__ void __launch_bounds__(32 * kTopkWarps)
sol_topk_kernel(const float* scores, uint8_t* mask, int rows, int num_blocks,
                int num_protected, int keep) {
  pdl_wait();
  pdl_release();
  const int row = blockIdx.x * kTopkWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= rows) return;
  const size_t base = static_cast<size_t>(row) * num_blocks;
  uint32_t key[PER_LANE];  // key block 32 * j + lane; larger float -> larger unsigned; 0 where nothing competes
#pragma unroll
  for (int j = 0; j < PER_LANE; ++j) {
    const int i = 32 * j + lane;
    key[j] = 0;
    if (i < num_blocks && i >= num_protected) {
      float x = scores[base + i];
      if (x == 0.f) x = 0.f;  // -0 and +0 rank equal
      const uint32_t bits = __float_as_uint(x);
      key[j] = (bits & 0x80000000u) ? ~bits : (bits | 0x80000000u);
    }
  }
  const bool all = keep >= num_blocks - num_protected;
  uint32_t cut = 0;    // at least `keep` elements are at or above it
  bool exact = false;  // exactly `keep` are
  for (int bit = 31; !all && !exact && bit >= 0; --bit) {
    const uint32_t candidate = cut | (1u << bit);
    int mine = 0;
#pragma unroll
    for (int j = 0; j < PER_LANE; ++j) mine += key[j] >= candidate;
    const int count = __reduce_add_sync(0xffffffffu, mine);
    if (count >= keep) cut = candidate;
    exact = count == keep;
  }
  int ties = 0;  // elements equal to the cut that belong to the k
  if (!all && !exact) {
    int mine = 0;
#pragma unroll
    for (int j = 0; j < PER_LANE; ++j) mine += key[j] > cut;
    ties = keep - __reduce_add_sync(0xffffffffu, mine);
  }
  int seen = 0;
#pragma unroll
  for (int j = 0; j < PER_LANE; ++j) {
    const int i = 32 * j + lane;
    const bool competes = i < num_blocks && i >= num_protected;
    bool chosen = i < num_protected || (competes && (all || (exact ? key[j] >= cut : key[j] > cut)));
    if (!all && !exact) {  // warp-uniform
      const uint32_t equal = __ballot_sync(0xffffffffu, competes && key[j] == cut);
      if (competes && key[j] == cut && seen + __popc(equal & ((1u << lane) - 1u)) < ties) chosen = true;
      seen += __popc(equal);
    }
    if (i < num_blocks) mask[base + i] = chosen ? 1 : 0;
  }
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

struct SelectLaunch {
  const __nv_bfloat16 *query, *pooled_key;
  const float* stats;
  uint8_t* mask;
  float* scores;
  int num_tokens, heads, block, num_blocks, num_protected;
  float tau;

  template <int ROWS, bool ALIGNED>
  int run_rows(cudaStream_t stream, const char* name) const {
    const size_t smem = sizeof(SelectShared<ROWS>);
    auto* kernel = sol_select_kernel<ROWS, ALIGNED>;
    const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess)
      return fail(kCudaError, "%s: cannot reserve %zu B of shared memory: %s", name, smem, cudaGetErrorString(err));
    return launch_pdl(name, kernel, dim3((num_blocks + 4 * ROWS - 1) / (4 * ROWS), heads), kSelectThreads, smem, stream,
                      query, pooled_key, stats, mask, scores, num_tokens, heads, block, num_blocks, num_protected, tau);
  }

  // 8 query blocks per lane read the least shared memory per product, 4 make twice the CTAs: where 32-block CTAs
  // would be fewer than two per SM the means of Q, a latency-bound pass, are what counts.
  int run(cudaStream_t stream, const char* name) const {
    const long long ctas = static_cast<long long>((num_blocks + 31) / 32) * heads;
    const bool aligned = aligned16(query) && aligned16(pooled_key);
    if (ctas >= 2 * 148) return aligned ? run_rows<8, true>(stream, name) : run_rows<8, false>(stream, name);
    return aligned ? run_rows<4, true>(stream, name) : run_rows<4, false>(stream, name);
  }
};

}  // namespace
}  // namespace nob200

using namespace nob200;

extern "C" int nob200_sol_pool(int num_tokens, const void* key, const void* value, const void* key_mean, void* output,
                               int heads, int block, void* stream) {
  NOB_REQUIRE(num_tokens > 0 && heads > 0, "sol_pool: sizes must be positive");
  NOB_REQUIRE(block == 64 || block == 128, "sol_pool: block must be 64 or 128 (got %d)", block);
  NOB_REQUIRE(key && value && output, "sol_pool: NULL tensor");
  NOB_REQUIRE(heads <= 65535, "sol_pool: heads exceed the grid limit");
  const int nb = (num_tokens + block - 1) / block;
  return launch_pdl("sol_pool", sol_pool_kernel, dim3(nb, heads), 64, 0, stream,
                    static_cast<const __nv_bfloat16*>(key), static_cast<const __nv_bfloat16*>(value),
                    static_cast<const float*>(key_mean), static_cast<__nv_bfloat16*>(output), num_tokens, heads, block, nb);
}

extern "C" int nob200_sol_stats(const void* pooled, void* output, int heads, int num_blocks, void* stream) {
  NOB_REQUIRE(heads > 0 && num_blocks > 0, "sol_stats: sizes must be positive");
  NOB_REQUIRE(pooled && output, "sol_stats: NULL tensor");
  auto* kernel = aligned16(pooled) ? sol_stats_kernel<true> : sol_stats_kernel<false>;
  return launch_pdl("sol_stats", kernel, dim3(heads, 128 / kStatsChannels), 256, 0, stream,
                    static_cast<const __nv_bfloat16*>(pooled), static_cast<float*>(output), num_blocks);
}

extern "C" size_t nob200_sol_select_workspace_bytes(int num_tokens, int heads, int block, int topk_blocks) {
  if (topk_blocks <= 0 || num_tokens <= 0 || heads <= 0 || block <= 0) return 0;
  const size_t nb = (static_cast<size_t>(num_tokens) + block - 1) / block;
  return nb * nb * heads * sizeof(float);
}

extern "C" int nob200_sol_select(int num_tokens, int num_protected_blocks, const void* query, const void* pooled_key,
                                 const void* stats, void* output, int heads, float tau, int block,
                                 int topk_blocks, void* workspace, size_t workspace_bytes, void* stream) {
  NOB_REQUIRE(num_tokens > 0 && heads > 0, "sol_select: sizes must be positive");
  NOB_REQUIRE(block == 64 || block == 128, "sol_select: block must be 64 or 128 (got %d)", block);
  NOB_REQUIRE(query && pooled_key && output, "sol_select: NULL tensor");
  NOB_REQUIRE(heads <= 65535, "sol_select: heads exceed the grid limit");
  const int nb = (num_tokens + block - 1) / block;
  NOB_REQUIRE(num_protected_blocks >= 0 && num_protected_blocks <= nb,
              "sol_select: num_protected_blocks %d outside [0, %d]", num_protected_blocks, nb);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  SelectLaunch launch = {static_cast<const __nv_bfloat16*>(query), static_cast<const __nv_bfloat16*>(pooled_key),
                         static_cast<const float*>(stats), nullptr, nullptr, num_tokens, heads, block, nb,
                         num_protected_blocks, tau};
  if (topk_blocks <= 0) {
    NOB_REQUIRE(stats, "sol_select: threshold routing needs the stats tensor");
    launch.mask = static_cast<uint8_t*>(output);
    return launch.run(s, "sol_select");
  }
  NOB_REQUIRE(nb <= kTopkMax, "sol_select: top-k routing supports at most %d blocks (got %d)", kTopkMax, nb);
  const size_t need = nob200_sol_select_workspace_bytes(num_tokens, heads, block, topk_blocks);
  NOB_REQUIRE(workspace && workspace_bytes >= need, "sol_select: top-k routing needs %zu B of workspace, %zu B given",
              need, workspace_bytes);
  launch.scores = static_cast<float*>(workspace);  // statistics are not read by top-k routing
  int rc = launch.run(s, "sol_select(scores)");
  if (rc) return rc;
  const int keep = topk_blocks < nb ? topk_blocks : nb;
  const int rows = nb * heads;  // at most 2048 * 65535
  auto* kernel = nb <= 256    ? sol_topk_kernel<8>
                 : nb <= 512  ? sol_topk_kernel<16>
                 : nb <= 1024 ? sol_topk_kernel<32>
                              : sol_topk_kernel<64>;
  return launch_pdl("sol_select(topk)", kernel, (rows + kTopkWarps - 1) / kTopkWarps, 32 * kTopkWarps, 0, stream,
                    launch.scores, static_cast<uint8_t*>(output), rows, nb, num_protected_blocks, keep);
}
