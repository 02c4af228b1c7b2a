// Dense non-causal int8-QK / fp8-PV attention forward for head_dim 128 on sm_100a.
//
// Replaces the reference program dense_int8_fp8_attention
// (src/nano_omni/kernels/attention/int8_fp8/dense.py:21-315):
//   S = Q8 K8^T in int32; s = S * qscale[row/32] * kscale[key/64] * log2e/sqrt(128);
//   online softmax in fp32; P scaled into the e4m3 range and rounded to e4m3;
//   O += P8 V8 (fp32 accumulation here, fp16 partials in the reference);
//   out = O * vscale[channel] / l.
// Operands: Q int8 [heads, Tq32, 128], K int8 [heads, Tk64, 128], V e4m3 [heads, 128, Tk64]
// (channel-major; inside every 16 tokens, stored position p holds token
// [0,1,8,9,2,3,10,11,4,5,12,13,6,7,14,15][p]), f32 scales, output bf16 [Tq, heads*128].
//
// CTA organisation of the bf16 kernel: 256 query rows of one head per CTA (tiles A and B), key tiles of 128, warps
// 0-3 / 4-7 softmax for A / B with one thread per row, warp 8 TMA producer, warp 9 issues the score MMAs, warp 10 the
// value MMAs.  QK is kind::i8 (K = 32 per MMA, 4 per tile) into ONE score buffer that A and B use in turn: it is free
// again as soon as a tile's softmax warps hold their rows in registers, so the next scores are computed during the
// exponentials.  PV is kind::f8f6f4 with P (e4m3, four keys per 32-bit TMEM column, two buffers per query tile) as the
// TMEM operand and the V tile K-major straight from TMA.
// TMEM columns: S 0-127, P_A 128-191, P_B 192-255, O_A 256-383, O_B 384-511.
// int32 scores are converted to fp32 exactly (|S| <= 128*128*128 < 2^24) before the row maximum.
// P is scaled by 448 / 2^3 and the running maximum is raised when it grew by more than
// 2^3, so P never exceeds 448 (e4m3's largest finite value).
#include <cuda.h>

#include "common.cuh"
#include "fa_common.cuh"
#include "tensor_map.cuh"
#include "../../include/nano_omni_b200.h"

namespace nob200 {
namespace {

constexpr int kTile = 128;
constexpr int kTileBytes = kTile * 128;  // 16 KiB: 128 rows of 128 one-byte elements
constexpr int kStages = 8;
constexpr int kThreads = 384;
constexpr int kProducerWarp = 8;
constexpr int kMmaWarp = 9;  // issues the score MMAs (S = Q K^T)
constexpr int kPvWarp = 10;  // issues the value MMAs (O += P V)
constexpr int kKeptScales = 8192;  // key scales (one per 64 keys) a CTA keeps in shared memory: 524288 keys
constexpr uint32_t kTmemCols = 512;
constexpr float kHeadroomLog2 = 3.0f;              // P <= 448 while the stale maximum lags by <= 2^3
constexpr float kLog2PScale = 8.807354922057604f - kHeadroomLog2;  // log2(448) - 3

constexpr uint32_t kColS = 0, kColP = 128, kColO = 256;  // P_t(j) at kColP + 64 t + 32 (j & 1), O_t at kColO + 128 t

struct __align__(1024) Shared {
  uint8_t q[2][kTileBytes];
  uint8_t kv[kStages][kTileBytes];
  uint64_t q_full;
  uint64_t kv_full[kStages];
  uint64_t kv_empty[kStages];
  uint64_t s_full[2];      // scores of tile t are in TMEM
  uint64_t s_taken[2];     // the softmax warps of tile t hold them in registers: the buffer is free
  uint64_t p_full[2][2];   // P_t(j) is written, by parity of j (the softmax may run a tile ahead of the value issuer)
  uint64_t pv_done[2][2];  // O_t += P_t(j) V_j is complete, by parity of j: that P buffer is free, O_t may be rescaled
  KeySplit::Share share;
  uint32_t tmem_base;
  uint32_t abort;
  float key_scale[kKeptScales];
};

// Register split after setmaxnreg: the CTA owns 384 x 168 registers; an increase beyond them would never return.
// Every register the issuing warps can spare goes to the softmax (88 instead of 56: +4 %, 104: +8 % in time).
constexpr int kServiceRegs = 56;
constexpr int kSoftmaxRegs = (384 * 168 - 128 * kServiceRegs) / 256 / 8 * 8;
static_assert(256 * kSoftmaxRegs + 128 * kServiceRegs <= 384 * 168, "setmaxnreg split exceeds the registers the CTA owns");

// four e4m3 bytes, `a` in bits 0-7
__device__ __forceinline__ uint32_t pack_e4m3x4(float a, float b, float c, float d) {
  uint32_t r;
  asm("{\n\t.reg .b16 lo, hi;\n\t"
      "cvt.rn.satfinite.e4m3x2.f32 lo, %2, %1;\n\t"
      "cvt.rn.satfinite.e4m3x2.f32 hi, %4, %3;\n\t"
      "mov.b32 %0, {lo, hi};\n\t}"
      : "=r"(r)
      : "f"(a), "f"(b), "f"(c), "f"(d));
  return r;
}
__global__ void __launch_bounds__(kThreads, 1)
fa_fwd_i8f8_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                   const __grid_constant__ CUtensorMap map_v, const float* query_scale,
                   const float* key_scale, const float* value_scale,
                   __nv_bfloat16* __restrict__ out, int num_query_tokens, int num_kv_tokens, int heads,
                   float scale_log2, uint32_t* status, int query_block, int key_block, const KeySplit split) {
  extern __shared__ uint8_t smem_raw[];
  Shared& S = *reinterpret_cast<Shared*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int n_kv_total = (num_kv_tokens + kTile - 1) / kTile;
  const KeySplit::Share share = split.share(blockIdx.x, n_kv_total);
  const int head = share.head;
  const int q0 = share.q_tile * split.unit_rows;
  const bool two = split.unit_rows > kTile && q0 + kTile < num_query_tokens;
  const int kv_begin = share.kv_begin;
  const int n_kv = share.kv_end - kv_begin;
  volatile uint32_t* abort_flag = &S.abort;

  if (threadIdx.x == 0) {
    mbar_init(&S.q_full, 1);
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&S.kv_full[s], 1);
      mbar_init(&S.kv_empty[s], 1);
    }
    for (int t = 0; t < 2; ++t) {
      mbar_init(&S.s_full[t], 1);
      mbar_init(&S.s_taken[t], 4);
      mbar_init(&S.p_full[t][0], 4);
      mbar_init(&S.p_full[t][1], 4);
      mbar_init(&S.pv_done[t][0], 1);
      mbar_init(&S.pv_done[t][1], 1);
    }
    S.share = share;
    S.abort = 0;
    mbar_fence_init();
  }
  if (warp == kProducerWarp) {
    tmem_alloc(&S.tmem_base, kTmemCols);
    tmem_relinquish();
  }
  pdl_wait();  // launched as a programmatic dependent: the set-up above overlaps the kernel before

  // Key scales of this CTA's keys, one per 64 keys (scales per `key_block`, 64 or 128 tokens), to shared memory: read
  // from global memory inside the loop they cost 4 % of the kernel.  Behind the wait, because the kernel before may be
  // the one that writes them.  Head and block count are worked out again for the few calls that read past the kept
  // scales: kept in registers over the key loop, they spill there.
  auto key_scale_of = [&](int in_head, int half64) {
    const int k_blocks = (num_kv_tokens + key_block - 1) / key_block;
    return key_scale[static_cast<size_t>(in_head) * k_blocks + min(key_block == 128 ? half64 >> 1 : half64, k_blocks - 1)];
  };
  for (int i = threadIdx.x; i < min(2 * n_kv, kKeptScales); i += kThreads) S.key_scale[i] = key_scale_of(head, 2 * kv_begin + i);

  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = S.tmem_base;
  pdl_release();  // the merge of the shares may be scheduled behind the last CTAs

  if (warp >= 8) {
    reg_dealloc<kServiceRegs>();
    if (warp == kProducerWarp) {
      // ------------------------------------------------------------ TMA producer
      if (lane == 0) {
        tma_prefetch_desc(&map_q);
        tma_prefetch_desc(&map_k);
        tma_prefetch_desc(&map_v);
        mbar_expect_tx(&S.q_full, two ? 2 * kTileBytes : kTileBytes);
        tma_load_3d(S.q[0], &map_q, &S.q_full, 0, q0, head);
        if (two) tma_load_3d(S.q[1], &map_q, &S.q_full, 0, q0 + kTile, head);
        const int loads = 2 * n_kv;  // K_j at 2j, V_j at 2j+1
        int issued = 0;
        for (int i = 0; i < loads; ++i) {
          const int st = i % kStages;
          if (i >= kStages) {
            if (!mbar_wait(&S.kv_empty[st], ((i / kStages) - 1) & 1, abort_flag, status, kWaitTimeoutRing)) break;
          }
          mbar_expect_tx(&S.kv_full[st], kTileBytes);
          const int tok = (kv_begin + (i >> 1)) * kTile;
          if (i & 1) {
            tma_load_3d(S.kv[st], &map_v, &S.kv_full[st], tok, 0, head);  // [channel][token] tile
          } else {
            tma_load_3d(S.kv[st], &map_k, &S.kv_full[st], 0, tok, head);  // [token][channel] tile
          }
          issued = i + 1;
        }
        if (*abort_flag) {
          for (int i = (issued > kStages ? issued - kStages : 0); i < issued; ++i) {
            uint64_t* bar = &S.kv_full[i % kStages];
            const uint32_t parity = (i / kStages) & 1;
            for (int spin = 0; spin < (1 << 16) && !mbar_try_wait(bar, parity); ++spin) {
            }
          }
        }
      }
    } else if (warp == kMmaWarp || warp == kPvWarp) {
      // --------------------------------------------------------- tcgen05 issuers
      // Whole warps in warp-uniform control flow, one elected lane issues a group of MMAs as one asm statement (see
      // elect_one()).  The tensor pipe is busy less than half of the time, so the two warps issue without regard to
      // each other.
      // All smem operands are K-major tiles of 128 rows x 128 bytes (one swizzle atom per row).
      const uint64_t desc = umma_smem_desc(0, 16, 1024, kSwizzle128B);
      const uint64_t kv_desc = desc + (smem_u32(S.kv[0]) >> 4);
      auto full_parity = [](int i) { return (uint32_t)((i / kStages) & 1); };
      auto spin = [&](uint64_t* bar, uint32_t parity, uint32_t bit) { return warp_poll(bar, parity, abort_flag, status, bit); };
      auto rest = [&](uint64_t* bar, uint32_t parity, uint32_t bit) { return warp_rest(bar, parity, abort_flag, status, bit); };
      if (warp == kMmaWarp) {
        constexpr uint32_t idesc_qk = umma_idesc(kDS32, kFmtS8, kFmtS8, 0, 0, kTile, kTile);
        const uint64_t q_desc[2] = {desc + (smem_u32(S.q[0]) >> 4), desc + (smem_u32(S.q[1]) >> 4)};
        // S = Q_t K_j^T: four MMAs of 32 channels (32 bytes of a row = 2 descriptor units), then the commits
        auto qk = [&](int t, int j, uint64_t* taken, uint32_t taken_parity) -> bool {
          const int ik = 2 * j, sk = ik % kStages;
          const uint64_t a = t ? q_desc[1] : q_desc[0], b = kv_desc + sk * (kTileBytes >> 4);
          if (t == 0 && !rest(&S.kv_full[sk], full_parity(ik), kWaitTimeoutLoad)) return false;
          if (taken && !spin(taken, taken_parity, kWaitTimeoutSoftmax)) return false;  // last: the critical hand-over
          tc_fence_after();
          if (elect_one()) {
            asm volatile(
                "{\n\t.reg .pred p0, p1;\n\t"
                "setp.ne.b32 p0, 0, 0;\n\tsetp.eq.b32 p1, 0, 0;\n\t"
                "tcgen05.mma.cta_group::1.kind::i8 [%0], %2, %6, %1, p0;\n\t"
                "tcgen05.mma.cta_group::1.kind::i8 [%0], %3, %7, %1, p1;\n\t"
                "tcgen05.mma.cta_group::1.kind::i8 [%0], %4, %8, %1, p1;\n\t"
                "tcgen05.mma.cta_group::1.kind::i8 [%0], %5, %9, %1, p1;\n\t}" ::"r"(tmem + kColS),
                "r"(idesc_qk), "l"(a), "l"(a + 2), "l"(a + 4), "l"(a + 6), "l"(b), "l"(b + 2), "l"(b + 4), "l"(b + 6)
                : "memory");
            tc_commit(&S.s_full[t]);
            if (t == 1 || !two) tc_commit(&S.kv_empty[sk]);  // last reader of K_j
          }
          return true;
        };
        bool ok = rest(&S.q_full, 0, kWaitTimeoutLoad) && qk(0, 0, nullptr, 0);
        for (int j = 0; ok && j < n_kv; ++j) {
          if (two && !(ok = qk(1, j, &S.s_taken[0], j & 1))) break;
          if (j + 1 < n_kv && !(ok = qk(0, j + 1, &S.s_taken[two ? 1 : 0], j & 1))) break;
        }
      } else {
        constexpr uint32_t idesc_pv = umma_idesc(kDF32, kFmtE4M3, kFmtE4M3, 0, 0, kTile, 128);
        // O_t += P_t(j) V_j: four MMAs of 32 keys (32 bytes of a V row; 8 columns of P), then the commits
        auto pv = [&](int t, int j) -> bool {
          const int iv = 2 * j + 1, sv = iv % kStages;
          const uint64_t b = kv_desc + sv * (kTileBytes >> 4);
          const uint32_t d = tmem + kColO + t * kTile, a = tmem + kColP + t * 64 + (j & 1) * 32;
          if (t == 0 && !rest(&S.kv_full[sv], full_parity(iv), kWaitTimeoutLoad)) return false;
          // asleep: with two P buffers there is slack, and a polling warp takes issue slots from the softmax warps of its
          // scheduler; .7 % (eight slices of 4096 x 30389 x 24 heads), not above what one run differs from the next on another GPU
          if (!rest(&S.p_full[t][j & 1], (j >> 1) & 1, kWaitTimeoutSoftmax)) return false;
          tc_fence_after();
          if (elect_one()) {
            asm volatile(
                "{\n\t.reg .pred p0, p1;\n\t"
                "setp.ne.b32 p0, %2, 0;\n\tsetp.eq.b32 p1, 0, 0;\n\t"
                "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], [%3], %7, %1, p0;\n\t"
                "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], [%4], %8, %1, p1;\n\t"
                "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], [%5], %9, %1, p1;\n\t"
                "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], [%6], %10, %1, p1;\n\t}" ::"r"(d),
                "r"(idesc_pv), "r"(j > 0 ? 1u : 0u), "r"(a), "r"(a + 8), "r"(a + 16), "r"(a + 24), "l"(b), "l"(b + 2),
                "l"(b + 4), "l"(b + 6)
                : "memory");
            tc_commit(&S.pv_done[t][j & 1]);
            if (t == 1 || !two) tc_commit(&S.kv_empty[sv]);  // last reader of V_j
          }
          return true;
        };
        bool ok = true;
        for (int j = 0; ok && j < n_kv; ++j) ok = pv(0, j) && (!two || pv(1, j));
      }
    }
  } else {
    // ------------------------------------------------- softmax + epilogue warps
    reg_alloc<kSoftmaxRegs>();
    auto poll = [&](uint64_t* bar, uint32_t parity, uint32_t bit) { return warp_poll(bar, parity, abort_flag, status, bit); };
    const int t = warp >> 2;
    if (t == 0 || two) {
      const int row = (warp & 3) * 32 + lane;
      const uint32_t lane_base = static_cast<uint32_t>((warp & 3) * 32) << 16;
      const uint32_t s_addr = tmem + lane_base + kColS;
      const uint32_t p_addr = tmem + lane_base + kColP + t * 64;
      const uint32_t o_addr = tmem + lane_base + kColO + t * kTile;
      const int token = q0 + t * kTile + row;
      // per-row factor: query scale of the row's block (32, 64 or 128 tokens) times log2e/sqrt(128)
      const int q_blocks = (num_query_tokens + query_block - 1) / query_block;
      const float qf = query_scale[static_cast<size_t>(head) * q_blocks + min(token / query_block, q_blocks - 1)] * scale_log2;
      float m_used = 0.f;
      uint64_t la = 0ull, lb = 0ull;  // four partial row sums as two fp32 pairs
      bool ok = true;
      for (int j = 0; j < n_kv; ++j) {
        const int jt = kv_begin + j;  // key tile in the whole sequence
        float ks0, ks1;
        if (2 * j + 1 < kKeptScales) {
          ks0 = S.key_scale[2 * j], ks1 = S.key_scale[2 * j + 1];
        } else {
          const int in_head = KeySplit::reload(S.share).head;
          ks0 = key_scale_of(in_head, 2 * jt), ks1 = key_scale_of(in_head, 2 * jt + 1);
        }
        ok = poll(&S.s_full[t], j & 1, kWaitTimeoutMma);
        if (!ok) break;
        tc_fence_after();
        uint32_t s[128];
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) tmem_ld32(s_addr + 32 * cc, *reinterpret_cast<uint32_t(*)[32]>(&s[32 * cc]));
        tc_wait_ld();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&S.s_taken[t]);
        // PV(j-2) read the P buffer of this tile: looked at early, so that the answer is there when P is stored
        bool p_free = j < 2 || mbar_test(&S.pv_done[t][j & 1], ((j - 2) >> 1) & 1);
#pragma unroll
        for (int i = 0; i < 128; ++i) s[i] = __float_as_uint(static_cast<float>(static_cast<int>(s[i])));
        const int valid = num_kv_tokens - jt * kTile;  // keys of this tile that exist (>= 1)
        if (valid < kTile) {
#pragma unroll
          for (int i = 0; i < 128; ++i)
            if (i >= valid) s[i] = 0xff800000u;  // -inf
        }
        float a0 = __uint_as_float(s[0]), a1 = __uint_as_float(s[64]), a2 = __uint_as_float(s[1]), a3 = __uint_as_float(s[65]);
#pragma unroll
        for (int i = 2; i < 62; i += 4) {
          a0 = max3(a0, __uint_as_float(s[i]), __uint_as_float(s[i + 1]));
          a1 = max3(a1, __uint_as_float(s[64 + i]), __uint_as_float(s[64 + i + 1]));
          a2 = max3(a2, __uint_as_float(s[i + 2]), __uint_as_float(s[i + 3]));
          a3 = max3(a3, __uint_as_float(s[64 + i + 2]), __uint_as_float(s[64 + i + 3]));
        }
        a0 = max3(a0, a2, fmaxf(__uint_as_float(s[62]), __uint_as_float(s[63])));
        a1 = max3(a1, a3, fmaxf(__uint_as_float(s[126]), __uint_as_float(s[127])));
        // factors of the two 64-key halves, kept positive so that the -inf of a key past the end stays -inf under them; a
        // scale that is not a number stays one and shows in the output
        const float f0 = max_nan(qf * ks0, 1e-30f), f1 = max_nan(qf * ks1, 1e-30f);
        const float mx = fmaxf(a0 * f0, a1 * f1);
        if (j == 0) {
          m_used = mx;
        } else if (__any_sync(0xffffffffu, mx > m_used + kHeadroomLog2)) {
          const float m_new = fmaxf(m_used, mx);
          const float alpha = ex2(m_used - m_new);
          const uint64_t alpha2 = pack2(alpha, alpha);
          la = mul2(la, alpha2);
          lb = mul2(lb, alpha2);
          // O_t += P_t V_{j-1} must have completed; the next PV waits for our arrival on p_full.
          ok = poll(&S.pv_done[t][(j - 1) & 1], ((j - 1) >> 1) & 1, kWaitTimeoutMma);
          if (!ok) break;
          p_free = true;
          tc_fence_after();
          tmem_scale_rows(o_addr, alpha);
          m_used = m_new;
        }
        const float cst = kLog2PScale - m_used;
        const uint64_t f2[2] = {pack2(f0, f0), pack2(f1, f1)}, cst2 = pack2(cst, cst);
        // Groups of 16 keys, the exponentials of a group ahead of the sums and conversions of the one before: the
        // special-function unit does not drain while a group is packed.
        float e[2][16];
        auto exponentials = [&](int g) {
#pragma unroll
          for (int i = 0; i < 16; i += 2) {
            float x0, x1;
            unpack2(fma2(pack2(__uint_as_float(s[16 * g + i]), __uint_as_float(s[16 * g + i + 1])), f2[g >> 2], cst2), x0, x1);
            e[g & 1][i] = ex2(x0);
            e[g & 1][i + 1] = ex2(x1);
          }
        };
        exponentials(0);
        uint32_t p[32];
#pragma unroll
        for (int g = 0; g < 8; ++g) {
          if (g < 7) exponentials(g + 1);
          const float* x = e[g & 1];
#pragma unroll
          for (int i = 0; i < 16; i += 4) {
            la = add2(la, pack2(x[i], x[i + 1]));
            lb = add2(lb, pack2(x[i + 2], x[i + 3]));
          }
          // stored order inside a group: 0,1,8,9 | 2,3,10,11 | ...
#pragma unroll
          for (int w = 0; w < 4; ++w) p[4 * g + w] = pack_e4m3x4(x[2 * w], x[2 * w + 1], x[8 + 2 * w], x[8 + 2 * w + 1]);
          if (g == 3) {
            if (!__all_sync(0xffffffffu, p_free)) {
              ok = poll(&S.pv_done[t][j & 1], ((j - 2) >> 1) & 1, kWaitTimeoutMma);
              if (!ok) break;
            }
            tc_fence_after();
            tmem_st16(p_addr + 32 * (j & 1), p);
          }
        }
        if (!ok) break;
        tmem_st16(p_addr + 32 * (j & 1) + 16, p + 16);
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&S.p_full[t][j & 1]);
      }
      if (ok) ok = poll(&S.pv_done[t][(n_kv - 1) & 1], ((n_kv - 1) >> 1) & 1, kWaitTimeoutMma);
      if (ok) {
        tc_fence_after();
        float l0, l1, l2, l3;
        unpack2(la, l0, l1);
        unpack2(lb, l2, l3);
        const float l = (l0 + l1) + (l2 + l3);
        const float inv = 1.0f / l;
        const KeySplit::Share at_end = KeySplit::reload(S.share);
        const int head = at_end.head, q0 = at_end.q_tile * split.unit_rows;
        const int token = q0 + t * kTile + (warp & 3) * 32 + lane;
        const float* vs = value_scale + head * 128;
        const bool divided = at_end.piece >= 0;
        bool store = token < num_query_tokens && NOB_CHECK(head < heads, status);
        __nv_bfloat16* dst = out + (static_cast<size_t>(store ? token : 0) * heads + head) * 128;
        size_t row_at = 0;
        if (divided) {
          // the probability scale 448/8 is common to all shares and cancels in the merge
          row_at = split.partial_row(at_end.piece, head, store ? token : q0, num_query_tokens);
          store = store && NOB_CHECK(row_at < static_cast<size_t>(split.splits) * split.tail_rows, status);
          if (store) split.lse[row_at] = m_used + log2f(l);
        }
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) {
          uint32_t o[32];
          tmem_ld32(o_addr + 32 * cc, o);
          tc_wait_ld();
          if (store) {
            float r[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) r[i] = __uint_as_float(o[i]) * vs[32 * cc + i] * inv;
            if (divided) {
              split.store(row_at, 32 * cc, r);
            } else {
#pragma unroll
              for (int i = 0; i < 32; i += 8)
                *reinterpret_cast<uint4*>(dst + 32 * cc + i) =
                    make_uint4(pack_bf16(r[i], r[i + 1]), pack_bf16(r[i + 2], r[i + 3]), pack_bf16(r[i + 4], r[i + 5]),
                               pack_bf16(r[i + 6], r[i + 7]));
            }
          }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == kProducerWarp) tmem_dealloc(tmem, kTmemCols);
}

int launch_dense_int8_fp8(int num_kv_tokens, int num_query_tokens, const void* query, const void* key, const void* value,
                          const void* query_scale, const void* key_scale, const void* value_scale, void* output, int heads,
                          int query_block, int key_block, int unit_rows, int kv_splits, int tail_units,
                          bool partial_f32, void* workspace, size_t workspace_bytes, void* stream) {
  NOB_REQUIRE(num_kv_tokens > 0 && num_query_tokens > 0 && heads > 0, "dense_int8_fp8_d128: sizes must be positive");
  NOB_REQUIRE(query && key && value && query_scale && key_scale && value_scale && output,
              "dense_int8_fp8_d128: NULL tensor");
  NOB_REQUIRE(query_block == 32 || query_block == 64 || query_block == 128,
              "dense_int8_fp8_d128: query scale block must be 32, 64 or 128 tokens (got %d)", query_block);
  NOB_REQUIRE(key_block == 64 || key_block == 128, "dense_int8_fp8_d128: key scale block must be 64 or 128 tokens (got %d)",
              key_block);
  KeySplit split;
  int rc;
  if ((rc = make_key_split(&split, "dense_int8_fp8_d128", num_query_tokens, num_kv_tokens, heads, unit_rows,
                           kv_splits, tail_units, partial_f32, workspace, workspace_bytes)))
    return rc;
  uint32_t* status = status_word_device_ptr();
  if (!status) return fail(kCudaError, "dense_int8_fp8_d128: no current CUDA device");
  const uint64_t q_rows = (static_cast<uint64_t>(num_query_tokens) + query_block - 1) / query_block * query_block;
  const uint64_t k_rows = (static_cast<uint64_t>(num_kv_tokens) + key_block - 1) / key_block * key_block;
  const uint64_t v_cols = (static_cast<uint64_t>(num_kv_tokens) + 63) / 64 * 64;  // the value quantiser pads to 64

  CUtensorMap mq, mk, mv;
  // Q, K: [heads][rows][128 bytes]; V: [heads][128 channels][v_cols bytes]
  if ((rc = make_tensor_map_3d(&mq, CU_TENSOR_MAP_DATA_TYPE_UINT8, query, 128, q_rows, heads, 128, q_rows * 128, 128,
                               kTile, 1)))
    return rc;
  if ((rc = make_tensor_map_3d(&mk, CU_TENSOR_MAP_DATA_TYPE_UINT8, key, 128, k_rows, heads, 128, k_rows * 128, 128,
                               kTile, 1)))
    return rc;
  if ((rc = make_tensor_map_3d(&mv, CU_TENSOR_MAP_DATA_TYPE_UINT8, value, v_cols, 128, heads, v_cols, v_cols * 128, 128,
                               kTile, 1)))
    return rc;

  const size_t smem = sizeof(Shared) + 1024;
  cudaError_t err =
      cudaFuncSetAttribute(fa_fwd_i8f8_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (err != cudaSuccess)
    return fail(kCudaError, "dense_int8_fp8_d128: cannot reserve %zu B of shared memory: %s", smem,
                cudaGetErrorString(err));
  const float scale_log2 = 0.08838834764831845f * 1.4426950408889634f;
  if ((rc = launch_pdl("dense_int8_fp8_d128", fa_fwd_i8f8_kernel, key_split_blocks(split, heads), kThreads, smem, stream, mq,
                       mk, mv, static_cast<const float*>(query_scale), static_cast<const float*>(key_scale),
                       static_cast<const float*>(value_scale), static_cast<__nv_bfloat16*>(output), num_query_tokens,
                       num_kv_tokens, heads, scale_log2, status, query_block, key_block, split)))
    return rc;
  if (!split.tail_rows) return kOk;
  OutRoute route = {};
  route.peer[0] = static_cast<__nv_bfloat16*>(output);
  return launch_merge_splits(split, route, num_query_tokens, heads, 0, stream);
}

}  // namespace
}  // namespace nob200

extern "C" int nob200_dense_int8_fp8_d128(int num_kv_tokens, int num_query_tokens, const void* query, const void* key,
                                          const void* value, const void* query_scale, const void* key_scale,
                                          const void* value_scale, void* output, int heads, void* stream) {
  return nob200::launch_dense_int8_fp8(num_kv_tokens, num_query_tokens, query, key, value, query_scale, key_scale,
                                       value_scale, output, heads, 32, 64, 2 * nob200::kTile, 1, 0, false, nullptr, 0, stream);
}

extern "C" int nob200_dense_int8_fp8_d128_splitkv(int num_kv_tokens, int num_query_tokens, const void* query,
                                                  const void* key, const void* value, const void* query_scale,
                                                  const void* key_scale, const void* value_scale, void* output,
                                                  int heads, int query_block, int key_block, int kv_splits,
                                                  void* workspace, size_t workspace_bytes, void* stream) {
  return nob200::launch_dense_int8_fp8(num_kv_tokens, num_query_tokens, query, key, value, query_scale, key_scale,
                                       value_scale, output, heads, query_block, key_block, 2 * nob200::kTile, kv_splits, 0,
                                       false, workspace,
                                       workspace_bytes, stream);
}

extern "C" int nob200_dense_int8_fp8_d128_units(int num_kv_tokens, int num_query_tokens, const void* query,
                                               const void* key, const void* value, const void* query_scale,
                                               const void* key_scale, const void* value_scale, void* output, int heads,
                                               int query_block, int key_block, int unit_rows, int kv_splits, int tail_units,
                                               void* workspace, size_t workspace_bytes, void* stream) {
  return nob200::launch_dense_int8_fp8(num_kv_tokens, num_query_tokens, query, key, value, query_scale, key_scale,
                                       value_scale, output, heads, query_block, key_block, unit_rows, kv_splits, tail_units, true,
                                       workspace, workspace_bytes, stream);
}

extern "C" int nob200_dense_int8_fp8_d128_blocks(int num_kv_tokens, int num_query_tokens, const void* query,
                                                 const void* key, const void* value, const void* query_scale,
                                                 const void* key_scale, const void* value_scale, void* output,
                                                 int heads, int query_block, int key_block, void* stream) {
  return nob200::launch_dense_int8_fp8(num_kv_tokens, num_query_tokens, query, key, value, query_scale, key_scale,
                                       value_scale, output, heads, query_block, key_block, 2 * nob200::kTile, 1, 0, false, nullptr, 0, stream);
}
