// Device helpers shared by the attention kernels: register reallocation between warpgroups,
// exp2 on the MUFU and on the FMA pipe, bf16 packing and packed fp32x2 arithmetic.
#pragma once

#include "common.cuh"

namespace nob200 {

template <int N>
__device__ __forceinline__ void reg_dealloc() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}
template <int N>
__device__ __forceinline__ void reg_alloc() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  uint32_t d;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}

// ---- packed fp32x2 arithmetic (two lanes of a 64-bit register pair)
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// NaN if either is (fmaxf returns the other one)
__device__ __forceinline__ float max_nan(float a, float b) {
  float d;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
  return d;
}
// 2^x for a pair on the FMA pipe: x = n + r with n = round(x), r in [-0.5, 0.5];
// 2^r by a degree-3 polynomial (relative error 7.5e-5, below bf16 resolution),
// n added into the exponent field.  x is clamped at -126 (result ~1e-38).
__device__ __forceinline__ void exp2_poly_pair(uint64_t x, float& y0, float& y1) {
  const uint64_t magic = pack2(12582912.f, 12582912.f);
  const uint64_t neg_magic = pack2(-12582912.f, -12582912.f);
  float x0, x1;
  unpack2(x, x0, x1);
  x = pack2(fmaxf(x0, -126.f), fmaxf(x1, -126.f));
  const uint64_t t = add2(x, magic);
  const uint64_t n = add2(t, neg_magic);
  const uint64_t r = fma2(n, pack2(-1.f, -1.f), x);
  uint64_t p = fma2(pack2(0.0551716648042202f, 0.0551716648042202f), r, pack2(0.2426111251115799f, 0.2426111251115799f));
  p = fma2(p, r, pack2(0.6932609677314758f, 0.6932609677314758f));
  p = fma2(p, r, pack2(0.9999280571937561f, 0.9999280571937561f));
  float t0, t1, p0, p1;
  unpack2(t, t0, t1);
  unpack2(p, p0, p1);
  y0 = __uint_as_float(__float_as_uint(p0) + (__float_as_uint(t0) << 23));
  y1 = __uint_as_float(__float_as_uint(p1) + (__float_as_uint(t1) << 23));
}

// The 128 accumulator columns of a warp's rows times `alpha` (each thread its row), in place.
__device__ __forceinline__ void tmem_scale_rows(uint32_t o_addr, float alpha) {
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint32_t o[32];
    tmem_ld32(o_addr + 32 * c, o);
    tc_wait_ld();
#pragma unroll
    for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
    tmem_st32(o_addr + 32 * c, o);
  }
  tc_wait_st();
}

// The same with all loads in flight at once, for a place where a tile's scores are no longer live in registers.
__device__ __forceinline__ void tmem_scale_rows_wide(uint32_t o_addr, float alpha) {
  uint32_t o[4][32];
#pragma unroll
  for (int c = 0; c < 4; ++c) tmem_ld32(o_addr + 32 * c, o[c]);
  tc_wait_ld();
  const uint64_t alpha2 = pack2(alpha, alpha);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
      float x, y;
      unpack2(mul2(pack2(__uint_as_float(o[c][i]), __uint_as_float(o[c][i + 1])), alpha2), x, y);
      o[c][i] = __float_as_uint(x), o[c][i + 1] = __float_as_uint(y);
    }
    tmem_st32(o_addr + 32 * c, o[c]);
  }
  tc_wait_st();
}

// ---- waits of the attention kernels (all 32 lanes of a converged warp call them; the result is warp-uniform)
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Gives up (warp-uniformly) when the CTA's abort flag is up or `start` lies more than the wait budget back; the
// first warp to give up raises the flag and records `bit` in the status word.
__device__ __forceinline__ bool warp_gives_up(uint64_t& start, volatile uint32_t* abort_flag, uint32_t* status,
                                              uint32_t bit) {
  const uint64_t now = global_timer_ns();
  if (start == 0) start = now;
  if (!__any_sync(0xffffffffu, *abort_flag != 0 || now - start > kWaitBudgetNs)) return false;
  if ((threadIdx.x & 31) == 0 && *abort_flag == 0) {
    *abort_flag = 1;
    atomicOr(status, bit);
  }
  return true;
}
// Polls mbarrier.test_wait.  For waits on the kernel's critical hand-overs: a warp suspended in try_wait was seen
// to resume hundreds of cycles after the phase completed, and the slowest warp of a tile sets the tile's pace.
__device__ __forceinline__ bool warp_poll(uint64_t* bar, uint32_t parity, volatile uint32_t* abort_flag,
                                          uint32_t* status, uint32_t bit) {
  uint64_t start = 0;
  for (uint32_t spins = 1; !__all_sync(0xffffffffu, mbar_test(bar, parity)); ++spins) {
    if ((spins & 0x3FF) == 0 && warp_gives_up(start, abort_flag, status, bit)) return false;
  }
  return true;
}
// Suspends in mbarrier.try_wait.  For waits with slack, where a polling warp takes issue slots from the softmax warps of
// its scheduler, and for the softmax warps' own waits in the bf16 kernels, which run at the power cap.
__device__ __forceinline__ bool warp_rest(uint64_t* bar, uint32_t parity, volatile uint32_t* abort_flag,
                                          uint32_t* status, uint32_t bit) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, status, bit));
}
// Waits until a shared-memory counter written by another warp of the CTA has reached `target`.
__device__ __forceinline__ bool warp_wait_counter(const uint32_t* counter, uint32_t target,
                                                  volatile uint32_t* abort_flag, uint32_t* status, uint32_t bit) {
  uint64_t start = 0;
  for (uint32_t spins = 1; !__all_sync(0xffffffffu, *reinterpret_cast<const volatile uint32_t*>(counter) >= target);
       ++spins) {
    __nanosleep(64);
    if ((spins & 0x3FF) == 0 && warp_gives_up(start, abort_flag, status, bit)) return false;
  }
  return true;
}
// One lane of a converged warp.  The issuing warps run all 32 lanes through warp-uniform control flow and put only
// the tcgen05 instructions themselves under this predicate: the compiler then keeps descriptors and addresses in
// uniform registers, which is where tcgen05.mma reads them from.  With a single active lane (`if (lane == 0)`)
// they live in ordinary registers and every MMA pays moves into uniform registers: about 100 instead of 64 cycles
// per MMA for the issuing thread.
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(pred));
  return pred != 0;
}

// Where output rows go.  tokens_per_rank == 0: all rows to peer[0] (the local output tensor).
// tokens_per_rank > 0: row `token` belongs to rank token / tokens_per_rank and is stored straight into
// that rank's output tensor (a peer pointer over NVLink) at its local row index: the head->sequence
// reshard of the multi-GPU path happens in the epilogue, without a collective.
constexpr int kMaxWorld = 8;
struct OutRoute {
  __nv_bfloat16* peer[kMaxWorld];
  int tokens_per_rank;
  __device__ __forceinline__ __nv_bfloat16* row(int token, int total_heads, int head) const {
    if (tokens_per_rank == 0) return peer[0] + (static_cast<size_t>(token) * total_heads + head) * 128;
    const int owner = token / tokens_per_rank;
    return peer[owner] + (static_cast<size_t>(token - owner * tokens_per_rank) * total_heads + head) * 128;
  }
};

// A scatter epilogue stores into other ranks' tensors only while no cross-rank barrier has timed out: after a
// timeout this rank's input was incomplete and its rows must not overwrite the peers' outputs.
__device__ __forceinline__ bool route_open(const OutRoute& route, const uint32_t* status) {
  if (route.tokens_per_rank == 0) return true;
  uint32_t word;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(word) : "l"(status));
  return (word & kWaitTimeoutPeer) == 0;
}

// How the units of a dense launch - `unit_rows` query rows of one head, numbered head by head - become CTAs.  256 rows
// are two query tiles that share their K / V tiles and overlap each other's phases; 128 rows (one tile, 0.72 of the
// time per key tile) double the units of a small call.  The first
// `full_units` are one CTA each; the key tiles of the rest are divided over `splits` CTAs, whose normalised partial
// results and log-sum-exps (log2 units) fa_merge_splits_kernel joins.  Dividing only the units of the last wave lets a
// launch end on all SMs together at the price of a few partial rows: 518 units on 148 SMs are 3.5 waves, not 4.
struct KeySplit {
  int unit_rows = 256, q_tiles = 0, full_units = 0, splits = 1;
  long long tail_base = 0;  // row (head * tokens + token) of the first divided unit
  long long tail_rows = 0;  // rows of all divided units
  void* partial = nullptr;  // [splits][tail_rows][128], f32 or bf16
  float* lse = nullptr;     // [splits][tail_rows]
  bool partial_f32 = false;

  struct Share {
    int head, q_tile, kv_begin, kv_end, piece;  // piece < 0: the whole unit
  };
  // A copy read back from shared memory: head, query tile and piece are needed before and after the key loop, and kept
  // in registers across it they would be spilled inside it.
  static __device__ __forceinline__ Share reload(const Share& kept) {
    const volatile Share& v = kept;
    return Share{v.head, v.q_tile, v.kv_begin, v.kv_end, v.piece};
  }
  __device__ __forceinline__ Share share(int block, int n_kv_total) const {
    Share r{0, 0, 0, n_kv_total, -1};
    int unit = block;
    if (block >= full_units) {
      const int k = (block - full_units) / splits;
      r.piece = block - full_units - k * splits;
      unit = full_units + k;
      r.kv_begin = static_cast<int>(static_cast<long long>(n_kv_total) * r.piece / splits);
      r.kv_end = static_cast<int>(static_cast<long long>(n_kv_total) * (r.piece + 1) / splits);
    }
    r.head = unit / q_tiles;
    r.q_tile = unit - r.head * q_tiles;
    return r;
  }
  __device__ __forceinline__ size_t partial_row(int piece, int head, int token, int num_tokens) const {
    return static_cast<size_t>(piece * tail_rows + (static_cast<long long>(head) * num_tokens + token - tail_base));
  }
  // 32 normalised channels of a partial row, from channel `c0` on
  __device__ __forceinline__ void store(size_t row, int c0, const float (&v)[32]) const {
    if (partial_f32) {
      float4* dst = reinterpret_cast<float4*>(static_cast<float*>(partial) + row * 128 + c0);
#pragma unroll
      for (int i = 0; i < 8; ++i) dst[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
    } else {
      uint4* dst = reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(partial) + row * 128 + c0);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        dst[i] = make_uint4(pack_bf16(v[8 * i], v[8 * i + 1]), pack_bf16(v[8 * i + 2], v[8 * i + 3]),
                            pack_bf16(v[8 * i + 4], v[8 * i + 5]), pack_bf16(v[8 * i + 6], v[8 * i + 7]));
    }
  }
};

// The split of a launch: `tail_units` 0 divides every unit.  Checks the arguments and the workspace.
int make_key_split(KeySplit* split, const char* name, int num_query_tokens, int num_kv_tokens, int heads, int unit_rows,
                   int kv_splits, int tail_units, bool partial_f32, void* workspace, size_t workspace_bytes);
inline int key_split_blocks(const KeySplit& s, int heads) {
  return s.full_units + (s.q_tiles * heads - s.full_units) * s.splits;
}
// Joins the shares of the divided units into the routed output; defined beside the bf16 attention kernel.
int launch_merge_splits(const KeySplit& split, const OutRoute& route, int num_tokens, int total_heads, int head_offset,
                        void* stream);

}  // namespace nob200
