// Per-head RMS norm and split-half RoPE of Q and K, alone (bf16 out) or fused into the int8 query quantiser.
// HBM-bound CUDA-core kernels: one pass over the projected activations instead of a bf16 round trip.
//
// Reference programs replaced here:
//   h3_head_norm_rope   src/nano_omni/kernels/specialized/h3_head_norm_rope.py:36-97
//   h3_query_prepare    src/nano_omni/kernels/specialized/h3_query_prepare.py:42-125
//
// For every (token, head) row x of 128 channels:
//   r = 1 / sqrt(sum(x^2) / 128 + 1e-5);  v = (x * r) * weight;
//   with RoPE, channels j < 48 and j + 48 form a pair rotated by (cos, sin)[token, j]:
//     out[j] = v[j] cos - v[j+48] sin,  out[j+48] = v[j] sin + v[j+48] cos;  channels 96..127 pass;
//   out is rounded to bf16 (stored, or quantised to int8 with one scale per head and 32 tokens).
// The reference leaves the order of the sum and the kind of reciprocal square root to its compiler (and its two
// ref_programs differ: mean of squares vs squared vector norm).  Here every step is an IEEE fp32 operation in a
// fixed order, which the CPU restatement repeats: a row is 16 chunks of 8 consecutive channels; a chunk adds
// its squares in channel order starting from 0, the 16 partial sums are combined by an xor butterfly with strides
// 8, 4, 2, 1; divide by 128, add 1e-5, square root, divide 1 by it; products and the sum or difference of the
// rotation are rounded one by one (no fused multiply-add).
#include "common.cuh"
#include "../../include/nano_omni_b200.h"

namespace nob200 {
namespace {

struct Row8 {
  float v[8];
};

__device__ __forceinline__ Row8 load_row8(const __nv_bfloat16* p) {
  const uint4 raw = *reinterpret_cast<const uint4*>(p);
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
  Row8 r;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    r.v[2 * i] = __uint_as_float(w[i] << 16);
    r.v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
  return r;
}

__device__ __forceinline__ Row8 row8_of(const uint4& raw) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
  Row8 r;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    r.v[2 * i] = __uint_as_float(w[i] << 16);
    r.v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
  return r;
}

__device__ __forceinline__ float round_bf16(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// A row lies on 8 lanes, each with two chunks of 8 channels: lanes 0-5 chunks t and t + 6, the two sides of the rotation's
// pairs, lanes 6 and 7 the chunks 12, 13 and 14, 15 that pass through.  The rotation then needs no exchange between
// lanes, and a row costs 5 shuffles per lane (the sum of squares) instead of 12 on twice as many lanes: shuffles and the
// divide / square root sequence, which every lane repeats, bounded the kernels (16 lanes per row, before / after:
// 9461 tokens x 14 heads 27 / 20 us, query quantiser 4096 x 24 24 / 20.6 us).
struct RowPart {
  Row8 a, b;
};
__device__ __forceinline__ int chunk_a(int lane8) { return lane8 < 6 ? lane8 : 2 * lane8; }
__device__ __forceinline__ int chunk_b(int lane8) { return lane8 < 6 ? lane8 + 6 : 2 * lane8 + 1; }

__device__ __forceinline__ RowPart load_part(const __nv_bfloat16* row, int lane8) {
  return {load_row8(row + 8 * chunk_a(lane8)), load_row8(row + 8 * chunk_b(lane8))};
}

__device__ __forceinline__ float sum_of_squares(const Row8& x) {
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) s = __fadd_rn(s, __fmul_rn(x.v[i], x.v[i]));
  return s;
}

// x[k]: this lane's part of row k; w: the norm weight of those channels.  On return x holds the normalised, rotated rows
// rounded to bf16 precision.  All lanes of the warp must call it.  N rows go through each stage together so that their
// loads, shuffles and the divide / square root sequences overlap.
template <int N, int NW = 1>  // NW = 1: one weight for all rows; NW = N: a weight per row
__device__ __forceinline__ void norm_rope_rows(RowPart (&x)[N], const RowPart (&w)[NW], const float* cosines,
                                               const float* sines, const int (&token)[N], int lane8,
                                               bool use_rope) {
  const bool rotates = use_rope && lane8 < 6;
  float4 c[N][2], s[N][2];
  if (rotates) {
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const int at = token[k] * 48 + 8 * lane8;
      c[k][0] = *reinterpret_cast<const float4*>(cosines + at);
      c[k][1] = *reinterpret_cast<const float4*>(cosines + at + 4);
      s[k][0] = *reinterpret_cast<const float4*>(sines + at);
      s[k][1] = *reinterpret_cast<const float4*>(sines + at + 4);
    }
  }
  // The sums p[0..15] of the chunks go through the butterfly with strides 8, 4, 2, 1: lane t first gets p[t] and p[t + 8].
  // p[6], p[7] are the second chunks of lanes 0, 1; p[8..11] those of lanes 2-5; p[12..15] lanes 6 and 7.
  const int from_b = lane8 < 4 ? lane8 + 2 : lane8 == 5 ? 6 : lane8 == 6 ? 0 : lane8 == 7 ? 1 : 4;
  const int from_a = lane8 == 4 ? 6 : lane8 == 6 ? 7 : lane8;
  float ss[N];
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const float sa = sum_of_squares(x[k].a), sb = sum_of_squares(x[k].b);
    const float other_b = __shfl_sync(0xffffffffu, sb, from_b, 8), other_a = __shfl_sync(0xffffffffu, sa, from_a, 8);
    const float low = lane8 < 6 ? sa : other_b;
    const float high = (lane8 == 4 || lane8 == 6) ? other_a : lane8 == 7 ? sb : other_b;
    ss[k] = __fadd_rn(low, high);
  }
#pragma unroll
  for (int m = 4; m > 0; m >>= 1) {
#pragma unroll
    for (int k = 0; k < N; ++k) ss[k] = __fadd_rn(ss[k], __shfl_xor_sync(0xffffffffu, ss[k], m));
  }
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const float r = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fmul_rn(ss[k], 0.0078125f), 1e-5f)));
    const RowPart& wk = w[NW == 1 ? 0 : k];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      x[k].a.v[i] = __fmul_rn(__fmul_rn(x[k].a.v[i], r), wk.a.v[i]);
      x[k].b.v[i] = __fmul_rn(__fmul_rn(x[k].b.v[i], r), wk.b.v[i]);
    }
    if (rotates) {
      const float cc[8] = {c[k][0].x, c[k][0].y, c[k][0].z, c[k][0].w, c[k][1].x, c[k][1].y, c[k][1].z, c[k][1].w};
      const float sn[8] = {s[k][0].x, s[k][0].y, s[k][0].z, s[k][0].w, s[k][1].x, s[k][1].y, s[k][1].z, s[k][1].w};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float first = x[k].a.v[i], second = x[k].b.v[i];
        x[k].a.v[i] = __fsub_rn(__fmul_rn(first, cc[i]), __fmul_rn(second, sn[i]));
        x[k].b.v[i] = __fadd_rn(__fmul_rn(first, sn[i]), __fmul_rn(second, cc[i]));
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      x[k].a.v[i] = round_bf16(x[k].a.v[i]);
      x[k].b.v[i] = round_bf16(x[k].b.v[i]);
    }
  }
}

__device__ __forceinline__ uint32_t pack_bf16_pair(float lo, float hi) {
  return (__float_as_uint(lo) >> 16) | (__float_as_uint(hi) & 0xffff0000u);  // both already bf16-representable
}

__device__ __forceinline__ uint4 pack_row8(const Row8& x) {
  return make_uint4(pack_bf16_pair(x.v[0], x.v[1]), pack_bf16_pair(x.v[2], x.v[3]), pack_bf16_pair(x.v[4], x.v[5]),
                    pack_bf16_pair(x.v[6], x.v[7]));
}

// 8 lanes per (token, head) row: 32 rows per CTA round.  TENSORS rows (of Q, or of Q and K, which share the rotary
// planes' entries) go through together.  In place is allowed.
struct NormRopeTensors {
  const __nv_bfloat16* src[2];
  const __nv_bfloat16* weight[2];
  __nv_bfloat16* dst[2];  // may be src
};

template <int TENSORS>
__global__ void __launch_bounds__(256)
norm_rope_kernel(const NormRopeTensors tensors, const float* cosines, const float* sines,
                 long long rows, int heads, int use_rope) {
  pdl_wait();
  pdl_release();
  const int lane8 = threadIdx.x & 7;
  const int at_a = 8 * chunk_a(lane8), at_b = 8 * chunk_b(lane8);
  RowPart w[TENSORS];
#pragma unroll
  for (int k = 0; k < TENSORS; ++k) w[k] = load_part(tensors.weight[k], lane8);
  const long long stride = static_cast<long long>(gridDim.x) * 32;
  // every lane of a warp runs the same number of rounds (the shuffles need all of them).  The pieces of the next
  // round are loaded before this round's shuffles, which the compiler would not move a load across: two rows of a
  // thread are in flight instead of one.  (In place: the next round's rows are other rows than this round's.)
  uint4 next[TENSORS][2];
  auto fetch = [&](long long base) {
    const long long row = base + (threadIdx.x >> 3);
#pragma unroll
    for (int k = 0; k < TENSORS; ++k) {
      const __nv_bfloat16* p = tensors.src[k] + (row < rows ? row : 0) * 128;
      next[k][0] = *reinterpret_cast<const uint4*>(p + at_a);
      next[k][1] = *reinterpret_cast<const uint4*>(p + at_b);
    }
  };
  const long long first_base = static_cast<long long>(blockIdx.x) * 32;
  if (first_base < rows) fetch(first_base);
  for (long long base = first_base; base < rows; base += stride) {
    const long long row = base + (threadIdx.x >> 3);
    const bool live = row < rows;
    const int tok = static_cast<int>((live ? row : 0) / heads);
    RowPart x[TENSORS];
    int token[TENSORS];
#pragma unroll
    for (int k = 0; k < TENSORS; ++k) {
      x[k] = {row8_of(next[k][0]), row8_of(next[k][1])};
      token[k] = tok;
    }
    if (base + stride < rows) fetch(base + stride);
    norm_rope_rows<TENSORS, TENSORS>(x, w, cosines, sines, token, lane8, use_rope != 0);
    if (live) {
#pragma unroll
      for (int k = 0; k < TENSORS; ++k) {
        __nv_bfloat16* p = tensors.dst[k] + row * 128;
        *reinterpret_cast<uint4*>(p + at_a) = pack_row8(x[k].a);
        *reinterpret_cast<uint4*>(p + at_b) = pack_row8(x[k].b);
      }
    }
  }
}

// One CTA per (32-token group, head): 128 threads, 16 rows per pass, 2 passes.
__global__ void __launch_bounds__(128)
query_prepare_kernel(const __nv_bfloat16* src, const __nv_bfloat16* weight,
                     const float* cosines, const float* sines,
                     int8_t* quantized, float* scales, int tokens, int heads, int groups,
                     int use_rope) {
  pdl_wait();
  pdl_release();
  const int head = blockIdx.x, group = blockIdx.y;  // heads fastest: CTAs in flight read whole rows of the source
  const int lane8 = threadIdx.x & 7, row_in_pass = threadIdx.x >> 3;
  const int at_a = 8 * chunk_a(lane8), at_b = 8 * chunk_b(lane8);
  const RowPart w[1] = {load_part(weight, lane8)};
  const size_t columns = static_cast<size_t>(heads) * 128;
  uint4 loaded[2][2];  // both rows' loads are in flight together; the shuffles below would keep them apart
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    const int t = group * 32 + p * 16 + row_in_pass;
    const __nv_bfloat16* row = src + static_cast<size_t>(t < tokens ? t : 0) * columns + head * 128;
    loaded[p][0] = *reinterpret_cast<const uint4*>(row + at_a);
    loaded[p][1] = *reinterpret_cast<const uint4*>(row + at_b);
  }
  RowPart x[2];
  float amax = 0.f;
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    const int t = group * 32 + p * 16 + row_in_pass;
    const bool live = t < tokens;
    const int token[1] = {live ? t : 0};
    RowPart now[1] = {{row8_of(loaded[p][0]), row8_of(loaded[p][1])}};
    norm_rope_rows<1>(now, w, cosines, sines, token, lane8, use_rope != 0);
    x[p] = now[0];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (!live) x[p].a.v[i] = x[p].b.v[i] = 0.f;  // rows past the end quantise to zero and do not count in the maximum
      amax = fmaxf(amax, fmaxf(fabsf(x[p].a.v[i]), fabsf(x[p].b.v[i])));
    }
  }
  __shared__ float warp_max[4];
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, m));
  if ((threadIdx.x & 31) == 0) warp_max[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = fmaxf(fmaxf(warp_max[0], warp_max[1]), fmaxf(warp_max[2], warp_max[3]));
  const float scale = fmaxf(amax / 127.0f, 1e-10f);
  const float inv_scale = __frcp_rn(scale);
  if (threadIdx.x == 0) scales[static_cast<size_t>(head) * groups + group] = scale;
  int8_t* dst_base = quantized + (static_cast<size_t>(head) * groups + group) * 32 * 128;
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    int8_t* dst = dst_base + (p * 16 + row_in_pass) * 128;
#pragma unroll
    for (int side = 0; side < 2; ++side) {
      uint32_t word[2] = {0, 0};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        // rint(RN(x / scale)): the product with RN(1/scale) rounds to the same integer unless it lies within 4e-5
        // of a half-integer; only then the IEEE division is done (as in the int8 Q/K quantiser).
        const float value = side ? x[p].b.v[i] : x[p].a.v[i];
        float a = value * inv_scale;
        float q = rintf(a);
        if (0.5f - fabsf(a - q) < 4e-5f) q = rintf(__fdiv_rn(value, scale));
        q = fminf(fmaxf(q, -128.f), 127.f);
        word[i >> 2] |= (static_cast<uint32_t>(static_cast<int>(q)) & 0xffu) << (8 * (i & 3));
      }
      *reinterpret_cast<uint2*>(dst + (side ? at_b : at_a)) = make_uint2(word[0], word[1]);
    }
  }
}

}  // namespace
}  // namespace nob200

extern "C" int nob200_h3_head_norm_rope(int tokens, const void* input, const void* weight, const void* cosines,
                                        const void* sines, void* output, int heads, void* stream) {
  using namespace nob200;
  NOB_REQUIRE(tokens > 0 && heads > 0, "h3_head_norm_rope: sizes must be positive");
  NOB_REQUIRE(input && weight && output, "h3_head_norm_rope: NULL tensor");
  NOB_REQUIRE((cosines == nullptr) == (sines == nullptr), "h3_head_norm_rope: cosines and sines come together");
  const long long rows = static_cast<long long>(tokens) * heads;
  const long long ctas = (rows + 31) / 32;
  const unsigned grid = static_cast<unsigned>(ctas < 148 * 8 ? ctas : 148 * 8);
  const NormRopeTensors tensors = {{static_cast<const __nv_bfloat16*>(input)},
                                   {static_cast<const __nv_bfloat16*>(weight)},
                                   {static_cast<__nv_bfloat16*>(output)}};
  return launch_pdl("h3_head_norm_rope", norm_rope_kernel<1>, grid, 256, 0, stream, tensors,
                    static_cast<const float*>(cosines), static_cast<const float*>(sines), rows, heads, cosines != nullptr);
}

extern "C" int nob200_h3_qk_norm_rope(int tokens, void* query, void* key, const void* query_weight,
                                      const void* key_weight, const void* cosines, const void* sines, int heads,
                                      void* stream) {
  using namespace nob200;
  NOB_REQUIRE(tokens > 0 && heads > 0, "h3_qk_norm_rope: sizes must be positive");
  NOB_REQUIRE(query && key && query_weight && key_weight && cosines && sines, "h3_qk_norm_rope: NULL tensor");
  const long long rows = static_cast<long long>(tokens) * heads;
  const long long ctas = (rows + 31) / 32;
  const unsigned grid = static_cast<unsigned>(ctas < 148 * 8 ? ctas : 148 * 8);
  auto *q = static_cast<__nv_bfloat16*>(query), *k = static_cast<__nv_bfloat16*>(key);
  const NormRopeTensors tensors = {
      {q, k}, {static_cast<const __nv_bfloat16*>(query_weight), static_cast<const __nv_bfloat16*>(key_weight)}, {q, k}};
  return launch_pdl("h3_qk_norm_rope", norm_rope_kernel<2>, grid, 256, 0, stream, tensors,
                    static_cast<const float*>(cosines), static_cast<const float*>(sines), rows, heads, 1);
}

extern "C" int nob200_h3_query_prepare(int tokens, const void* source, const void* weight, const void* cosines,
                                       const void* sines, void* quantized, void* scales, int heads, void* stream) {
  using namespace nob200;
  NOB_REQUIRE(tokens > 0 && heads > 0, "h3_query_prepare: sizes must be positive");
  NOB_REQUIRE(source && weight && quantized && scales, "h3_query_prepare: NULL tensor");
  NOB_REQUIRE((cosines == nullptr) == (sines == nullptr), "h3_query_prepare: cosines and sines come together");
  const int groups = (tokens + 31) / 32;
  NOB_REQUIRE(groups <= 65535, "h3_query_prepare: %d token groups exceed the grid limit", groups);
  return launch_pdl("h3_query_prepare", query_prepare_kernel, dim3(heads, groups), 128, 0, stream,
                    static_cast<const __nv_bfloat16*>(source), static_cast<const __nv_bfloat16*>(weight),
                    static_cast<const float*>(cosines), static_cast<const float*>(sines), static_cast<int8_t*>(quantized),
                    static_cast<float*>(scales), tokens, heads, groups, cosines != nullptr);
}

// ------------------------------------------------- row-wise int8 of the projection inputs, with group rotation
// Replaces int8_rowwise (src/nano_omni/kernels/quantization/int8_rowwise.py:107-116) and convrot_int8
// (src/nano_omni/kernels/quantization/convrot_int8.py:130-161): optionally rotate every group of 256 columns by
// B (x) B (x) B (x) B / 16 with B = [[1,1,1,-1],[1,1,-1,1],[1,-1,1,1],[-1,1,1,1]], round to bf16, then one scale per
// row, max(amax / 127, 1e-30), and round-half-even to int8 in [-127, 127].
// The reference multiplies by the 256 x 256 matrix and leaves the summation order to the GEMM; here the rotation is
// four radix-4 stages over the base-4 digits of the column index, lowest digit first, each stage computing from
// (a, b, c, d) = the values at digit 0..3:  p = a + b, q = a - b, r = c + d, u = c - d;  y0 = p + u, y1 = p - u,
// y2 = q + r, y3 = r - q  (every operation rounded to fp32); the CPU restatement repeats that.
namespace nob200 {
namespace {

// Two columns at a time, one of each of two groups: the packed operations round their halves one by one.
struct Pair {
  uint64_t v;
};
__device__ __forceinline__ Pair pair_of(float lo, float hi) {
  Pair r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void halves(Pair p, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(p.v));
}
__device__ __forceinline__ Pair operator+(Pair a, Pair b) {
  Pair r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ Pair operator*(Pair a, Pair b) {
  Pair r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ Pair operator-(Pair a, Pair b) {  // b * -1 is exact: one rounding, that of the difference
  Pair r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(b.v), "l"(0xbf800000bf800000ull), "l"(a.v));
  return r;
}

__device__ __forceinline__ void radix4(Pair& a, Pair& b, Pair& c, Pair& d) {
  const Pair p = a + b, q = a - b, r = c + d, u = c - d;
  a = p + u;
  b = p - u;
  c = q + r;
  d = r - q;
}

// One CTA per row; a group of 256 columns lies on 16 lanes with 16 consecutive columns each, and a half-warp rotates two
// groups at once.  The kernel is bound by its instructions, about 30 per column one by one; with the packed rotation,
// packed rounding and the boundary test below about half (15104 x 7168: 135 us, now 105 us; 50 us of traffic).
__global__ void __launch_bounds__(128)
rowwise_int8_kernel(const __nv_bfloat16* src, int8_t* dst, float* scales,
                    int columns, int rotate) {
  pdl_wait();
  pdl_release();
  extern __shared__ __align__(16) __nv_bfloat16 rotated[];  // the row after rotation and bf16 rounding
  __shared__ float warp_max[4];
  __shared__ uint64_t transpose[8][16 * 17];  // two 256-column groups per half-warp
  const size_t row = blockIdx.x;
  const int lane16 = threadIdx.x & 15, half_warp = threadIdx.x >> 4;
  const __nv_bfloat16* in = src + row * columns;
  float amax = 0.f;
  const int groups = columns / 256;
  if (rotate) {
    // both half-warps of a warp run every round (the warp synchronises around the transpose); a group past the last
    // one is group 0 again, its result discarded.  The next round's loads are in flight during this round.
    uint4 next[2][2];
    auto fetch = [&](int first) {
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int g = first + 8 * s + half_warp;
        const uint4* at = reinterpret_cast<const uint4*>(in + (g < groups ? g : 0) * 256 + 16 * lane16);
        next[s][0] = at[0];
        next[s][1] = at[1];
      }
    };
    fetch(0);
    __nv_bfloat162 top = __floats2bfloat162_rn(0.f, 0.f);
    for (int first = 0; first < groups; first += 16) {
      const int ga = first + half_warp, gb = ga + 8;
      Pair x[16];
      const Row8 a0 = row8_of(next[0][0]), a1 = row8_of(next[0][1]), b0 = row8_of(next[1][0]), b1 = row8_of(next[1][1]);
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = pair_of(a0.v[i], b0.v[i]), x[8 + i] = pair_of(a1.v[i], b1.v[i]);
      if (first + 16 < groups) fetch(first + 16);
#pragma unroll
      for (int i = 0; i < 16; i += 4) radix4(x[i], x[i + 1], x[i + 2], x[i + 3]);  // digit 0: column stride 1
#pragma unroll
      for (int i = 0; i < 4; ++i) radix4(x[i], x[i + 4], x[i + 8], x[i + 12]);  // digit 1: column stride 4
      // digits 2 and 3 (column strides 16 and 64) lie across the lanes: transpose through shared memory so that a
      // lane holds columns lane16 + 16 r, r = 0..15, and they become register digits too (rows padded to 17 pairs)
      uint64_t* scratch = transpose[half_warp];
#pragma unroll
      for (int i = 0; i < 16; ++i) scratch[17 * lane16 + i] = x[i].v;
      __syncwarp();
#pragma unroll
      for (int r = 0; r < 16; ++r) x[r].v = scratch[17 * r + lane16];
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 16; i += 4) radix4(x[i], x[i + 1], x[i + 2], x[i + 3]);  // digit 2
#pragma unroll
      for (int i = 0; i < 4; ++i) radix4(x[i], x[i + 4], x[i + 8], x[i + 12]);  // digit 3
      const bool live_a = ga < groups, live_b = gb < groups;
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        float a, b;
        halves(x[r] * pair_of(0.0625f, 0.0625f), a, b);
        // a discarded group repeats group 0, whose maximum counts anyway
        const __nv_bfloat162 rounded = __floats2bfloat162_rn(a, b);
        top = __hmax2(top, __habs2(rounded));
        if (live_a) rotated[ga * 256 + lane16 + 16 * r] = rounded.x;
        if (live_b) rotated[gb * 256 + lane16 + 16 * r] = rounded.y;
      }
    }
    amax = fmaxf(__bfloat162float(top.x), __bfloat162float(top.y));
  } else {
    for (int c = 8 * threadIdx.x; c < columns; c += 8 * 128) {  // columns is a multiple of 8
      const uint4 raw = *reinterpret_cast<const uint4*>(in + c);
      const Row8 v = row8_of(raw);
#pragma unroll
      for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(v.v[i]));
      *reinterpret_cast<uint4*>(rotated + c) = raw;
    }
  }
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, m));
  if ((threadIdx.x & 31) == 0) warp_max[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = fmaxf(fmaxf(warp_max[0], warp_max[1]), fmaxf(warp_max[2], warp_max[3]));
  const float scale = fmaxf(amax / 127.0f, 1e-30f);
  const float inv_scale = __frcp_rn(scale);
  if (threadIdx.x == 0) scales[row] = scale;
  int8_t* out = dst + row * columns;
  const Pair inverse = pair_of(inv_scale, inv_scale), magic = pair_of(12582912.f, 12582912.f);  // 2^23 * 1.5
  for (int c = 8 * threadIdx.x; c < columns; c += 8 * 128) {
    const Row8 v = load_row8(rotated + c);
    // rint(RN(x / scale)) as in the other int8 quantisers: the product with RN(1 / scale) rounds to the same integer
    // unless it lies within 4e-5 of a half-integer (or is not finite); only then the IEEE division is done.  The adder
    // rounds to nearest even, and the low byte of product + 2^23 * 1.5 is the code (|product| <= 127 and an ulp).
    uint32_t code[8];
    bool near = false;
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      const Pair product = pair_of(v.v[i], v.v[i + 1]) * inverse;
      const Pair moved = product + magic;
      float d0, d1, t0, t1;
      halves(product - (moved - magic), d0, d1);
      halves(moved, t0, t1);
      near = near || !(fabsf(d0) <= 0.5f - 4e-5f) || !(fabsf(d1) <= 0.5f - 4e-5f);
      code[i] = __float_as_uint(t0);
      code[i + 1] = __float_as_uint(t1);
    }
    if (near) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float a = v.v[i] * inv_scale;
        float q = rintf(a);
        if (!(0.5f - fabsf(a - q) >= 4e-5f)) q = rintf(__fdiv_rn(v.v[i], scale));
        code[i] = static_cast<uint32_t>(static_cast<int>(fminf(fmaxf(q, -127.f), 127.f)));
      }
    }
    uint32_t word[2];
#pragma unroll
    for (int w = 0; w < 2; ++w)
      word[w] = __byte_perm(__byte_perm(code[4 * w], code[4 * w + 1], 0x0040),
                            __byte_perm(code[4 * w + 2], code[4 * w + 3], 0x0040), 0x5410);
    *reinterpret_cast<uint2*>(out + c) = make_uint2(word[0], word[1]);
  }
}

}  // namespace
}  // namespace nob200

extern "C" int nob200_int8_rowwise(int num_tokens, const void* input, void* output, void* scales, int columns,
                                   int rotation_group, void* stream) {
  using namespace nob200;
  NOB_REQUIRE(num_tokens > 0 && columns > 0, "int8_rowwise: sizes must be positive");
  NOB_REQUIRE(input && output && scales, "int8_rowwise: NULL tensor");
  NOB_REQUIRE(rotation_group == 0 || rotation_group == 256, "int8_rowwise: rotation group must be 0 (none) or 256 (got %d)",
              rotation_group);
  NOB_REQUIRE(columns % 8 == 0 && (rotation_group == 0 || columns % 256 == 0),
              "int8_rowwise: columns (%d) must be a multiple of 8, and of the rotation group", columns);
  NOB_REQUIRE(columns <= 65536, "int8_rowwise: at most 65536 columns (the row is staged in shared memory)");
  const size_t smem = static_cast<size_t>(columns) * 2;
  if (smem + 18 * 1024 > 48 * 1024) {  // the kernel also holds 17 KiB of static shared memory (the transpose)
    cudaError_t err = cudaFuncSetAttribute(rowwise_int8_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess)
      return fail(kCudaError, "int8_rowwise: cannot reserve %zu B of shared memory: %s", smem, cudaGetErrorString(err));
  }
  return launch_pdl("int8_rowwise", rowwise_int8_kernel, num_tokens, 128, smem, stream,
                    static_cast<const __nv_bfloat16*>(input), static_cast<int8_t*>(output), static_cast<float*>(scales),
                    columns, rotation_group == 256);
}
