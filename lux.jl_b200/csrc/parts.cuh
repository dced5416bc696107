// A Float32 operand of the tensor-core kernels as three bf16 parts.
//
// x = x1 + x2 + x3, 8 significant bits each; the sum is exact for |x| >= 2^-110 (8e-34; below, the third part falls under the
// smallest bf16 and x is off by up to 2^-134). Of the nine products of two operands the six
// x1*y1, x1*y2, x2*y1, x1*y3, x3*y1, x2*y2 are formed; the three left out are below 2^-25 of x*y. (Two tf32 parts leave a bit
// of x over in every fourth value, 4e-8 of it, and their 22-bit products lose bits where the tensor core aligns them; an 8-bit
// product loses next to nothing. Six bf16 products take the tensor core as long as three tf32 products.)
//
// The tensor core truncates when it adds into TMEM. A kernel therefore takes x1*y1 out after every k-block of 32 and adds it
// round-to-nearest in fp32 registers, gathers the small products in an accumulator of their own, and puts back what the
// truncation takes away on average (parts_unbias).
#pragma once
#include "tc_ptx.cuh"

namespace lb2 {

struct Parts { uint16_t a, b, c; };
__device__ __forceinline__ float part_f32(uint16_t h) { return __uint_as_float((uint32_t)h << 16); }
__device__ __forceinline__ uint16_t part_rn(float v) { return __bfloat16_as_ushort(__float2bfloat16_rn(v)); }

// Not-a-number and infinity give what a sum of fp32 products gives. An infinity is (+-1, 0, +-Inf), NaN (1, 0, NaN): the third
// part meets only the other operand's first, so that an infinite term is formed once, with its own sign (0 * Inf included);
// where both are infinite the ones carry the sign.
__device__ __forceinline__ Parts split_parts(float v) {
  Parts p;
  const uint32_t u = __float_as_uint(v);
  if ((u & 0x7F800000u) == 0x7F800000u) {
    const bool nan = (u & 0x007FFFFFu) != 0;
    p.a = nan ? 0x3F80u : (uint16_t)(((u >> 16) & 0x8000u) | 0x3F80u);
    p.b = 0;
    p.c = nan ? 0x7FC0u : (uint16_t)(u >> 16);
    return p;
  }
  p.a = part_rn(v);
  if ((p.a & 0x7FFFu) == 0x7F80u) p.a = (uint16_t)(u >> 16);   // finite, but rounded up to infinity
  const float r = v - part_f32(p.a);
  p.b = part_rn(r);
  p.c = part_rn(r - part_f32(p.b));
  return p;
}
__device__ __forceinline__ float join_parts(const uint16_t* p, int64_t part_stride) {
  return (part_f32(__ldg(p)) + part_f32(__ldg(p + part_stride))) + part_f32(__ldg(p + 2 * part_stride));
}
// four values: one 8-byte store per part; eight: one 16-byte store
__device__ __forceinline__ void pack_parts4(const float* v, uint32_t (&w)[3][2]) {
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const Parts l = split_parts(v[2 * k]), h = split_parts(v[2 * k + 1]);
    w[0][k] = l.a | ((uint32_t)h.a << 16);
    w[1][k] = l.b | ((uint32_t)h.b << 16);
    w[2][k] = l.c | ((uint32_t)h.c << 16);
  }
}
__device__ __forceinline__ void store_parts4(uint16_t* dst, int64_t part_stride, const float (&v)[4]) {
  uint32_t w[3][2];
  pack_parts4(v, w);
#pragma unroll
  for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2*>(dst + i * part_stride) = make_uint2(w[i][0], w[i][1]);
}
__device__ __forceinline__ void store_parts8(uint16_t* dst, int64_t part_stride, const float (&v)[8]) {
  uint32_t l[3][2], h[3][2];
  pack_parts4(v, l);
  pack_parts4(v + 4, h);
#pragma unroll
  for (int i = 0; i < 3; ++i) *reinterpret_cast<uint4*>(dst + i * part_stride) = make_uint4(l[i][0], l[i][1], h[i][0], h[i][1]);
}

// The products of one k-block of 32 (two k-steps), to be issued by one lane: x1*y1 into `main`, the others into `small`
// (added to what it holds, or replacing it).
__device__ __forceinline__ void parts_issue(uint32_t main, uint32_t small, uint64_t a, uint64_t b, uint32_t a_part, uint32_t b_part,
                                            uint32_t a_step, uint32_t b_step, uint32_t idesc, bool replace, uint64_t* main_done) {
  umma<false>(main, a, b, idesc, 0u);
  umma<false>(main, a + a_step, b + b_step, idesc, 1u);
  if (main_done != nullptr) umma_commit(main_done);
#pragma unroll
  for (int ks = 0; ks < 2; ++ks) {
    const uint64_t a1 = a + ks * a_step, b1 = b + ks * b_step;
    umma<false>(small, a1, b1 + 2 * b_part, idesc, replace && ks == 0 ? 0u : 1u);
    umma<false>(small, a1 + 2 * a_part, b1, idesc, 1u);
    umma<false>(small, a1 + a_part, b1 + b_part, idesc, 1u);
    umma<false>(small, a1, b1 + b_part, idesc, 1u);
    umma<false>(small, a1 + a_part, b1, idesc, 1u);
  }
}

// What the truncation of the x1*y1 accumulators (two k-steps each) takes from a sum on average, put back: kPartsLost of it
// (measured on convolutions of 18 to 4608 terms; the loss of a partial sum is proportional to it, so that of the sum of all is
// too), by way of the small products, whose last bits can hold it. It is below half a unit of the sum's own last place: a sum
// that was exact stays as it is.
constexpr float kPartsLost = 2.5e-8f;
__device__ __forceinline__ float parts_unbias(float sum, float small) { return sum + fmaf(sum, kPartsLost, small); }

}  // namespace lb2
