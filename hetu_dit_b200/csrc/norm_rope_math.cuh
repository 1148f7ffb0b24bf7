// Per-head RMSNorm / LayerNorm and rotary embedding of eight consecutive elements in the linear kernel's epilogue
// (gemm_sm100.cu), with the rounding points of norm_rope_kernel (norm_rope.cu), so that both give the same bits.
//
// Rounding follows the reference's eager sequence: normalise in fp32, round to the 16-bit type, multiply by the 16-bit
// weight and round, rotate in fp32 with separately rounded products, round once more. Roundings are done two at a
// time (cvt.rn.bf16x2.f32 / f16x2) and the multiplication by the weight as one packed 16-bit multiplication: the fp32
// product of two 16-bit operands is exact, so rounding it is what the packed instruction does.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

namespace hdit {

template <bool FP16>
__device__ __forceinline__ uint32_t nr_pack(float lo, float hi) {
  if constexpr (FP16) {
    const __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
  } else {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
  }
}
template <bool FP16>
__device__ __forceinline__ void nr_unpack(uint32_t v, float& lo, float& hi) {
  if constexpr (FP16) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&v));
    lo = f.x;
    hi = f.y;
  } else {
    lo = __uint_as_float(v << 16);
    hi = __uint_as_float(v & 0xffff0000u);
  }
}
template <bool FP16>
__device__ __forceinline__ void nr_unpack8(const uint4& v, float (&f)[8]) {
  nr_unpack<FP16>(v.x, f[0], f[1]);
  nr_unpack<FP16>(v.y, f[2], f[3]);
  nr_unpack<FP16>(v.z, f[4], f[5]);
  nr_unpack<FP16>(v.w, f[6], f[7]);
}
template <bool FP16>
__device__ __forceinline__ uint4 nr_pack8(const float (&f)[8]) {
  return make_uint4(nr_pack<FP16>(f[0], f[1]), nr_pack<FP16>(f[2], f[3]), nr_pack<FP16>(f[4], f[5]), nr_pack<FP16>(f[6], f[7]));
}
// a * b, rounded to the 16-bit type, for two packed values
template <bool FP16>
__device__ __forceinline__ uint32_t nr_mul2(uint32_t a, uint32_t b) {
  if constexpr (FP16) {
    const __half2 v = __hmul2_rn(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b));
    return *reinterpret_cast<const uint32_t*>(&v);
  } else {
    const __nv_bfloat162 v =
        __hmul2_rn(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
    return *reinterpret_cast<const uint32_t*>(&v);
  }
}

// RMSNorm of eight elements: round(x * rstd), times the packed weight when has_w.
template <bool FP16>
__device__ __forceinline__ uint4 nr_rms8(const float (&f)[8], float rstd, bool has_w, const uint4& w) {
  uint4 y = make_uint4(nr_pack<FP16>(__fmul_rn(f[0], rstd), __fmul_rn(f[1], rstd)),
                       nr_pack<FP16>(__fmul_rn(f[2], rstd), __fmul_rn(f[3], rstd)),
                       nr_pack<FP16>(__fmul_rn(f[4], rstd), __fmul_rn(f[5], rstd)),
                       nr_pack<FP16>(__fmul_rn(f[6], rstd), __fmul_rn(f[7], rstd)));
  if (has_w) {
    y.x = nr_mul2<FP16>(y.x, w.x);
    y.y = nr_mul2<FP16>(y.y, w.y);
    y.z = nr_mul2<FP16>(y.z, w.z);
    y.w = nr_mul2<FP16>(y.w, w.w);
  }
  return y;
}

// LayerNorm of eight elements (d = x - mean): fp32 throughout, one rounding, as torch's layer_norm does for 16-bit inputs.
template <bool FP16>
__device__ __forceinline__ uint4 nr_layer8(const float (&d)[8], float rstd, bool has_w, const uint4& w, bool has_b,
                                           const uint4& b) {
  float wf[8], bf[8], o[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) wf[i] = 1.f, bf[i] = 0.f;
  if (has_w) nr_unpack8<FP16>(w, wf);
  if (has_b) nr_unpack8<FP16>(b, bf);
#pragma unroll
  for (int i = 0; i < 8; ++i) o[i] = fmaf(d[i] * rstd, wf[i], bf[i]);
  return nr_pack8<FP16>(o);
}

// Rotation of four adjacent pairs by the table rows c0, c1 (cosines) and s0, s1 (sines) of these eight elements.
template <bool FP16>
__device__ __forceinline__ uint4 nr_rotate8(const uint4& v, const float4& c0, const float4& c1, const float4& s0,
                                            const float4& s1) {
  float f[8], o[8];
  nr_unpack8<FP16>(v, f);
  const float cs[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
  const float sn[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
#pragma unroll
  for (int i = 0; i < 8; i += 2) {
    o[i] = __fadd_rn(__fmul_rn(f[i], cs[i]), __fmul_rn(-f[i + 1], sn[i]));
    o[i + 1] = __fadd_rn(__fmul_rn(f[i + 1], cs[i + 1]), __fmul_rn(f[i], sn[i + 1]));
  }
  return nr_pack8<FP16>(o);
}

}  // namespace hdit
