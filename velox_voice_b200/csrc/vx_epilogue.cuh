// Device-side arithmetic of the fused epilogues: Swish and GLU on accumulator registers, and the quantization of a finished
// 32-column chunk of one row (shared by the GEMM kernels and the whole-encoder kernel of short passes).
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "vx_common.cuh"
#include "vx_ptx.cuh"
#include "vx_quant_math.cuh"

namespace vx {

// sigmoid(g) = 1 / (1 + 2^(-g log2 e)) via ex2.approx + rcp.approx (relative error ~1e-6).  Alternatives measured and
// rejected: tanh.approx (one MUFU operation, but its 2^-11 error flips FP4 codes / bf16
// roundings of the re-quantized activations often enough to move CTC argmaxes), and a Newton
// reciprocal on the FMA pipe (one MUFU operation less, six instructions more: 20 % slower).
// ex2 / rcp with the .ftz qualifier are single MUFU instructions (the default forms wrap them
// in range fix-ups for denormal inputs / results).  Results are the same here: a flushed
// 2^x only ever feeds 1 + 2^x, and the reciprocal of a denominator above 2^126 belongs to
// |z| > 87, whose product rounds to zero in bf16 / FP4 either way.
__device__ __forceinline__ float ex2_ftz(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp_ftz(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float sigmoid_f(float z) { return rcp_ftz(1.0f + ex2_ftz(-1.4426950408889634f * z)); }
// Four Swish values z * sigmoid(z), held as two packed pairs za = (z0, z1), zb = (z2, z3), with
// ONE reciprocal (the special-function unit is the busiest pipe of the Swish epilogues) and packed
// fp32x2 arithmetic (their cost is instruction issue):
//   d = 1 + 2^min(-z log2 e, 30)                          mul.f32x2, min, ex2 (MUFU), add.f32x2
//   A = (d0, d1), B = (d2, d3), P = A * B = (d0 d2, d1 d3), r = 1 / (P.lo P.hi)
//   (r P.hi, r P.lo) * B = (1/d0, 1/d1),   (r P.hi, r P.lo) * A = (1/d2, 1/d3)
// -- 1.25 special-function operations per value, seven packed / scalar multiplies per four.
// The exponent is capped at 2^30 so the product of four cannot overflow; a sigmoid below 2^-30
// only occurs for z < -20.8, where z * sigmoid(z) is below 1e-7 in magnitude either way.
// Every Swish of the library goes through this function, so the fp32 / bf16 outputs and the FP4
// re-quantized output of the same GEMM see the same bits.
__device__ __forceinline__ float tanh_approx(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// The TANH form on h = z / 2 (already halved).
__device__ __forceinline__ void swish4p_half(uint64_t& ha, uint64_t& hb) {
  float h0, h1, h2, h3;
  unpack_f32x2(ha, h0, h1);
  unpack_f32x2(hb, h2, h3);
  ha = fma_f32x2(ha, pack_f32x2(tanh_approx(h0), tanh_approx(h1)), ha);
  hb = fma_f32x2(hb, pack_f32x2(tanh_approx(h2), tanh_approx(h3)), hb);
}
//
// TANH = true: z sigmoid(z) = h + h tanh(h), h = z / 2, with tanh.approx -- one special-function
// operation, one packed multiply and one packed fused multiply-add per pair: 2 instructions per value
// instead of 5 (these epilogues are bound by instruction issue).  Used by the GEMMs whose operands carry
// power-of-two block scales (MX32, per-row): there the activation is re-quantized with power-of-two
// scales too, which absorbs the difference -- the 12-block MX32 stack still reproduces the CPU
// oracle's logits bit for bit (T = 1000) and agrees in every arg-max at M = 24000.  The formats with
// fp32 / E4M3 scales (NV16, FP8) keep the exponential form: their scales move with the last bits of a
// block maximum, and the same swap costs them arg-max agreement over 12 blocks (NV16 1.000 -> 0.991,
// FP8 0.992 -> 0.966 against the oracle in kernel order).
template <bool TANH>
__device__ __forceinline__ void swish4p(uint64_t& za, uint64_t& zb) {
  if constexpr (TANH) {
    const uint64_t half2 = pack_f32x2(0.5f, 0.5f);
    za = mul_f32x2(za, half2);
    zb = mul_f32x2(zb, half2);
    swish4p_half(za, zb);
    return;
  }
  const uint64_t nl2e = pack_f32x2(-1.4426950408889634f, -1.4426950408889634f);
  const uint64_t one2 = pack_f32x2(1.0f, 1.0f);
  float t0, t1, t2, t3;
  unpack_f32x2(mul_f32x2(za, nl2e), t0, t1);
  unpack_f32x2(mul_f32x2(zb, nl2e), t2, t3);
  const uint64_t da = add_f32x2(pack_f32x2(ex2_ftz(fminf(t0, 30.0f)), ex2_ftz(fminf(t1, 30.0f))), one2);
  const uint64_t db = add_f32x2(pack_f32x2(ex2_ftz(fminf(t2, 30.0f)), ex2_ftz(fminf(t3, 30.0f))), one2);
  float p0, p1;
  unpack_f32x2(mul_f32x2(da, db), p0, p1);
  const float rr = rcp_ftz(__fmul_rn(p0, p1));
  const uint64_t rp = mul_f32x2(pack_f32x2(p1, p0), pack_f32x2(rr, rr));
  za = mul_f32x2(za, mul_f32x2(rp, db));
  zb = mul_f32x2(zb, mul_f32x2(rp, da));
}
template <bool TANH>
__device__ __forceinline__ void silu4_f(float& z0, float& z1, float& z2, float& z3) {
  uint64_t za = pack_f32x2(z0, z1), zb = pack_f32x2(z2, z3);
  swish4p<TANH>(za, zb);
  unpack_f32x2(za, z0, z1);
  unpack_f32x2(zb, z2, z3);
}

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// Swish + re-quantization of one 32-column chunk of one output row, straight from the accumulator
// registers to E2M1 codes: the epilogue of the FFN up-projection, whose cost is instruction issue
// (one thread per row, 32 values each), so everything that can is done two values per
// instruction with the packed fp32x2 forms:
//   z = acc (* tensor scales) + bias                      add.f32x2 (mul.f32x2)
//   s = z * sigmoid(z)                                    swish4p, four values at a time
//   block maximum with three-input max; the E2M1 encode of e2m1_pack8p.
// NV16 = false: one UE8M0 scale for the 32 values; true: two E4M3 scales (16 values each).
// Returns the scale byte(s), little end first.
// Eight accumulator values r[8 g .. 8 g + 7] -> (* tensor scales) + bias -> Swish, as four packed pairs.
template <bool NV16, bool BIAS>
__device__ __forceinline__ void swish_group8(const uint32_t (&r)[32], int g, const float* bias_s, bool scale_acc,
                                             uint64_t g2, uint64_t (&out)[4]) {
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int q4 = 2 * g + i;
    uint64_t za = pack_f32x2(__uint_as_float(r[4 * q4]), __uint_as_float(r[4 * q4 + 1]));
    uint64_t zb = pack_f32x2(__uint_as_float(r[4 * q4 + 2]), __uint_as_float(r[4 * q4 + 3]));
    if (NV16 && scale_acc) {
      za = mul_f32x2(za, g2);
      zb = mul_f32x2(zb, g2);
    }
    if constexpr (!NV16) {
      // (acc + bias) / 2 = fma(acc, 1/2, bias / 2) bit for bit; the caller's table holds bias / 2
      const uint64_t half2 = pack_f32x2(0.5f, 0.5f);
      if constexpr (BIAS) {
        uint64_t ba, bb;
        ld_shared_pairs(smem_u32(bias_s) + 16 * q4, ba, bb);
        za = fma_f32x2(za, half2, ba);
        zb = fma_f32x2(zb, half2, bb);
      } else {
        za = mul_f32x2(za, half2);
        zb = mul_f32x2(zb, half2);
      }
      swish4p_half(za, zb);
    } else {
      if constexpr (BIAS) {
        uint64_t ba, bb;
        ld_shared_pairs(smem_u32(bias_s) + 16 * q4, ba, bb);
        za = add_f32x2(za, ba);
        zb = add_f32x2(zb, bb);
      }
      swish4p<false>(za, zb);
    }
    out[2 * i] = za;
    out[2 * i + 1] = zb;
  }
}
// Block scale(s) of 32 finished values (16 packed pairs): the scale byte(s), little end first, and
// the reciprocal(s) to normalise with (NV16: rcp0 for values 0..15, rcp1 for 16..31).
template <bool NV16>
__device__ __forceinline__ uint32_t chunk_scales_p(const uint64_t (&sv)[16], const Nv16Tensor& nv, const float* nv_tab, float& rcp0, float& rcp1) {
  if constexpr (!NV16) {
    float a = 0.0f;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      float lo, hi;
      unpack_f32x2(sv[j], lo, hi);
      a = max3(a, fabsf(lo), fabsf(hi));
    }
    uint32_t byte;
    ue8m0_from_amax(a, byte, rcp0);
    rcp1 = rcp0;
    return byte;
  } else {
    uint32_t sb = 0;
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      float a = 0.0f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float lo, hi;
        unpack_f32x2(sv[8 * hh + j], lo, hi);
        a = max3(a, fabsf(lo), fabsf(hi));
      }
      uint32_t byte;
      float rcp;
      nv.block(a, nv_tab, byte, rcp);
      if (hh == 0) rcp0 = rcp; else rcp1 = rcp;
      sb |= byte << (8 * hh);
    }
    return sb;
  }
}
// Codes of values 8 g .. 8 g + 7 of a finished chunk.
template <bool NV16>
__device__ __forceinline__ uint32_t encode_group8(const uint64_t (&sv)[16], int g, float rcp0, float rcp1) {
  const uint64_t v[4] = {sv[4 * g], sv[4 * g + 1], sv[4 * g + 2], sv[4 * g + 3]};
  return e2m1_pack8p<false, true>(v, NV16 && g >= 2 ? rcp1 : rcp0);
}

// ... in two steps: the Swish values of the chunk, and their scales and codes.
template <bool NV16>
__device__ __forceinline__ void swish_chunk(const uint32_t (&r)[32], const float* bias_s, bool scale_acc, float g_ab, uint64_t (&sv)[16]) {
  const uint64_t g2 = pack_f32x2(g_ab, g_ab);
  // (the bias test once per chunk, not once per four values: the epilogue is bound by instruction issue)
  if (bias_s) {
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      uint64_t o[4];
      swish_group8<NV16, true>(r, g, bias_s, scale_acc, g2, o);
#pragma unroll
      for (int j = 0; j < 4; ++j) sv[4 * g + j] = o[j];
    }
  } else {
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      uint64_t o[4];
      swish_group8<NV16, false>(r, g, bias_s, scale_acc, g2, o);
#pragma unroll
      for (int j = 0; j < 4; ++j) sv[4 * g + j] = o[j];
    }
  }
}
template <bool NV16>
__device__ __forceinline__ uint32_t quant_chunk(const uint64_t (&sv)[16], const Nv16Tensor& nv, const float* nv_tab, uint32_t (&w)[4]) {
  float rcp0, rcp1;
  const uint32_t sbytes = chunk_scales_p<NV16>(sv, nv, nv_tab, rcp0, rcp1);
#pragma unroll
  for (int g = 0; g < 4; ++g) w[g] = encode_group8<NV16>(sv, g, rcp0, rcp1);
  return sbytes;
}
template <bool NV16>
__device__ __forceinline__ uint32_t swish_quant_chunk(const uint32_t (&r)[32], const float* bias_s, bool scale_acc,
                                                      float g_ab, const Nv16Tensor& nv, const float* nv_tab, uint32_t (&w)[4]) {
  uint64_t sv[16];
  swish_chunk<NV16>(r, bias_s, scale_acc, g_ab, sv);
  return quant_chunk<NV16>(sv, nv, nv_tab, w);
}

// z += 32 bias values cached in shared memory (all lanes read the same words), two at a time: each half rounds like the scalar addition.
// (Scalar additions of a float4: GLU of 90,000 x 512 x 1,024 37.8 us and 34.3 like this, FP8 q | k | v 129.9 and 126.2, FFN-down 68.6 and 67.8,
// fp32 results of 1,537 rows 6.50 and 6.20.)  PAIRS = false, one at a time, for the residual epilogue whose output is chosen at run time: there the pairs cost
// registers of its long tail.  NVFP4 residual with fp32 output, 512 x 512, pairs / one at a time: 90,000 rows 74.4 and 63.7 us, 24,000 21.5 and 19.5, 1,537 6.27
// and 5.99; MX32 1,537 rows 6.31 and 5.98, 90,000 61.7 and 62.8; FP8 with an fp32 residual 1,537 rows 16.3 and 15.9.
template <bool PAIRS = true>
__device__ __forceinline__ void add_bias32(float (&z)[32], const float* bias_s) {
  if constexpr (!PAIRS) {
#pragma unroll
    for (int i = 0; i < 32; i += 4) {
      const float4 b = *reinterpret_cast<const float4*>(bias_s + i);
      z[i] = __fadd_rn(z[i], b.x); z[i + 1] = __fadd_rn(z[i + 1], b.y);
      z[i + 2] = __fadd_rn(z[i + 2], b.z); z[i + 3] = __fadd_rn(z[i + 3], b.w);
    }
    return;
  }
  const uint32_t addr = smem_u32(bias_s);
#pragma unroll
  for (int i = 0; i < 32; i += 4) {
    uint64_t ba, bb;
    ld_shared_pairs(addr + 4 * i, ba, bb);
    unpack_f32x2(add_f32x2(pack_f32x2(z[i], z[i + 1]), ba), z[i], z[i + 1]);
    unpack_f32x2(add_f32x2(pack_f32x2(z[i + 2], z[i + 3]), bb), z[i + 2], z[i + 3]);
  }
}

// The bf16 values of a 32-column chunk quantized to E2M1 as the stand-alone quantizer does it on a bf16 tensor: codes and
// scale bytes (1 or 2, little end first).
__device__ __forceinline__ uint32_t quant_bf16_chunk(const int out_fmt, const float (&z)[32], float g_out, uint32_t (&w)[4]) {
  uint64_t v[4][4];
  float a[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t pk = pack_bf16x2(z[8 * q + 2 * i], z[8 * q + 2 * i + 1]);
      v[q][i] = pack_f32x2(__uint_as_float(pk << 16), __uint_as_float(pk & 0xffff0000u));
    }
    a[q] = amax8p(v[q]);
  }
  uint32_t byte;
  float rcp;
  if (out_fmt == VX_FMT_MX32) {
    ue8m0_from_amax(fmaxf(max3(a[0], a[1], a[2]), a[3]), byte, rcp);
#pragma unroll
    for (int q = 0; q < 4; ++q) w[q] = e2m1_pack8p<true, false>(v[q], rcp);
    return byte;
  }
  uint32_t sbytes = 0;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    nv16_block(fmaxf(a[2 * h], a[2 * h + 1]), g_out, byte, rcp);
#pragma unroll
    for (int q = 0; q < 2; ++q) w[2 * h + q] = e2m1_pack8p<true, true>(v[2 * h + q], rcp);
    sbytes |= byte << (8 * h);
  }
  return sbytes;
}

}  // namespace vx
