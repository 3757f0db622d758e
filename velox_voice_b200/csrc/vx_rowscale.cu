// One linear of the reference's per-row-scaled FP4 lane on plain activations: out f32 [M, N] = quantize(x) . W^T * scales + bias.
//
// Two routes.  Ordinary sizes: the quantizer, then the tcgen05 GEMM (vx_gemm.cu).  Few rows (a streaming chunk): ONE launch,
// below.  What bounds a call of 16 rows is not work but launches: 3 us of host time each, and on the GPU a quantizer of 2.2 us
// in front of a GEMM of 6.2 us whose time is set-up, tensor maps, tensor memory and the staged store.
//
// rowscale_small_kernel: every CTA quantizes all rows itself (they come from L2; the codes stay in shared memory) while its
// slice of the weight is already on the way into registers, and multiplies with mma.sync m16n8k16 on E2M1 values
// converted to f16.  Codes are multiples of 1/2 up to 6, so products and sums are exact in fp32 and the result has the bits
// of the two-launch route whatever the order.  A warp owns 8 columns and every KW-th 128-wide chunk of K; a lane reads
// 16 bytes (32 codes) of its column's row and of its two activation rows per chunk and feeds them to the MMAs in
// memory order -- the contraction does not care which k an MMA calls which, as long as both operands agree.
// A call of 16 x 512 -> 2048 fp32, launches overlapped: 8.2 us with two -> 5.3 us; one row of 9,728 -> 512: 7.1 us.

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "vx_common.cuh"
#include "vx_ptx.cuh"
#include "vx_quant_math.cuh"

namespace vx {
namespace {

constexpr int RS_WARPS = 8;
constexpr int RS_MAX_ROWS = 64;
constexpr int64_t RS_MAX_ELEMENTS = 32768;  // rows x K that every CTA quantizes: about 1 us

struct RsParams {
  const void* x;
  int64_t ldx;
  const uint8_t* w;
  int64_t ldw;
  const uint8_t* ws;
  const float* bias;
  float* out;
  int64_t ldo;
  int M, N, K, kw_log2;  // 2^kw_log2 warps share a column group
};

// two E2M1 values (one byte) -> f16x2, four bytes at a time
__device__ __forceinline__ void e2m1_to_f16x2(uint32_t codes, uint32_t (&h)[4]) {
  asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
      "mov.b32 {b0, b1, b2, b3}, %4;\n\t"
      "cvt.rn.f16x2.e2m1x2 %0, b0;\n\t"
      "cvt.rn.f16x2.e2m1x2 %1, b1;\n\t"
      "cvt.rn.f16x2.e2m1x2 %2, b2;\n\t"
      "cvt.rn.f16x2.e2m1x2 %3, b3;\n\t}"
      : "=r"(h[0]), "=r"(h[1]), "=r"(h[2]), "=r"(h[3])
      : "r"(codes));
}
__device__ __forceinline__ void mma_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// MT: 16-row tiles.  Dynamic shared memory: codes [M][pitch], then the partial sums [warp][MT][lane] (KW > 1).
template <typename T, int MT>
__global__ void __launch_bounds__(RS_WARPS * 32) rowscale_small_kernel(const RsParams p) {
  extern __shared__ __align__(16) uint8_t smem[];
  __shared__ float row_scale_s[16 * MT], seg_max_s[RS_WARPS];
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int KW = 1 << p.kw_log2, kw = warp & (KW - 1), group = warp >> p.kw_log2;
  const int pitch = (((p.K >> 1) + 127) & ~127) + 64;  // 64 mod 128: a phase of eight lanes reads two rows without conflicts
  const int g = lane >> 2, t = lane & 3;
  const int n0 = (static_cast<int>(blockIdx.x) * (RS_WARPS >> p.kw_log2) + group) * 8;
  const int chunks = p.K >> 7;
  const int n = n0 + g < p.N ? n0 + g : p.N - 1;  // (columns beyond N: computed on the last row, not stored)
  const uint8_t* const wrow = p.w + static_cast<int64_t>(n) * p.ldw + t * 16;

  // the warp's first weight pieces (constants of the model) leave before the wait for the previous launch
  constexpr int PF = 4;
  uint4 wv[PF];
#pragma unroll
  for (int i = 0; i < PF; ++i) {
    const int c = kw + i * KW;
    wv[i] = c < chunks ? __ldg(reinterpret_cast<const uint4*>(wrow + c * 64)) : make_uint4(0, 0, 0, 0);
  }
  const int nc = n0 + 2 * t;  // this lane's two output columns
  pdl_wait();
  float col_scale[2], bias[2];  // (behind the wait: the launch before may have written the bias)
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int c = nc + i < p.N ? nc + i : p.N - 1;
    col_scale[i] = ue8m0_to_float(__ldg(p.ws + c));
    bias[i] = p.bias ? __ldg(p.bias + c) : 0.0f;
  }

  // ---- quantize: a warp per row (up to four rows: 2, 4 or 8 warps share one, every wpr-th 256-element chunk each), lane l
  // owns elements [8 l, 8 l + 8) of a chunk (as quant_kernel does)
  const int wpr = p.M > 4 ? 1 : (p.M > 2 ? 2 : (p.M > 1 ? 4 : 8)), seg = warp & (wpr - 1);
  const int kstep = 256 * wpr;
  for (int r = warp / wpr; r < p.M || wpr > 1; r += RS_WARPS) {  // (wpr > 1: one round, which every warp takes)
    const bool row_ok = r < p.M;
    const T* const x = static_cast<const T*>(p.x) + (row_ok ? r : 0) * p.ldx + lane * 8;
    constexpr int KEEP = 2;  // chunks held in registers between the two passes
    Raw8<T> keep[KEEP];
    float a = 0.0f;
    auto amax = [&](const Raw8<T>& raw) {
      uint64_t v[4];
      raw.get(v);
      a = fmaxf(a, amax8p(v));
    };
#pragma unroll
    for (int c = 0; c < KEEP; ++c) {
      const int k = seg * 256 + c * kstep;
      if (k + lane * 8 < p.K) keep[c].load(x + k);
      else keep[c].zero();
    }
#pragma unroll
    for (int c = 0; c < KEEP; ++c) amax(keep[c]);
#pragma unroll 4
    for (int k = seg * 256 + KEEP * kstep; k < p.K; k += kstep) {
      Raw8<T> raw;
      if (k + lane * 8 < p.K) raw.load(x + k);
      else raw.zero();
      amax(raw);
    }
    a = warp_max(a);
    if (wpr > 1) {
      if (lane == 0) seg_max_s[warp] = a;
      __syncthreads();
      for (int i = 0; i < wpr; ++i) a = fmaxf(a, seg_max_s[(warp & ~(wpr - 1)) + i]);
      if (!row_ok) break;
    }
    uint32_t byte;
    float rcp;
    ue8m0_from_amax(a, byte, rcp);
    if (lane == 0 && seg == 0) row_scale_s[r] = ue8m0_to_float(byte);
    uint8_t* const dst = smem + r * pitch + lane * 4;
    auto encode = [&](const Raw8<T>& raw, int k) {
      uint64_t v[4];
      raw.get(v);
      if (k + lane * 8 < p.K) *reinterpret_cast<uint32_t*>(dst + (k >> 1)) = e2m1_pack8p<true, sizeof(T) == 4>(v, rcp);
    };
#pragma unroll
    for (int c = 0; c < KEEP; ++c) encode(keep[c], seg * 256 + c * kstep);
#pragma unroll 4
    for (int k = seg * 256 + KEEP * kstep; k < p.K; k += kstep) {
      Raw8<T> raw;
      if (k + lane * 8 < p.K) raw.load(x + k);
      else raw.zero();
      encode(raw, k);
    }
    if (wpr > 1) break;
  }
  __syncthreads();

  // ---- multiply (rows beyond M: computed on the last row, not stored)
  float acc[MT][4] = {};
  auto chunk = [&](int c, const uint4& wc) {
    const uint32_t wr[4] = {wc.x, wc.y, wc.z, wc.w};
    uint32_t bh[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) e2m1_to_f16x2(wr[i], bh[i]);
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      const uint8_t* const a_src = smem + c * 64 + t * 16;
      const uint4 lo = *reinterpret_cast<const uint4*>(a_src + min(m * 16 + g, p.M - 1) * pitch);
      const uint4 hi = *reinterpret_cast<const uint4*>(a_src + min(m * 16 + 8 + g, p.M - 1) * pitch);
      const uint32_t lw[4] = {lo.x, lo.y, lo.z, lo.w}, hw[4] = {hi.x, hi.y, hi.z, hi.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        uint32_t al[4], ah[4];
        e2m1_to_f16x2(lw[i], al);
        e2m1_to_f16x2(hw[i], ah);
        mma_f16(acc[m], al[0], ah[0], al[1], ah[1], bh[i][0], bh[i][1]);
        mma_f16(acc[m], al[2], ah[2], al[3], ah[3], bh[i][2], bh[i][3]);
      }
    }
  };
#pragma unroll
  for (int i = 0; i < PF; ++i)
    if (kw + i * KW < chunks) chunk(kw + i * KW, wv[i]);
  for (int c = kw + PF * KW; c < chunks; c += 2 * KW) {
    const uint4 w0 = __ldg(reinterpret_cast<const uint4*>(wrow + c * 64));
    const bool two = c + KW < chunks;
    const uint4 w1 = two ? __ldg(reinterpret_cast<const uint4*>(wrow + (c + KW) * 64)) : w0;
    chunk(c, w0);
    if (two) chunk(c + KW, w1);
  }
  if (KW > 1) {
    float4* const part = reinterpret_cast<float4*>(smem + p.M * pitch);
#pragma unroll
    for (int m = 0; m < MT; ++m) part[(warp * MT + m) * 32 + lane] = make_float4(acc[m][0], acc[m][1], acc[m][2], acc[m][3]);
    __syncthreads();
    if (kw != 0) return;
    for (int o = 1; o < KW; ++o)
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        const float4 v = part[((warp + o) * MT + m) * 32 + lane];
        acc[m][0] += v.x; acc[m][1] += v.y; acc[m][2] += v.z; acc[m][3] += v.w;
      }
  }
  const bool pair = nc + 1 < p.N && ((p.ldo & 1) == 0) && ((reinterpret_cast<uintptr_t>(p.out) & 7) == 0);
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = m * 16 + h * 8 + g;
      if (r < p.M && nc < p.N) {
        const float rs = row_scale_s[r];
        // the order of the GEMM's epilogue: product * row scale * column scale, then the bias
        float z0 = acc[m][2 * h] * rs * col_scale[0], z1 = acc[m][2 * h + 1] * rs * col_scale[1];
        if (p.bias) {
          z0 = __fadd_rn(z0, bias[0]);
          z1 = __fadd_rn(z1, bias[1]);
        }
        float* const o = p.out + r * p.ldo + nc;
        if (pair) {
          *reinterpret_cast<float2*>(o) = make_float2(z0, z1);
        } else {
          o[0] = z0;
          if (nc + 1 < p.N) o[1] = z1;
        }
      }
    }
}

template <typename T, int MT>
int launch_small(const RsParams& p, int grid, cudaStream_t st) {
  const size_t pitch = (((p.K >> 1) + 127) & ~127) + 64;
  const size_t smem = p.M * pitch + (p.kw_log2 ? RS_WARPS * MT * 32 * 16 : 0);  // at most 45 KB
  VX_CUDA_OK(launch_dependent(rowscale_small_kernel<T, MT>, dim3(grid), dim3(RS_WARPS * 32), smem, st, p));
  return 0;
}

bool small_route(int64_t M, int64_t N, int64_t K) {
  return M <= RS_MAX_ROWS && K % 128 == 0 && M * K <= RS_MAX_ELEMENTS && N < (1 << 30);
}

}  // namespace
}  // namespace vx

extern "C" {

int64_t vx_rowscale_linear_scratch(int64_t M, int64_t N, int64_t K) { return vx::small_route(M, N, K) ? 0 : M * (K / 2 + 1); }

int vx_rowscale_linear(const void* x, int x_dtype, int64_t M, int64_t K, int64_t ldx, const void* w_codes, int64_t ldw,
                       const void* w_scales, int64_t N, const float* bias, void* scratch, float* out, int64_t ldo, void* stream) {
  using namespace vx;
  if (x_dtype != VX_F32 && x_dtype != VX_BF16) return fail(-1, "x_dtype must be VX_F32 or VX_BF16");
  if (M < 0 || N < 0 || K <= 0) return fail(-1, "bad shape M=%lld N=%lld K=%lld", (long long)M, (long long)N, (long long)K);
  if (M == 0 || N == 0) return 0;
  if (small_route(M, N, K)) {
    const int64_t esz = x_dtype == VX_BF16 ? 2 : 4;
    if (!x || !aligned16(x) || ldx < K || (ldx * esz) % 16 != 0) return fail(-1, "x rows must be 16-byte aligned (ldx=%lld)", (long long)ldx);
    if (!w_codes || !aligned16(w_codes) || ldw % 16 != 0 || ldw < K / 2) return fail(-1, "weight rows must be 16-byte aligned and at least K / 2 bytes");
    if (!w_scales || !out || ldo < N) return fail(-1, "w_scales and out must not be NULL, ldo >= N");
    RsParams p{};
    p.x = x; p.ldx = ldx;
    p.w = static_cast<const uint8_t*>(w_codes); p.ldw = ldw;
    p.ws = static_cast<const uint8_t*>(w_scales);
    p.bias = bias;
    p.out = out; p.ldo = ldo;
    p.M = static_cast<int>(M); p.N = static_cast<int>(N); p.K = static_cast<int>(K);
    // as many warps on one column group as there are chunks of K, while the CTAs stay within two rounds
    const int groups = static_cast<int>((N + 7) / 8), chunks = static_cast<int>(K / 128);
    auto ctas = [&](int lg) { return (groups + (RS_WARPS >> lg) - 1) / (RS_WARPS >> lg); };
    while (p.kw_log2 < 3 && (2 << p.kw_log2) <= chunks && ctas(p.kw_log2 + 1) <= 2 * sm_count()) ++p.kw_log2;
    const int grid = ctas(p.kw_log2), mt = M <= 16 ? 1 : (M <= 32 ? 2 : 4);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (x_dtype == VX_BF16)
      return mt == 1 ? launch_small<__nv_bfloat16, 1>(p, grid, st) : (mt == 2 ? launch_small<__nv_bfloat16, 2>(p, grid, st) : launch_small<__nv_bfloat16, 4>(p, grid, st));
    return mt == 1 ? launch_small<float, 1>(p, grid, st) : (mt == 2 ? launch_small<float, 2>(p, grid, st) : launch_small<float, 4>(p, grid, st));
  }
  if (!scratch || !aligned16(scratch)) return fail(-1, "scratch must be 16-byte aligned");
  uint8_t* const codes = static_cast<uint8_t*>(scratch);
  uint8_t* const scales = codes + M * (K / 2);
  const int rc = quantize_rowscale_activation(x, x_dtype, M, K, ldx, codes, scales, stream);
  if (rc) return rc;
  vx_gemm_desc d{};
  d.struct_size = static_cast<int32_t>(sizeof(d));
  d.fmt = VX_FMT_ROWSCALE;
  d.M = M; d.N = N; d.K = K;
  d.a_codes = codes; d.lda = K / 2;
  d.b_codes = w_codes; d.ldb = ldw;
  d.a_scales = scales; d.b_scales = w_scales;
  d.epilogue = bias ? VX_EPI_BIAS : VX_EPI_NONE;
  d.bias = bias;
  d.out_dtype = VX_F32; d.out = out; d.ldo = ldo;
  d.flags = VX_GEMM_CONST_B;
  return vx_bsgemm(&d, stream);
}

}  // extern "C"
