// Relative-position attention of the Conformer encoder on the folded operands of the attention
// fold pack (vx_qkv_pack / the QKV GEMM's fold-pack epilogue):
//
//   q2[h, t, :] = ((q + pos_u) | (q + pos_v)) / sqrt(dk)      k2[h, t, :] = k | p      v2[h, t, 0:dk] = v
//   out[t, h dk : (h + 1) dk] = softmax_j(q2[h, t, :] . k2[h, j, :]) v[h, j, :]        (keys j < kv_len)
//
// i.e. what the model computes with scaled_dot_product_attention(q2, k2, v2, scale = 1)[..., :dk] followed
// by transpose(1, 2).reshape (veloxvoice/models/wenet/torch_conformer.py:514-519; the reference's own
// CUDA kernel for the chunked case is veloxvoice/kernels/csrc/velox_chunk_rel_pos_attn.cu:23-114).  The zero
// half of v2 is never read and the result lands token-major, ready for the output projection's quantizer.
//
// One CTA = 128 queries of one head, TWO CTAs PER SM (half the shared and tensor memory each), all on the 5th-generation
// tensor cores (tcgen05.mma kind::f16, bf16 operands, fp32 accumulators in tensor memory):
//   warps 0..3  softmax, one query row per thread straight out of tensor memory, 64 keys per step;
//   warp 4      TMA producer: K and V tiles of 64 keys through two four-stage rings;
//   warp 5      MMA issuer: S = Q K^T (128 x 64 x 128), O += P V (128 x 64 x 64; V is read in its natural [key][dv] layout
//               as an MN-major operand).
// Q and P are A operands in TENSOR MEMORY: Q is put there once by the softmax warps, P (bf16) each step, so the MMAs read
// only K and V from shared memory (with Q there too they were bound by it) and no proxy fence stands between the softmax
// and P V.  P has columns of its own, so that S of step j + 1 is issued as soon as the softmax of step j has READ its S, and
// is there when the softmax gets to it.
// Tensor memory (256 columns): S (64) | P0 | P1 (32 each) | O (64) | Q (64).
// One pass over the keys with a lazily updated reference maximum: p = 2^((s - m_ref) log2 e) is formed
// against the reference m_ref the row has used so far, at first the maximum of its first 128 keys, which only moves when a
// step's maximum exceeds it by more than 2^8 (so p never exceeds 256 and nothing overflows in bf16 or fp32).  When it moves -- in
// few rows and steps -- the row sum and the row's O accumulator are multiplied by 2^((m_old - m_new) log2 e)
// (tcgen05.ld / tcgen05.st) before the next P V product is released.  O is divided by the row sum once at the end.
// What bounds it: the two softmax warps of an SM partition and the special-function unit that they share (64 exponentials per
// row and step, 16 lanes per cycle and SM: 512 cycles per CTA and step; the MMAs take 400).  3,750 frames and 8 heads: 99 us
// with one CTA per SM, P through shared memory and a maximum exchange between two warps per row (3,200 cycles per 128 x 128
// tile); 62 us with two CTAs and P over S, where the round trip of a buffer -- P V, then the S behind it -- made the softmax
// wait 340 cycles a step; 58 us with the maximum of the first 64 keys as reference, 60 with that of 128, 58 without a wait of its own for the buffer of P.  (The shared maximum in every
// pair of steps: 70 us, the softmax then waits for the second S.)  Neither eight softmax warps per CTA in two independent groups (73 us) nor a
// quarter of the exponentials as polynomials on the fp32 pipe (64 us) helped.
// Every mbarrier wait is bounded.

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "vx_common.cuh"
#include "vx_ptx.cuh"
#include "vx_quant_math.cuh"
#include "vx_tmap.cuh"

namespace vx {
namespace {

constexpr int AT_BM = 128;   // queries per CTA = TMEM lanes
constexpr int AT_BN = 64;    // keys per tile
constexpr int AT_D = 128;    // folded head dimension (2 dk)
constexpr int AT_DV = 64;    // value dimension (dk)
constexpr int AT_K_PANEL = AT_BN * 128;           // one 64-column bf16 panel of a K tile: 8 KB
constexpr int AT_K_BYTES = 2 * AT_K_PANEL;
constexpr int AT_V_BYTES = AT_BN * AT_DV * 2;     // 8 KB
constexpr int AT_NS = 4;                          // K and V tiles in flight
constexpr int AT_SMEM = AT_NS * (AT_K_BYTES + AT_V_BYTES) + 1024;
constexpr int AT_SOFTMAX_WARPS = 4;
constexpr int AT_THREADS = (AT_SOFTMAX_WARPS + 2) * 32;
constexpr uint32_t AT_TM_S = 0, AT_TM_P = 64, AT_TM_O = 128, AT_TM_Q = 192, AT_TM_COLS = 256;

struct AttnParams {
  int64_t T;        // queries and keys per head
  int64_t kv_len;   // keys j >= kv_len are masked
  int heads;
  const __nv_bfloat16* q;
  __nv_bfloat16* out;
  int64_t ldo;
  int* status;
};

struct AttnBarriers {
  uint64_t q_full, k_full[AT_NS], k_empty[AT_NS], v_full[AT_NS], v_empty[AT_NS], s_full, s_empty, p_full[2], pv_done[2], o_full;
  uint32_t tmem_base;
};

// bf16 x bf16 -> fp32, A K-major; B K-major or MN-major (b_mn)
__host__ __device__ constexpr uint32_t make_idesc_bf16(int M, int N, bool b_mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((b_mn ? 1u : 0u) << 16) | (static_cast<uint32_t>(N >> 3) << 17) |
         (static_cast<uint32_t>(M >> 4) << 24);
}
// A from tensor memory (lane = row, two consecutive K elements per 32-bit column), B from shared memory
__device__ __forceinline__ void mma_bf16_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tc_st_32x32b_x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
      "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
      "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ float ex2f(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ uint32_t bf16x2(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

__global__ void __launch_bounds__(AT_THREADS, 2)
relpos_attn_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v, const AttnParams p) {
  pdl_launch_dependents();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* const k_s = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* const v_s = k_s + AT_NS * AT_K_BYTES;
  __shared__ AttnBarriers bar;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int head = blockIdx.y;
  const int64_t q0 = static_cast<int64_t>(blockIdx.x) * AT_BM;
  const int steps = static_cast<int>((p.kv_len + AT_BN - 1) / AT_BN);
  const int row_base = static_cast<int>(head * p.T);  // this head's token 0 in the [heads * T, 128] views

  if (threadIdx.x == 0) {
    mbar_init(&bar.q_full, AT_SOFTMAX_WARPS);
    mbar_init(&bar.s_full, 1);
    mbar_init(&bar.s_empty, AT_SOFTMAX_WARPS);
    mbar_init(&bar.o_full, 1);
    for (int s = 0; s < AT_NS; ++s) {
      mbar_init(&bar.k_full[s], 1);
      mbar_init(&bar.k_empty[s], 1);
      mbar_init(&bar.v_full[s], 1);
      mbar_init(&bar.v_empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bar.p_full[s], AT_SOFTMAX_WARPS);
      mbar_init(&bar.pv_done[s], 1);
    }
    mbar_fence_init();
    prefetch_tmap(&tm_k);
    prefetch_tmap(&tm_v);
  }
  if (warp == AT_SOFTMAX_WARPS + 1) {
    tmem_alloc(&bar.tmem_base, AT_TM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bar.tmem_base;
  pdl_wait();  // set-up done: from here on the kernel touches what the previous kernel of the stream produced

  if (warp == AT_SOFTMAX_WARPS) {
    // =========================== TMA producer ===========================
    if (lane == 0) {
      auto load_k = [&](int j) {
        const int s = j % AT_NS;
        if (!mbar_wait(&bar.k_empty[s], ((j / AT_NS) & 1) ^ 1, p.status, 20)) return false;
        uint8_t* const dst = k_s + s * AT_K_BYTES;
        mbar_expect_tx(&bar.k_full[s], AT_K_BYTES);
        tma_load_2d(dst, &tm_k, 0, row_base + j * AT_BN, &bar.k_full[s]);
        tma_load_2d(dst + AT_K_PANEL, &tm_k, 64, row_base + j * AT_BN, &bar.k_full[s]);
        return true;
      };
      bool ok = load_k(0);
      for (int j = 0; j < steps && ok; ++j) {  // K runs one tile ahead of V
        if (j + 1 < steps && !load_k(j + 1)) break;
        const int s = j % AT_NS;
        if (!mbar_wait(&bar.v_empty[s], ((j / AT_NS) & 1) ^ 1, p.status, 29)) break;
        mbar_expect_tx(&bar.v_full[s], AT_V_BYTES);
        tma_load_2d(v_s + s * AT_V_BYTES, &tm_v, 0, row_base + j * AT_BN, &bar.v_full[s]);
      }
    }
  } else if (warp == AT_SOFTMAX_WARPS + 1) {
    // =========================== MMA issuer ===========================
    // (warp-uniform control flow; descriptors are one 32-bit add each: low word = shared address >> 4, constant high word)
    const bool leader = elect_one();
    const uint32_t idesc_s = make_idesc_bf16(AT_BM, AT_BN, false);
    const uint32_t idesc_o = make_idesc_bf16(AT_BM, AT_DV, true);
    const uint32_t desc_hi = (1024u >> 4) | (1u << 14) | (2u << 29);
    auto desc = [&](uint32_t lo) { return (static_cast<uint64_t>(desc_hi) << 32) | lo; };
    const uint32_t k_lo = smem_u32(k_s) >> 4, v_lo = smem_u32(v_s) >> 4;
    bool ok = mbar_wait_spin(&bar.q_full, 0, p.status, 21);
    uint32_t ks = 0, kph = 0, vs = 0, vph = 0;  // ring positions
    auto issue_s = [&]() {  // S of the next tile
      if (!mbar_wait_spin(&bar.k_full[ks], kph, p.status, 22)) return false;
      tc_fence_after();
      const uint32_t kt = k_lo + ks * (AT_K_BYTES >> 4);
#pragma unroll
      for (int i = 0; i < AT_D / 16; ++i)
        if (leader)
          mma_bf16_ta(tmem_base + AT_TM_S, tmem_base + AT_TM_Q + i * 8, desc(kt + (i >> 2) * (AT_K_PANEL >> 4) + (i & 3) * 2), idesc_s, i != 0);
      if (leader) {
        tc_commit(&bar.s_full);
        tc_commit(&bar.k_empty[ks]);
      }
      if (++ks == AT_NS) { ks = 0; kph ^= 1; }
      return true;
    };
    if (ok) ok = issue_s();
    for (int j = 0; j < steps && ok; ++j) {
      const uint32_t b = j & 1, par = (j >> 1) & 1;
      if (j + 1 < steps) {
        // the softmax of this step has read its S
        if (!mbar_wait_spin(&bar.s_empty, j & 1, p.status, 23)) { ok = false; break; }
        tc_fence_after();
        ok = issue_s();
        if (!ok) break;
      }
      if (!mbar_wait_spin(&bar.v_full[vs], vph, p.status, 30) || !mbar_wait_spin(&bar.p_full[b], par, p.status, 24)) { ok = false; break; }
      tc_fence_after();
      // V tile as TMA wrote it: one 128-byte row of 64 dv values per key, 8-key swizzle atoms 1 KB apart
      // (the stride offset of the MN-major operand); 64 dv values are one group along N, so the leading
      // offset is not used.  A K = 16 step is two atoms.
      const uint32_t vt = v_lo + vs * (AT_V_BYTES >> 4), pt = tmem_base + AT_TM_P + b * (AT_BN / 2);
#pragma unroll
      for (int i = 0; i < AT_BN / 16; ++i)
        if (leader) mma_bf16_ta(tmem_base + AT_TM_O, pt + i * 8, desc(vt + i * ((16 * 128) >> 4)), idesc_o, (j | i) != 0);
      if (leader) {
        tc_commit(&bar.pv_done[b]);
        tc_commit(&bar.v_empty[vs]);
        if (j == steps - 1) tc_commit(&bar.o_full);
      }
      if (++vs == AT_NS) { vs = 0; vph ^= 1; }
    }
  } else {
    // =========================== softmax: warps 0..3, thread = query row ===========================
    const int row = warp * 32 + lane;
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(warp * 32) << 16);
    const int64_t tq = q0 + row;
    constexpr float L2E = 1.4426950408889634f;
    const float NEG_INF = __int_as_float(0xff800000);
    {
      // this row's Q: 128 bf16 -> 64 columns
      const uint4* src = reinterpret_cast<const uint4*>(p.q + (static_cast<int64_t>(row_base) + (tq < p.T ? tq : 0)) * AT_D);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t r[32];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const uint4 u = src[h * 8 + i];
          r[4 * i] = u.x; r[4 * i + 1] = u.y; r[4 * i + 2] = u.z; r[4 * i + 3] = u.w;
        }
        tc_st_32x32b_x32(lane_addr + AT_TM_Q + h * 32, r);
      }
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar.q_full);
    }
    float m_ref = NEG_INF;  // reference maximum of the row, in units of log2 (s * log2 e)
    uint64_t la[2] = {0ull, 0ull}, lb[2] = {0ull, 0ull};  // row sums of the even and the odd steps, four partial sums each as packed pairs
    bool ok = true;
    // S of step j into registers; keys beyond kv_len (the last step of a span whose length is not a multiple of 64) count as -inf
    auto read_s = [&](int j, uint32_t (&s)[2][32]) {
      if (!__all_sync(0xffffffffu, mbar_wait_spin(&bar.s_full, j & 1, p.status, 25))) return false;
      tc_fence_after();
      tc_ld_32x32b_x32(lane_addr + AT_TM_S, s[0]);
      tc_ld_32x32b_x32(lane_addr + AT_TM_S + 32, s[1]);
      tc_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar.s_empty);  // S is in registers: that of the next step may be written
      const int n_valid = static_cast<int>(p.kv_len - static_cast<int64_t>(j) * AT_BN);  // >= 64: the whole step
      if (n_valid < AT_BN) {
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (c * 32 + i >= n_valid) s[c][i] = 0xff800000u;
      }
      return true;
    };
    auto max_s = [&](const uint32_t (&s)[2][32]) {
      float m4[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t* v = &s[q >> 1][(q & 1) * 16];
        float m = fmaxf(__uint_as_float(v[0]), __uint_as_float(v[1]));
#pragma unroll
        for (int i = 2; i < 16; i += 2) m = max3(m, __uint_as_float(v[i]), __uint_as_float(v[i + 1]));
        m4[q] = m;
      }
      return fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
    };
    // P of step j against the row's reference, its sum into l, P V released
    auto put_p = [&](int j, const uint32_t (&s)[2][32], uint64_t (&l)[2]) {
      const uint64_t k2 = pack_f32x2(L2E, L2E), n2 = pack_f32x2(-m_ref, -m_ref);
      uint32_t pk[32];
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          float x0, x1;
          unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(s[c][i]), __uint_as_float(s[c][i + 1])), k2, n2), x0, x1);
          x0 = ex2f(x0);
          x1 = ex2f(x1);
          l[(i >> 1) & 1] = add_f32x2(l[(i >> 1) & 1], pack_f32x2(x0, x1));
          pk[c * 16 + (i >> 1)] = bf16x2(x0, x1);
        }
      // (P V of step j - 2 has read this buffer: it was issued before S of step j, and the arrival that says that S is complete says so of
      // everything issued before it.  A wait of its own took 120 of 1,410 cycles a step.)
      tc_st_32x32b_x32(lane_addr + AT_TM_P + (j & 1) * (AT_BN / 2), pk);
      tc_wait_st();
      tc_fence_before();  // P and the O correction before the P V product that the arrival releases
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar.p_full[j & 1]);
    };
    int j = 0;
    {
      // The first two steps share their maximum: most rows never move their reference again, and with the first 64 keys alone
      // a row whose largest probability lies among the next 64 would have it rounded instead of exactly 1 (relative error
      // against fp64 for 128 keys, scores of standard deviation 3: 2.04e-3, 1.75e-3 like this).
      uint32_t s0[2][32], s1[2][32];
      ok = read_s(0, s0);
      if (ok) {
        float m = max_s(s0);
        if (steps > 1) ok = read_s(1, s1);
        if (steps > 1 && ok) m = fmaxf(m, max_s(s1));
        m_ref = __fmul_rn(m, L2E);
        if (ok) put_p(0, s0, la);
        if (ok && steps > 1) put_p(1, s1, lb);
      }
      j = steps > 1 ? 2 : 1;
    }
    for (; ok && j < steps; ++j) {
      uint32_t s[2][32];
      ok = read_s(j, s);
      if (!ok) break;
      const float m_step = __fmul_rn(max_s(s), L2E);
      // The reference of a row moves when the step's maximum exceeds it by more than 8.  Then the row sum and the row's O are
      // scaled by 2^(m_ref - m_step).  The tensor-memory accesses are warp-wide, so the warp goes through them when any of
      // its rows moves; the other rows scale by one.
      const bool moves = m_step > m_ref + 8.0f;
      if (__any_sync(0xffffffffu, moves)) {
        const float alpha = moves ? ex2f(m_ref - m_step) : 1.0f;  // 0 for m_ref = -inf
        if (moves) m_ref = m_step;
        const uint64_t a2 = pack_f32x2(alpha, alpha);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          la[i] = mul_f32x2(la[i], a2);
          lb[i] = mul_f32x2(lb[i], a2);
        }
        ok = __all_sync(0xffffffffu, mbar_wait_spin(&bar.pv_done[(j & 1) ^ 1], ((j - 1) >> 1) & 1, p.status, 26));  // P V of the previous step complete
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t o[32];
          tc_ld_32x32b_x32(lane_addr + AT_TM_O + h * 32, o);
          tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
          tc_st_32x32b_x32(lane_addr + AT_TM_O + h * 32, o);
        }
      }
      put_p(j, s, la);
#pragma unroll
      for (int i = 0; i < 2; ++i) {  // the other sum is next
        const uint64_t t = la[i];
        la[i] = lb[i];
        lb[i] = t;
      }
    }
    // O / l -> bf16 -> out[t, head * dk + :]
    if (ok) {
      ok = __all_sync(0xffffffffu, mbar_wait_spin(&bar.o_full, 0, p.status, 27));
    }
    if (ok) {
      tc_fence_after();
      auto sum4 = [](const uint64_t (&l)[2]) {
        float a0, a1, b0, b1;
        unpack_f32x2(l[0], a0, a1);
        unpack_f32x2(l[1], b0, b1);
        return (a0 + a1) + (b0 + b1);
      };
      const float inv = 1.0f / (sum4(la) + sum4(lb));
      __nv_bfloat16* const dst = p.out + tq * p.ldo + head * AT_DV;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t r[32];
        tc_ld_32x32b_x32(lane_addr + AT_TM_O + h * 32, r);
        tc_wait_ld();
        if (tq < p.T) {
#pragma unroll
          for (int g = 0; g < 4; ++g)
            reinterpret_cast<uint4*>(dst)[h * 4 + g] =
                make_uint4(bf16x2(__uint_as_float(r[8 * g]) * inv, __uint_as_float(r[8 * g + 1]) * inv),
                           bf16x2(__uint_as_float(r[8 * g + 2]) * inv, __uint_as_float(r[8 * g + 3]) * inv),
                           bf16x2(__uint_as_float(r[8 * g + 4]) * inv, __uint_as_float(r[8 * g + 5]) * inv),
                           bf16x2(__uint_as_float(r[8 * g + 6]) * inv, __uint_as_float(r[8 * g + 7]) * inv));
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == AT_SOFTMAX_WARPS + 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, AT_TM_COLS);
  }
}

}  // namespace
}  // namespace vx

extern "C" int vx_relpos_attention(const void* q2, const void* k2, const void* v2, int64_t T, int heads, int head_dim,
                                   int64_t kv_len, void* out, int64_t ldo, void* stream) {
  using namespace vx;
  if (T < 0 || heads <= 0) return fail(-1, "bad shape T=%lld heads=%d", (long long)T, heads);
  if (T == 0) return 0;
  if (head_dim != AT_DV) return fail(-1, "head_dim must be %d (got %d)", AT_DV, head_dim);
  if (!q2 || !k2 || !v2 || !out) return fail(-1, "q2, k2, v2 and out must not be NULL");
  if (kv_len <= 0 || kv_len > T) kv_len = T;
  if (static_cast<int64_t>(heads) * T + AT_BM >= (1ll << 31)) return fail(-1, "heads * T must stay below 2^31");
  if (!aligned16(q2) || !aligned16(k2) || !aligned16(v2) || !aligned16(out) || ldo < static_cast<int64_t>(heads) * AT_DV || (ldo * 2) % 16 != 0)
    return fail(-1, "operands must be 16-byte aligned, out rows at least heads * head_dim wide");
  CUtensorMap tk, tv;
  const int64_t rows = static_cast<int64_t>(heads) * T;
  int rc = make_tmap_2d(&tk, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, k2, rows, AT_D, AT_D * 2, 64, AT_BN);
  if (rc) return rc;
  rc = make_tmap_2d(&tv, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, v2, rows, AT_D, AT_D * 2, 64, AT_BN);
  if (rc) return rc;
  AttnParams p{};
  p.T = T; p.kv_len = kv_len; p.heads = heads;
  p.q = static_cast<const __nv_bfloat16*>(q2);
  p.out = static_cast<__nv_bfloat16*>(out); p.ldo = ldo;
  p.status = device_status_ptr();
  int dev = 0;
  VX_CUDA_OK(cudaGetDevice(&dev));
  static std::atomic<uint64_t> attr_done{0};
  const bool dev_cached = dev >= 0 && dev < 64;
  if (!dev_cached || !(attr_done.load(std::memory_order_acquire) & (1ull << dev))) {
    VX_CUDA_OK(cudaFuncSetAttribute(relpos_attn_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, AT_SMEM));
    if (dev_cached) attr_done.fetch_or(1ull << dev, std::memory_order_release);
  }
  const dim3 grid(static_cast<unsigned>((T + AT_BM - 1) / AT_BM), static_cast<unsigned>(heads));
  VX_CUDA_OK(launch_dependent(relpos_attn_kernel, grid, dim3(AT_THREADS), AT_SMEM, static_cast<cudaStream_t>(stream), tk, tv, p));
  return 0;
}
