// Top-k of the CTC log-probabilities through bf16 logits that never leave the L2 cache.
//
// The prefix beam search takes torch.topk(log_softmax(ctc_lo(x)), k).  The head's GEMM writes the bf16 logits of a block
// of rows (vx_ctc_topk_rows, about 60 MB: half of the L2) into a scratch buffer, and the kernel below reads them back from
// L2, one warp per row: log-sum-exp and the k largest values.  Against the route without
// logits (two launches of the head, the second with a candidate test in its epilogue, a threshold kernel, a finish
// kernel and a host check for overflowed candidate lists) that is half the matrix work and no synchronisation.

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "vx_common.cuh"
#include "vx_ptx.cuh"
#include "vx_quant_math.cuh"

namespace vx {
namespace {

constexpr int TK_WARPS = 8;
constexpr int TK_CAND = 128;  // candidate list of a row; more (many equal logits): exact rescans instead

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// order-preserving bits of a bf16 value held as fp32, lowest column first among equals
__device__ __forceinline__ unsigned long long topk_key(float z, int col) {
  const uint32_t x = __float_as_uint(z);
  const uint32_t u = x ^ (static_cast<uint32_t>(static_cast<int32_t>(x) >> 31) | 0x80000000u);
  return (static_cast<unsigned long long>(u) << 32) | (0xffffffffu - static_cast<uint32_t>(col));
}
__device__ __forceinline__ unsigned long long warp_max_u64(unsigned long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
    v = w > v ? w : v;
  }
  return v;
}
__device__ __forceinline__ void unpack8(const uint4& u, float (&z)[8]) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    z[2 * i] = __uint_as_float(w[i] << 16);
    z[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}

// One warp per row.  Pass 1: every lane's running (max, sum of 2^((z - max) log2 e)) over its 16-byte pieces, merged into the
// row's log-sum-exp.  The k-th largest of the 32 lane maxima is a threshold that at least k logits reach and each of the k
// largest does; pass 2 (the row again, from L1) collects what reaches it -- a few more than k -- and the k largest of the
// list are taken in order.  Bound by instruction issue: 1,670 warp instructions per row of 1,000 columns.
__global__ void __launch_bounds__(TK_WARPS * 32) topk_rows_kernel(const __nv_bfloat16* logits, int64_t ld, int N, int M,
                                                                  int k, float* logp, int64_t* ids) {
  __shared__ unsigned long long cand_s[TK_WARPS][TK_CAND];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int row = static_cast<int>(blockIdx.x) * TK_WARPS + w;
  pdl_launch_dependents();
  pdl_wait();
  if (row >= M) return;
  constexpr float L2E = 1.4426950408889634f;
  const uint4* const src = reinterpret_cast<const uint4*>(logits + static_cast<int64_t>(row) * ld);
  const int pieces = (N + 7) >> 3;
  auto load = [&](int c, float (&z)[8]) {
    unpack8(src[c], z);
    if (8 * c + 8 > N) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (8 * c + i >= N) z[i] = -INFINITY;
    }
  };
  float m = -INFINITY, s = 0.0f, nb = 0.0f;  // nb = -m log2 e; 0 while only masked columns came: they add 2^-inf = 0
#pragma unroll 4
  for (int c = lane; c < pieces; c += 32) {
    float z[8];
    load(c, z);
    float cm = max3(z[0], z[1], z[2]);
    cm = max3(cm, z[3], z[4]);
    cm = max3(cm, z[5], z[6]);
    cm = max3(cm, z[7], m);
    if (cm > m) {
      s *= ex2_approx((m - cm) * L2E);  // m = -inf: 0
      m = cm;
      nb = -m * L2E;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) s += ex2_approx(fmaf(z[i], L2E, nb));
  }
  // The maximum itself adds 1 to s.  With columns masked by a large negative value the rounding of m log2 e is no longer small
  // against 1, or the product overflows: s is then not the sum of at most N ones, or no number, and is formed again from the
  // exact differences (as a branch in the loop above that took 51.9 us for 3,750 frames, 49.3 without).
  if (m > -INFINITY && !(s >= 0.5f && s <= 2.0f * static_cast<float>(N))) {
    s = 0.0f;
    for (int c = lane; c < pieces; c += 32) {
      float z[8];
      load(c, z);
#pragma unroll
      for (int i = 0; i < 8; ++i) s += ex2_approx((z[i] - m) * L2E);
    }
  }
  float rm = m;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) rm = fmaxf(rm, __shfl_xor_sync(0xffffffffu, rm, o));
  float rs = m > -INFINITY ? s * ex2_approx((m - rm) * L2E) : 0.0f;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) rs += __shfl_xor_sync(0xffffffffu, rs, o);
  const float lse = rm + logf(rs);
  // threshold: the lane maximum of rank k - 1
  int rank = 0;
#pragma unroll
  for (int l = 0; l < 32; ++l) {
    const float o = __shfl_sync(0xffffffffu, m, l);
    rank += (o > m || (o == m && l < lane)) ? 1 : 0;
  }
  const uint32_t who = __ballot_sync(0xffffffffu, rank == k - 1);
  const float thr = __shfl_sync(0xffffffffu, m, __ffs(who) - 1);

  int n = 0;  // candidates of the row
  for (int c0 = 0; c0 < pieces; c0 += 32) {
    const int c = c0 + lane;
    float z[8];
    float cm = -INFINITY;
    if (c < pieces) {
      load(c, z);
      cm = max3(z[0], z[1], z[2]);
      cm = max3(cm, z[3], z[4]);
      cm = max3(cm, z[5], z[6]);
      cm = fmaxf(cm, z[7]);
    }
    if (__any_sync(0xffffffffu, c < pieces && cm >= thr)) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const bool hit = c < pieces && 8 * c + i < N && z[i] >= thr;
        const uint32_t b = __ballot_sync(0xffffffffu, hit);
        const int at = n + __popc(b & ((1u << lane) - 1u));
        if (hit && at < TK_CAND) cand_s[w][at] = topk_key(z[i], 8 * c + i);
        n += __popc(b);
      }
    }
  }
  __syncwarp();
  unsigned long long mine[TK_CAND / 32];
#pragma unroll
  for (int j = 0; j < TK_CAND / 32; ++j) mine[j] = j * 32 + lane < n ? cand_s[w][j * 32 + lane] : 0ull;
  unsigned long long last = ~0ull;
  for (int j = 0; j < k; ++j) {
    unsigned long long best = 0;
    if (n <= TK_CAND) {
#pragma unroll
      for (int t = 0; t < TK_CAND / 32; ++t)
        if (mine[t] < last && mine[t] > best) best = mine[t];
    } else {
      for (int c = lane; c < pieces; c += 32) {
        float z[8];
        load(c, z);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const unsigned long long e = topk_key(z[i], 8 * c + i);
          if (8 * c + i < N && e < last && e > best) best = e;
        }
      }
    }
    best = warp_max_u64(best);
    last = best;
    if (lane == 0) {
      const uint32_t u = static_cast<uint32_t>(best >> 32);
      const float z = __uint_as_float((u & 0x80000000u) ? (u ^ 0x80000000u) : ~u);
      ids[static_cast<int64_t>(row) * k + j] = best ? static_cast<int64_t>(0xffffffffu - static_cast<uint32_t>(best)) : -1;
      logp[static_cast<int64_t>(row) * k + j] = best ? z - lse : -INFINITY;
    }
  }
}

// The same for rows of 1,025 to 6,144 columns, which a warp holds in registers (8, 16 or 24 pieces of 16 bytes a lane): the row is read
// once, with all loads of a lane in flight, maxima are taken on packed bf16 pairs, the log-sum-exp against the row's maximum
// without running rescales.  The threshold is found by one integer reduction per rank; the pieces that hold a value reaching it
// (few more than k) are listed, and only their values are looked at one by one.  About 1,670 warp instructions per row of 5,538
// where two passes over the row with a running maximum issued 3,300.  Head's GEMM, selection and LayerNorm quantizer of 3,750 rows:
// 49 us with two passes, 33.4 like this.  (Four warps per row, 2.5 us more: what each repeats costs more than the shorter chain gives.)
constexpr int TR_WARPS = 8, TR_LIST = 64, TR_MIN_N = 1024;
template <int PIECES, int BLOCKS>
__global__ void __launch_bounds__(TR_WARPS * 32, BLOCKS) topk_regs_kernel(const __nv_bfloat16* logits, int64_t ld, int N, int M, int k,
                                                                          float* logp, int64_t* ids) {
  __shared__ unsigned long long cand_s[TR_WARPS][TK_CAND];
  __shared__ int list_s[TR_WARPS][TR_LIST];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t row = static_cast<int64_t>(blockIdx.x) * TR_WARPS + w;
  pdl_launch_dependents();
  pdl_wait();
  if (row >= M) return;
  constexpr float L2E = 1.4426950408889634f;
  const __nv_bfloat16* const z0 = logits + row * ld;
  const uint4* const src = reinterpret_cast<const uint4*>(z0);
  const int full = N >> 3, pieces = (N + 7) >> 3;
  constexpr uint32_t NONE = 0xff80ff80u;  // two bf16 -inf
  // Piece j * 32 + lane in slot j.  A ragged last piece goes to the last slot, lane 0, unless that holds it anyway: so only one slot
  // is masked (all of them, 24 pieces: 15,000 rows of 1,025 columns 51 us, where 1,032 columns took 40).
  constexpr int LAST = PIECES - 1;
  const bool moved = pieces <= LAST * 32;
  const int last_c = !moved ? LAST * 32 + lane : (lane == 0 ? full : pieces);  // (N a multiple of 8: full == pieces, none)
  uint4 u[PIECES];
#pragma unroll
  for (int j = 0; j < PIECES; ++j) {
    const int c = j == LAST ? last_c : j * 32 + lane;
    u[j] = make_uint4(NONE, NONE, NONE, NONE);
    if (c < (j == LAST ? pieces : full)) u[j] = src[c];
  }
  if (last_c == full && full < pieces) {
    uint32_t* const x = reinterpret_cast<uint32_t*>(&u[LAST]);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int valid = (N & 7) - 2 * i;
      if (valid <= 0) x[i] = NONE;
      else if (valid == 1) x[i] = (x[i] & 0xffffu) | (NONE & 0xffff0000u);
    }
  }
  auto used = [&](int j) { return j == LAST ? !moved || full < pieces : j * 32 < pieces; };  // (the same for all lanes)
  auto b2 = [](const uint32_t& x) { return *reinterpret_cast<const __nv_bfloat162*>(&x); };
  __nv_bfloat162 m4[4] = {b2(u[0].x), b2(u[0].y), b2(u[0].z), b2(u[0].w)};
#pragma unroll
  for (int j = 1; j < PIECES; ++j) {
    if (used(j)) {
      m4[0] = __hmax2(m4[0], b2(u[j].x));
      m4[1] = __hmax2(m4[1], b2(u[j].y));
      m4[2] = __hmax2(m4[2], b2(u[j].z));
      m4[3] = __hmax2(m4[3], b2(u[j].w));
    }
  }
  const __nv_bfloat162 mm = __hmax2(__hmax2(m4[0], m4[1]), __hmax2(m4[2], m4[3]));
  const float m = fmaxf(fmaxf(__low2float(mm), __high2float(mm)), -INFINITY);  // (a lane of NaNs only: -inf)
  // order-preserving bits of the lane's maximum in the high half, the lane below: all different
  uint32_t key, top = 0, kth = 0;
  {
    const uint32_t x = __float_as_uint(__fadd_rn(m, 0.0f));
    key = ((x ^ (static_cast<uint32_t>(static_cast<int32_t>(x) >> 31) | 0x80000000u)) & 0xffff0000u) | static_cast<uint32_t>(31 - lane);
  }
  for (int r = 0; r < k; ++r) {
    kth = __reduce_max_sync(0xffffffffu, key);
    if (r == 0) top = kth;
    if (key == kth) key = 0;
  }
  auto value = [](uint32_t kk) {
    const uint32_t x = kk & 0xffff0000u;
    return __uint_as_float((x & 0x80000000u) ? (x ^ 0x80000000u) : ~x & 0xffff0000u);
  };
  const float rm = value(top), thr = value(kth);
  // The exponents are x log2 e + nb, nb = -rm log2 e rounded: the rounding, the same for the whole row, is known exactly and leaves the
  // logarithm again (mean error against 64 bits, N = 1,500, logits around -40: 8.5e-7 without that, 4.9e-7 with it, 5.0e-7 for the
  // kernel above, whose 32 lanes round 32 products).
  const float nb = __fmul_rn(-rm, L2E);
  float off = __fmul_rn(fmaf(rm, L2E, nb), 0.6931471805599453f);
  const uint64_t l2 = pack_f32x2(L2E, L2E), nb2 = pack_f32x2(nb, nb);
  uint64_t sa = pack_f32x2(0.0f, 0.0f), sb = sa;
  int listed = 0;  // pieces that reach the threshold
#pragma unroll
  for (int j = 0; j < PIECES; ++j) {
    if (used(j)) {
      const uint32_t x[4] = {u[j].x, u[j].y, u[j].z, u[j].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float a, b;
        unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(x[i] << 16), __uint_as_float(x[i] & 0xffff0000u)), l2, nb2), a, b);
        const uint64_t e = pack_f32x2(ex2_approx(a), ex2_approx(b));
        if (i & 1) sb = add_f32x2(sb, e); else sa = add_f32x2(sa, e);
      }
      const __nv_bfloat162 pm = __hmax2(__hmax2(b2(x[0]), b2(x[1])), __hmax2(b2(x[2]), b2(x[3])));
      const int c = j == LAST ? last_c : j * 32 + lane;
      const bool hit = c < (j == LAST ? pieces : full) && fmaxf(__low2float(pm), __high2float(pm)) >= thr;
      const uint32_t who = __ballot_sync(0xffffffffu, hit);
      if (who) {
        const int at = listed + __popc(who & ((1u << lane) - 1u));
        if (hit && at < TR_LIST) list_s[w][at] = c;
        listed += __popc(who);
      }
    }
  }
  float s0, s1;
  unpack_f32x2(add_f32x2(sa, sb), s0, s1);
  float rs = s0 + s1;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) rs += __shfl_xor_sync(0xffffffffu, rs, o);
  // (as there: a sum that is not one of at most N ones is formed again from the exact differences)
  if (rm > -INFINITY && !(rs >= 0.5f && rs <= 2.0f * static_cast<float>(N))) {
    rs = off = 0.0f;
    for (int c = lane; c < pieces; c += 32) {
      float z[8];
      unpack8(src[c], z);
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (8 * c + i < N) rs += ex2_approx((z[i] - rm) * L2E);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) rs += __shfl_xor_sync(0xffffffffu, rs, o);
  }
  if (!(rm > -INFINITY)) rs = 0.0f;
  const float lse = rm + (logf(rs) - off);
  // the listed pieces value by value, four pieces at a time
  __syncwarp();
  int n = listed <= TR_LIST ? 0 : TK_CAND + 1;
  if (listed <= TR_LIST)
    for (int p0 = 0; p0 < listed; p0 += 4) {
      const int p = p0 + (lane >> 3);
      const int col = p < listed ? 8 * list_s[w][p] + (lane & 7) : N;
      const float z = col < N ? __bfloat162float(z0[col]) : 0.0f;
      const bool hit = col < N && z >= thr;
      const uint32_t who = __ballot_sync(0xffffffffu, hit);
      const int at = n + __popc(who & ((1u << lane) - 1u));
      if (hit && at < TK_CAND) cand_s[w][at] = topk_key(z, col);
      n += __popc(who);
    }
  __syncwarp();
  auto put = [&](int j, unsigned long long e) {
    const uint32_t x = static_cast<uint32_t>(e >> 32);
    const float z = __uint_as_float((x & 0x80000000u) ? (x ^ 0x80000000u) : ~x);
    ids[row * k + j] = e ? static_cast<int64_t>(0xffffffffu - static_cast<uint32_t>(e)) : -1;
    logp[row * k + j] = e ? z - lse : -INFINITY;
  };
  if (n <= 64 && n >= k) {  // as a rule: every lane counts the entries above its own one or two and writes them where that says
    for (int t = lane; t < n; t += 32) {
      const unsigned long long mine = cand_s[w][t];
      int rank = 0;
      for (int i = 0; i < n; ++i) rank += cand_s[w][i] > mine ? 1 : 0;
      if (rank < k) put(rank, mine);
    }
    return;
  }
  unsigned long long last = ~0ull;
  for (int j = 0; j < k; ++j) {
    unsigned long long best = 0;
    if (n <= TK_CAND) {
      for (int t = lane; t < n; t += 32) {
        const unsigned long long e = cand_s[w][t];
        if (e < last && e > best) best = e;
      }
    } else {
      for (int c = lane; c < pieces; c += 32) {
        float z[8];
        unpack8(src[c], z);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const unsigned long long e = topk_key(z[i], 8 * c + i);
          if (8 * c + i < N && z[i] >= thr && e < last && e > best) best = e;  // (no NaN, as in the list)
        }
      }
    }
    best = warp_max_u64(best);
    last = best;
    if (lane == 0) put(j, best);
  }
}

}  // namespace
}  // namespace vx

extern "C" {

// Rows per block: about 60 MB of bf16 logits, whole 128-row tiles.
int64_t vx_ctc_topk_rows(int64_t N) {
  if (N <= 0) return 0;
  const int64_t tile_bytes = (N + 7) / 8 * 8 * 2 * 128;
  const int64_t tiles = (60ll << 20) / tile_bytes;
  return 128 * (tiles < 1 ? 1 : tiles);
}

int vx_ctc_topk(const vx_gemm_desc* desc, int k, void* logits, int64_t rows, float* logp, int64_t* ids, void* stream) {
  using namespace vx;
  if (!desc) return fail(-1, "desc must not be NULL");
  if (desc->struct_size != static_cast<int32_t>(sizeof(vx_gemm_desc)))
    return fail(-1, "vx_gemm_desc.struct_size=%d, expected %d", desc->struct_size, (int)sizeof(vx_gemm_desc));
  const int64_t M = desc->M, N = desc->N, K = desc->K;
  if (M < 0 || N <= 0 || N > 0x7fffffffll) return fail(-1, "bad shape");
  if (k <= 0 || k > 16 || k > N) return fail(-1, "k must be in 1..16 and at most N");
  if (desc->fmt == VX_FMT_FP8_1X128) return fail(-1, "vx_ctc_topk runs on the FP4 formats");
  if (M == 0) return 0;
  if (!logits || !logp || !ids || !aligned16(logits)) return fail(-1, "logits (16-byte aligned), logp and ids must not be NULL");
  if (rows <= 0 || (rows < M && rows % 128 != 0)) return fail(-1, "rows must cover M or be a multiple of 128");
  const int64_t ld = (N + 7) / 8 * 8;
  for (int64_t r0 = 0; r0 < M; r0 += rows) {
    const int64_t m = M - r0 < rows ? M - r0 : rows;
    vx_gemm_desc d = *desc;
    d.M = m;
    d.a_codes = static_cast<const uint8_t*>(desc->a_codes) + r0 * desc->lda;
    d.a_scales = static_cast<const uint8_t*>(desc->a_scales) +
                 (desc->fmt == VX_FMT_ROWSCALE ? r0 : r0 / 128 * vx_sf_kgroups(desc->fmt, K) * 512);
    d.epilogue = desc->bias ? VX_EPI_BIAS : VX_EPI_NONE;
    d.out_dtype = VX_BF16; d.out = logits; d.ldo = ld;
    const int rc = vx_bsgemm(&d, stream);
    if (rc) return rc;
    auto regs = [&](auto kernel) {
      return launch_dependent(kernel, dim3(static_cast<unsigned>((m + TR_WARPS - 1) / TR_WARPS)), dim3(TR_WARPS * 32), 0,
                              static_cast<cudaStream_t>(stream), static_cast<const __nv_bfloat16*>(logits), ld, static_cast<int>(N),
                              static_cast<int>(m), k, logp + r0 * k, ids + r0 * k);
    };
    // As many pieces a lane as the row needs, in steps of 8, so that 32, 24 or 16 warps per SM wait for them (15,000 rows, k = 1: N = 1,032
    // 36 us with 24 pieces, 25 with 8, 30 with two passes; N = 2,049 46, 39 with 16, 44).  Two passes below: N = 300 29 us, 42 with 24 pieces.
    if (N > TR_MIN_N && N <= 24 * 256) {
      VX_CUDA_OK(N <= 8 * 256 ? regs(topk_regs_kernel<8, 4>) : N <= 16 * 256 ? regs(topk_regs_kernel<16, 3>) : regs(topk_regs_kernel<24, 2>));
      continue;
    }
    VX_CUDA_OK(launch_dependent(topk_rows_kernel, dim3(static_cast<unsigned>((m + TK_WARPS - 1) / TK_WARPS)), dim3(TK_WARPS * 32), 0,
                                static_cast<cudaStream_t>(stream), static_cast<const __nv_bfloat16*>(logits), ld, static_cast<int>(N),
                                static_cast<int>(m), k, logp + r0 * k, ids + r0 * k));
  }
  return 0;
}

}  // extern "C"
