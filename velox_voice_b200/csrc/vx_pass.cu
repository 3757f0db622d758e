// Every linear, LayerNorm and quantizer of a run of Conformer blocks in ONE launch, for passes of few frames (MX32, d_model 512).
//
// What bounds a short pass is not its work but its launches: twelve blocks are 144 dependent launches, and each takes about 5 us
// for set-up, the latency of its first load, one tile, its stores and the hand-over (375 frames: 752 us of which 7 us are work).
// Rows depend on their own row only, so here a CLUSTER of CPC CTAs takes a block of 128 rows through all layers: a layer's
// result is handed to the next one by stores to a scratch block that stays in L2 and an mbarrier arrival in every CTA of the
// cluster, about a microsecond instead of a launch, and the weights of the layers ahead are loaded meanwhile.
//
// CTA r of the cluster owns columns [CW r, CW r + CW), CW = 512 / CPC, of everything that is 512 wide -- the residual stream x
// among them, which stays in its tensor memory (bf16 pairs) from the first layer to the last -- and the same share of the wider
// layers.  Layers of a block (one phase each; every phase is an MMA with N = CW or 128 columns per job):
//   UP1    x^ -> h = quantize(swish(w1 x^ + b))                         2048 columns, jobs of 128
//   DOWN1  x += 0.5 (w2 h + b);             x^ = quantize(LN_mha(x))
//   QKV    q | k | v = w x^ + b (stored);   c  = quantize(v)            three jobs of CW columns
//   LO     x += w c + b;                    x^ = quantize(LN_conv(x))
//   PW1    c  = quantize(value sigmoid(gate))                           a job of value and a job of gate columns
//   PW2    x += w c + b;                    x^ = quantize(LN_ff(x))
//   UP2    as UP1
//   DOWN2  x += 0.5 (w2 h + b);  x = LN_final(x);  x^ = quantize(LN_next(x))
// The statistics of a LayerNorm need whole rows: every thread sends the sums of its 32-column block to all CTAs of the cluster
// (st.async into a table in distributed shared memory, mbarrier completion), and each combines the sixteen blocks of its row.
//
// Warps: 0..15 epilogue, warp (q, g) = tensor-memory lane quadrant q, 32-column unit g of a job (a thread is a row); 16 loads
// activations, 17 issues the MMAs (one elected lane), 18 and 19 load weights and the biases and LayerNorm parameters, which depend on
// no layer and run ahead of them through rings of four and three slots.  Accumulators: a ring of three times 128 columns.
//
// Measured, whole greedy pass of 12 blocks, captured, separate launches / this: 375 frames 632 / 550 us, 1,920 frames (the most for
// clusters of eight) 773 / 564, 4,000 frames (clusters of four) 890 / 687, 4,200 frames 937 / 724 (its twelve positional projections are launches of their own).  What bounds
// it now, of 88,000 cycles a block (45 us, clusters of eight): the hand-over of an operand, 4,000 a phase -- the release waits 1,750 for the stores, fence and loads take
// 1,900 --, the issue of the MMAs, 500 to 700 cycles per stage of four, and the chain accumulator -> sums -> exchange -> quantize of
// the four LayerNorms, 4,000 each.  Tried and not kept: operands pushed to the other CTAs' shared memory by st.async (630 us) or bulk
// copies (590; shared memory leaves an SM at 14 to 16 bytes a cycle, what L2 delivers enters at 90), jobs of 64 columns for the
// up-projection, registers moved to the epilogue warps (the loaders spill).
//
// Every value takes the operations of the separate kernels in their order (the accumulation of vx_gemm.cu, the LayerNorm and
// quantizer of rows2_kernel as in vx_gemm_ln.cu, the epilogues of vx_epilogue.cuh), so the results are the same bits.
// Every mbarrier wait is bounded; all CTAs reach the closing cluster barrier on every path.

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "vx_common.cuh"
#include "vx_epilogue.cuh"
#include "vx_ptx.cuh"
#include "vx_quant_math.cuh"
#include "vx_tmap.cuh"

namespace vx {
namespace {

constexpr int PS_D = 512;
constexpr int PS_BM = 128;
constexpr int PS_ROW_BLOCKS = PS_D / 32;  // 32-column blocks of a row: one E2M1 scale each
// A operands in the scratch block and in shared memory, as the MMA reads them (K-major without swizzle): block j of the rows = 128 rows
// x 16 bytes, contiguous, so that what a warp makes of 32 rows is one piece of 512 bytes; scale factors: an atom of 512 bytes per K
// step of 64 (two blocks, in the low half of a word).  A stage of K = 256 is one piece of 18 KB and comes by one bulk copy.
constexpr int PS_BLOCK = PS_BM * 16;
constexpr int PS_STAGE_SF = 8 * PS_BLOCK;
constexpr int PS_STAGE = PS_STAGE_SF + 4 * 512;
constexpr int PS_A_SLOTS = 5;
constexpr int PS_B_SLOTS = 4, PS_B_SLOT = 18 * 1024;  // weights: 256 of K x 128 rows, or 512 of K x 64 rows, and scale factors
constexpr int PS_EPI_WARPS = 16, PS_WARP_A = 16, PS_WARP_MMA = 17, PS_WARP_B = 18, PS_WARP_P = 19;
constexpr int PS_THREADS = 20 * 32;
constexpr int PS_P_SLOTS = 3;
constexpr int PS_MAX_BLOCKS = 16;  // 1.3 KB of kernel parameters each
constexpr int PS_MAX_FFN = 2048;
constexpr uint32_t PS_XCH_BYTES = PS_ROW_BLOCKS * 32 * 8;  // sums of a lane quadrant's rows: 16 blocks x 32 rows x 8 bytes
constexpr int PS_ACCS = 3;
// tensor-memory columns: accumulators of 128, x (16 per unit), scale factors of A (two stages) and B (ring of four stages)
constexpr uint32_t PS_TM_X = 384, PS_TM_SFA = 448, PS_TM_SFB = 480;

enum { PH_UP1, PH_DOWN1, PH_QKV, PH_LO, PH_PW1, PH_PW2, PH_UP2, PH_DOWN2, PH_COUNT };
static_assert(PH_COUNT == VX_PASS_LINEARS, "one weight per phase");
enum { READY_X, READY_H, READY_C, READY_COUNT };

struct PassBlock {
  CUtensorMap w[PH_COUNT];
  const uint8_t* sf[PH_COUNT];
  const float* bias[PH_COUNT];
  const float* gamma[5];  // LN_ffm, LN_mha, LN_conv, LN_ff, LN_final
  const float* beta[5];
};
struct PassParams {
  PassBlock blk[PS_MAX_BLOCKS];
  int blocks, m_tiles, ffn;
  int b_const;  // 1: the weights may be loaded ahead of the wait for the previous launch
  int64_t M;
  float eps;
  const __nv_bfloat16* src;
  int64_t ld_src;
  __nv_bfloat16* x;
  int64_t ldx;
  __nv_bfloat16* qkv;   // [M, 3 * 512]
  const float *after_gamma, *after_beta;
  uint8_t* scratch;     // per cluster: x^ and c (two stages each), h (ffn / 256 stages)
  uint8_t* codes;       // quantize(LN_after(x)): [M, 256] and scale-factor atoms
  uint8_t* sf_out;
  int* status;
};

__device__ __forceinline__ bool is_up(int ph) { return ph == PH_UP1 || ph == PH_UP2; }
__device__ __forceinline__ bool is_down(int ph) { return ph == PH_DOWN1 || ph == PH_DOWN2; }
__device__ __forceinline__ int phase_stages(int ph, int ffn) { return is_down(ph) ? ffn >> 8 : 2; }
__device__ __forceinline__ uint32_t bf16_pair(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

__host__ __device__ constexpr int64_t pass_scratch_stages(int64_t ffn) { return 4 + ffn / 256; }

template <int CPC>
struct Geo {
  static constexpr int CW = PS_D / CPC;      // this CTA's columns of a 512-wide layer
  static constexpr int UNITS = CW / 32;
  static constexpr int P_FLOATS = 5 * CW;    // parameters of a phase: bias, gamma, beta, gamma2, beta2, or the biases of its jobs
  static_assert(PS_MAX_FFN / CPC <= P_FLOATS, "biases of the up-projection");
  // A phase is jobs of `cols` accumulator columns; the more columns, the less its issue costs (an MMA of 64 columns takes the issuing
  // thread 49 cycles, one of 128 65)
  static __device__ __forceinline__ int cols(int ph) { return is_up(ph) ? 128 : CW; }
  static __device__ __forceinline__ int slot_stages(int ph) { return is_up(ph) ? 1 : 128 / CW; }  // K stages of a weight slot
  static __device__ __forceinline__ int jobs(int ph, int ffn) { return is_up(ph) ? ffn / (CPC * 128) : (ph == PH_QKV ? 3 : (ph == PH_PW1 ? 2 : 1)); }
  // first weight row of job j
  static __device__ __forceinline__ int row0(int ph, int j, int rank, int ffn) {
    if (is_up(ph)) return rank * (ffn / CPC) + 128 * j;
    const int c = rank * CW;
    if (ph == PH_QKV) return j * PS_D + c;
    if (ph == PH_PW1) return (c >> 7) * 256 + (c & 127) + 128 * j;  // (rows interleaved per 256: 128 of value, 128 of gate)
    return c;
  }
};

template <int CPC>
struct __align__(1024) PassSmem {
  using G = Geo<CPC>;
  uint8_t a[PS_A_SLOTS][PS_STAGE];
  uint8_t b[PS_B_SLOTS][PS_B_SLOT];
  float2 part[2][PS_ROW_BLOCKS][PS_BM];  // [LayerNorm of the phase][32-column block of the row][row]: (sum, sum of squares)
  uint8_t out[PS_EPI_WARPS / 2][2048];   // q | k | v on their way out, warps 8..15; warps 0..7 use the second table of `part`
  float par[PS_P_SLOTS][G::P_FLOATS];
  float half_bias[PS_EPI_WARPS][32];
  uint64_t a_full[PS_A_SLOTS], a_empty[PS_A_SLOTS], b_full[PS_B_SLOTS], b_empty[PS_B_SLOTS], p_full[PS_P_SLOTS], p_empty[PS_P_SLOTS];
  uint64_t tm_full[PS_ACCS], tm_empty[PS_ACCS];
  uint64_t ready[READY_COUNT];           // the operand is complete in the scratch block: an arrival per writing warp of the cluster
  uint64_t xch[2][4];                    // [LayerNorm of the phase][lane quadrant]
  uint32_t tmem_base;
};

template <int CPC>
__global__ void __launch_bounds__(PS_THREADS, 1) conformer_pass_kernel(const __grid_constant__ PassParams p) {
  using G = Geo<CPC>;
  constexpr int CW = G::CW, UNITS = G::UNITS;
  extern __shared__ uint8_t smem_raw[];
  // (the same offset in every CTA of the cluster: map_to_cta relies on it)
  PassSmem<CPC>& sm = *reinterpret_cast<PassSmem<CPC>*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_rank());
  const int cluster = static_cast<int>(blockIdx.x) / CPC, nclusters = static_cast<int>(gridDim.x) / CPC;
  const int ffn = p.ffn;

  // ---- set-up
  if (threadIdx.x == 0) {
    for (int s = 0; s < PS_A_SLOTS; ++s) { mbar_init(&sm.a_full[s], 1); mbar_init(&sm.a_empty[s], 1); }
    for (int s = 0; s < PS_B_SLOTS; ++s) { mbar_init(&sm.b_full[s], 1); mbar_init(&sm.b_empty[s], 1); }
    for (int s = 0; s < PS_P_SLOTS; ++s) { mbar_init(&sm.p_full[s], 1); mbar_init(&sm.p_empty[s], PS_EPI_WARPS); }
    for (int s = 0; s < PS_ACCS; ++s) { mbar_init(&sm.tm_full[s], 1); mbar_init(&sm.tm_empty[s], PS_EPI_WARPS); }
    mbar_init(&sm.ready[READY_X], PS_ROW_BLOCKS * 4);
    mbar_init(&sm.ready[READY_H], PS_EPI_WARPS * CPC);
    mbar_init(&sm.ready[READY_C], PS_ROW_BLOCKS * 4);
    // exchange barriers: the one arrival is the arming here / after each use; the sums arrive as bytes
    for (int t = 0; t < 2; ++t)
      for (int qq = 0; qq < 4; ++qq) {
        mbar_init(&sm.xch[t][qq], 1);
        mbar_expect_tx(&sm.xch[t][qq], PS_XCH_BYTES);
      }
    mbar_fence_init();
  }
  if (warp == PS_WARP_MMA) {
    tmem_alloc(&sm.tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  cluster_sync_all();  // every CTA's barriers exist before anything is sent to them
  const uint32_t tmem_base = sm.tmem_base;
  // (Only weights are read ahead, if the caller calls them constant: biases and LayerNorm parameters may be what the launch before
  // wrote, as for the separate launches.  The trigger: behind the wait, by warps that have waited, as in vx_gemm.cu; the head's
  // CTAs set up on the SMs this grid leaves idle.)
  if (warp != PS_WARP_B) {
    pdl_wait();
    pdl_launch_dependents();
  } else if (!p.b_const) {
    pdl_wait();
  }
  uint8_t* const img_x = p.scratch + cluster * pass_scratch_stages(ffn) * PS_STAGE;
  uint8_t* const img_c = img_x + 2 * PS_STAGE;
  uint8_t* const img_h = img_x + 4 * PS_STAGE;

  if (warp == PS_WARP_B) {
    // =========================== weights ===========================
    if (lane == 0) {
      uint32_t s = 0, par = 1;
      bool ok = true, waited = !p.b_const;
#pragma unroll 1
      for (int mt = cluster; mt < p.m_tiles && ok; mt += nclusters)
#pragma unroll 1
        for (int b = 0; b < p.blocks && ok; ++b)
#pragma unroll 1
          for (int ph = 0; ph < PH_COUNT && ok; ++ph) {
            const CUtensorMap* const map = &p.blk[b].w[ph];
            const uint8_t* const sf = p.blk[b].sf[ph];
            const int stages = phase_stages(ph, ffn), jobs = G::jobs(ph, ffn), n = G::slot_stages(ph), tile = G::cols(ph) * 128;
#pragma unroll 1
            for (int j = 0; j < jobs && ok; ++j) {
              const int row0 = G::row0(ph, j, rank, ffn);
              const uint8_t* const sf_row = sf + static_cast<int64_t>(row0 >> 7) * stages * 1024;
#pragma unroll 1
              for (int ks = 0; ks < stages; ks += n) {
                if (!par && !waited) { pdl_wait(); waited = true; }  // a ring ahead; the limit of the waits is not for the previous launch
                if (!mbar_wait(&sm.b_empty[s], par, p.status, 41)) { ok = false; break; }
                mbar_expect_tx(&sm.b_full[s], n * (tile + 1024));
                tma_load_2d(sm.b[s], map, ks * 128, row0, &sm.b_full[s]);
                if (n == 2) tma_load_2d(sm.b[s] + tile, map, ks * 128 + 128, row0, &sm.b_full[s]);
                bulk_load(sm.b[s] + n * tile, sf_row + ks * 1024, n * 1024, &sm.b_full[s]);
                if (++s == PS_B_SLOTS) { s = 0; par ^= 1; }
              }
            }
          }
    }
  } else if (warp == PS_WARP_P) {
    // =========================== biases and LayerNorm parameters ===========================
    if (lane == 0) {
      uint32_t s = 0, par = 1;
      bool ok = true;
      auto part = [&](int at, const float* src, int n) { bulk_load(sm.par[s] + at, src, n * 4, &sm.p_full[s]); };
      const int col = rank * CW;
#pragma unroll 1
      for (int mt = cluster; mt < p.m_tiles && ok; mt += nclusters)
#pragma unroll 1
        for (int b = 0; b < p.blocks && ok; ++b)
#pragma unroll 1
          for (int ph = b == 0 ? -1 : 0; ph < PH_COUNT; ++ph) {
            if (!mbar_wait(&sm.p_empty[s], par, p.status, 53)) { ok = false; break; }
            const PassBlock& B = p.blk[b];
            if (ph >= 0 && is_up(ph)) {
              mbar_expect_tx(&sm.p_full[s], ffn / CPC * 4);
              part(0, B.bias[ph] + rank * (ffn / CPC), ffn / CPC);
            } else if (ph == PH_QKV || ph == PH_PW1) {
              const int jobs = ph == PH_QKV ? 3 : 2;
              mbar_expect_tx(&sm.p_full[s], jobs * CW * 4);
#pragma unroll 1
              for (int j = 0; j < jobs; ++j) part(j * CW, B.bias[ph] + G::row0(ph, j, rank, ffn), CW);
            } else {
              const int n = ph < 0 ? 0 : (ph == PH_DOWN1 ? 1 : (ph == PH_LO ? 2 : (ph == PH_PW2 ? 3 : 4)));
              mbar_expect_tx(&sm.p_full[s], (2 + (ph >= 0) + 2 * (ph == PH_DOWN2)) * CW * 4);
              if (ph >= 0) part(0, B.bias[ph] + col, CW);
              part(CW, B.gamma[n] + col, CW);
              part(2 * CW, B.beta[n] + col, CW);
              if (ph == PH_DOWN2) {
                const bool last = b + 1 == p.blocks;
                part(3 * CW, (last ? p.after_gamma : p.blk[b + 1].gamma[0]) + col, CW);
                part(4 * CW, (last ? p.after_beta : p.blk[b + 1].beta[0]) + col, CW);
              }
            }
            if (++s == PS_P_SLOTS) { s = 0; par ^= 1; }
          }
    }
  } else if (warp == PS_WARP_A) {
    // =========================== activations ===========================
    if (lane == 0) {
      uint32_t s = 0, par = 1, rpar = 0;  // bit r of rpar: parity of ready[r]
      bool ok = true;
#pragma unroll 1
      for (int mt = cluster; mt < p.m_tiles && ok; mt += nclusters)
#pragma unroll 1
        for (int i = 0; i < PH_COUNT * p.blocks && ok; ++i) {
          const int ph = i & (PH_COUNT - 1);
          const int r = is_down(ph) ? READY_H : (ph == PH_LO || ph == PH_PW2 ? READY_C : READY_X);
          const uint8_t* const img = r == READY_H ? img_h : (r == READY_C ? img_c : img_x);
          const int stages = phase_stages(ph, ffn);
          if (!mbar_wait_cluster(&sm.ready[r], (rpar >> r) & 1, p.status, 42)) { ok = false; break; }
          rpar ^= 1u << r;
          fence_proxy_async_all();  // what other SMs wrote with ordinary stores is read by bulk copies
#pragma unroll 1
          for (int ks = 0; ks < stages; ++ks) {
            if (!mbar_wait(&sm.a_empty[s], par, p.status, 43)) { ok = false; break; }
            mbar_expect_tx(&sm.a_full[s], PS_STAGE);
            bulk_load(sm.a[s], img + ks * PS_STAGE, PS_STAGE, &sm.a_full[s]);
            if (++s == PS_A_SLOTS) { s = 0; par ^= 1; }
          }
        }
    }
  } else if (warp == PS_WARP_MMA) {
    // =========================== MMA issuer ===========================
    // (one thread: lanes that wait together could part where a limit runs out, unless they vote, 587 us for 375 frames against 580)
    if (elect_one()) {
      const uint32_t b_hi = (1024u >> 4) | (1u << 14) | (2u << 29);  // rows of 128 bytes, 128-byte swizzle
      const uint32_t a_hi = (128u >> 4) | (1u << 14);                // no swizzle: 128 bytes to the next eight rows ...
      const uint32_t a_lbo = static_cast<uint32_t>(PS_BLOCK >> 4) << 16;  // ... and a block to the next 16 bytes of K
      const uint32_t sf_hi = (128u >> 4) | (1u << 14);
      auto desc = [](uint32_t lo, uint32_t hi) -> uint64_t { return (static_cast<uint64_t>(hi) << 32) | lo; };
      const uint32_t a_lo0 = smem_u32(sm.a) >> 4, b_lo0 = smem_u32(sm.b) >> 4;
      uint32_t as = 0, apar = 0, bs = 0, bpar = 0, acc = 0, accpar = 1, sfsel = 0;
      bool ok = true;
#pragma unroll 1
      for (int mt = cluster; mt < p.m_tiles && ok; mt += nclusters)
#pragma unroll 1
        for (int i = 0; i < PH_COUNT * p.blocks && ok; ++i) {
          const int ph = i & (PH_COUNT - 1);
          const int stages = phase_stages(ph, ffn), jobs = G::jobs(ph, ffn), n = G::slot_stages(ph);
          const uint32_t tile = G::cols(ph) * 128 >> 4, idesc = make_idesc_mxf4(PS_BM, G::cols(ph), true);
#pragma unroll 1
          for (int j = 0; j < jobs && ok; ++j) {
            // a job's weight rows may be part of a 128-row scale-factor tile: column of their first group of 32 rows
            const uint32_t sfc = static_cast<uint32_t>(G::row0(ph, j, rank, ffn) & 127) >> 5;
            if (!mbar_wait(&sm.tm_empty[acc], accpar, p.status, 44)) { ok = false; break; }
            uint32_t s = as, par = apar, in_slot = 0;
#pragma unroll 1
            for (int ks = 0; ks < stages; ++ks) {
              if (in_slot == 0 && !mbar_wait(&sm.b_full[bs], bpar, p.status, 45)) { ok = false; break; }
              // (jobs behind the first find the phase's two stages in place; the last one releases them)
              if (j == 0 && !mbar_wait(&sm.a_full[s], par, p.status, 46)) { ok = false; break; }
              tc_fence_after();
              const uint32_t a_lo = a_lo0 + s * (PS_STAGE >> 4);
              const uint32_t slot_lo = b_lo0 + bs * (PS_B_SLOT >> 4), b_lo = slot_lo + in_slot * tile, b_sf = slot_lo + n * tile + in_slot * 64;
              const uint32_t sfa = tmem_base + PS_TM_SFA + (ks & 1) * 16, sfb = tmem_base + PS_TM_SFB + sfsel * 8;
              const bool slot_done = in_slot + 1 == static_cast<uint32_t>(n);
              if (j == 0) {  // (scale factors of the two stages of K = 512 stay in tensor memory for the other jobs)
#pragma unroll
                for (int t = 0; t < 4; ++t) tc_cp_32x128b_warpx4(sfa + t * 4, desc((a_lo + (PS_STAGE_SF >> 4) + t * 32) & 0x3fffu, sf_hi));
              }
#pragma unroll
              for (int t = 0; t < 2; ++t) tc_cp_32x128b_warpx4(sfb + t * 4, desc((b_sf + t * 32) & 0x3fffu, sf_hi));
#pragma unroll
              for (int k4 = 0; k4 < 4; ++k4)
                mma_mxf4<2>(tmem_base + acc * 128, desc(((a_lo + k4 * (2 * PS_BLOCK >> 4)) & 0x3fffu) | a_lbo, a_hi),
                            desc((b_lo + 2 * k4) & 0x3fffu, b_hi), idesc_with_sf_id(idesc, 0, (k4 & 1) * 2), sfa + k4 * 4,
                            sfb + (k4 >> 1) * 4 + sfc, static_cast<uint32_t>((ks | k4) != 0));
              if (slot_done) tc_commit(&sm.b_empty[bs]);
              if (j == jobs - 1) tc_commit(&sm.a_empty[s]);
              if (ks == stages - 1) tc_commit(&sm.tm_full[acc]);
              sfsel = (sfsel + 1) & 3;
              ++in_slot;
              if (slot_done) {
                in_slot = 0;
                if (++bs == PS_B_SLOTS) { bs = 0; bpar ^= 1; }
              }
              if (++s == PS_A_SLOTS) { s = 0; par ^= 1; }
            }
            if (j == jobs - 1) { as = s; apar = par; }
            if (++acc == PS_ACCS) { acc = 0; accpar ^= 1; }
          }
        }
    }
  } else {
    // =========================== epilogue ===========================
    const int q = warp & 3, g = warp >> 2;
    const int row_in = q * 32 + lane;
    const uint32_t lane_addr = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
    const bool owner = g < UNITS;  // warps that hold columns of x: 32-column block `jblk` of the row
    const int jblk = rank * UNITS + (g & (UNITS - 1));
    // piece (8 columns) handled at step c of the block: the order in which the stand-alone LayerNorm kernel sums them
    const int rot = (jblk >> 1) & 3;
    int piece[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) piece[c] = (c + rot) & 3;
    uint32_t es = 0, epar = 0;             // accumulator read next, parity of the wait for it
    uint32_t ps = 0, ppar = 0;             // the same for the parameters
    uint32_t xpar = 0;                     // bit t: parity of exchange barrier t
    bool ok = true;
    const Nv16Tensor nv{};

    auto acc_wait = [&](int site) -> bool {
      const bool full = __all_sync(0xffffffffu, mbar_wait(&sm.tm_full[es], epar, p.status, site));
      tc_fence_after();
      return full;
    };
    auto acc_release = [&] {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.tm_empty[es]);
      if (++es == PS_ACCS) { es = 0; epar ^= 1; }
    };
    auto read_acc = [&](int unit, float (&z)[32]) {
      uint32_t r[32];
      tc_ld_32x32b_x32(lane_addr + es * 128 + unit * 32, r);
      tc_wait_ld();
#pragma unroll
      for (int i = 0; i < 32; ++i) z[i] = __uint_as_float(r[i]);
    };
    // codes and scale byte of block `jb` of this row -> the operand's image in the scratch block
    auto store_block = [&](uint8_t* img, int jb, const uint32_t (&w)[4], uint32_t byte) {
      uint8_t* const st = img + (jb >> 3) * PS_STAGE;
      *reinterpret_cast<uint4*>(st + (jb & 7) * PS_BLOCK + row_in * 16) = make_uint4(w[0], w[1], w[2], w[3]);
      st[PS_STAGE_SF + ((jb >> 1) & 3) * 512 + lane * 16 + q * 4 + (jb & 1)] = static_cast<uint8_t>(byte);
    };
    // this warp's part of an operand is written: an arrival in every CTA of the cluster, which releases the writes of all lanes
    auto publish = [&](int r) {
      __syncwarp();
      if (lane < CPC) mbar_arrive_cluster(map_to_cta(smem_u32(&sm.ready[r]), lane));
    };
    // bf16 pairs of a block -> this thread's (sum, sum of squares), in the order of the stand-alone kernel
    auto block_sums = [&](const uint32_t (&xp)[16], float& sum, float& sq) {
      uint64_t S = pack_f32x2(0.0f, 0.0f), Q = S;
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const uint64_t v = pack_f32x2(__uint_as_float(xp[e] << 16), __uint_as_float(xp[e] & 0xffff0000u));
        S = add_f32x2(S, v);
        Q = fma_f32x2(v, v, Q);
      }
      float s0, s1, q0, q1;
      unpack_f32x2(S, s0, s1);
      unpack_f32x2(Q, q0, q1);
      sum = __fadd_rn(s0, s1);
      sq = __fadd_rn(q0, q1);
    };
    // sums of the row -> all CTAs, and back: (rstd, -mean rstd) as packed pairs
    auto exchange = [&](int t, float sum, float sq, uint64_t& R2, uint64_t& N2) -> bool {
      const float2* const table = &sm.part[t][0][0];
      const uint32_t mine = smem_u32(table + jblk * PS_BM + row_in), bar = smem_u32(&sm.xch[t][q]);
#pragma unroll
      for (int d = 0; d < CPC; ++d) st_async_f2(map_to_cta(mine, d), sum, sq, map_to_cta(bar, d));
      if (!__all_sync(0xffffffffu, mbar_wait_cluster(&sm.xch[t][q], (xpar >> t) & 1, p.status, 47))) return false;
      xpar ^= 1u << t;
      if (g == 0 && lane == 0) mbar_expect_tx(&sm.xch[t][q], PS_XCH_BYTES);  // armed for the next use
      float s[8], qq[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {  // blocks j and j ^ 8 first, then xor 4, 2, 1
        const float2 lo = table[e * PS_BM + row_in], hi = table[(e + 8) * PS_BM + row_in];
        s[e] = __fadd_rn(lo.x, hi.x);
        qq[e] = __fadd_rn(lo.y, hi.y);
      }
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) {
#pragma unroll
        for (int e = 0; e < o; ++e) {
          s[e] = __fadd_rn(s[e], s[e + o]);
          qq[e] = __fadd_rn(qq[e], qq[e + o]);
        }
      }
      const float mean = __fmul_rn(s[0], 1.0f / 512.0f);
      const float ex2 = __fmul_rn(qq[0], 1.0f / 512.0f);
      const float var = fmaxf(__fmaf_rn(-mean, mean, ex2), 0.0f);
      const float rstd = __frsqrt_rn(__fadd_rn(var, p.eps));
      const float nmr = __fmul_rn(-mean, rstd);
      R2 = pack_f32x2(rstd, rstd);
      N2 = pack_f32x2(nmr, nmr);
      return true;
    };
    // four LayerNorm outputs (values 4 hh .. of piece c) as two packed pairs
    auto normed = [&](const uint32_t (&xp)[16], int c, int hh, const float* ga, const float* be, uint64_t R2, uint64_t N2, uint64_t& y0,
                      uint64_t& y1) {
      uint64_t g0, g1, b0, b1;
      ld_shared_pairs(smem_u32(ga + piece[c] * 8 + 4 * hh), g0, g1);
      ld_shared_pairs(smem_u32(be + piece[c] * 8 + 4 * hh), b0, b1);
      const uint32_t w0 = xp[4 * c + 2 * hh], w1 = xp[4 * c + 2 * hh + 1];
      const uint64_t x0 = pack_f32x2(__uint_as_float(w0 << 16), __uint_as_float(w0 & 0xffff0000u));
      const uint64_t x1 = pack_f32x2(__uint_as_float(w1 << 16), __uint_as_float(w1 & 0xffff0000u));
      y0 = fma_f32x2(fma_f32x2(x0, R2, N2), g0, b0);
      y1 = fma_f32x2(fma_f32x2(x1, R2, N2), g1, b1);
    };

#pragma unroll 1
    for (int mt = cluster; mt < p.m_tiles && ok; mt += nclusters) {
      const int64_t row = static_cast<int64_t>(mt) * PS_BM + row_in;
      const bool row_ok = row < p.M;
      // step -1: the features come in; then PH_COUNT phases per block
      int b = 0, ph = -1;
#pragma unroll 1
      while (b < p.blocks) {
        const bool last = ph == PH_DOWN2 && b + 1 == p.blocks;
        ok = __all_sync(0xffffffffu, mbar_wait(&sm.p_full[ps], ppar, p.status, 54));
        if (!ok) break;
        const float* const par = sm.par[ps];
        if (ph >= 0 && is_up(ph)) {
          const int jobs = G::jobs(ph, ffn);
#pragma unroll 1
          for (int j = 0; j < jobs; ++j) {
            sm.half_bias[warp][lane] = 0.5f * par[j * 128 + g * 32 + lane];  // see swish_group8
            __syncwarp();
            ok = acc_wait(48);
            if (!ok) break;
            uint32_t r[32];
            tc_ld_32x32b_x32(lane_addr + es * 128 + g * 32, r);
            tc_wait_ld();
            acc_release();
            uint32_t w[4];
            const uint32_t byte = swish_quant_chunk<false>(r, sm.half_bias[warp], false, 1.0f, nv, nullptr, w);
            store_block(img_h, (rank * (ffn / CPC) + j * 128) / 32 + g, w, byte);
            __syncwarp();
          }
          if (!ok) break;
          publish(READY_H);
        } else if (ph == PH_QKV || ph == PH_PW1) {
          // q, k, v in turn, the units going round the warps; or value and gate, both in the warp that owns the columns
          const bool glu = ph == PH_PW1;
          const int jobs = glu ? 2 : 3;
          float value[32];
#pragma unroll 1
          for (int j = 0; j < jobs; ++j) {
            const int u = glu ? g : (g - j * UNITS) & 3;
            ok = acc_wait(49);
            if (!ok) break;
            if (u >= UNITS) {
              acc_release();
              continue;
            }
            float z[32];
            read_acc(u, z);
            acc_release();
            add_bias32(z, par + j * CW + u * 32);
            const int col = rank * CW + u * 32;
            if (glu) {
              if (j == 0) {
#pragma unroll
                for (int i = 0; i < 32; ++i) value[i] = z[i];
                continue;
              }
#pragma unroll
              for (int i = 0; i < 32; ++i) z[i] = value[i] * sigmoid_f(z[i]);
            }
            if (j == jobs - 1) {
              uint32_t w[4];
              const uint32_t byte = quant_bf16_chunk(VX_FMT_MX32, z, 1.0f, w);
              store_block(img_c, col >> 5, w, byte);
              publish(READY_C);
            }
            if (!glu) {
              // q | k | v as bf16, by way of shared memory: 64 bytes of a row per four lanes instead of 16 bytes of 32 rows per store
              uint8_t* const st = warp < 8 ? reinterpret_cast<uint8_t*>(sm.part[1]) + warp * 2048 : sm.out[warp - 8];
#pragma unroll
              for (int v = 0; v < 4; ++v)
                *reinterpret_cast<uint4*>(st + lane * 64 + ((v ^ ((lane >> 1) & 3)) << 4)) =
                    make_uint4(bf16_pair(z[8 * v], z[8 * v + 1]), bf16_pair(z[8 * v + 2], z[8 * v + 3]),
                               bf16_pair(z[8 * v + 4], z[8 * v + 5]), bf16_pair(z[8 * v + 6], z[8 * v + 7]));
              __syncwarp();
#pragma unroll
              for (int v = 0; v < 4; ++v) {
                const int r = 8 * v + (lane >> 2), c4 = lane & 3;
                const int64_t orow = static_cast<int64_t>(mt) * PS_BM + q * 32 + r;
                if (orow < p.M)
                  *reinterpret_cast<uint4*>(p.qkv + orow * (3 * PS_D) + j * PS_D + col + c4 * 8) =
                      *reinterpret_cast<const uint4*>(st + r * 64 + ((c4 ^ ((r >> 1) & 3)) << 4));
              }
              __syncwarp();
            }
          }
          if (!ok) break;
        } else if (!owner) {
          if (ph >= 0) {
            ok = acc_wait(51);
            if (!ok) break;
            acc_release();
          }
        } else {
          // features (ph < 0) or a residual GEMM, then the LayerNorm(s) in front of the next layer
          const int col = jblk * 32;
          const float *ga = par + CW + g * 32, *be = par + 2 * CW + g * 32;
          uint32_t xp[16];
          if (ph < 0) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              uint4 u = make_uint4(0, 0, 0, 0);
              if (row_ok) u = *reinterpret_cast<const uint4*>(p.src + row * p.ld_src + col + piece[c] * 8);
              xp[4 * c] = u.x; xp[4 * c + 1] = u.y; xp[4 * c + 2] = u.z; xp[4 * c + 3] = u.w;
            }
          } else {
            ok = acc_wait(52);
            if (!ok) break;
            uint32_t z[4][8];
#pragma unroll
            for (int c = 0; c < 4; ++c) tc_ld_x8(lane_addr + es * 128 + g * 32 + piece[c] * 8, z[c]);
            tc_ld_x16(lane_addr + PS_TM_X + g * 16, xp);
            tc_wait_ld();
            acc_release();
            // x = bf16(alpha (acc + bias) + x)
            const float alpha = is_down(ph) ? 0.5f : 1.0f;
            const uint64_t A2 = pack_f32x2(alpha, alpha);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const uint32_t bs = smem_u32(par + g * 32 + piece[c] * 8);
              uint64_t bb[4];
              ld_shared_pairs(bs, bb[0], bb[1]);
              ld_shared_pairs(bs + 16, bb[2], bb[3]);
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const uint32_t rw = xp[4 * c + e];
                const uint64_t zz = add_f32x2(pack_f32x2(__uint_as_float(z[c][2 * e]), __uint_as_float(z[c][2 * e + 1])), bb[e]);
                const uint64_t xx = fma_f32x2(A2, zz, pack_f32x2(__uint_as_float(rw << 16), __uint_as_float(rw & 0xffff0000u)));
                float lo, hi;
                unpack_f32x2(xx, lo, hi);
                xp[4 * c + e] = bf16_pair(lo, hi);
              }
            }
          }
          uint64_t R2, N2;
#pragma unroll 1
          for (int t = 0;; ++t) {
            float sum, sq;
            block_sums(xp, sum, sq);
            if (t == (ph == PH_DOWN2) && !last) tc_st_x16(lane_addr + PS_TM_X + g * 16, xp);
            ok = exchange(t, sum, sq, R2, N2);
            if (!ok || t == (ph == PH_DOWN2)) break;
            // x = bf16(LN_final(x)), and on to the LayerNorm behind it
#pragma unroll
            for (int c = 0; c < 4; ++c)
#pragma unroll
              for (int hh = 0; hh < 2; ++hh) {
                uint64_t y0, y1;
                normed(xp, c, hh, ga, be, R2, N2, y0, y1);
                float a0, a1, a2, a3;
                unpack_f32x2(y0, a0, a1);
                unpack_f32x2(y1, a2, a3);
                xp[4 * c + 2 * hh] = bf16_pair(a0, a1);
                xp[4 * c + 2 * hh + 1] = bf16_pair(a2, a3);
              }
            ga += 2 * CW;
            be += 2 * CW;
          }
          if (!ok) break;
          uint64_t v[4][4];
          float a[4];
#pragma unroll
          for (int c = 0; c < 4; ++c) {
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) normed(xp, c, hh, ga, be, R2, N2, v[c][2 * hh], v[c][2 * hh + 1]);
            a[c] = amax8p(v[c]);
          }
          uint32_t byte;
          float rcp;
          ue8m0_from_amax(fmaxf(max3(a[0], a[1], a[2]), a[3]), byte, rcp);
          uint32_t wd[4];
#pragma unroll
          for (int c = 0; c < 4; ++c) wd[c] = e2m1_pack8p<false, true>(v[c], rcp);
          // word of step c belongs to piece (c + rot) & 3: rotate the four words back
          if (rot & 1) { const uint32_t t = wd[3]; wd[3] = wd[2]; wd[2] = wd[1]; wd[1] = wd[0]; wd[0] = t; }
          if (rot & 2) { uint32_t t = wd[0]; wd[0] = wd[2]; wd[2] = t; t = wd[1]; wd[1] = wd[3]; wd[3] = t; }
          if (!last) {
            store_block(img_x, jblk, wd, byte);
            publish(READY_X);
          } else {
            // x, and the head's operand; rows beyond M read as zero scale factors
            if (row_ok) {
#pragma unroll
              for (int c = 0; c < 4; ++c)
                *reinterpret_cast<uint4*>(p.x + row * p.ldx + col + piece[c] * 8) = make_uint4(xp[4 * c], xp[4 * c + 1], xp[4 * c + 2], xp[4 * c + 3]);
              *reinterpret_cast<uint4*>(p.codes + row * (PS_D / 2) + jblk * 16) = make_uint4(wd[0], wd[1], wd[2], wd[3]);
            }
            p.sf_out[(static_cast<int64_t>(mt) * 4 + (jblk >> 2)) * 512 + lane * 16 + q * 4 + (jblk & 3)] = static_cast<uint8_t>(row_ok ? byte : 0u);
          }
          tc_wait_st_all();  // x is in tensor memory before the next phase reads it
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.p_empty[ps]);
        if (++ps == PS_P_SLOTS) { ps = 0; ppar ^= 1; }
        if (++ph == PH_COUNT) { ph = 0; ++b; }
      }
    }
  }

  // ---- tear-down
  tc_fence_before();
  __syncthreads();
  if (warp == PS_WARP_MMA) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
  cluster_sync_all();  // no CTA leaves while another may still write into its shared memory
}

template <int CPC>
constexpr size_t kPassSmem = sizeof(PassSmem<CPC>) + 1024;
static_assert(kPassSmem<8> <= 232448 && kPassSmem<4> <= 232448, "shared memory of one CTA");

// Clusters of CPC such CTAs that the current device runs at a time (0: none), asked once per device.
template <int CPC>
int max_clusters() {
  static std::atomic<int> cache[64] = {};  // answer + 1
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  if (const int c = cache[dev].load(std::memory_order_acquire)) return c - 1;
  int n = 0;
  if (cudaFuncSetAttribute(conformer_pass_kernel<CPC>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kPassSmem<CPC>)) == cudaSuccess) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(CPC);
    cfg.blockDim = dim3(PS_THREADS);
    cfg.dynamicSmemBytes = kPassSmem<CPC>;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CPC;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, conformer_pass_kernel<CPC>, &cfg) != cudaSuccess) n = 0;
  }
  if (n == 0) cudaGetLastError();
  cache[dev].store(n + 1, std::memory_order_release);
  return n;
}

template <int CPC>
int launch_pass(PassParams& p, const vx_pass_desc* d, cudaStream_t st) {
  constexpr int CW = PS_D / CPC;
  for (int b = 0; b < d->blocks; ++b)
    for (int l = 0; l < PH_COUNT; ++l) {
      const bool up = l == PH_UP1 || l == PH_UP2, down = l == PH_DOWN1 || l == PH_DOWN2;
      const int64_t n = up ? d->ffn : (l == PH_QKV ? 3 * PS_D : (l == PH_PW1 ? 2 * PS_D : PS_D));
      const int64_t k = down ? d->ffn : PS_D;
      const vx_pass_linear& w = d->block[b].lin[l];
      const int rc = make_tmap_2d(&p.blk[b].w[l], CU_TENSOR_MAP_DATA_TYPE_UINT8, w.codes, n, k / 2, w.ld, 128, up ? 128 : CW);
      if (rc) return rc;
    }
  int clusters = max_clusters<CPC>();
  if (clusters > p.m_tiles) clusters = p.m_tiles;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(CPC * clusters);
  cfg.blockDim = dim3(PS_THREADS);
  cfg.dynamicSmemBytes = kPassSmem<CPC>;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CPC;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  VX_CUDA_OK(cudaLaunchKernelEx(&cfg, conformer_pass_kernel<CPC>, p));
  return 0;
}

// CTAs per cluster for a pass of `tiles` row blocks: eight while all row blocks run at once (15 on a B200), as a Conformer block takes 47 us
// instead of 58; four up to 33 row blocks.
int pass_cluster(int64_t tiles) { return tiles <= max_clusters<8>() ? 8 : 4; }

}  // namespace
}  // namespace vx

extern "C" {

int vx_conformer_pass_supported(int fmt, int64_t d_model, int64_t ffn, int64_t conv_pw, int64_t blocks) {
  using namespace vx;
  return fmt == VX_FMT_MX32 && d_model == PS_D && ffn >= 1024 && ffn % 1024 == 0 && ffn <= PS_MAX_FFN && conv_pw == 2 * PS_D && blocks >= 1 &&
         blocks <= PS_MAX_BLOCKS;
}

// One round of clusters of four.  Separate launches / one launch: 4,200 frames 937 / 724 us; a second round would take as long again, about 1,450 us, where the launches
// that pipeline over many row blocks take 954 (4,608 frames).
int64_t vx_conformer_pass_frames(void) {
  return static_cast<int64_t>(vx::max_clusters<4>()) * vx::PS_BM;
}

int64_t vx_conformer_pass_scratch(int64_t M, int64_t ffn) {
  using namespace vx;
  const int64_t tiles = (M + PS_BM - 1) / PS_BM, most = sm_count() / 4;
  return (tiles < most ? tiles : most) * pass_scratch_stages(ffn) * PS_STAGE;
}

int vx_conformer_pass(const vx_pass_desc* d, void* stream) {
  using namespace vx;
  if (!d) return fail(-1, "desc must not be NULL");
  if (d->struct_size != static_cast<int32_t>(sizeof(vx_pass_desc)))
    return fail(-1, "vx_pass_desc.struct_size=%d, expected %d", d->struct_size, (int)sizeof(vx_pass_desc));
  if (!vx_conformer_pass_supported(VX_FMT_MX32, PS_D, d->ffn, 2 * PS_D, d->blocks))
    return fail(-1, "vx_conformer_pass: 1 to %d blocks, ffn 1,024 or 2,048 (see vx_conformer_pass_supported)", PS_MAX_BLOCKS);
  if (d->M < 0) return fail(-1, "negative shape");
  if (d->M == 0) return 0;
  if ((d->M + PS_BM - 1) / PS_BM > 0x7fffffff / PS_BM) return fail(-1, "too many rows");
  if (!d->block || !d->src || !d->x || !d->qkv || !d->scratch || !d->codes || !d->scales_sf || !d->after_gamma || !d->after_beta || !aligned16(d->after_gamma) ||
      !aligned16(d->after_beta))
    return fail(-1, "vx_conformer_pass: NULL pointer, or after_gamma / after_beta not 16-byte aligned");
  if (!aligned16(d->src) || !aligned16(d->x) || !aligned16(d->qkv) || !aligned16(d->scratch) || !aligned16(d->codes) || d->ld_src % 8 != 0 ||
      d->ldx % 8 != 0 || d->ld_src < PS_D || d->ldx < PS_D)
    return fail(-1, "rows of src and x must be 16-byte aligned and at least 512 elements; qkv, scratch and codes 16-byte aligned");
  PassParams p;
  for (int b = 0; b < d->blocks; ++b) {
    const vx_pass_block& B = d->block[b];
    for (int l = 0; l < PH_COUNT; ++l) {
      const vx_pass_linear& w = B.lin[l];
      const int64_t k = l == PH_DOWN1 || l == PH_DOWN2 ? d->ffn : PS_D;
      if (!w.codes || !w.scales_sf || !aligned16(w.codes) || !aligned16(w.scales_sf) || w.ld % 16 != 0 || w.ld < k / 2)
        return fail(-1, "weight rows must be 16-byte aligned and whole, scale-factor atoms 16-byte aligned");
      if (!w.bias || !aligned16(w.bias)) return fail(-1, "biases must be 16-byte aligned");
      p.blk[b].sf[l] = static_cast<const uint8_t*>(w.scales_sf);
      p.blk[b].bias[l] = w.bias;
    }
    for (int n = 0; n < 5; ++n) {
      if (!B.gamma[n] || !B.beta[n] || !aligned16(B.gamma[n]) || !aligned16(B.beta[n])) return fail(-1, "gamma and beta must be 16-byte aligned");
      p.blk[b].gamma[n] = B.gamma[n];
      p.blk[b].beta[n] = B.beta[n];
    }
  }
  p.blocks = d->blocks;
  p.m_tiles = static_cast<int>((d->M + PS_BM - 1) / PS_BM);
  p.ffn = static_cast<int>(d->ffn);
  p.b_const = d->const_weights != 0;
  p.M = d->M;
  p.eps = d->eps;
  p.src = static_cast<const __nv_bfloat16*>(d->src); p.ld_src = d->ld_src;
  p.x = static_cast<__nv_bfloat16*>(d->x); p.ldx = d->ldx;
  p.qkv = static_cast<__nv_bfloat16*>(d->qkv);
  p.after_gamma = d->after_gamma; p.after_beta = d->after_beta;
  p.scratch = static_cast<uint8_t*>(d->scratch);
  p.codes = static_cast<uint8_t*>(d->codes); p.sf_out = static_cast<uint8_t*>(d->scales_sf);
  p.status = device_status_ptr();
  if (max_clusters<4>() == 0) return fail(-2, "this device runs no cluster of four such CTAs");
  const cudaStream_t st = static_cast<cudaStream_t>(stream);
  return pass_cluster(p.m_tiles) == 8 ? launch_pass<8>(p, d, st) : launch_pass<4>(p, d, st);
}

}  // extern "C"
