// Filterbank projection of the audio front-end: power spectrum -> mel GEMM -> log -> CMVN, one pass.
//
//   out[t, m] = (log(max(sum_f (re[t,f]^2 + im[t,f]^2) * mel[m, f], 2^-23)) - mean[m]) * istd[m]
//
// Replaces power_mel_log (veloxvoice/kernels/ops/cuda_ops.py:82-135) and its kernel
// (veloxvoice/kernels/csrc/dgx/dgx_power_mel_log.cu:20-79, dgx/block/nv_block_power_mel_log.h:35-190:
// mma.sync m16n8k8 tf32, at most 48 CTAs).  Here the product runs on the 5th-generation tensor cores
// (tcgen05.mma kind::tf32, accumulator in tensor memory) and the kernel is shaped by what bounds it,
// the 2 KB of complex spectrum per frame that have to come out of HBM.  Contiguous spectra with an ordinary filterbank
// run on power_mel_log_dense_kernel (further down); this is the general kernel (strided rows, larger filterbanks):
//
//   warps 0..3    epilogue: tcgen05.ld of the fp32 accumulator (one frame per thread), log, CMVN, store;
//   warps 4..11   loaders: read the spectrum with coalesced 8-byte loads (one complex bin per lane, sixteen
//                 rows per stage, the loads of the next stage in flight while the current one is
//                 processed), form re^2 + im^2 and write it straight into the 128-byte-swizzled
//                 K-major tile layout the MMA reads -- the power spectrum never exists in global memory;
//   warp 12       MMA issuer: four K = 8 MMAs per 32-bin stage, tcgen05.commit hands ring slots back and
//                 publishes finished accumulators (two of them, so the epilogue of frame tile i runs under the
//                 loads and MMAs of tile i + 1).
// The filterbank (at most 256 mel rows, zero-padded to a multiple of 16) stays resident in shared memory in
// the same swizzled layout for the whole kernel.  fp32 operands are read by the tensor core as tf32 (the low
// 13 mantissa bits are ignored), which is the reference kernel's precision contract
// (tests/kernels/test_power_mel_log.py:1-16).  Every mbarrier wait is bounded.

#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "vx_common.cuh"
#include "vx_ptx.cuh"

namespace vx {
namespace {

constexpr int MEL_BM = 128;             // frames per tile = TMEM lanes
constexpr int MEL_KS = 32;              // spectrum bins per K stage (128 bytes of fp32)
constexpr int MEL_SLOT = MEL_BM * 128;  // bytes of one A stage
constexpr int MEL_RING_MAX = 4;         // A stages in flight: as many (2..4) as fit beside the filterbank
constexpr int MEL_LOADERS = 8;          // loader warps, 16 frames each
constexpr int MEL_THREADS = (4 + MEL_LOADERS + 1) * 32;
constexpr int MEL_MAX_SMEM = 220 * 1024;

struct MelParams {
  const float2* spec;
  int64_t T, F, ld_spec;
  const float* mel;
  int64_t M, ld_mel;
  const float* mean;
  const float* istd;
  float* out;
  int64_t ldo;
  int n_pad, stages, tiles, ring;
  int bank_off, early;  // dense kernel: where the filterbank passes through shared memory, ring slots in front of it
  int* status;
};

// byte offset of element (row, k) of a K-major tile of 128-byte rows with the 128-byte swizzle
__device__ __forceinline__ uint32_t sw128(int row, int k) {
  return static_cast<uint32_t>(row) * 128u + ((static_cast<uint32_t>(k >> 2) ^ (static_cast<uint32_t>(row) & 7u)) << 4) +
         (static_cast<uint32_t>(k & 3) << 2);
}

__host__ __device__ constexpr uint32_t make_idesc_tf32(int M, int N) {
  // fp32 accumulate (c_format 1), A and B tf32 (format 2), both K-major
  return (1u << 4) | (2u << 7) | (2u << 10) | (static_cast<uint32_t>(N >> 3) << 17) | (static_cast<uint32_t>(M >> 4) << 24);
}

__device__ __forceinline__ void mma_tf32(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void tc_ld_32x32b_x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

struct MelBarriers {
  uint64_t full[MEL_RING_MAX];
  uint64_t empty[MEL_RING_MAX];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint32_t tmem_base;
  int abort_flag;
};

__global__ void __launch_bounds__(MEL_THREADS, 1) power_mel_log_kernel(const MelParams p) {
  pdl_launch_dependents();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* const ring = base;                                  // p.ring x 16 KB
  uint8_t* const bres = base + p.ring * MEL_SLOT;              // stages x n_pad x 128 B (n_pad % 8 == 0: 1 KB atoms hold)
  __shared__ MelBarriers bar;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  volatile int* const abortp = &bar.abort_flag;
  const int my_tiles = static_cast<int>(blockIdx.x) < p.tiles ? (p.tiles - static_cast<int>(blockIdx.x) + gridDim.x - 1) / gridDim.x : 0;
  const uint32_t b_stage_bytes = static_cast<uint32_t>(p.n_pad) * 128u;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.ring; ++s) {
      mbar_init(&bar.full[s], MEL_LOADERS);
      mbar_init(&bar.empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&bar.acc_full[a], 1);
      mbar_init(&bar.acc_empty[a], 4);
    }
    bar.abort_flag = 0;
    mbar_fence_init();
  }
  pdl_wait();  // the launch before may have written the filterbank, too
  // the filterbank, zero-padded, into its resident swizzled tiles: element (n, k) of stage k / 32
  for (int64_t i = threadIdx.x; i < static_cast<int64_t>(p.stages) * p.n_pad * MEL_KS; i += blockDim.x) {
    const int kk = static_cast<int>(i % MEL_KS);
    const int n = static_cast<int>((i / MEL_KS) % p.n_pad);
    const int ks = static_cast<int>(i / (static_cast<int64_t>(MEL_KS) * p.n_pad));
    const int64_t k = static_cast<int64_t>(ks) * MEL_KS + kk;
    const float v = (n < p.M && k < p.F) ? p.mel[n * p.ld_mel + k] : 0.0f;
    *reinterpret_cast<float*>(bres + ks * b_stage_bytes + sw128(n, kk)) = v;
  }
  fence_proxy_async_smem();
  if (warp == 4 + MEL_LOADERS) {
    tmem_alloc(&bar.tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bar.tmem_base;

  if (warp >= 4 && warp < 4 + MEL_LOADERS) {
    // =========================== loaders ===========================
    // The (tile, stage) items of this CTA form one sequence; the sixteen loads of item n + 1 are in
    // flight while item n is squared and written to its ring slot.
    const int lw = warp - 4;
    const int64_t items = static_cast<int64_t>(my_tiles) * p.stages;
    auto fetch = [&](int64_t n, float2 (&c)[16]) {
      const int64_t tile = static_cast<int64_t>(blockIdx.x) + (n / p.stages) * gridDim.x;
      const int64_t row0 = tile * MEL_BM + lw * 16;
      const int64_t f = (n % p.stages) * MEL_KS + lane;
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        const int64_t row = row0 + r;
        c[r] = (n < items && row < p.T && f < p.F) ? p.spec[row * p.ld_spec + f] : make_float2(0.0f, 0.0f);
      }
    };
    auto publish = [&](uint32_t s, const float2 (&c)[16]) {
      uint8_t* const slot = ring + s * MEL_SLOT;
#pragma unroll
      for (int r = 0; r < 16; ++r)  // two rounded squares and one rounded add, as spec.real**2 + spec.imag**2
        *reinterpret_cast<float*>(slot + sw128(lw * 16 + r, lane)) = __fadd_rn(__fmul_rn(c[r].x, c[r].x), __fmul_rn(c[r].y, c[r].y));
      fence_proxy_async_smem();  // generic-proxy writes -> visible to the tensor core's reads
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar.full[s]);
    };
    uint32_t s = 0, ph = 0;
    bool ok = true;
    float2 ca[16], cb[16];
    fetch(0, ca);
    for (int64_t n = 0; n < items && ok; n += 2) {
      fetch(n + 1, cb);
      ok = __all_sync(0xffffffffu, mbar_wait<true>(&bar.empty[s], ph ^ 1, p.status, 11, abortp));
      if (!ok) break;
      publish(s, ca);
      if (++s == static_cast<uint32_t>(p.ring)) { s = 0; ph ^= 1; }
      if (n + 1 >= items) break;
      fetch(n + 2, ca);
      ok = __all_sync(0xffffffffu, mbar_wait<true>(&bar.empty[s], ph ^ 1, p.status, 11, abortp));
      if (!ok) break;
      publish(s, cb);
      if (++s == static_cast<uint32_t>(p.ring)) { s = 0; ph ^= 1; }
    }
    if (!ok) bar.abort_flag = 1;
  } else if (warp == 4 + MEL_LOADERS) {
    // =========================== MMA issuer ===========================
    if (my_tiles > 0) {
      const bool leader = elect_one();
      const uint32_t idesc = make_idesc_tf32(MEL_BM, p.n_pad);
      const uint32_t ring_u32 = smem_u32(ring), b_u32 = smem_u32(bres);
      uint32_t s = 0, ph = 0;
      bool ok = true;
      for (int i = 0; i < my_tiles && ok; ++i) {
        const uint32_t a = i & 1;
        ok = __all_sync(0xffffffffu, mbar_wait_spin(&bar.acc_empty[a], ((i >> 1) & 1) ^ 1, p.status, 12, abortp));
        if (!ok) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + a * 256;
        for (int ks = 0; ks < p.stages; ++ks) {
          ok = __all_sync(0xffffffffu, mbar_wait_spin(&bar.full[s], ph, p.status, 13, abortp));
          if (!ok) break;
          tc_fence_after();
          if (leader) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
              mma_tf32(d_tmem, make_desc_k128(ring_u32 + s * MEL_SLOT + j * 32), make_desc_k128(b_u32 + ks * b_stage_bytes + j * 32), idesc,
                       (ks | j) != 0);
            tc_commit(&bar.empty[s]);
          }
          __syncwarp();
          if (++s == static_cast<uint32_t>(p.ring)) { s = 0; ph ^= 1; }
        }
        if (ok && leader) tc_commit(&bar.acc_full[a]);
        __syncwarp();
      }
      if (!ok && leader) bar.abort_flag = 1;
    }
  } else {
    // =========================== epilogue (warps 0..3 = lane quadrants 0..3) ===========================
    bool ok = true;
    for (int i = 0; i < my_tiles && ok; ++i) {
      const uint32_t a = i & 1;
      ok = __all_sync(0xffffffffu, mbar_wait<true>(&bar.acc_full[a], (i >> 1) & 1, p.status, 14, abortp));
      if (!ok) break;
      tc_fence_after();
      const int64_t row = (static_cast<int64_t>(blockIdx.x) + static_cast<int64_t>(i) * gridDim.x) * MEL_BM + warp * 32 + lane;
      const uint32_t taddr = tmem_base + a * 256 + (static_cast<uint32_t>(warp * 32) << 16);
      for (int c0 = 0; c0 < p.n_pad; c0 += 16) {
        uint32_t r[16];
        tc_ld_32x32b_x16(taddr + c0, r);
        tc_wait_ld();
        if (row < p.T) {
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const int m = c0 + j;
            if (m < p.M) {
              float v = __logf(fmaxf(__uint_as_float(r[j]), 1.1920929e-7f));
              if (p.mean) v = (v - __ldg(p.mean + m)) * __ldg(p.istd + m);
              p.out[row * p.ldo + m] = v;
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar.acc_empty[a]);
    }
    if (!ok) bar.abort_flag = 1;
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 4 + MEL_LOADERS) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}


// ---------------------------------------------------------------------------------------
// The dense spectrum (rows back to back, what torch.fft.rfft returns), at most 128 mel rows and 448 bins: the product is
// formed transposed, D[mel][frame] = filterbank . power^T, so that
//   * the filterbank is the M = 128 operand and stays in TENSOR MEMORY for the whole kernel (one column per bin): the MMAs
//     read only the frames from shared memory.  With both operands in shared memory the 4 KB of filterbank per K = 8
//     step bounded the kernel (201 us, see below), and the filterbank took the 92 KB that the ring of raw rows wants;
//   * the input comes as bulk asynchronous copies of eight whole rows (any even number of rows of 8 F bytes starts and
//     ends on a 16-byte boundary even where a single row does not): the bytes in flight are set by shared memory, and
//     every DRAM page is read once and in order;
//   * a transform warp turns one row of a chunk into one row of the K-major operand tile (32 frames, all of F), so
//     nothing waits for 128 frames to gather;
//   * a lane of the epilogue holds one mel row: a warp stores 32 consecutive outputs of a frame with one instruction
//     (frame-per-lane stores touch 32 sectors each), and the CMVN constants of a lane stay in registers.
// Bound by HBM.  360,000 x 257 -> 80 (855 MB): 290 us (frames as the M operand, 8-byte loads) -> 132 us = 6.47 TB/s; 60,000
// frames 50 -> 28 us, 200 frames 23 -> 6 us.
constexpr int MT_ROWS = 8;     // rows per chunk
constexpr int MT_N = 32;       // frames per tile
constexpr int MT_RING_MAX = 8;
constexpr int MT_XF = 16;      // transform warps: one per row of two chunks
constexpr int MT_THREADS = (4 + MT_XF + 2) * 32;  // epilogue, transform, MMA issuer, producer
constexpr int MT_TM_D = 0, MT_TM_A = 2 * MT_N;    // tensor-memory columns: two accumulators, then the filterbank
constexpr int MT_MAX_F = 512 - MT_TM_A;

struct MtBarriers {
  uint64_t raw_full[MT_RING_MAX], raw_empty[MT_RING_MAX];
  uint64_t b_full[2], b_empty[2], acc_full[2], acc_empty[2], bank_full;
  uint32_t tmem_base;
  int abort_flag;
};

__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
// A from tensor memory (lane = row, one 32-bit column per K element), B from shared memory
__device__ __forceinline__ void mma_tf32_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tc_st_32x32b_x8(uint32_t taddr, const float (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "f"(v[0]), "f"(v[1]),
               "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
               : "memory");
}

__global__ void __launch_bounds__(MT_THREADS, 1) power_mel_log_dense_kernel(const MelParams p) {
  pdl_launch_dependents();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* const base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  // [operand tiles: 2 x stages x 32 x 128 B][ring of raw chunks]; during set-up the filterbank passes through the end of the memory
  uint8_t* const tiles_s = base;
  const uint32_t tile_bytes = static_cast<uint32_t>(p.stages) * MT_N * 128u;
  uint8_t* const ring = tiles_s + 2 * tile_bytes;
  const uint32_t row_bytes = static_cast<uint32_t>(p.F) * 8u, chunk_bytes = MT_ROWS * row_bytes;
  __shared__ MtBarriers bar;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  volatile int* const abortp = &bar.abort_flag;
  const int my_tiles = static_cast<int>(blockIdx.x) < p.tiles ? (p.tiles - static_cast<int>(blockIdx.x) + gridDim.x - 1) / gridDim.x : 0;
  const int F = static_cast<int>(p.F), M = static_cast<int>(p.M), ksteps = (F + 7) / 8;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.ring; ++s) {
      mbar_init(&bar.raw_full[s], 1);
      mbar_init(&bar.raw_empty[s], MT_ROWS);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&bar.b_full[a], MT_XF);
      mbar_init(&bar.b_empty[a], 1);
      mbar_init(&bar.acc_full[a], 1);
      mbar_init(&bar.acc_empty[a], 4);
    }
    mbar_init(&bar.bank_full, 1);
    bar.abort_flag = 0;
    mbar_fence_init();
  }
  // Tile i of this CTA covers frames [32 t, 32 t + 32), t = blockIdx.x + i gridDim.x, as up to four chunks of eight rows.
  auto chunks_of = [&](int64_t t0) { const int64_t left = p.T - t0; return left >= MT_N ? MT_N / MT_ROWS : static_cast<int>((left + MT_ROWS - 1) / MT_ROWS); };
  auto tile_frame = [&](int i) { return (static_cast<int64_t>(blockIdx.x) + static_cast<int64_t>(i) * gridDim.x) * MT_N; };
  auto load_chunk = [&](int64_t row, uint32_t s) {
    const int64_t rows = p.T - row < MT_ROWS ? p.T - row : MT_ROWS;
    // (an odd number of rows, the end of the input only, may leave 8 bytes: the transform warp fetches them itself)
    const uint32_t bytes = (static_cast<uint32_t>(rows) * row_bytes) & ~15u;
    mbar_expect_tx(&bar.raw_full[s], bytes);
    if (bytes) bulk_load(ring + s * chunk_bytes, p.spec + row * p.F, bytes, &bar.raw_full[s]);
  };

  // Filterbank -> shared memory, behind the wait: the launch before may have written it, too.  Rows of F | 1 words (an odd pitch: the column
  // reads below are conflict-free); a dense bank of odd F lies like this already and comes in one copy.  It passes through the end of the memory, so that
  // the chunks of the first tile whose slots lie in front of it come in meanwhile.  64 frames right behind another call: 4.1 us with
  // the filterbank read ahead of the wait, 7.7 behind it word by word, 5.6 like this, 1,000 frames 7.5 and 6.2, 20,000 33.6 and 32.3; behind torch's rfft,
  // which triggers nothing early, 64 frames 10.3 and 8.2, 3,750 14.6 and 12.3.
  pdl_wait();
  const int pitch = F | 1;
  float* const bank_s = reinterpret_cast<float*>(base + p.bank_off);
  const bool one_copy = pitch == F && p.ld_mel == F && M * F >= 4 && (reinterpret_cast<uintptr_t>(p.mel) & 15) == 0;
  if (one_copy) {
    const int whole = (M * F) & ~3;
    if (threadIdx.x == 0) {
      mbar_expect_tx(&bar.bank_full, whole * 4u);
      bulk_load(bank_s, p.mel, whole * 4u, &bar.bank_full);
    }
    if (threadIdx.x < static_cast<unsigned>(M * F - whole)) bank_s[whole + threadIdx.x] = p.mel[whole + threadIdx.x];
  } else {
    for (int n = warp; n < M; n += MT_THREADS / 32)
      for (int k = lane; k < F; k += 32) cp_async4(smem_u32(bank_s + n * pitch + k), p.mel + n * p.ld_mel + k);
  }
  const int early = p.early < chunks_of(tile_frame(0)) ? p.early : chunks_of(tile_frame(0));
  if (threadIdx.x == 0)
    for (int c = 0; c < early; ++c) load_chunk(tile_frame(0) + c * MT_ROWS, c);
  if (warp == 4 + MT_XF) {
    tmem_alloc(&bar.tmem_base, 512);
    tmem_relinquish();
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = bar.tmem_base;
  // -> tensor memory: lane m of quadrant `warp` holds filterbank row m, zero beyond M and F
  if (warp < 4 && (!one_copy || __all_sync(0xffffffffu, mbar_wait<true>(&bar.bank_full, 0, p.status, 17, abortp)))) {
    const int m = warp * 32 + lane;
    const uint32_t ta = tmem_base + MT_TM_A + (static_cast<uint32_t>(warp * 32) << 16);
    const float* const src = bank_s + (m < M ? m : 0) * pitch;
    int k0 = 0;
#pragma unroll 4
    for (; k0 + 8 <= F; k0 += 8) {
      float v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = src[k0 + j];
      if (m >= M) {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = 0.0f;
      }
      tc_st_32x32b_x8(ta + k0, v);
    }
    if (k0 < F) {
      float v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = m < M && k0 + j < F ? src[k0 + j] : 0.0f;
      tc_st_32x32b_x8(ta + k0, v);
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  // operand tiles: the bins beyond F, in the last stage, are never written, they must read as zero (rows of frames beyond T only reach columns
  // that are not stored)
  if (F % MEL_KS != 0)
    for (uint32_t i = threadIdx.x; i < 2 * MT_N * 8; i += MT_THREADS)
      reinterpret_cast<uint4*>(tiles_s + (i / (MT_N * 8)) * tile_bytes + (p.stages - 1) * (MT_N * 128))[i % (MT_N * 8)] = make_uint4(0, 0, 0, 0);
  fence_proxy_async_smem();
  __syncthreads();

  if (warp == 4 + MT_XF + 1) {
    // =========================== producer ===========================
    if (lane == 0) {
      uint32_t s = early == p.ring ? 0 : early, ph = early == p.ring ? 1 : 0;
      bool ok = true;
      for (int i = 0; i < my_tiles && ok; ++i) {
        const int64_t t0 = tile_frame(i);
        const int nc = chunks_of(t0);
        for (int c = i == 0 ? early : 0; c < nc; ++c) {
          if (!mbar_wait<true>(&bar.raw_empty[s], ph ^ 1, p.status, 11, abortp)) { ok = false; break; }
          load_chunk(t0 + c * MT_ROWS, s);
          if (++s == static_cast<uint32_t>(p.ring)) { s = 0; ph ^= 1; }
        }
      }
      if (!ok) bar.abort_flag = 1;
    }
  } else if (warp >= 4 && warp < 4 + MT_XF) {
    // =========================== transform: rows w and w + 16 of every tile ===========================
    const int w = warp - 4, lw = w % MT_ROWS;  // lw: row of the chunk
    constexpr int STEP = MT_XF / MT_ROWS;      // this warp takes every second chunk
    uint32_t s = w / MT_ROWS, ph = 0;          // its ring slot (the ring holds at least two chunks)
    bool ok = true;
    const int full_stages = F / MEL_KS, rest = F % MEL_KS;
    // two rounded squares and one rounded add, as spec.real**2 + spec.imag**2
    auto power = [](float2 v) { return __fadd_rn(__fmul_rn(v.x, v.x), __fmul_rn(v.y, v.y)); };
    for (int i = 0; i < my_tiles && ok; ++i) {
      const int64_t t0 = tile_frame(i);
      const int b = i & 1, nc = chunks_of(t0);
      ok = __all_sync(0xffffffffu, mbar_wait<true>(&bar.b_empty[b], ((i >> 1) & 1) ^ 1, p.status, 12, abortp));
      if (!ok) break;
      for (int r = w; r < MT_N && r / MT_ROWS < nc; r += MT_XF) {
        ok = __all_sync(0xffffffffu, mbar_wait<true>(&bar.raw_full[s], ph, p.status, 13, abortp));
        if (!ok) break;
        const int64_t row = t0 + r;
        if (row < p.T) {
          const float2* const src = reinterpret_cast<const float2*>(ring + s * chunk_bytes + lw * row_bytes) + lane;
          uint8_t* const dst = tiles_s + b * tile_bytes + sw128(r, lane);
          int ks = 0;
          for (; ks + 8 <= full_stages; ks += 8) {
            float2 v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = src[(ks + u) * MEL_KS];
#pragma unroll
            for (int u = 0; u < 8; ++u) *reinterpret_cast<float*>(dst + (ks + u) * (MT_N * 128)) = power(v[u]);
          }
          for (; ks < full_stages; ++ks) *reinterpret_cast<float*>(dst + ks * (MT_N * 128)) = power(src[ks * MEL_KS]);
          if (lane < rest) {
            const int k = full_stages * MEL_KS + lane;
            // the last value of the input when the chunk's bytes were rounded down
            const bool cut = row == p.T - 1 && k == F - 1 && (((lw + 1) * row_bytes) & 15u);
            const float2 v = cut ? p.spec[row * p.F + k] : src[full_stages * MEL_KS];
            *reinterpret_cast<float*>(dst + full_stages * (MT_N * 128)) = power(v);
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar.raw_empty[s]);
        s += STEP;
        if (s >= static_cast<uint32_t>(p.ring)) { s -= p.ring; ph ^= 1; }
      }
      if (!ok) break;
      fence_proxy_async_smem();  // generic-proxy writes -> visible to the tensor core's reads
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar.b_full[b]);
    }
    if (!ok) bar.abort_flag = 1;
  } else if (warp == 4 + MT_XF) {
    // =========================== MMA issuer ===========================
    const bool leader = elect_one();
    const uint32_t idesc = make_idesc_tf32(128, MT_N);
    // descriptors are formed with one 32-bit add (low word: shared address >> 4; the high word is constant)
    const uint32_t desc_hi = (1024u >> 4) | (1u << 14) | (2u << 29);
    auto desc = [&](uint32_t lo) { return (static_cast<uint64_t>(desc_hi) << 32) | lo; };
    const uint32_t tiles_lo = smem_u32(tiles_s) >> 4;
    const int whole = ksteps >> 2;
    bool ok = true;
    for (int i = 0; i < my_tiles && ok; ++i) {
      const int b = i & 1;
      const uint32_t par = (i >> 1) & 1;
      // (No vote and no __syncwarp below: a lane that gives up a wait leaves the others to theirs.  With votes 64 frames took 3.93 us, 3.83 without.)
      if (!mbar_wait_spin(&bar.acc_empty[b], par ^ 1, p.status, 14, abortp) || !mbar_wait_spin(&bar.b_full[b], par, p.status, 15, abortp)) {
        ok = false;
        break;
      }
      tc_fence_after();
      if (leader) {
        const uint32_t d = tmem_base + MT_TM_D + b * MT_N;
        uint32_t a = tmem_base + MT_TM_A, b_lo = tiles_lo + b * (tile_bytes >> 4);
        for (int k = 0; k < whole; ++k) {
#pragma unroll
          for (int j = 0; j < 4; ++j) mma_tf32_ta(d, a + 8 * j, desc(b_lo + 2 * j), idesc, (k | j) != 0);
          a += MEL_KS;
          b_lo += (MT_N * 128) >> 4;
        }
        for (int j = 0; j < (ksteps & 3); ++j) mma_tf32_ta(d, a + 8 * j, desc(b_lo + 2 * j), idesc, (whole | j) != 0);
        tc_commit(&bar.b_empty[b]);
        tc_commit(&bar.acc_full[b]);
      }
    }
    if (!ok && leader) bar.abort_flag = 1;
  } else {
    // =========================== epilogue: warps 0..3, lane = mel row ===========================
    const int m = warp * 32 + lane;
    const bool mine = m < M;
    const float mean = p.mean && mine ? __ldg(p.mean + m) : 0.0f, istd = p.mean && mine ? __ldg(p.istd + m) : 1.0f;
    bool ok = true;
    for (int i = 0; i < my_tiles && ok; ++i) {
      const int b = i & 1;
      ok = __all_sync(0xffffffffu, mbar_wait<true>(&bar.acc_full[b], (i >> 1) & 1, p.status, 16, abortp));
      if (!ok) break;
      tc_fence_after();
      uint32_t r[MT_N];
      tc_ld_32x32b_x32(tmem_base + MT_TM_D + b * MT_N + (static_cast<uint32_t>(warp * 32) << 16), r);
      tc_wait_ld();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar.acc_empty[b]);
      const int64_t t0 = tile_frame(i);
      const int n = p.T - t0 < MT_N ? static_cast<int>(p.T - t0) : MT_N;
      if (mine) {
        float* const o = p.out + t0 * p.ldo + m;
        // (all logarithms before the first store or test: they overlap each other's latency)
        float v[MT_N];
#pragma unroll
        for (int j = 0; j < MT_N; ++j) v[j] = __logf(fmaxf(__uint_as_float(r[j]), 1.1920929e-7f));
        if (p.mean) {
#pragma unroll
          for (int j = 0; j < MT_N; ++j) v[j] = (v[j] - mean) * istd;
        }
        if (n == MT_N) {
#pragma unroll
          for (int j = 0; j < MT_N; ++j) o[j * p.ldo] = v[j];
        } else {
#pragma unroll
          for (int j = 0; j < MT_N; ++j)
            if (j < n) o[j * p.ldo] = v[j];
        }
      }
    }
    if (!ok) bar.abort_flag = 1;
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 4 + MT_XF) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace
}  // namespace vx

namespace vx {
namespace {
// shared memory the kernel needs for an M x F filterbank with `ring` A stages; 0 when M is too large
size_t mel_smem_bytes(int64_t F, int64_t M, int ring) {
  if (M <= 0 || F <= 0 || M > 256) return 0;
  const size_t n_pad = static_cast<size_t>((M + 15) / 16 * 16), stages = static_cast<size_t>((F + MEL_KS - 1) / MEL_KS);
  return stages * n_pad * 128 + 1024 + static_cast<size_t>(ring) * MEL_SLOT;
}
}  // namespace
}  // namespace vx

extern "C" int vx_power_mel_log_supported(int64_t F, int64_t M) {
  const size_t need = vx::mel_smem_bytes(F, M, 2);
  return need != 0 && need <= static_cast<size_t>(vx::MEL_MAX_SMEM);
}

extern "C" int vx_power_mel_log(const void* spec, int64_t T, int64_t F, int64_t ld_spec, const float* mel, int64_t M,
                                int64_t ld_mel, const float* cmvn_mean, const float* cmvn_istd, float* out, int64_t ldo,
                                void* stream) {
  using namespace vx;
  if (T < 0 || F <= 0 || M <= 0) return fail(-1, "bad shape T=%lld F=%lld M=%lld", (long long)T, (long long)F, (long long)M);
  if (T == 0) return 0;
  if (!spec || !mel || !out) return fail(-1, "spec, mel and out must not be NULL");
  if ((cmvn_mean == nullptr) != (cmvn_istd == nullptr)) return fail(-1, "cmvn_mean and cmvn_istd go together");
  if (reinterpret_cast<uintptr_t>(spec) & 7) return fail(-1, "spec must be 8-byte aligned (complex64)");
  if (ld_spec < F || ld_mel < F || ldo < M) return fail(-1, "row strides are smaller than the rows");
  if (M > 256) return fail(-1, "at most 256 mel rows (M=%lld)", (long long)M);
  MelParams p{};
  p.spec = static_cast<const float2*>(spec);
  p.T = T; p.F = F; p.ld_spec = ld_spec;
  p.mel = mel; p.M = M; p.ld_mel = ld_mel;
  p.mean = cmvn_mean; p.istd = cmvn_istd;
  p.out = out; p.ldo = ldo;
  p.n_pad = static_cast<int>((M + 15) / 16 * 16);
  p.stages = static_cast<int>((F + MEL_KS - 1) / MEL_KS);
  p.tiles = static_cast<int>((T + MEL_BM - 1) / MEL_BM);
  const size_t bank = static_cast<size_t>(p.stages) * p.n_pad * 128 + 1024;
  p.ring = MEL_RING_MAX;
  while (p.ring > 2 && bank + static_cast<size_t>(p.ring) * MEL_SLOT > static_cast<size_t>(MEL_MAX_SMEM)) --p.ring;
  const size_t smem = bank + static_cast<size_t>(p.ring) * MEL_SLOT;
  if (smem > static_cast<size_t>(MEL_MAX_SMEM))
    return fail(-1, "filterbank of %lld x %lld does not fit in shared memory (%zu bytes needed, %d available)", (long long)M,
                (long long)F, smem, MEL_MAX_SMEM);
  p.status = device_status_ptr();
  // dense rows, at most 128 mel rows and 448 bins: the transposed product (see power_mel_log_dense_kernel)
  {
    const size_t tiles_bytes = 1024 + 2 * static_cast<size_t>(p.stages) * MT_N * 128, chunk = static_cast<size_t>(MT_ROWS) * F * 8;
    const size_t room = 225 * 1024, bank_bytes = 1024 + static_cast<size_t>(M) * (F | 1) * 4;
    const int ring = tiles_bytes < room ? static_cast<int>((room - tiles_bytes) / chunk) : 0;
    if (ld_spec == F && aligned16(spec) && M <= 128 && F <= MT_MAX_F && ring >= 2 && bank_bytes <= room) {
      p.ring = ring < MT_RING_MAX ? ring : MT_RING_MAX;
      p.tiles = static_cast<int>((T + MT_N - 1) / MT_N);
      const size_t need = tiles_bytes + p.ring * chunk;
      size_t bytes = need > bank_bytes ? need : bank_bytes;
      const size_t four = tiles_bytes + MT_N / MT_ROWS * chunk + bank_bytes;  // a tile's chunks in front of the filterbank, where that fits
      if (four > bytes) bytes = four < room ? four : room;
      p.bank_off = static_cast<int>((bytes - bank_bytes) & ~static_cast<size_t>(127));
      const int64_t front = p.bank_off - static_cast<int64_t>(tiles_bytes - 1024);
      p.early = front <= 0 ? 0 : static_cast<int>(front / static_cast<int64_t>(chunk) < p.ring ? front / static_cast<int64_t>(chunk) : p.ring);
      static std::atomic<uint64_t> dense_done{0};
      int dv = 0;
      VX_CUDA_OK(cudaGetDevice(&dv));
      if (dv >= 64 || !(dense_done.load(std::memory_order_acquire) & (1ull << dv))) {
        VX_CUDA_OK(cudaFuncSetAttribute(power_mel_log_dense_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(room)));
        if (dv < 64) dense_done.fetch_or(1ull << dv, std::memory_order_release);
      }
      const int g = p.tiles < sm_count() ? p.tiles : sm_count();
      VX_CUDA_OK(launch_dependent(power_mel_log_dense_kernel, dim3(g), dim3(MT_THREADS), bytes, static_cast<cudaStream_t>(stream), p));
      return 0;
    }
  }
  int dev = 0;
  VX_CUDA_OK(cudaGetDevice(&dev));
  const int sms = sm_count();
  static std::atomic<uint64_t> attr_done{0};
  const bool dev_cached = dev >= 0 && dev < 64;
  if (!dev_cached || !(attr_done.load(std::memory_order_acquire) & (1ull << dev))) {
    VX_CUDA_OK(cudaFuncSetAttribute(power_mel_log_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MEL_MAX_SMEM));
    if (dev_cached) attr_done.fetch_or(1ull << dev, std::memory_order_release);
  }
  const int grid = p.tiles < sms ? p.tiles : sms;
  VX_CUDA_OK(launch_dependent(power_mel_log_kernel, dim3(grid), dim3(MEL_THREADS), smem, static_cast<cudaStream_t>(stream), p));
  return 0;
}
