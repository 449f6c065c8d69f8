// bf16 GEMM on 5th-generation tensor cores (sm_100a): C[M,N] = A * B^T (+ bias) (+ C), fp32 accumulation in TMEM.
//
// One persistent CTA per SM, warp-specialised:
//   warp 0   : TMA producer  (one elected lane issues cp.async.bulk.tensor loads, 128-byte swizzle, no multicast)
//   warp 1   : MMA issuer    (one elected lane issues tcgen05.mma; owns the TMEM allocation)
//   warps 2-9: epilogue      (tcgen05.ld TMEM -> registers -> bf16 -> shared memory -> global), two per TMEM lane quarter
// Tile 128 x 256 x 64, 4-stage shared-memory ring (48 KB per stage), two 256-column TMEM accumulators so
// the epilogue of tile i overlaps the main loop of tile i+1.
//
// Operand layouts ("major" = which dim is contiguous in global memory):
//   A K-major : A[M, K]   (activations in a forward projection, dY in dgrad)
//   A MN-major: A^T[K, M] (dY in wgrad: the reduction dim T is the row index)
//   B K-major : B[N, K]   (weights in a forward projection)
//   B MN-major: B^T[K, N] (weights in dgrad, X in wgrad)
// MN-major tiles are fetched as 64x64 boxes so that the shared-memory image is the canonical
// MN-major 128B-swizzle layout (64-element blocks LBO apart, 8-row groups SBO apart).
//
// Every launch is a programmatic dependent of the kernel before it (pdl.cuh, the second kind): the launch, the barriers, the tensor memory and
// the descriptors of a GEMM are ready when the last block of that kernel leaves, or long before where that kernel lets its successor start
// early, and all its warps wait for the kernel's results before they touch memory.
// Back to back, us: [2048 x 512] K = 256 6.2 -> 3.9, [768 x 256] K = 2048 9.3 -> 7.3, [1024 x 2048] K = 2048 12.4 -> 9.8,
// [8192 x 4096] K = 512 35.1 -> 32.9, [512 x 4096] K = 8192 31 -> 28.4.  A GEMM does not let its successor start before its own last CTA
// ends (let_next_start): the CTAs of a successor of one wave then took whatever SMs were idle, and the last of these sizes 31.4, probably
// because neighbouring tiles no longer met in one half of the L2 cache (CTA pairs would gain 0.5 of 33).
//
// All waits are bounded (sm100.cuh); on a timeout the kernel records a status word, every role unwinds,
// TMEM is freed and the kernel returns.
#include <cuda_fp8.h>

#include "entries.h"
#include "pdl.cuh"
#include "sm100.cuh"

namespace sb {

constexpr int BM = 128, BN = 256, BK = 64;
constexpr int EPI_WARPS = 8;                      // two per TMEM lane quarter, each takes half of a tile's columns
constexpr int A_STAGE = BM * BK * 2;              // 16 KB
constexpr int EPI_OFF = 4 * 48 * 1024 + 256;      // behind the stages and the barriers
constexpr int SMEM_BYTES = EPI_OFF + EPI_WARPS * 32 * 64 /*EPI_BYTES*/ + 1024 /*align*/;
constexpr int TMEM_COLS = 512;
constexpr int GROUP_M = 16;                       // raster: 16 m-tiles share the concurrently running n-tiles
constexpr int NUM_THREADS = 64 + 32 * EPI_WARPS;

struct GemmParams {
  __nv_bfloat16* C;
  const __nv_bfloat16* bias;   // [N] or null
  const __nv_bfloat16* residual;  // [M, N] (leading dim ldr) added in the epilogue, or null
  int M, N, K, ldc, ldr;
  int beta;                    // 1: C += result (bf16 read-modify-write)
  uint32_t* status;
  const float* alpha;          // device scalar multiplied into the accumulator (fp8 de-quantisation), or null
  const float* alpha2;         // second device scalar (the other operand's de-quantisation factor), or null
  int a_fmt, b_fmt;            // fp8 operand formats for the instruction descriptor: 0 = e4m3, 1 = e5m2
  // gated-MLP epilogue of the CTA-pair kernel (GLU mode): B = [w1 ; w2] with F rows each, C = [a | b] (ldc >= 2 F);
  // besides C the epilogue writes q = e4m3(silu(a) * b) [M, F] under delayed scaling (ring `hist` of `slots` floats,
  // this call's slot `cur`, de-quantisation factor to `scale_inv`)
  uint8_t* glu_q;
  int glu_F;
  float* glu_hist;
  int glu_slots, glu_cur;
  float* glu_scale_inv;
  // gate backward in the epilogue of the w3 input-gradient product (GLU = 2): C is not written; with g = the product's
  // result and [a | b] read from glu_ab (leading dimension glu_ld_ab), the epilogue writes q [M, 2 F] =
  // e5m2(g * b * silu'(a) | g * silu(a)) under delayed scaling (same ring protocol)
  const __nv_bfloat16* glu_ab;
  int glu_ld_ab;
};

__device__ __forceinline__ void tile_coords(int tile, int m_tiles, int n_tiles, int& mt, int& nt) {
  const int per_group = GROUP_M * n_tiles;
  const int g = tile / per_group;
  const int first_m = g * GROUP_M;
  const int gsz = min(GROUP_M, m_tiles - first_m);
  const int r = tile - g * per_group;
  mt = first_m + r % gsz;
  nt = r / gsz;
}

// A warp's 32 rows x 32 columns on their way to memory.  A lane holds a row (that is how tensor memory is read); stored from there, a
// 16-byte store touches 32 lines and half a sector of each, and a 256 x 256 tile took 5.6 us to leave: more than the products of a tile need
// at K = 512.  Through 2 KB of shared memory four lanes store 64 consecutive bytes of a row, eight rows at a time.  The 16-byte chunks of a row
// are permuted so that neither side meets a bank twice.
constexpr int EPI_WARP_BYTES = 32 * 64, EPI_BYTES = EPI_WARPS * EPI_WARP_BYTES;
__device__ __forceinline__ void epi_put(uint32_t at, const uint4 v) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ uint4 epi_get(uint32_t at) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at) : "memory");
  return v;
}
// bf16: out = the lane's row, 4 x 8 columns from col0 on; rows row0 .. row0 + 31 of dst (leading dimension ld)
__device__ __forceinline__ void store_rows(uint32_t stage, const uint4 (&out)[4], __nv_bfloat16* dst, int ld, int row0, int rows, int col0,
                                           int cols, int lane) {
#pragma unroll
  for (int v = 0; v < 4; ++v) epi_put(stage + lane * 64 + ((v ^ (lane >> 1 & 3)) << 4), out[v]);
  __syncwarp();
  const int c = lane & 3, col = col0 + 8 * c;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = 8 * i + (lane >> 2);
    const uint4 v = epi_get(stage + r * 64 + ((c ^ (r >> 1 & 3)) << 4));
    if (row0 + r < rows && col + 8 <= cols) *reinterpret_cast<uint4*>(dst + size_t(row0 + r) * ld + col) = v;
  }
  __syncwarp();
}
// one byte a value: 2 x 16 columns
__device__ __forceinline__ void store_rows_u8(uint32_t stage, const uint4 a, const uint4 b, uint8_t* dst, int ld, int row0, int rows, int col0,
                                              int lane) {
  epi_put(stage + lane * 32 + ((lane >> 2 & 1) << 4), a);
  epi_put(stage + lane * 32 + ((lane >> 2 & 1 ^ 1) << 4), b);
  __syncwarp();
  const int c = lane & 1;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r = 16 * i + (lane >> 1);
    const uint4 v = epi_get(stage + r * 32 + ((c ^ (r >> 2 & 1)) << 4));
    if (row0 + r < rows) *reinterpret_cast<uint4*>(dst + size_t(row0 + r) * ld + col0 + 16 * c) = v;
  }
  __syncwarp();
}

// Epilogue of 32 accumulator columns of one row: scale, + bias, + residual, (+ C), bf16.  Most products have none of the additions: without
// the tests for them between its columns a chunk takes 400 cycles less (a tile of 128 x 256 per warp has four).
__device__ __forceinline__ void finish_chunk(const GemmParams& p, bool plain, int row, int col0, const uint32_t (&r)[32], float alpha,
                                             uint4 (&out)[4]) {
  if (plain) {
    __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&out[0]);
#pragma unroll
    for (int j = 0; j < 16; ++j) o2[j] = __floats2bfloat162_rn(__uint_as_float(r[2 * j]) * alpha, __uint_as_float(r[2 * j + 1]) * alpha);
    return;
  }
  const __nv_bfloat16* crow = p.C + size_t(row) * p.ldc;
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    const int col = col0 + v * 8;
    const bool live = row < p.M && col + 8 <= p.N;
    float f[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = __uint_as_float(r[v * 8 + j]) * alpha;
    if (p.bias && live) {
      const uint4 bv = *reinterpret_cast<const uint4*>(p.bias + col);
      const __nv_bfloat162* b2 = reinterpret_cast<const __nv_bfloat162*>(&bv);
#pragma unroll
      for (int j = 0; j < 4; ++j) { float2 t = __bfloat1622float2(b2[j]); f[2 * j] += t.x; f[2 * j + 1] += t.y; }
    }
    if (p.residual && live) {
      const uint4 rv = *reinterpret_cast<const uint4*>(p.residual + size_t(row) * p.ldr + col);
      const __nv_bfloat162* r2 = reinterpret_cast<const __nv_bfloat162*>(&rv);
#pragma unroll
      for (int j = 0; j < 4; ++j) { float2 t = __bfloat1622float2(r2[j]); f[2 * j] += t.x; f[2 * j + 1] += t.y; }
    }
    if (p.beta && live) {
      const uint4 ov = *reinterpret_cast<const uint4*>(crow + col);
      const __nv_bfloat162* o2 = reinterpret_cast<const __nv_bfloat162*>(&ov);
#pragma unroll
      for (int j = 0; j < 4; ++j) { float2 t = __bfloat1622float2(o2[j]); f[2 * j] += t.x; f[2 * j + 1] += t.y; }
    }
    __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&out[v]);
#pragma unroll
    for (int j = 0; j < 4; ++j) o2[j] = __floats2bfloat162_rn(f[2 * j], f[2 * j + 1]);
  }
}

// EB = bytes per operand element: 2 = bf16 (kind::f16), 1 = fp8 e4m3 / e5m2 (kind::f8f6f4).  A shared-memory row is
// always 128 bytes, so a k-block holds 64 bf16 or 128 fp8 values and every MMA consumes 32 bytes of K.
// BN = tile width: 256, or 128 / 64 for outputs with too few 256-wide tiles to fill the chip (see pick_tile); the same
// 192 KB of shared memory then hold 6 / 8 stages.
template <int A_MN, int B_MN, int EB, int BN = 256>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, GemmParams p) {
  constexpr int B_STAGE = BN * 128, STAGE_BYTES = A_STAGE + B_STAGE, STAGES = 4 * 48 * 1024 / STAGE_BYTES;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  // barrier block after the stages
  const uint32_t bar_base = smem_base + STAGES * STAGE_BYTES;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
  auto tfull_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + a); };
  auto tempty_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + 2 + a); };
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem_gen + STAGES * STAGE_BYTES + 8 * (2 * STAGES + 4));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_gen + STAGES * STAGE_BYTES + 8 * (2 * STAGES + 4) + 8);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int m_tiles = (p.M + BM - 1) / BM, n_tiles = (p.N + BN - 1) / BN;
  const int num_tiles = m_tiles * n_tiles;
  constexpr int BKE = 128 / EB;                      // elements of K per k-block
  constexpr int MNB = 128 / EB;                      // MN elements per 128-byte row of an MN-major box
  constexpr int MN_BOX_BYTES = BKE * 128;            // one MN-major box: BKE k-rows of 128 bytes
  const int num_kb = (p.K + BKE - 1) / BKE;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(tfull_bar(a), 1); mbar_init(tempty_bar(a), EPI_WARPS); }
    *abort_flag = 0;
    fence_barrier_init();
    prefetch_tmap(&tmA);
    prefetch_tmap(&tmB);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  wait_for_previous();

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      int stage = 0; uint32_t phase = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
        int mt, nt; tile_coords(tile, m_tiles, n_tiles, mt, nt);
        const int m0 = mt * BM, n0 = nt * BN;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag, p.status, ST_TIMEOUT_EMPTY)) { ok = false; break; }
          const uint32_t a_dst = smem_base + stage * STAGE_BYTES;
          const uint32_t b_dst = a_dst + A_STAGE;
          mbar_expect_tx(full_bar(stage), STAGE_BYTES);
          const int k0 = kb * BKE;
          if (A_MN == 0) {
            tma_load_2d(a_dst, &tmA, k0, m0, full_bar(stage));
          } else {
#pragma unroll
            for (int j = 0; j < BM / MNB; ++j) tma_load_2d(a_dst + j * MN_BOX_BYTES, &tmA, m0 + MNB * j, k0, full_bar(stage));
          }
          if (B_MN == 0) {
            tma_load_2d(b_dst, &tmB, k0, n0, full_bar(stage));
          } else {
#pragma unroll
            for (int j = 0; j < BN / MNB; ++j) tma_load_2d(b_dst + j * MN_BOX_BYTES, &tmB, n0 + MNB * j, k0, full_bar(stage));
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        }
      }
      if (!ok) {
        // let loads that are still in flight land before the CTA exits
        const unsigned long long t0 = globaltimer();
        while (globaltimer() - t0 < 200000ull) { __nanosleep(1000); }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      constexpr int UK = 32 / EB;                       // K elements per MMA (32 bytes)
      const uint32_t idesc = EB == 2 ? umma_idesc_bf16(BM, BN, A_MN, B_MN)
                                     : umma_idesc_fp8(BM, BN, A_MN, B_MN, p.a_fmt, p.b_fmt);
      constexpr uint32_t a_lbo = A_MN ? (uint32_t)MN_BOX_BYTES : 16u, a_step = A_MN ? (UK * 128u) >> 4 : 2u;
      constexpr uint32_t b_lbo = B_MN ? (uint32_t)MN_BOX_BYTES : 16u, b_step = B_MN ? (UK * 128u) >> 4 : 2u;
      int stage = 0; uint32_t phase = 0;
      uint32_t acc_phase[2] = {0u, 0u};
      int local = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x, ++local) {
        const int acc = local & 1;
        if (!mbar_wait(tempty_bar(acc), acc_phase[acc] ^ 1u, abort_flag, p.status, ST_TIMEOUT_TMEM_EMPTY)) { ok = false; break; }
        acc_phase[acc] ^= 1u;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(full_bar(stage), phase, abort_flag, p.status, ST_TIMEOUT_FULL)) { ok = false; break; }
          tc_fence_after();
          const uint32_t a_addr = smem_base + stage * STAGE_BYTES;
          const uint64_t adesc = umma_smem_desc(a_addr, a_lbo, 1024u);
          const uint64_t bdesc = umma_smem_desc(a_addr + A_STAGE, b_lbo, 1024u);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            if (EB == 2) umma_bf16(d_tmem, adesc + k * a_step, bdesc + k * b_step, idesc, (kb | k) != 0 ? 1u : 0u);
            else umma_fp8(d_tmem, adesc + k * a_step, bdesc + k * b_step, idesc, (kb | k) != 0 ? 1u : 0u);
          }
          umma_commit(empty_bar(stage));
          if (++stage == STAGES) { stage = 0; phase ^= 1u; }
        }
        if (ok) umma_commit(tfull_bar(acc));
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2..9)
    const int q = warp & 3;                         // TMEM lane quarter this warp may access
    const int half = (warp - 2) >> 2;               // its half of the columns
    const uint32_t stage_w = smem_base + EPI_OFF + (warp - 2) * EPI_WARP_BYTES;
    uint32_t acc_phase[2] = {0u, 0u};
    int local = 0;
    bool ok = true;
    const float alpha = (p.alpha ? p.alpha[0] : 1.f) * (p.alpha2 ? p.alpha2[0] : 1.f);
    const bool plain = !p.bias && !p.residual && !p.beta;
    for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x, ++local) {
      const int acc = local & 1;
      int mt, nt; tile_coords(tile, m_tiles, n_tiles, mt, nt);
      if (!mbar_wait(tfull_bar(acc), acc_phase[acc], abort_flag, p.status, ST_TIMEOUT_TMEM_FULL)) { ok = false; break; }
      acc_phase[acc] ^= 1u;
      tc_fence_after();
      const int row0 = mt * BM + q * 32;
      const int n0 = nt * BN;
      const uint32_t t_row = tmem_base + (uint32_t(q * 32) << 16) + acc * BN;
#pragma unroll 1
      for (int c = half * (BN / 64); c < (half + 1) * (BN / 64); ++c) {
        uint32_t r[32];
        tmem_ld_32x32(t_row + c * 32, r);
        tmem_wait_ld();
        uint4 out[4];
        finish_chunk(p, plain, row0 + lane, n0 + c * 32, r, alpha, out);
        store_rows(stage_w, out, p.C, p.ldc, row0, p.M, n0 + c * 32, p.N, lane);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(tempty_bar(acc));
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}


// ------------------------------------------------------------------------------------ CTA-pair kernel (cta_group::2)
// Two CTAs of a cluster (an SM pair) work on one 256 x 256 output tile.  CTA r of the pair stages rows [128 r, 128 r + 128)
// of the A tile and rows [128 r, 128 r + 128) of the B tile (32 KB per stage instead of 48 KB: six stages, and a third
// less shared-memory traffic per FLOP, which is what bounds one-byte operands on a single SM); its TMEM holds the 128
// accumulator rows of its half.  The even CTA's MMA thread issues tcgen05.mma.cta_group::2 for both; its commits
// arrive on the stage barriers of both CTAs.  Loads complete on the even CTA's `full` barrier.  No multicast loads.
constexpr int P_STAGES = 6;
constexpr int P_A_STAGE = 128 * 128;                 // 16 KB: this CTA's 128 rows of A (128-byte rows)
constexpr int P_B_STAGE = 128 * 128;                 // 16 KB: this CTA's 128 rows of B
constexpr int P_STAGE_BYTES = P_A_STAGE + P_B_STAGE;
constexpr int P_EPI_OFF = P_STAGES * P_STAGE_BYTES + 256;
constexpr int P_SMEM_BYTES = P_EPI_OFF + EPI_BYTES + 1024;
constexpr int P_GROUP_M = 8;

__device__ __forceinline__ void pair_tile_coords(int tile, int m_tiles, int n_tiles, int& mt, int& nt) {
  const int per_group = P_GROUP_M * n_tiles;
  const int g = tile / per_group;
  const int first_m = g * P_GROUP_M;
  const int gsz = min(P_GROUP_M, m_tiles - first_m);
  const int r = tile - g * per_group;
  mt = first_m + r % gsz;
  nt = r / gsz;
}

// GLU = 1 (K-major one-byte operands only): output tile t covers features [128 t, 128 t + 128) of BOTH halves of the
// packed gate projection: the even CTA stages the w1 rows of those features, the odd CTA the w2 rows, so accumulator
// columns 0-127 hold a and 128-255 hold b of the same features, and the epilogue applies the gate on the spot: it
// stores a and b (bf16, for the backward) and the e4m3 operand of the following projection, which the separate gate
// kernel otherwise produces by re-reading [a | b] from memory.
template <int A_MN, int B_MN, int EB, int GLU = 0>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, GemmParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  const uint32_t bar_base = smem_base + P_STAGES * P_STAGE_BYTES;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (P_STAGES + s); };
  auto tfull_bar = [&](int a) { return bar_base + 8u * (2 * P_STAGES + a); };
  auto tempty_bar = [&](int a) { return bar_base + 8u * (2 * P_STAGES + 2 + a); };
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem_gen + P_STAGES * P_STAGE_BYTES + 8 * (2 * P_STAGES + 4));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_gen + P_STAGES * P_STAGE_BYTES + 8 * (2 * P_STAGES + 4) + 8);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();             // 0: issues the MMAs, 1: partner
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
  const int m_tiles = (p.M + 255) / 256, n_tiles = GLU == 1 ? p.glu_F / 128 : (p.N + BN - 1) / BN;
  const int num_tiles = m_tiles * n_tiles;
  constexpr int BKE = 128 / EB;
  constexpr int MNB = 128 / EB;
  constexpr int MN_BOX_BYTES = BKE * 128;
  const int num_kb = (p.K + BKE - 1) / BKE;

  if (threadIdx.x == 0) {
    for (int s = 0; s < P_STAGES; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(tfull_bar(a), 1); mbar_init(tempty_bar(a), 2 * EPI_WARPS); }   // of both CTAs
    *abort_flag = 0;
    fence_barrier_init();
    prefetch_tmap(&tmA);
    prefetch_tmap(&tmB);
  }
  if (warp == 1) {
    tmem_alloc_pair(smem_u32(const_cast<uint32_t*>(tmem_slot)), TMEM_COLS);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  // barriers of both CTAs are initialised before either signals the other
  cluster_arrive();
  cluster_wait();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  wait_for_previous();

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (both CTAs)
    if (elect_one()) {
      int stage = 0; uint32_t phase = 0;
      bool ok = true;
      for (int tile = pair; tile < num_tiles && ok; tile += npairs) {
        int mt, nt; pair_tile_coords(tile, m_tiles, n_tiles, mt, nt);
        const int m0 = mt * 256 + int(rank) * 128;
        const int n0 = GLU == 1 ? nt * 128 + int(rank) * p.glu_F : nt * BN + int(rank) * 128;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(empty_bar(stage), phase ^ 1u, abort_flag, p.status, ST_TIMEOUT_EMPTY)) { ok = false; break; }
          const uint32_t a_dst = smem_base + stage * P_STAGE_BYTES;
          const uint32_t b_dst = a_dst + P_A_STAGE;
          const uint32_t bar = map_to_cta(full_bar(stage), 0);         // the even CTA counts both CTAs' bytes
          if (rank == 0) mbar_expect_tx(full_bar(stage), 2 * P_STAGE_BYTES);
          const int k0 = kb * BKE;
          if (A_MN == 0) {
            tma_load_2d_pair(a_dst, &tmA, k0, m0, bar);
          } else {
#pragma unroll
            for (int j = 0; j < 128 / MNB; ++j) tma_load_2d_pair(a_dst + j * MN_BOX_BYTES, &tmA, m0 + MNB * j, k0, bar);
          }
          if (B_MN == 0) {
            tma_load_2d_pair(b_dst, &tmB, k0, n0, bar);
          } else {
#pragma unroll
            for (int j = 0; j < 128 / MNB; ++j) tma_load_2d_pair(b_dst + j * MN_BOX_BYTES, &tmB, n0 + MNB * j, k0, bar);
          }
          if (++stage == P_STAGES) { stage = 0; phase ^= 1u; }
        }
      }
      if (!ok) {
        const unsigned long long t0 = globaltimer();
        while (globaltimer() - t0 < 200000ull) { __nanosleep(1000); }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (even CTA only)
    if (rank == 0 && elect_one()) {
      constexpr int UK = 32 / EB;
      const uint32_t idesc = EB == 2 ? umma_idesc_bf16(256, BN, A_MN, B_MN)
                                     : umma_idesc_fp8(256, BN, A_MN, B_MN, p.a_fmt, p.b_fmt);
      constexpr uint32_t a_lbo = A_MN ? (uint32_t)MN_BOX_BYTES : 16u, a_step = A_MN ? (UK * 128u) >> 4 : 2u;
      constexpr uint32_t b_lbo = B_MN ? (uint32_t)MN_BOX_BYTES : 16u, b_step = B_MN ? (UK * 128u) >> 4 : 2u;
      int stage = 0; uint32_t phase = 0;
      uint32_t acc_phase[2] = {0u, 0u};
      int local = 0;
      bool ok = true;
      for (int tile = pair; tile < num_tiles && ok; tile += npairs, ++local) {
        const int acc = local & 1;
        if (!mbar_wait(tempty_bar(acc), acc_phase[acc] ^ 1u, abort_flag, p.status, ST_TIMEOUT_TMEM_EMPTY)) { ok = false; break; }
        acc_phase[acc] ^= 1u;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(full_bar(stage), phase, abort_flag, p.status, ST_TIMEOUT_FULL)) { ok = false; break; }
          tc_fence_after();
          const uint32_t a_addr = smem_base + stage * P_STAGE_BYTES;
          const uint64_t adesc = umma_smem_desc(a_addr, a_lbo, 1024u);
          const uint64_t bdesc = umma_smem_desc(a_addr + P_A_STAGE, b_lbo, 1024u);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            if (EB == 2) umma_bf16_pair(d_tmem, adesc + k * a_step, bdesc + k * b_step, idesc, (kb | k) != 0 ? 1u : 0u);
            else umma_fp8_pair(d_tmem, adesc + k * a_step, bdesc + k * b_step, idesc, (kb | k) != 0 ? 1u : 0u);
          }
          umma_commit_pair(empty_bar(stage));          // frees this stage in both CTAs
          if (++stage == P_STAGES) { stage = 0; phase ^= 1u; }
        }
        if (ok) umma_commit_pair(tfull_bar(acc));      // wakes the epilogue warps of both CTAs
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2..9 of both CTAs)
    const int q = warp & 3;
    const int half = (warp - 2) >> 2;
    const uint32_t stage_w = smem_base + P_EPI_OFF + (warp - 2) * EPI_WARP_BYTES;
    uint32_t acc_phase[2] = {0u, 0u};
    int local = 0;
    bool ok = true;
    const float alpha = (p.alpha ? p.alpha[0] : 1.f) * (p.alpha2 ? p.alpha2[0] : 1.f);
    const bool plain = !p.bias && !p.residual && !p.beta;
    float q_scale = 1.f, q_amax = 0.f;
    if (GLU) {
      // delayed scaling of the gated output: scale from the amax ring (all slots but this call's and the next one's)
      const int nxt = p.glu_cur + 1 == p.glu_slots ? 0 : p.glu_cur + 1;
      float a = 0.f;
      for (int j = 0; j < p.glu_slots; ++j) {
        if (j == p.glu_cur || j == nxt) continue;
        const float h = p.glu_hist[j];
        if (h > a && h < 3.0e38f) a = h;
      }
      const float fmax_q = GLU == 2 ? 57344.f : 448.f;          // e5m2 gradients, e4m3 activations
      if (!(a > 0.f)) a = fmax_q;
      if (blockIdx.x == 0 && warp == 2 && lane == 0) { p.glu_scale_inv[0] = a / fmax_q; p.glu_hist[nxt] = 0.f; }
      q_scale = fmax_q / a;
    }
    for (int tile = pair; tile < num_tiles && ok; tile += npairs, ++local) {
      const int acc = local & 1;
      int mt, nt; pair_tile_coords(tile, m_tiles, n_tiles, mt, nt);
      if (!mbar_wait(tfull_bar(acc), acc_phase[acc], abort_flag, p.status, ST_TIMEOUT_TMEM_FULL)) { ok = false; break; }
      acc_phase[acc] ^= 1u;
      tc_fence_after();
      const int row0 = mt * 256 + int(rank) * 128 + q * 32, row = row0 + lane;
      const int n0 = nt * BN;
      const uint32_t t_row = tmem_base + (uint32_t(q * 32) << 16) + acc * BN;
      if (GLU == 2) {
        const int F = p.glu_F;
#pragma unroll 1
        for (int c = half * (BN / 64); c < (half + 1) * (BN / 64); ++c) {
          uint32_t r[32];
          tmem_ld_32x32(t_row + c * 32, r);
          const int f = n0 + c * 32;
          const bool live = row < p.M && f < F;
          uint4 av[4], bv[4];
          if (live) {
            const uint4* pa = reinterpret_cast<const uint4*>(p.glu_ab + size_t(row) * p.glu_ld_ab + f);
            const uint4* pb = reinterpret_cast<const uint4*>(p.glu_ab + size_t(row) * p.glu_ld_ab + F + f);
#pragma unroll
            for (int v = 0; v < 4; ++v) { av[v] = pa[v]; bv[v] = pb[v]; }
          }
          tmem_wait_ld();
          uint32_t qa[8], qb[8];
          if (live) {
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              const __nv_bfloat162* a2 = reinterpret_cast<const __nv_bfloat162*>(&av[v]);
              const __nv_bfloat162* b2 = reinterpret_cast<const __nv_bfloat162*>(&bv[v]);
              float da[8], db[8];
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const float2 af = __bfloat1622float2(a2[j]), bf = __bfloat1622float2(b2[j]);
                // g as the separate product would have stored it (bf16), then the gate backward's arithmetic
                const float g0 = __bfloat162float(__float2bfloat16_rn(__uint_as_float(r[v * 8 + 2 * j]) * alpha));
                const float g1 = __bfloat162float(__float2bfloat16_rn(__uint_as_float(r[v * 8 + 2 * j + 1]) * alpha));
                const float s0 = __fdividef(1.f, 1.f + __expf(-af.x)), s1 = __fdividef(1.f, 1.f + __expf(-af.y));
                const float f0 = af.x * s0, f1 = af.y * s1;
                const float d0 = s0 + f0 * (1.f - s0), d1 = s1 + f1 * (1.f - s1);
                da[2 * j] = __bfloat162float(__float2bfloat16_rn(g0 * bf.x * d0));
                da[2 * j + 1] = __bfloat162float(__float2bfloat16_rn(g1 * bf.y * d1));
                db[2 * j] = __bfloat162float(__float2bfloat16_rn(g0 * f0));
                db[2 * j + 1] = __bfloat162float(__float2bfloat16_rn(g1 * f1));
                q_amax = fmaxf(q_amax, fmaxf(fmaxf(fabsf(da[2 * j]), fabsf(da[2 * j + 1])), fmaxf(fabsf(db[2 * j]), fabsf(db[2 * j + 1]))));
              }
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const unsigned short x0 = __nv_cvt_float2_to_fp8x2(make_float2(da[4 * h] * q_scale, da[4 * h + 1] * q_scale), __NV_SATFINITE, __NV_E5M2);
                const unsigned short x1 = __nv_cvt_float2_to_fp8x2(make_float2(da[4 * h + 2] * q_scale, da[4 * h + 3] * q_scale), __NV_SATFINITE, __NV_E5M2);
                const unsigned short y0 = __nv_cvt_float2_to_fp8x2(make_float2(db[4 * h] * q_scale, db[4 * h + 1] * q_scale), __NV_SATFINITE, __NV_E5M2);
                const unsigned short y1 = __nv_cvt_float2_to_fp8x2(make_float2(db[4 * h + 2] * q_scale, db[4 * h + 3] * q_scale), __NV_SATFINITE, __NV_E5M2);
                qa[2 * v + h] = uint32_t(x0) | (uint32_t(x1) << 16);
                qb[2 * v + h] = uint32_t(y0) | (uint32_t(y1) << 16);
              }
            }
          }
          if (f < F) {
            store_rows_u8(stage_w, make_uint4(qa[0], qa[1], qa[2], qa[3]), make_uint4(qa[4], qa[5], qa[6], qa[7]), p.glu_q, 2 * F, row0, p.M, f, lane);
            store_rows_u8(stage_w, make_uint4(qb[0], qb[1], qb[2], qb[3]), make_uint4(qb[4], qb[5], qb[6], qb[7]), p.glu_q, 2 * F, row0, p.M, F + f, lane);
          }
        }
      } else if (GLU) {
        const int f0 = nt * 128;
#pragma unroll 1
        for (int c = 2 * half; c < 2 * half + 2; ++c) {
          uint32_t ra[32], rb[32];
          tmem_ld_32x32(t_row + c * 32, ra);
          tmem_ld_32x32(t_row + 128 + c * 32, rb);
          tmem_wait_ld();
          {
            const int f = f0 + c * 32;
            uint32_t qw[8];
            uint4 oa[4], ob[4];
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              __nv_bfloat162* a2 = reinterpret_cast<__nv_bfloat162*>(&oa[v]);
              __nv_bfloat162* b2 = reinterpret_cast<__nv_bfloat162*>(&ob[v]);
              float o[8];
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                a2[j] = __floats2bfloat162_rn(__uint_as_float(ra[v * 8 + 2 * j]) * alpha, __uint_as_float(ra[v * 8 + 2 * j + 1]) * alpha);
                b2[j] = __floats2bfloat162_rn(__uint_as_float(rb[v * 8 + 2 * j]) * alpha, __uint_as_float(rb[v * 8 + 2 * j + 1]) * alpha);
                // the gate on the bf16-rounded a and b (what the backward re-reads), its result rounded to bf16 as the
                // separate gate kernel's is
                const float2 af = __bfloat1622float2(a2[j]), bf = __bfloat1622float2(b2[j]);
                o[2 * j] = __bfloat162float(__float2bfloat16_rn(af.x * __fdividef(1.f, 1.f + __expf(-af.x)) * bf.x));
                o[2 * j + 1] = __bfloat162float(__float2bfloat16_rn(af.y * __fdividef(1.f, 1.f + __expf(-af.y)) * bf.y));
                if (row < p.M) q_amax = fmaxf(q_amax, fmaxf(fabsf(o[2 * j]), fabsf(o[2 * j + 1])));
              }
              const unsigned short h0 = __nv_cvt_float2_to_fp8x2(make_float2(o[0] * q_scale, o[1] * q_scale), __NV_SATFINITE, __NV_E4M3);
              const unsigned short h1 = __nv_cvt_float2_to_fp8x2(make_float2(o[2] * q_scale, o[3] * q_scale), __NV_SATFINITE, __NV_E4M3);
              const unsigned short h2 = __nv_cvt_float2_to_fp8x2(make_float2(o[4] * q_scale, o[5] * q_scale), __NV_SATFINITE, __NV_E4M3);
              const unsigned short h3 = __nv_cvt_float2_to_fp8x2(make_float2(o[6] * q_scale, o[7] * q_scale), __NV_SATFINITE, __NV_E4M3);
              qw[2 * v] = uint32_t(h0) | (uint32_t(h1) << 16);
              qw[2 * v + 1] = uint32_t(h2) | (uint32_t(h3) << 16);
            }
            store_rows(stage_w, oa, p.C, p.ldc, row0, p.M, f, p.N, lane);
            store_rows(stage_w, ob, p.C, p.ldc, row0, p.M, p.glu_F + f, p.N, lane);
            store_rows_u8(stage_w, make_uint4(qw[0], qw[1], qw[2], qw[3]), make_uint4(qw[4], qw[5], qw[6], qw[7]), p.glu_q, p.glu_F, row0, p.M, f, lane);
          }
        }
      } else {
#pragma unroll 1
      for (int c = half * (BN / 64); c < (half + 1) * (BN / 64); ++c) {
        uint32_t r[32];
        tmem_ld_32x32(t_row + c * 32, r);
        tmem_wait_ld();
        uint4 out[4];
        finish_chunk(p, plain, row, n0 + c * 32, r, alpha, out);
        store_rows(stage_w, out, p.C, p.ldc, row0, p.M, n0 + c * 32, p.N, lane);
      }
      }
      tc_fence_before();
      __syncwarp();
      // the MMA thread of the even CTA waits for the epilogue warps of both CTAs
      if (lane == 0) mbar_arrive_cluster(map_to_cta(tempty_bar(acc), 0));
    }
    if (GLU) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) q_amax = fmaxf(q_amax, __shfl_xor_sync(0xffffffffu, q_amax, o));
      if (lane == 0 && q_amax > 0.f) atomicMax(reinterpret_cast<unsigned int*>(p.glu_hist + p.glu_cur), __float_as_uint(q_amax));
    }
  }
  tc_fence_before();
  __syncthreads();
  // neither CTA may free tensor memory or leave while its partner can still signal it or read its shared memory
  cluster_arrive();
  cluster_wait();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
}

// ------------------------------------------------------------------------------------ host side

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) != cudaSuccess ||
        qres != cudaDriverEntryPointSuccess) {
      return nullptr;
    }
    fn = reinterpret_cast<EncodeTiledFn>(ptr);
  }
  return fn;
}

static int g_last_encode_result = 0;

// 2-D bf16 tensor map: `inner` contiguous elements per row, `outer` rows, row stride `ld` elements.
int make_tmap_2d_bf16(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer, uint64_t ld,
                      uint32_t box_inner, uint32_t box_outer) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return -1;
  cuuint64_t dims[2] = {inner, outer};
  cuuint64_t strides[1] = {ld * 2};
  cuuint32_t box[2] = {box_inner, box_outer};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) g_last_encode_result = (int)r;
  return r == CUDA_SUCCESS ? 0 : -2;
}

// 2-D one-byte tensor map (fp8 operands)
int make_tmap_2d_u8(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer, uint64_t ld, uint32_t box_inner,
                    uint32_t box_outer) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return -1;
  cuuint64_t dims[2] = {inner, outer};
  cuuint64_t strides[1] = {ld};
  cuuint32_t box[2] = {box_inner, box_outer};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) g_last_encode_result = (int)r;
  return r == CUDA_SUCCESS ? 0 : -2;
}

static int g_num_sms = 0;
static int g_last_detail = 0;   // (which operand << 16) | CUresult of the last failed tensor-map encode

static int g_pair_mode = 3;      // CTA-pair kernel 0: never, 1: for one-byte operands, 2: for every GEMM, 3: where pick_tile chooses it

// Tile of a GEMM on `sms` SMs: 0 = the CTA-pair kernel's 256 x 256, or the width of a single-CTA tile 128 x {128, 64}, for
// outputs with too few 256 x 256 tiles to fill the chip.  Compared are waves times cycles of a tile per 128-byte k-block: an SM
// pair spends 512 on its 256 x 256 tile; a single-CTA tile is bound by shared memory, which takes both operands in and reads
// them once (32 KB a k-block: 256 cycles and their share of latency, 320; 24 KB: 260).  A narrower tile has to win by an
// eighth, because it reads its operands more often.  Back to back, us, pair -> chosen: [999 x 1024] K = 5632 32 -> 16 and
// K = 2816 20 -> 11 (64 wide), [512 x 4096] K = 8192 48 -> 28 (128 wide), weight gradients of a 256-wide model 18 -> 7;
// [999 x 5632] K = 1024 keeps the pair (17 with either).  `b_box128`: B comes in boxes of 128 columns (one-byte
// MN-major operand), 64 is not possible.
static int pick_tile(int M, int N, int sms, bool b_box128) {
  const long long m1 = (M + 127) / 128, m2 = (M + 255) / 256;
  auto waves = [](long long tiles, long long slots) { return (tiles + slots - 1) / slots; };
  const long long pair = waves(m2 * ((N + 255) / 256), sms / 2) * 512;
  const long long w128 = waves(m1 * ((N + 127) / 128), sms) * 320, w64 = waves(m1 * ((N + 63) / 64), sms) * 260;
  if (8 * (w64 < w128 && !b_box128 ? w64 : w128) > 7 * pair) return 0;
  return 8 * w64 <= 7 * w128 && !b_box128 ? 64 : 128;
}

// The kernel that a GEMM takes in the present mode: 0 = the CTA pair, else the width of a single-CTA tile.
static int chosen_tile(int M, int N, int sms, bool one_byte, bool b_mn, int max_ctas) {
  if (g_pair_mode < (one_byte ? 1 : 2) || max_ctas > 0) return BN;
  return g_pair_mode == 3 ? pick_tile(M, N, sms, one_byte && b_mn) : 0;
}

// A launch in clusters of `cluster` CTAs, as a programmatic dependent of the kernel before it (see the kernels' wait_for_previous).
static int launch_behind(void (*kern)(const CUtensorMap, const CUtensorMap, GemmParams), int grid, int cluster, int smem, cudaStream_t stream,
                         const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmParams& p) {
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(NUM_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  if (cudaLaunchKernelEx(&cfg, kern, tmA, tmB, p) == cudaSuccess) return 0;
  (void)cudaGetLastError();              // reported here, as in launch_chained
  return -6;
}

// Launch the single-CTA kernel with tile width BNT.
template <int EB, int BNT>
static int launch_single(const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmParams& p, int a_mn, int b_mn, int max_ctas,
                         cudaStream_t stream) {
  const int tiles = ((p.M + BM - 1) / BM) * ((p.N + BNT - 1) / BNT);
  int grid = tiles < g_num_sms ? tiles : g_num_sms;
  if (max_ctas > 0 && grid > max_ctas) grid = max_ctas;
  void (*kern)(const CUtensorMap, const CUtensorMap, GemmParams);
  constexpr int BN_MN = EB == 1 && BNT < 128 ? 128 : BNT;          // never chosen (see pick_tile), but instantiated
  if (!a_mn && !b_mn) kern = gemm_bf16_kernel<0, 0, EB, BNT>;
  else if (!a_mn && b_mn) kern = gemm_bf16_kernel<0, 1, EB, BN_MN>;
  else if (a_mn && b_mn) kern = gemm_bf16_kernel<1, 1, EB, BN_MN>;
  else kern = gemm_bf16_kernel<1, 0, EB, BNT>;
  static bool attr_set[4] = {false, false, false, false};
  const int idx = a_mn * 2 + b_mn;
  if (!attr_set[idx]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) != cudaSuccess) return -5;
    attr_set[idx] = true;
  }
  return launch_behind(kern, grid, 1, SMEM_BYTES, stream, tmA, tmB, p);
}

// Launch the CTA-pair kernel (cluster of 2) on tensor maps whose boxes are 128 rows (K-major) / 128-byte MN boxes.
template <int EB>
static int launch_pair(const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmParams& p, int a_mn, int b_mn,
                       cudaStream_t stream) {
  void (*kern)(const CUtensorMap, const CUtensorMap, GemmParams);
  if (!a_mn && !b_mn) kern = gemm_pair_kernel<0, 0, EB>;
  else if (!a_mn && b_mn) kern = gemm_pair_kernel<0, 1, EB>;
  else if (a_mn && b_mn) kern = gemm_pair_kernel<1, 1, EB>;
  else kern = gemm_pair_kernel<1, 0, EB>;
  static bool attr_set[4] = {false, false, false, false};
  const int idx = a_mn * 2 + b_mn;
  if (!attr_set[idx]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, P_SMEM_BYTES) != cudaSuccess) return -5;
    attr_set[idx] = true;
  }
  const int tiles = ((p.M + 255) / 256) * ((p.N + BN - 1) / BN);
  int pairs = g_num_sms / 2;
  if (tiles < pairs) pairs = tiles;
  return launch_behind(kern, 2 * pairs, 2, P_SMEM_BYTES, stream, tmA, tmB, p);
}

}  // namespace sb

extern "C" int sb_gemm_last_error_detail() { return sb::g_last_detail; }
// 0: single-CTA tiles only; 1: CTA pairs (cta_group::2) for fp8 operands; 2: CTA pairs for bf16 operands too; 3 (default): by size
extern "C" int sb_gemm_set_pair_mode(int mode) { sb::g_pair_mode = mode; return 0; }
// What a GEMM of this size runs on a chip of `sms` SMs in the present mode: 0 = CTA pairs, else the width of a 128-row tile.
extern "C" int sb_gemm_tile(int M, int N, int one_byte, int b_mn, int max_ctas, int sms) {
  return sb::chosen_tile(M, N, sms, one_byte != 0, b_mn != 0, max_ctas);
}

// C = A * B^T (+bias) (+residual) (+C).  a_mn = 0: A is [M, K] row-major with leading dim lda; a_mn = 1: A is stored
// transposed as [K, M] with leading dim lda.  b_mn likewise for B ([N, K] or [K, N]).  All leading dims and
// base addresses must be 16-byte aligned; N a multiple of 8, and K too unless both operands are MN-major.  Returns 0 on a successful launch.
extern "C" int sb_gemm_bf16(const void* A, const void* B, void* C, const void* bias, const void* residual, int M, int N,
                            int K, int lda, int ldb, int ldc, int ldr, int a_mn, int b_mn, int beta, unsigned int* status,
                            int max_ctas, cudaStream_t stream) {
  using namespace sb;
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  // The tensor-map encoder is a driver call and needs a current context; a thread that has made no runtime call
  // yet (e.g. an autograd worker on its first launch) has none until the runtime binds the primary context.
  static thread_local bool ctx_bound = false;
  if (!ctx_bound) { cudaFree(0); ctx_bound = true; }
  // K only has to be a multiple of 8 where it is the contiguous dim of an operand (a K-major one)
  if ((N % 8) || (lda % 8) || (ldb % 8) || (ldc % 8) || ((!a_mn || !b_mn) && (K % 8))) return -3;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C)) & 15) return -4;
  if (!g_num_sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
  }
  const int width = chosen_tile(M, N, g_num_sms, false, b_mn != 0, max_ctas);
  CUtensorMap tmA, tmB;
  int rc;
  if (!a_mn) rc = make_tmap_2d_bf16(&tmA, A, K, M, lda, BK, BM);
  else       rc = make_tmap_2d_bf16(&tmA, A, M, K, lda, 64, BK);
  if (rc) { g_last_detail = (1 << 16) | (g_last_encode_result & 0xffff); return rc; }
  if (!b_mn) rc = make_tmap_2d_bf16(&tmB, B, K, N, ldb, BK, width ? width : 128);      // a pair: 128 B rows per CTA
  else       rc = make_tmap_2d_bf16(&tmB, B, N, K, ldb, 64, BK);
  if (rc) { g_last_detail = (2 << 16) | (g_last_encode_result & 0xffff); return rc; }
  if (residual && ((ldr % 8) || (reinterpret_cast<uintptr_t>(residual) & 15))) return -4;
  GemmParams p{reinterpret_cast<__nv_bfloat16*>(C), reinterpret_cast<const __nv_bfloat16*>(bias),
               reinterpret_cast<const __nv_bfloat16*>(residual), M, N, K, ldc, ldr, beta, status, nullptr, nullptr, 0, 0};
  if (width == 0) return launch_pair<2>(tmA, tmB, p, a_mn, b_mn, stream);
  if (width == 64) return launch_single<2, 64>(tmA, tmB, p, a_mn, b_mn, 0, stream);
  if (width == 128) return launch_single<2, 128>(tmA, tmB, p, a_mn, b_mn, 0, stream);
  return launch_single<2, 256>(tmA, tmB, p, a_mn, b_mn, max_ctas, stream);
}

// Gate projection of the gated MLP with the gate in the epilogue (CTA-pair kernel, GLU mode): AB [M, 2 F] bf16 =
// alpha * A [M, K] * W12 [2 F, K]^T with e4m3 operands, and Q [M, F] = e4m3(silu(a) * b) under delayed scaling (ring
// protocol of sb_quantize_fp8_delayed: `hist` of `slots` floats, slot `cur` collects this call's amax, `scale_inv`
// receives the de-quantisation factor).  F % 128 == 0, K % 16 == 0.
extern "C" int sb_gemm_fp8_glu(const void* A, const void* W12, void* AB, void* Q, const float* alpha, const float* alpha2, int M,
                               int F, int K, int lda, int ldb, int ldab, float* hist, int slots, int cur, float* scale_inv,
                               unsigned int* status, cudaStream_t stream) {
  using namespace sb;
  if (M <= 0 || F <= 0 || K <= 0) return 0;
  static thread_local bool ctx_bound = false;
  if (!ctx_bound) { cudaFree(0); ctx_bound = true; }
  if ((F % 128) || (K % 16) || (lda % 16) || (ldb % 16) || (ldab % 8) || ldab < 2 * F || slots < 3 || cur < 0 || cur >= slots) return -3;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W12) | reinterpret_cast<uintptr_t>(AB) |
       reinterpret_cast<uintptr_t>(Q)) & 15) return -4;
  CUtensorMap tmA, tmB;
  int rc;
  if ((rc = make_tmap_2d_u8(&tmA, A, K, M, lda, 128, BM))) return rc;
  if ((rc = make_tmap_2d_u8(&tmB, W12, K, 2 * F, ldb, 128, 128))) return rc;
  if (!g_num_sms) { int dev = 0; cudaGetDevice(&dev); cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev); }
  GemmParams p{reinterpret_cast<__nv_bfloat16*>(AB), nullptr, nullptr, M, 2 * F, K, ldab, 0, 0, status, alpha, alpha2, 0, 0,
               reinterpret_cast<uint8_t*>(Q), F, hist, slots, cur, scale_inv};
  auto kern = gemm_pair_kernel<0, 0, 1, 1>;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, P_SMEM_BYTES) != cudaSuccess) return -5;
    attr_set = true;
  }
  const int tiles = ((M + 255) / 256) * (F / 128);
  int pairs = g_num_sms / 2;
  if (tiles < pairs) pairs = tiles;
  return launch_behind(kern, 2 * pairs, 2, P_SMEM_BYTES, stream, tmA, tmB, p);
}

// Input-gradient product of the gated MLP's output projection with the gate backward in the epilogue (GLU = 2):
// g [M, F] = alpha * G [M, D] (e5m2) * W3 [D, F] (e4m3, rows of F contiguous) is not stored; with [a | b] = AB [M, 2 F]
// the epilogue writes Q [M, 2 F] = e5m2(g * b * silu'(a) | g * silu(a)) under delayed scaling.  F % 16 == 0, D % 16 == 0.
extern "C" int sb_gemm_fp8_glu_bwd(const void* G, const void* W3, const void* AB, void* Q, const float* alpha, const float* alpha2,
                                   int M, int F, int D, int ldg, int ldw, int ldab, float* hist, int slots, int cur,
                                   float* scale_inv, unsigned int* status, cudaStream_t stream) {
  using namespace sb;
  if (M <= 0 || F <= 0 || D <= 0) return 0;
  static thread_local bool ctx_bound = false;
  if (!ctx_bound) { cudaFree(0); ctx_bound = true; }
  if ((F % 32) || (D % 16) || (ldg % 16) || (ldw % 16) || (ldab % 8) || ldab < 2 * F || slots < 3 || cur < 0 || cur >= slots) return -3;
  if ((reinterpret_cast<uintptr_t>(G) | reinterpret_cast<uintptr_t>(W3) | reinterpret_cast<uintptr_t>(AB) |
       reinterpret_cast<uintptr_t>(Q)) & 15) return -4;
  CUtensorMap tmA, tmB;
  int rc;
  if ((rc = make_tmap_2d_u8(&tmA, G, D, M, ldg, 128, BM))) return rc;
  if ((rc = make_tmap_2d_u8(&tmB, W3, F, D, ldw, 128, 128))) return rc;          // MN-major operand: boxes of 128 x 128
  if (!g_num_sms) { int dev = 0; cudaGetDevice(&dev); cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev); }
  GemmParams p{nullptr, nullptr, nullptr, M, F, D, 0, 0, 0, status, alpha, alpha2, 1, 0,
               reinterpret_cast<uint8_t*>(Q), F, hist, slots, cur, scale_inv, reinterpret_cast<const __nv_bfloat16*>(AB), ldab};
  auto kern = gemm_pair_kernel<0, 1, 1, 2>;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, P_SMEM_BYTES) != cudaSuccess) return -5;
    attr_set = true;
  }
  const int tiles = ((M + 255) / 256) * ((F + BN - 1) / BN);
  int pairs = g_num_sms / 2;
  if (tiles < pairs) pairs = tiles;
  return launch_behind(kern, 2 * pairs, 2, P_SMEM_BYTES, stream, tmA, tmB, p);
}

// fp8 GEMM: C[M,N] (bf16) = alpha * A * B^T (+bias) (+residual) (+C) with one-byte operands (e4m3 = 0 / e5m2 = 1) and
// fp32 accumulation; `alpha` and `alpha2` are device scalars (the operands' de-quantisation factors; either may be
// null) whose product scales the accumulator.  Leading dims and contiguous extents must be multiples of 16 elements.
extern "C" int sb_gemm_fp8(const void* A, const void* B, void* C, const void* bias, const void* residual, const float* alpha,
                           const float* alpha2, int M, int N, int K, int lda, int ldb, int ldc, int ldr, int a_mn, int b_mn, int a_fmt, int b_fmt,
                           int beta, unsigned int* status, cudaStream_t stream) {
  using namespace sb;
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  static thread_local bool ctx_bound = false;
  if (!ctx_bound) { cudaFree(0); ctx_bound = true; }
  if ((N % 8) || (lda % 16) || (ldb % 16) || (ldc % 8) || ((!a_mn || !b_mn) && (K % 16))) return -3;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C)) & 15) return -4;
  if (!g_num_sms) { int dev = 0; cudaGetDevice(&dev); cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev); }
  const int width = chosen_tile(M, N, g_num_sms, true, b_mn != 0, 0);
  CUtensorMap tmA, tmB;
  int rc;
  if (!a_mn) rc = make_tmap_2d_u8(&tmA, A, K, M, lda, 128, BM);
  else       rc = make_tmap_2d_u8(&tmA, A, M, K, lda, 128, 128);
  if (rc) { g_last_detail = (1 << 16) | (g_last_encode_result & 0xffff); return rc; }
  if (!b_mn) rc = make_tmap_2d_u8(&tmB, B, K, N, ldb, 128, width ? width : 128);       // a pair: 128 B rows per CTA
  else       rc = make_tmap_2d_u8(&tmB, B, N, K, ldb, 128, 128);
  if (rc) { g_last_detail = (2 << 16) | (g_last_encode_result & 0xffff); return rc; }
  if (residual && ((ldr % 8) || (reinterpret_cast<uintptr_t>(residual) & 15))) return -4;
  GemmParams p{reinterpret_cast<__nv_bfloat16*>(C), reinterpret_cast<const __nv_bfloat16*>(bias),
               reinterpret_cast<const __nv_bfloat16*>(residual), M, N, K, ldc, ldr, beta, status, alpha, alpha2, a_fmt, b_fmt};
  if (width == 0) return launch_pair<1>(tmA, tmB, p, a_mn, b_mn, stream);
  if (width == 64) return launch_single<1, 64>(tmA, tmB, p, a_mn, b_mn, 0, stream);
  if (width == 128) return launch_single<1, 128>(tmA, tmB, p, a_mn, b_mn, 0, stream);
  return launch_single<1, 256>(tmA, tmB, p, a_mn, b_mn, 0, stream);
}
