// Hyena-MR on tensor cores: the causal FIR of <= 128 taps shared by the 16+ channels of a group is a product
// with a banded Toeplitz matrix, so a [16 time x 16 channel] output block is
//     Y[i0] = sum_{d = 0..8} A_d * U[i0 - 16 d],      A_d[r][c] = h[16 d + r - c]   (zero outside 0..K-1)
// i.e. nine m16n8k16 bf16 MMAs per 8 channels with the A fragments (functions of the filter only) held in
// registers for the whole kernel and the B fragments read from a shared-memory image of u = x2*v with
// ldmatrix.  (The group width of 16 channels is too narrow for a tcgen05 tile — its minimum useful N at M = 128
// would leave the Toeplitz operand, 64 KB per group, as the only thing in shared memory — so this operator uses
// the warp-level MMA path; the wide GEMMs and attention use tcgen05.)  fp32 accumulation; u and h are rounded to
// bf16 for the product, like every other tensor-core operand in the model.
//
//   mr_tc_fwd : z = x1 * (h*u + bias*u)
//   mr_tc_bwd : dfeat = (dz*y, du*v, du*x2), du = h (*) g + bias*g (anticausal), g = dz*x1;
//               dh[s] += sum g[t] u[t-s]  (as P_d = G_blk^T-contracted-over-channels MMAs), dbias += sum g*u;
//               y recomputed instead of saved
// Both walk a segment of 32-row tiles of 64 channels.
//
// Calls without halo rows take mr_conv_umma.cu, but for forwards with short filters (autograd_native.cpp: short_filter).
// Measured at B = 1, L = 8192, D = 4096, K = 128 on a B200 (us; in brackets the kernels these replace, which staged 128-row
// tiles with their halo, or rebuilt 72 fragment registers from global memory for every 64-row tile): forward 71 (108),
// backward 256 (475), forward and backward with their host side 589 -> 333.  Copying the data takes 40 and 71 us.  What bounds
// them now is issue slots and latency at four (two) blocks per SM: of the first streaming version (106 and 411 us) most of
// the difference was address arithmetic of the copies, unpacking to fp32 for the gates, and spilled fragments.
// Rows before the sequence start come from `halo` [B, K-1, 3D] (context-parallel shards) or are zero; the
// backward kernel also produces the halo rows' gradient.  Requires dg % 16 == 0 (a warp's 16-channel slab shares
// one filter); other group widths use the CUDA-core kernels in mr_conv.cu.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "entries.h"
#include "halo_src.cuh"

#include "device_info.h"

namespace sb {
typedef __nv_bfloat16 bf16;

constexpr int TC_CH = 64;                 // channels per tile (4 slabs of 16)
constexpr int TC_LD = 72;                 // padded row of a u / g ring (elements) -> 144 B, conflict-free ldmatrix
constexpr int TC_TT = 32;                 // rows per tile step
constexpr int TC_HALO = 128;              // rows of u behind (g ahead of) the tile
constexpr int TC_RING = TC_HALO + TC_TT;  // 160 rows: ten 16-row blocks, a block never wraps
constexpr int RAW_LD = 200;               // padded row of a staged feature tile (elements): 400 B, so that the 8 rows x 4
                                          // channel pairs of an MMA fragment fall into 32 different banks
constexpr int FWD_THREADS = 128;          // one warp per 16-channel slab
constexpr int BWD_THREADS = 256;          // two warps per slab
constexpr int ND = 9;                     // Toeplitz block diagonals d = 0..8
constexpr int NF = 2 * ND + 1;            // distinct fragment registers of all diagonals (see toeplitz_frags)

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float2 unpack2(uint32_t u) {
  return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&u));
}
__device__ __forceinline__ float tap(const float* h, int K, int s) { return (s >= 0 && s < K) ? h[s] : 0.f; }

// A fragments of the Toeplitz block diagonals for this thread.  CAUSAL: A_d[r][c] = h[16d + r - c];  otherwise
// A_d[r][c] = h[16d + c - r] (the anticausal product of the backward pass).  Register q of diagonal d holds the taps at
// 16 d + base + {0, 8, -8, 0}[q] (signs swapped when anticausal): the off-diagonal 8 x 8 quarter of one diagonal is the
// next one's, so the nine diagonals share 19 registers and stay resident over a whole segment.
template <bool CAUSAL>
__device__ __forceinline__ void toeplitz_frags(uint32_t (&f)[NF], const float* h, int K, int lane) {
  const int g = lane >> 2, t = lane & 3, base = CAUSAL ? g - 2 * t : 2 * t - g;
#pragma unroll
  for (int m = 0; m < NF; ++m) {
    const int s = 8 * (m - 1) + base;
    f[m] = pack2(tap(h, K, s), tap(h, K, CAUSAL ? s - 1 : s + 1));
  }
}
template <bool CAUSAL>
__device__ __forceinline__ void toeplitz_mma(float (&d)[4], const uint32_t (&f)[NF], int diag, uint32_t b0, uint32_t b1) {
  const uint32_t a[4] = {f[2 * diag + 1], f[2 * diag + (CAUSAL ? 2 : 0)], f[2 * diag + (CAUSAL ? 0 : 2)], f[2 * diag + 1]};
  mma16816(d, a, b0, b1);
}

struct MrArgs {
  const bf16* feat; HaloSrc halo; const float* h; const float* bias;
  int L, D, K, dg;
  // context-parallel backward: rows [L, L + K - 1) of x1 and dz come from the next chunk's staged head (peer memory)
  int ahead_mode; HaloSrc ahead_f, ahead_g;
};

// Feature row t of batch row b: the sequence, the rows before it, or null (zeros).
__device__ __forceinline__ const bf16* mr_row(const MrArgs& a, int b, int t) {
  if (t >= 0) return t < a.L ? a.feat + ((size_t)b * a.L + t) * 3 * a.D : nullptr;
  return t >= -(a.K - 1) ? halo_row(a.halo, b, t + a.K - 1, a.K - 1, (size_t)3 * a.D) : nullptr;
}
// Three words of two channels' interleaved triples (x1 x2 | v x1 | x2 v) -> packed pairs.  bf16 products of bf16 values round
// once, exactly as the fp32 product rounded to bf16 does.
__device__ __forceinline__ uint32_t tri_x1(uint32_t w0, uint32_t w1) { return __byte_perm(w0, w1, 0x7610); }
__device__ __forceinline__ uint32_t tri_x2(uint32_t w0, uint32_t w2) { return __byte_perm(w0, w2, 0x5432); }
__device__ __forceinline__ uint32_t tri_v(uint32_t w1, uint32_t w2) { return __byte_perm(w1, w2, 0x7610); }
__device__ __forceinline__ uint32_t mul_bf2(uint32_t a, uint32_t b) {
  __nv_bfloat162 r = __hmul2(*reinterpret_cast<__nv_bfloat162*>(&a), *reinterpret_cast<__nv_bfloat162*>(&b));
  return *reinterpret_cast<uint32_t*>(&r);
}
// u = x2 v of eight channels from their 48 staged bytes
__device__ __forceinline__ uint4 gate_u(const uint4* p) {
  const uint4 a = p[0], b = p[1], c = p[2];
  return make_uint4(mul_bf2(tri_x2(a.x, a.z), tri_v(a.y, a.z)), mul_bf2(tri_x2(a.w, b.y), tri_v(b.x, b.y)),
                    mul_bf2(tri_x2(b.z, c.x), tri_v(b.w, c.x)), mul_bf2(tri_x2(c.y, c.w), tri_v(c.z, c.w)));
}
// g = dz x1 of eight channels
__device__ __forceinline__ uint4 gate_g(const uint4* p, const uint4 z) {
  const uint4 a = p[0], b = p[1], c = p[2];
  return make_uint4(mul_bf2(tri_x1(a.x, a.y), z.x), mul_bf2(tri_x1(a.w, b.x), z.y), mul_bf2(tri_x1(b.z, b.w), z.z),
                    mul_bf2(tri_x1(c.y, c.z), z.w));
}
__device__ __forceinline__ void mr_cp_async16(void* dst, const void* src, int nbytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(nbytes) : "memory");
}
__device__ __forceinline__ void mr_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void mr_cp_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// Issue the asynchronous copies of feature rows t .. t + TC_TT - 1, channels [c_base, c_base + 64), into dst[TC_TT][RAW_LD]:
// 96 threads, four rows of 24 chunks side by side.  Tiles inside the sequence walk one pointer.
__device__ __forceinline__ void mr_stage_feat(bf16* dst, const MrArgs& a, int b, int t, int c_base, int tid) {
  const int r0 = tid / 24, c = tid - r0 * 24;
  if (r0 >= 4) return;
  const bool live = 3 * c_base + c * 8 < 3 * a.D;
  bf16* d = dst + r0 * RAW_LD + c * 8;
  if (t >= 0 && t + TC_TT <= a.L) {
    const size_t ld = (size_t)3 * a.D;
    const bf16* p = live ? a.feat + ((size_t)b * a.L + t + r0) * ld + 3 * c_base + c * 8 : a.feat;
    const size_t step = live ? 4 * ld : 0;
    const int nb = live ? 16 : 0;
#pragma unroll
    for (int j = 0; j < TC_TT / 4; ++j, p += step, d += 4 * RAW_LD) mr_cp_async16(d, p, nb);
  } else {
    for (int j = 0; j < TC_TT / 4; ++j, d += 4 * RAW_LD) {
      const bf16* row = mr_row(a, b, t + r0 + 4 * j);
      const bool ok = row && live;
      mr_cp_async16(d, ok ? row + 3 * c_base + c * 8 : a.feat, ok ? 16 : 0);
    }
  }
}

// ------------------------------------------------------------------------------------ forward
// A block owns 64 channels and a segment of consecutive 32-row tiles.  The tile's features land in shared memory by
// asynchronous copies one step ahead; u = x2*v goes into a bf16 ring of 160 rows (128 behind the tile), the Toeplitz MMAs
// read it from there, and z = x1 (y + bias u) is formed in fp32 from the accumulators and the staged features.  Every
// feature row is read once per segment plus the 128 rows behind its start.  48 KB of shared memory and 4 warps: four
// blocks per SM.
constexpr int FWD_SMEM = (2 * TC_TT * RAW_LD + TC_RING * TC_LD) * 2;

template <bool FULL>       // FULL: all nine diagonals (K > 112), so that the loads and MMAs of the diagonals interleave
__global__ void __launch_bounds__(FWD_THREADS, 4)
mr_tc_fwd_kernel(MrArgs a, bf16* __restrict__ z, int n_tiles, int tiles_per_seg) {
  extern __shared__ __align__(16) uint8_t smraw[];
  bf16* sRaw = reinterpret_cast<bf16*>(smraw);                 // [2][TT][RAW_LD]
  bf16* sU = sRaw + 2 * TC_TT * RAW_LD;                        // [RING][LD]
  const int tid = threadIdx.x, lane = tid & 31, slab = tid >> 5;
  const int c_base = blockIdx.x * TC_CH, b = blockIdx.z;
  const int k0 = blockIdx.y * tiles_per_seg, k1 = min(k0 + tiles_per_seg, n_tiles);
  if (k0 >= k1) return;
  const int seg_t0 = k0 * TC_TT;
  const int ch0 = c_base + slab * 16;
  const int nd = min(ND, (a.K - 1) / 16 + 2);
  const int g = lane >> 2, tq = lane & 3;
  const int lm_row = (lane & 7) + ((lane >> 3) & 1) * 8, lm_col = slab * 16 + (lane >> 4) * 8;
  // The 128 rows behind the segment run through the same pipeline as tiles that produce no output; diagonals beyond nd are
  // never read, so filters shorter than 128 taps start closer to the segment.
  const int lead = min(TC_HALO / TC_TT, (16 * (nd - 1) + TC_TT - 1) / TC_TT);
  mr_stage_feat(sRaw, a, b, seg_t0 - lead * TC_TT, c_base, tid);
  mr_cp_commit();
  uint32_t F[NF];
  toeplitz_frags<true>(F, a.h + (size_t)(min(ch0, a.D - 1) / a.dg) * a.K, a.K, lane);
  float bias[2][2];
#pragma unroll
  for (int nt = 0; nt < 2; ++nt)
#pragma unroll
    for (int e = 0; e < 2; ++e) { const int c = ch0 + nt * 8 + 2 * tq + e; bias[nt][e] = c < a.D ? a.bias[c] : 0.f; }
  int rel = (TC_RING - lead * TC_TT) % TC_RING;                // ring row of the step's first row
  for (int k = k0 - lead; k < k1; ++k) {
    bf16* raw = sRaw + ((k - k0 + lead) & 1) * TC_TT * RAW_LD;
    mr_cp_wait_all();
    __syncthreads();                                           // tile k is here; all reads of tile k - 1 (raw, ring) are done
    if (k + 1 < k1) mr_stage_feat(sRaw + ((k - k0 + lead + 1) & 1) * TC_TT * RAW_LD, a, b, (k + 1) * TC_TT, c_base, tid);
    mr_cp_commit();
#pragma unroll
    for (int j = 0; j < TC_TT * 8 / FWD_THREADS; ++j) {
      const int i = tid + j * FWD_THREADS, r = i >> 3, cv = i & 7;
      *reinterpret_cast<uint4*>(sU + (rel + r) * TC_LD + cv * 8) = gate_u(reinterpret_cast<const uint4*>(raw + r * RAW_LD + cv * 24));
    }
    __syncthreads();
    if (k >= k0) {
      float acc[2][2][4];
#pragma unroll
      for (int i = 0; i < 16; ++i) acc[i >> 3][(i >> 2) & 1][i & 3] = 0.f;
      // input block e (rows 16 e behind the tile's second output block) feeds diagonal e of block 1 and e - 1 of block 0
#pragma unroll
      for (int e = 0; e <= ND; ++e) {
        if (FULL || e <= nd) {
          int row = rel + 16 - 16 * e;
          if (row < 0) row += TC_RING;
          uint32_t bf[4];
          ldsm_x4_t(bf, smem_addr(sU + (row + lm_row) * TC_LD + lm_col));
          if (e < ND && (FULL || e < nd)) {
            toeplitz_mma<true>(acc[1][0], F, e < ND ? e : 0, bf[0], bf[1]);
            toeplitz_mma<true>(acc[1][1], F, e < ND ? e : 0, bf[2], bf[3]);
          }
          if (e > 0) {
            toeplitz_mma<true>(acc[0][0], F, e > 0 ? e - 1 : 0, bf[0], bf[1]);
            toeplitz_mma<true>(acc[0][1], F, e > 0 ? e - 1 : 0, bf[2], bf[3]);
          }
        }
      }
      // z = x1 (y + bias u) in fp32 at the fragment positions; the four lanes of a row store 16 consecutive bytes
#pragma unroll
      for (int blk = 0; blk < 2; ++blk)
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {
            const int row = blk * 16 + g + hh * 8, c = slab * 16 + nt * 8 + 2 * tq;
            uint32_t* w = reinterpret_cast<uint32_t*>(raw + row * RAW_LD + 3 * c);
            const float2 p0 = unpack2(w[0]), p1 = unpack2(w[1]), p2 = unpack2(w[2]);      // (x1 x2) (v x1) (x2 v)
            const float z0 = p0.x * (acc[blk][nt][hh * 2] + bias[nt][0] * (p0.y * p1.x));
            const float z1 = p1.y * (acc[blk][nt][hh * 2 + 1] + bias[nt][1] * (p2.x * p2.y));
            const int t = k * TC_TT + row, cg = c_base + c;
            if (t < a.L && cg < a.D) *reinterpret_cast<uint32_t*>(z + ((size_t)b * a.L + t) * a.D + cg) = pack2(z0, z1);
          }
    }
    rel += TC_TT;
    if (rel >= TC_RING) rel -= TC_RING;
  }
}

// ------------------------------------------------------------------------------------ backward
// A block owns 64 channels and a segment of consecutive 32-row tiles.  Two rings of 160 rows hold bf16 u = x2*v (the tile
// and 128 rows behind it) and g = dz*x1 (the tile and 128 rows ahead).  A step stages two raw tiles by asynchronous copies
// that are issued one step ahead: the front rows (t0 + 128 ..), from which g is formed, and the tile itself, from which u is
// formed and which stays until the end of the step: y and du come out of the accumulators in fp32, are combined with the
// tile's x2, v and dz at their fragment positions and replace the features in place, and the tile leaves as 16-byte
// chunks.  The filter-gradient accumulators stay in registers over the segment (one flush per block).  Every input row is
// read twice (the second time from L2).
constexpr int RAWG_LD = 72;                                    // padded row of a staged dz tile
constexpr int RAW_TILE = TC_TT * (RAW_LD + RAWG_LD);           // elements of a staged (features, dz) tile
constexpr int BWD_SMEM = (3 * RAW_TILE + 2 * TC_RING * TC_LD) * 2 + (4 * 128 + TC_CH + 4 * NF * 32) * 4;

// dz row t, or null: the sequence, or (context-parallel look-ahead) the next chunk's first rows
__device__ __forceinline__ void mr_rows_fg(const MrArgs& a, const bf16* dz, int b, int t, const bf16*& fr, const bf16*& gr) {
  gr = nullptr;
  if (t >= a.L) {
    fr = nullptr;
    if (a.ahead_mode && t < a.L + a.K - 1) {
      fr = halo_row(a.ahead_f, b, t - a.L, a.K - 1, (size_t)3 * a.D);
      gr = halo_row(a.ahead_g, b, t - a.L, a.K - 1, (size_t)a.D);
    }
    return;
  }
  fr = mr_row(a, b, t);
  if (t >= 0) gr = dz + ((size_t)b * a.L + t) * a.D;
}
// Features and dz of rows t .. t + TC_TT - 1: threads 0-191 copy features (eight rows of 24 chunks side by side), the other 64
// dz (eight rows of 8 chunks).
__device__ __forceinline__ void mr_stage_fg(bf16* dst, const MrArgs& a, const bf16* dz, int b, int t, int c_base, int tid) {
  const bool fe = tid < 192;
  const int i = fe ? tid : tid - 192, per = fe ? 24 : 8, r0 = fe ? i / 24 : i >> 3, c = i - r0 * per;
  const size_t ld = fe ? (size_t)3 * a.D : (size_t)a.D;
  const int col = (fe ? 3 * c_base : c_base) + c * 8, dld = fe ? RAW_LD : RAWG_LD;
  const bool live = col < (int)ld;
  bf16* d = dst + (fe ? 0 : TC_TT * RAW_LD) + r0 * dld + c * 8;
  if (t >= 0 && t + TC_TT <= a.L) {
    const bf16* p = live ? (fe ? a.feat : dz) + ((size_t)b * a.L + t + r0) * ld + col : a.feat;
    const size_t step = live ? 8 * ld : 0;
    const int nb = live ? 16 : 0;
#pragma unroll
    for (int j = 0; j < TC_TT / 8; ++j, p += step, d += 8 * dld) mr_cp_async16(d, p, nb);
  } else {
    for (int j = 0; j < TC_TT / 8; ++j, d += 8 * dld) {
      const bf16 *fr, *gr;
      mr_rows_fg(a, dz, b, t + r0 + 8 * j, fr, gr);
      const bf16* row = fe ? fr : gr;
      const bool ok = row && live;
      mr_cp_async16(d, ok ? row + col : a.feat, ok ? 16 : 0);
    }
  }
}

template <bool FULL>
__global__ void __launch_bounds__(BWD_THREADS, 2)
mr_tc_bwd_kernel(MrArgs a, const bf16* __restrict__ dz, bf16* __restrict__ dfeat, bf16* __restrict__ dhalo,
                 float* __restrict__ dh, float* __restrict__ dbias, int n_halo_tiles, int n_tiles, int tiles_per_seg) {
  extern __shared__ __align__(16) uint8_t smraw[];
  bf16* sT = reinterpret_cast<bf16*>(smraw);                   // the tile, double buffered
  bf16* sF = sT + 2 * RAW_TILE;                                // the front rows
  bf16* sU = sF + RAW_TILE;
  bf16* sG = sU + TC_RING * TC_LD;
  float* sdh = reinterpret_cast<float*>(sG + TC_RING * TC_LD);      // [4 slabs][128]
  float* sdb = sdh + 4 * 128;                                        // [64]
  uint32_t* sFa = reinterpret_cast<uint32_t*>(sdb + TC_CH);          // [4 slabs][NF][32] anticausal fragments
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int c_base = blockIdx.x * TC_CH, b = blockIdx.z;
  const int k0 = blockIdx.y * tiles_per_seg, k1 = min(k0 + tiles_per_seg, n_tiles);
  if (k0 >= k1) return;
  const int seg_t0 = (k0 - n_halo_tiles) * TC_TT;              // halo tiles have negative times
  for (int i = tid; i < 4 * 128 + TC_CH; i += BWD_THREADS) sdh[i] = 0.f;
  const int slab = warp & 3, half = warp >> 2;
  const int ch0 = c_base + slab * 16;
  const int nd = min(ND, (a.K - 1) / 16 + 2);
  const int g = lane >> 2, tq = lane & 3;
  const int lm_row = (lane & 7) + ((lane >> 3) & 1) * 8, lm_col = slab * 16 + (lane >> 4) * 8;
  const int b_row = (lane & 7) + (lane >> 4) * 8, b_col = slab * 16 + ((lane >> 3) & 1) * 8;
  // fill the rings: steps -4 .. -1 stage rows behind the segment (u) and the segment's first 128 rows ahead (g)
  constexpr int LEAD = TC_HALO / TC_TT;
  mr_stage_fg(sT, a, dz, b, seg_t0 - LEAD * TC_TT, c_base, tid);
  mr_stage_fg(sF, a, dz, b, seg_t0, c_base, tid);
  mr_cp_commit();
  // causal fragments in registers, anticausal ones in shared memory: both in registers would spill
  uint32_t Fc[NF];
  const uint32_t* Fa = sFa + slab * NF * 32 + lane;
  {
    const float* hg = a.h + (size_t)(min(ch0, a.D - 1) / a.dg) * a.K;
    if (half == 0) {
      toeplitz_frags<false>(Fc, hg, a.K, lane);
#pragma unroll
      for (int m = 0; m < NF; ++m) sFa[(slab * NF + m) * 32 + lane] = Fc[m];
    }
    toeplitz_frags<true>(Fc, hg, a.K, lane);
  }
  // filter-gradient accumulators: this warp covers diagonals d = half, half + 2, ... for both row blocks of the tile
  constexpr int NDH = (ND + 1) / 2;
  float P[NDH][2][4];
#pragma unroll
  for (int i = 0; i < NDH * 8; ++i) P[i >> 3][(i >> 2) & 1][i & 3] = 0.f;
  float db[2][2] = {{0.f, 0.f}, {0.f, 0.f}};

  int rel = TC_RING - LEAD * TC_TT;                            // ring row of the step's first row (row t <-> (t - seg_t0) mod RING)
  for (int k = k0 - LEAD; k < k1; ++k) {
    const int t0 = (k - n_halo_tiles) * TC_TT;
    bf16* raw = sT + ((k - k0 + LEAD) & 1) * RAW_TILE;
    bf16* rawg = raw + TC_TT * RAW_LD;
    mr_cp_wait_all();
    __syncthreads();                                           // staged rows are here; reads of step k - 1 (raw, rings) are done
    {
      const int r = tid >> 3, cv = tid & 7;                    // 32 rows x 8 vectors of 8 channels
      *reinterpret_cast<uint4*>(sU + (rel + r) * TC_LD + cv * 8) = gate_u(reinterpret_cast<const uint4*>(raw + r * RAW_LD + cv * 24));
      int fr = rel + TC_HALO;
      if (fr >= TC_RING) fr -= TC_RING;
      *reinterpret_cast<uint4*>(sG + (fr + r) * TC_LD + cv * 8) =
          gate_g(reinterpret_cast<const uint4*>(sF + r * RAW_LD + cv * 24),
                 *reinterpret_cast<const uint4*>(sF + TC_TT * RAW_LD + r * RAWG_LD + cv * 8));
    }
    __syncthreads();                                           // rings complete; the front buffer is free
    if (k + 1 < k1) {
      mr_stage_fg(sT + ((k - k0 + LEAD + 1) & 1) * RAW_TILE, a, dz, b, t0 + TC_TT, c_base, tid);
      mr_stage_fg(sF, a, dz, b, t0 + TC_TT + TC_HALO, c_base, tid);
    }
    mr_cp_commit();
    if (k >= k0) {
      const int i0 = rel + half * 16;                          // ring row of this warp's output block
      float ya[2][4], da[2][4];
#pragma unroll
      for (int i = 0; i < 8; ++i) { ya[i >> 2][i & 3] = 0.f; da[i >> 2][i & 3] = 0.f; }
#pragma unroll
      for (int d = 0; d < ND; ++d) {
        if (FULL || d < nd) {
          int ru = i0 - 16 * d, rg = i0 + 16 * d;
          if (ru < 0) ru += TC_RING;
          if (rg >= TC_RING) rg -= TC_RING;
          uint32_t bu[4], bg[4];
          ldsm_x4_t(bu, smem_addr(sU + (ru + lm_row) * TC_LD + lm_col));
          ldsm_x4_t(bg, smem_addr(sG + (rg + lm_row) * TC_LD + lm_col));
          toeplitz_mma<true>(ya[0], Fc, d, bu[0], bu[1]);
          toeplitz_mma<true>(ya[1], Fc, d, bu[2], bu[3]);
          const uint32_t fm = Fa[(2 * d + 1) * 32], fa[4] = {fm, Fa[2 * d * 32], Fa[(2 * d + 2) * 32], fm};
          mma16816(da[0], fa, bg[0], bg[1]);
          mma16816(da[1], fa, bg[2], bg[3]);
        }
      }
      // filter gradient: P_d[i][j] += sum_c G[i0+i][c] U[i0-16d+j][c] over the two row blocks, d = half, half+2, ..
      if (t0 >= 0) {
#pragma unroll
        for (int blk = 0; blk < 2; ++blk) {
          uint32_t af[4];
          ldsm_x4(af, smem_addr(sG + (rel + blk * 16 + lm_row) * TC_LD + lm_col));
#pragma unroll
          for (int dd = 0; dd < NDH; ++dd) {
            const int d = 2 * dd + half;
            if (FULL ? d < ND : d < nd) {
              int ru = rel + blk * 16 - 16 * d;
              if (ru < 0) ru += TC_RING;
              uint32_t bf[4];
              ldsm_x4(bf, smem_addr(sU + (ru + b_row) * TC_LD + b_col));
              mma16816(P[dd][0], af, bf[0], bf[1]);
              mma16816(P[dd][1], af, bf[2], bf[3]);
            }
          }
        }
      }
      // combine at the fragment positions; the gradient replaces the features in place (each thread its own words)
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        const int c = slab * 16 + nt * 8 + 2 * tq;
        const float b0 = c_base + c < a.D ? a.bias[c_base + c] : 0.f, b1 = c_base + c + 1 < a.D ? a.bias[c_base + c + 1] : 0.f;
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          const int row = half * 16 + g + hh * 8;
          uint32_t* w = reinterpret_cast<uint32_t*>(raw + row * RAW_LD + 3 * c);
          const float2 p0 = unpack2(w[0]), p1 = unpack2(w[1]), p2 = unpack2(w[2]);        // (x1 x2) (v x1) (x2 v)
          const float2 gz = unpack2(*reinterpret_cast<const uint32_t*>(rawg + row * RAWG_LD + c));
          const float u0 = p0.y * p1.x, u1 = p2.x * p2.y, g0 = gz.x * p0.x, g1 = gz.y * p1.y;
          const float y0 = ya[nt][hh * 2] + b0 * u0, y1 = ya[nt][hh * 2 + 1] + b1 * u1;
          const float d0 = da[nt][hh * 2] + b0 * g0, d1 = da[nt][hh * 2 + 1] + b1 * g1;
          db[nt][0] += g0 * u0;                                // rows outside the sequence carry dz = 0
          db[nt][1] += g1 * u1;
          w[0] = pack2(gz.x * y0, d0 * p1.x);
          w[1] = pack2(d0 * p0.y, gz.y * y1);
          w[2] = pack2(d1 * p2.y, d1 * p2.x);
        }
      }
      __syncthreads();
#pragma unroll
      for (int j = 0; j < TC_TT * 24 / BWD_THREADS; ++j) {
        const int i = tid + j * BWD_THREADS, r = i / 24, q = i - r * 24;
        const int t = t0 + r, c3 = 3 * c_base + q * 8;
        if (c3 >= 3 * a.D) continue;
        const uint4 val = *reinterpret_cast<const uint4*>(raw + r * RAW_LD + q * 8);
        if (t >= 0 && t < a.L) *reinterpret_cast<uint4*>(dfeat + ((size_t)b * a.L + t) * 3 * a.D + c3) = val;
        else if (t < 0 && t >= -(a.K - 1) && dhalo) *reinterpret_cast<uint4*>(dhalo + ((size_t)b * (a.K - 1) + (t + a.K - 1)) * 3 * a.D + c3) = val;
      }
    }
    rel += TC_TT;
    if (rel >= TC_RING) rel -= TC_RING;
  }

  // ---- flush: filter gradient (once per block), bias gradient
#pragma unroll
  for (int dd = 0; dd < NDH; ++dd) {
    const int d = 2 * dd + half;
    if (d < nd) {
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int i = g + ((q & 2) ? 8 : 0), j = nt * 8 + 2 * tq + (q & 1);
          const int s = 16 * d + i - j;
          if (s >= 0 && s < a.K) atomicAdd(&sdh[slab * 128 + s], P[dd][nt][q]);
        }
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) atomicAdd(&sdb[slab * 16 + (j >> 1) * 8 + 2 * tq + (j & 1)], db[j >> 1][j & 1]);
  __syncthreads();
  for (int i = tid; i < 4 * 128; i += BWD_THREADS) {
    const int sl = i >> 7, s = i & 127;
    const int c = c_base + sl * 16;
    if (s < a.K && c < a.D) atomicAdd(dh + (size_t)(c / a.dg) * a.K + s, sdh[i]);
  }
  for (int i = tid; i < TC_CH; i += BWD_THREADS)
    if (c_base + i < a.D) atomicAdd(dbias + c_base + i, sdb[i]);
}

// Segments per (channel tile, batch row): as many as fit in one wave of `per_sm` blocks per SM (a partial second wave would
// cost a whole segment time), but no shorter than 4 tiles (a segment's lead-in stages 4 tiles of rows).
static inline int mr_tiles_per_seg(int n_tiles, int D, int B, int per_sm) {
  int segs = (per_sm * num_sms()) / (((D + TC_CH - 1) / TC_CH) * B);
  if (segs > (n_tiles + 3) / 4) segs = (n_tiles + 3) / 4;
  if (segs < 1) segs = 1;
  return (n_tiles + segs - 1) / segs;
}

static int mr_launch_fwd(const MrArgs& a, void* z, int B, cudaStream_t st) {
  auto kern = a.K > 16 * (ND - 2) ? mr_tc_fwd_kernel<true> : mr_tc_fwd_kernel<false>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, FWD_SMEM) != cudaSuccess) return -5;
  const int n_tiles = (a.L + TC_TT - 1) / TC_TT, tps = mr_tiles_per_seg(n_tiles, a.D, B, 4);
  const dim3 grid((a.D + TC_CH - 1) / TC_CH, (n_tiles + tps - 1) / tps, B);
  kern<<<grid, FWD_THREADS, FWD_SMEM, st>>>(a, (bf16*)z, n_tiles, tps);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

static int mr_launch_bwd(const MrArgs& a, const void* dz, void* dfeat, void* dhalo, float* dh, float* dbias, int n_halo, int B,
                         cudaStream_t st) {
  auto kern = a.K > 16 * (ND - 2) ? mr_tc_bwd_kernel<true> : mr_tc_bwd_kernel<false>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, BWD_SMEM) != cudaSuccess) return -5;
  const int n_tiles = (a.L + TC_TT - 1) / TC_TT + n_halo, tps = mr_tiles_per_seg(n_tiles, a.D, B, 2);
  const dim3 grid((a.D + TC_CH - 1) / TC_CH, (n_tiles + tps - 1) / tps, B);
  kern<<<grid, BWD_THREADS, BWD_SMEM, st>>>(a, (const bf16*)dz, (bf16*)dfeat, (bf16*)dhalo, dh, dbias, n_halo, n_tiles, tps);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // namespace sb

using namespace sb;

extern "C" int sb_mr_tc_supported(int D, int G, int K) {
  const int dg = D / G;
  return (D % G == 0) && (dg % 16 == 0) && K >= 1 && K <= 128 && (D % 8 == 0);
}

extern "C" int sb_mr_tc_fwd(const void* feat, const void* halo, const float* h, const float* bias, void* z, int B, int L,
                            int D, int G, int K, cudaStream_t st) {
  if (!sb_mr_tc_supported(D, G, K)) return -1;
  if (B * L == 0) return 0;
  return mr_launch_fwd(MrArgs{(const bf16*)feat, halo_local(halo), h, bias, L, D, K, D / G, 0, halo_local(nullptr), halo_local(nullptr)},
                       z, B, st);
}

// Context-parallel forward: feat [2B, L, 3D] (two zigzag chunks per sequence), rows before each chunk read in place
// from the neighbours' staged tails (`before`, see halo_src.cuh).
extern "C" int sb_mr_tc_fwd_cp(const void* feat, const HaloSrc* before, const float* h, const float* bias, void* z, int B2,
                               int L, int D, int G, int K, cudaStream_t st) {
  if (!sb_mr_tc_supported(D, G, K) || !before) return -9;
  if (B2 * L == 0) return 0;
  return mr_launch_fwd(MrArgs{(const bf16*)feat, *before, h, bias, L, D, K, D / G, 0, halo_local(nullptr), halo_local(nullptr)}, z, B2,
                       st);
}

// Context-parallel backward: the look-ahead of dz * x1 past each chunk's end comes from the next chunk's staged head
// (`ahead_feat`, `ahead_dz`), so the gradients of the chunk's tail rows are complete and no halo gradient is produced.
// L must be a multiple of 64 (whole tiles: a look-ahead row never shares a tile with chunk rows).
extern "C" int sb_mr_tc_bwd_cp(const void* feat, const HaloSrc* before, const float* h, const float* bias, const void* dz,
                               const HaloSrc* ahead_feat, const HaloSrc* ahead_dz, void* dfeat, float* dh, float* dbias, int B2,
                               int L, int D, int G, int K, cudaStream_t st) {
  if (!sb_mr_tc_supported(D, G, K) || !before || !ahead_feat || !ahead_dz || (L % 64)) return -9;
  if (B2 * L == 0) return 0;
  return mr_launch_bwd(MrArgs{(const bf16*)feat, *before, h, bias, L, D, K, D / G, 1, *ahead_feat, *ahead_dz}, dz, dfeat, nullptr, dh,
                       dbias, 0, B2, st);
}

extern "C" int sb_mr_tc_bwd(const void* feat, const void* halo, const float* h, const float* bias, const void* dz,
                            void* dfeat, void* dhalo, float* dh, float* dbias, int B, int L, int D, int G, int K,
                            cudaStream_t st) {
  if (!sb_mr_tc_supported(D, G, K)) return -1;
  if (B * L == 0) return 0;
  const int n_halo = (halo && dhalo) ? (K - 1 + TC_TT - 1) / TC_TT : 0;
  return mr_launch_bwd(MrArgs{(const bf16*)feat, halo_local(halo), h, bias, L, D, K, D / G, 0, halo_local(nullptr), halo_local(nullptr)},
                       dz, dfeat, dhalo, dh, dbias, n_halo, B, st);
}
