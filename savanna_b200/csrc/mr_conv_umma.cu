// Hyena-MR on the fifth-generation tensor cores: the causal FIR of <= 128 taps that the channels of a group share, as a product with
// a Toeplitz matrix of 128 x 256 taps,
//     y[t] = sum_r T1[t][r] u_prev[r] + T0[t][r] u_cur[r],      T0[t][r] = h[t - r],  T1[t][r] = h[128 + t - r]   (zero outside 0..K-1)
// over the 128-row tile of t and the one before it; the backward's du is the same product with T0 and T1 transposed, over the tile and
// the one behind it, of g = dz x1, and the tap gradient is the product G U^T over the channels, summed along its diagonals at the end.
// A block takes 16 channels (one filter) of a run of 128-row tiles: features come by TMA (96 bytes a row), u and g go into shared memory
// as bf16, [rows][16 channels] in 32-byte rows, and the 16 channels of two tiles are the N = 32 columns of one tcgen05.mma, whose A
// operand, the Toeplitz matrix, lies in tensor memory for the whole run.  The rows of u and g serve as N of the Toeplitz products
// (MN-major) and as K of the tap gradient (K-major) from the same bytes, in the 32-byte swizzle.  fp32 accumulation; u, g and the taps are
// rounded to bf16 for the products, gates and bias are fp32: the roundings of mr_conv_tc.cu.
//
// The Toeplitz product takes twice the multiplications of the 16-row blocks of mr_conv_tc.cu, whose mma.sync fragments were bound by issue
// slots and their latency (a thousand warp instructions for 16 x 16 outputs of the backward; here 350).  Measured on a B200, B = 1, L = 8192, D = 4096,
// K = 128, us, L2 flushed: forward 71 -> 65 (copying the data 41), backward 256 -> 107 (72); [3 x 777 x 512] 12 -> 10 and 36 -> 17, [2 x 1024 x 256]
// 11 -> 7 and 29 -> 15, [2048 x 2048] of 64 taps 14.5 -> 14.5 and 45 -> 23.  Forwards of up to 32 taps are mostly faster there (autograd_native.cpp:
// short_filter).  What bounds these is memory: DRAM moves the case's own bytes and nothing else (ncu: backward 269 MB read, 163 written, 48 % of
// the issue slots, forward 202, 45 and 35 %).  The backward has one block per SM, moves 5.2 TB/s while all of them run, and its 256 runs are
// 1.7 waves; the forward has two, and its 256 runs are one wave that leaves 40 SMs with one block.  Runs of equal length keep neighbouring blocks, which
// share 128-byte lines, at the same rows: dealing the tiles out evenly instead (132 -> 116 tiles a block) took 207 for the backward.  Shorter runs
// pay for their first tiles and for the operands again (16 tiles: 131).  The backward as one chain of steps per block, with rows kept in
// registers and T' in shared memory, took 170; with two groups of warps forming u and g, so that registers spill, 123.
// A run's tap gradient adds up in one accumulator, so the rounding of its fp32 sum grows with the run (32 tiles 1.2e-6, 64 2.4e-6; u and g
// rounded to bf16 2.3e-3).
//
// A Toeplitz product multiplies whole tiles, zero taps included, so an Inf or NaN would spread over its tile and the next, and into taps whose
// lag reaches beyond the sequence, where the tap gradient multiplies zero rows: once one has been seen, results that are not finite are
// formed again, tap by tap or row by row.
//
// Halo rows and the context-parallel forms stay with mr_conv_tc.cu, group widths that are not a multiple of 16 with mr_conv.cu.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "entries.h"
#include "sm100.cuh"

namespace sb {
namespace mru {
typedef __nv_bfloat16 bf16;

constexpr int TILE = 128, CH = 16;
constexpr int THREADS = 320, ROWS_T = 256;        // forward: 8 warps of rows, loader, MMA issuer
constexpr uint32_t IMG = TILE * CH * 2;           // a tile of u or g: 4 KB
constexpr uint32_t RING = 5 * IMG;                // slots 0..3 and a second copy of slot 0 behind slot 3, so that pairs are contiguous
constexpr uint32_t FEAT_B = TILE * 3 * CH * 2, DZ_B = TILE * CH * 2;

// barriers (offsets in the barrier block)
enum { RAW_FULL = 0, RAW_FREE = 32, UG_READY = 64, ACC_FULL = 72, ABORT = 80, TMEM_SLOT = 84, BAD = 88, BAR_BYTES = 128 };

struct Params {
  const float* h;
  const float* bias;
  float* dh;
  float* dbias;
  const bf16 *feat, *dz;
  int B, L, K, dg, slabs, tiles, tps, units;
  uint32_t* status;
};
struct Unit { int slab, b, j0, n; };
__device__ __forceinline__ Unit unit_of(const Params& p, int u) {
  Unit r;
  r.slab = u % p.slabs;
  const int q = u / p.slabs;
  r.b = q % p.B;
  r.j0 = q / p.B * p.tps;
  r.n = min(p.tps, p.tiles - r.j0);
  return r;
}

__device__ __forceinline__ uint64_t desc_sw32(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return uint64_t((addr & 0x3FFFFu) >> 4) | uint64_t((lbo >> 4) & 0x3FFFu) << 16 | uint64_t((sbo >> 4) & 0x3FFFu) << 32 | 1ull << 46 |
         6ull << 61;
}
// 16 rows (the contraction) x 16 channels of two tiles that are IMG apart
__device__ __forceinline__ uint64_t desc_pair(uint32_t slot, int kk) { return desc_sw32(slot + kk * 512u, IMG, 256u); }
// 128 rows x 16 channels (the contraction)
__device__ __forceinline__ uint64_t desc_rows(uint32_t slot) { return desc_sw32(slot, 16u, 256u); }

__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void tma_store_3d(const void* tmap, uint32_t src, int x, int y, int z) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%1, %2, %3}], [%4];"
               ::"l"(reinterpret_cast<uint64_t>(tmap)), "r"(x), "r"(y), "r"(z), "r"(src) : "memory");
}
__device__ __forceinline__ void tmem_ld_16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                 "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(taddr) : "memory");
}
// Volatile, so that it stays in front of the arrival that hands the buffer back to the loader.  That alone is not enough: the refill is a write
// of the async proxy, which the arrival's release does not order behind reads of the generic proxy (tiles were overwritten under loads in
// flight).  A load is over once its value has been used: the test for Inf and NaN takes in every word that was loaded, and has to stay
// in front of the arrival.
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.volatile.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void sts128(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__device__ __forceinline__ uint32_t pk(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
__device__ __forceinline__ __nv_bfloat162 b2(uint32_t w) { return *reinterpret_cast<__nv_bfloat162*>(&w); }
__device__ __forceinline__ uint32_t w2(__nv_bfloat162 v) { return *reinterpret_cast<uint32_t*>(&v); }
// Two channels' interleaved triples in three words, (x1 x2 | v x1 | x2 v) -> packed products.  A bf16 product of bf16 values rounds
// once, exactly as the fp32 product rounded to bf16 does.
__device__ __forceinline__ uint32_t gate_u(uint32_t w0, uint32_t w1, uint32_t w2_) {
  return w2(__hmul2(b2(__byte_perm(w0, w2_, 0x5432)), b2(__byte_perm(w1, w2_, 0x7610))));
}
__device__ __forceinline__ uint32_t gate_g(uint32_t w0, uint32_t w1, uint32_t dz) {
  return w2(__hmul2(b2(__byte_perm(w0, w1, 0x7610)), b2(dz)));
}
// byte offset of channel chunk c (8 channels) of row r inside a tile image
__device__ __forceinline__ uint32_t img_chunk(int r, int c) { return uint32_t(r) * 32u + (uint32_t(c ^ ((r >> 2) & 1)) << 4); }

// Words of two taps, in shared memory: x even first, then x odd, of the array f(x), f(x + 1).
template <class F>
__device__ __forceinline__ void tap_words(uint32_t* dst, F f, int tid, int threads) {
  for (int i = tid; i < 384; i += threads) {
    const int x = i < 192 ? 2 * i : 2 * (i - 192) + 1;
    dst[i] = pk(f(x), f(x + 1));
  }
}
// Row `x0` .. of such an array into tensor memory: 64 taps, 32 columns.
__device__ __forceinline__ void taps_to_tmem(uint32_t dst, const uint32_t* words, int x0) {
  const uint32_t* tb = words + ((x0 & 1) ? 192 : 0) + (x0 >> 1);
  uint32_t w[32];
#pragma unroll
  for (int e = 0; e < 32; ++e) w[e] = tb[e];
  tmem_st_32x32(dst, w);
}

__device__ __forceinline__ bool finite(float v) { return (__float_as_uint(v) & 0x7f800000u) != 0x7f800000u; }
// A result that an Inf or NaN elsewhere in its tiles has spoilt, tap by tap: y (DIR = -1) or du (DIR = 1) of one channel of row t.
template <int DIR>
__device__ __noinline__ float fir_element(const bf16* feat, const bf16* dz, const float* h, int K, int L, int D, int t, int c) {
  float y = 0.f;
  for (int s = 0; s < K && y == y; ++s) {              // a NaN stays one: a row of them takes one step an element, not K
    const int q = t + DIR * s;
    if (q < 0 || q >= L) break;
    const bf16* f = feat + (size_t)q * 3 * D + 3 * c;
    const __nv_bfloat16 u = DIR < 0 ? __hmul(f[1], f[2]) : __hmul(dz[(size_t)q * D + c], f[0]);
    y += __bfloat162float(__float2bfloat16_rn(h[s])) * __bfloat162float(u);
  }
  return y;
}
// The gradient of tap s over rows t0 .. t1 - 1 and the 16 channels from c0 on, by the products that exist: a zero row beyond the sequence times
// an Inf or NaN has spoilt the sum of the tensor cores.
__device__ __noinline__ float tap_gradient(const bf16* feat, const bf16* dz, int t0, int t1, int D, int c0, int s) {
  float sum = 0.f;
  for (int t = max(t0, s); t < t1 && sum == sum; ++t) {
    const uint4* f = reinterpret_cast<const uint4*>(feat + (size_t)t * 3 * D + 3 * c0);
    const uint4* q = reinterpret_cast<const uint4*>(feat + (size_t)(t - s) * 3 * D + 3 * c0);
    const uint4* z = reinterpret_cast<const uint4*>(dz + (size_t)t * D + c0);
    float row = 0.f;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      uint4 fv[3], qv[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) { fv[k] = f[3 * half + k]; qv[k] = q[3 * half + k]; }
      const uint4 zv = z[half];
      const uint32_t *fw = reinterpret_cast<const uint32_t*>(fv), *qw = reinterpret_cast<const uint32_t*>(qv), *zw = reinterpret_cast<const uint32_t*>(&zv);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint32_t g = gate_g(fw[3 * k], fw[3 * k + 1], zw[k]), u = gate_u(qw[3 * k], qw[3 * k + 1], qw[3 * k + 2]);
        row += lo(g) * lo(u) + hi(g) * hi(u);
      }
    }
    sum += row;
  }
  return sum;
}

__device__ __forceinline__ void linger() {            // copies of this block may still be in flight: not before they have landed
  const unsigned long long t0 = globaltimer();
  while (globaltimer() - t0 < 200000ull) __nanosleep(1000);
}

// ------------------------------------------------------------------------------------ forward
// z = x1 (h * u + bias u).  A step takes two tiles, a thread a row: u into shared memory, then z from the accumulators and from the
// features, which the thread has kept in registers; the steps of the two blocks of an SM fill each other's waits.  A step needs u of the
// tile before it, so a run starts with that tile alone.  Warp 8 loads, warp 9 issues the products.
constexpr uint32_t F_RAW = RING, F_OUT = F_RAW + 4 * FEAT_B, F_BAR = F_OUT + 2 * IMG, F_MISC = F_BAR + BAR_BYTES,
                   F_SMEM = F_MISC + 384 * 4 + CH * 4 + 1024;
constexpr uint32_t F_TMEM = 256, F_T = 0, F_Y = 128;

__global__ void __launch_bounds__(THREADS, 2)
mr_umma_fwd_kernel(const __grid_constant__ CUtensorMap tmF, const __grid_constant__ CUtensorMap tmZ, Params p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t bar = base + F_BAR;
  uint32_t* sR = reinterpret_cast<uint32_t*>(gen + F_MISC);
  float* sBias = reinterpret_cast<float*>(sR + 384);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gen + F_BAR + ABORT);
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gen + F_BAR + TMEM_SLOT);
  volatile int* bad = reinterpret_cast<volatile int*>(gen + F_BAR + BAD);
  const int tid = threadIdx.x, warp = tid >> 5;
  if (tid == 0) {
    for (int i = 0; i < 4; ++i) { mbar_init(bar + RAW_FULL + 8 * i, 1); mbar_init(bar + RAW_FREE + 8 * i, 128); }
    mbar_init(bar + UG_READY, ROWS_T); mbar_init(bar + ACC_FULL, 1);
    *abort_flag = 0; *bad = 0;
    fence_barrier_init();
    prefetch_tmap(&tmF); prefetch_tmap(&tmZ);
  }
  if (warp == 9) { tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), F_TMEM); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 8) {
    if (elect_one()) {
      bool ok = true;
      uint32_t cnt[2] = {0, 0};
      for (int u = blockIdx.x; u < p.units && ok; u += gridDim.x) {
        const Unit un = unit_of(p, u);
        for (int i = -1; i < un.n && ok; ++i) {
          const int w = i & 1;
          const uint32_t c = cnt[w]++, slot = 2 * w + (c & 1);
          if (c >= 2) ok = mbar_wait(bar + RAW_FREE + 8 * slot, ((c >> 1) & 1) ^ 1u, abort_flag, p.status, ST_MR_FWD);
          if (!ok) break;
          mbar_expect_tx(bar + RAW_FULL + 8 * slot, FEAT_B);
          tma_load_3d(base + F_RAW + slot * FEAT_B, &tmF, 3 * CH * un.slab, (un.j0 + i) * TILE, un.b, bar + RAW_FULL + 8 * slot);
        }
      }
      if (!ok) linger();
    }
  } else if (warp == 9) {
    if (elect_one()) {
      const uint32_t idesc = umma_idesc_bf16(128, 32, 0, 1);
      uint32_t gs = 0;
      bool ok = true;
      for (int u = blockIdx.x; u < p.units && ok; u += gridDim.x) {
        const Unit un = unit_of(p, u);
        for (int k = 1; k <= (un.n + 1) / 2; ++k, ++gs) {
          ok = mbar_wait(bar + UG_READY, gs & 1u, abort_flag, p.status, ST_MR_FWD + 1);
          if (!ok) break;
          tc_fence_after();
          const uint32_t prev = base + ((2 * k - 3) & 3) * IMG, cur = base + ((2 * k - 2) & 3) * IMG;
#pragma unroll
          for (int kk = 0; kk < 16; ++kk)
            umma_bf16_ts(tmem + F_Y, tmem + F_T + kk * 8, desc_pair(kk < 8 ? prev : cur, kk & 7), idesc, kk ? 1u : 0u);
          umma_commit(bar + ACC_FULL);
        }
      }
    }
  } else {
    const int w = warp >> 2, r = tid & 127;
    const uint32_t lane_off = uint32_t((warp & 3) * 32) << 16, out = base + F_OUT + w * IMG;
    uint32_t cnt = 0, ga = 0;
    int group = -1;
    bool ok = true;
    for (int u = blockIdx.x; u < p.units; u += gridDim.x) {
      const Unit un = unit_of(p, u);
      const int g = un.slab * CH / p.dg;
      bar_sync(1, ROWS_T);                             // the unit before is through with the tables
      const float* h = p.h + (size_t)g * p.K;
      if (g != group) tap_words(sR, [&](int x) { return x > 255 - p.K && x < 256 ? h[255 - x] : 0.f; }, tid, ROWS_T);
      if (tid < CH) sBias[tid] = p.bias[un.slab * CH + tid];
      bar_sync(1, ROWS_T);
      if (g != group) {                                // warps 0-3 write T1, 4-7 T0
#pragma unroll
        for (int part = 0; part < 2; ++part)
          taps_to_tmem(tmem + lane_off + F_T + w * 64 + part * 32, sR, (w ? 255 : 127) - r + 64 * part);
        tmem_wait_st();
      }
      group = g;
      for (int k = 0; k <= (un.n + 1) / 2; ++k) {
        const int i = 2 * (k - 1) + w;                 // this thread's tile of the step
        const bool live = i >= -1 && i < un.n;
        uint4 x[6];
        if (live) {
          const uint32_t slot = 2 * w + (cnt & 1);
          if (ok) ok = mbar_wait(bar + RAW_FULL + 8 * slot, (cnt >> 1) & 1u, abort_flag, p.status, ST_MR_FWD + 2);
          ++cnt;
          const uint32_t src = base + F_RAW + slot * FEAT_B + r * 96u;
#pragma unroll
          for (int q = 0; q < 6; ++q) x[q] = lds128(src + q * 16);
          const uint32_t* xw = reinterpret_cast<const uint32_t*>(x);
          uint32_t uw[8];
          __nv_bfloat162 chk = __floats2bfloat162_rn(0.f, 0.f);
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            uw[q] = gate_u(xw[3 * q], xw[3 * q + 1], xw[3 * q + 2]);
            chk = __hfma2(b2(uw[q]), __floats2bfloat162_rn(0.f, 0.f), chk);
          }
          if (w2(chk) & 0x7fff7fffu) *bad = 1;         // 0 x Inf, 0 x NaN
          mbar_arrive(bar + RAW_FREE + 8 * slot);
          const uint32_t d0 = base + (i & 3) * IMG + img_chunk(r, 0), d1 = base + (i & 3) * IMG + img_chunk(r, 1);
          sts128(d0, uw[0], uw[1], uw[2], uw[3]);
          sts128(d1, uw[4], uw[5], uw[6], uw[7]);
          if ((i & 3) == 0) {
            sts128(d0 + 4 * IMG, uw[0], uw[1], uw[2], uw[3]);
            sts128(d1 + 4 * IMG, uw[4], uw[5], uw[6], uw[7]);
          }
        }
        fence_proxy_async();
        tc_fence_before();
        if (k > 0) {
          mbar_arrive(bar + UG_READY);
          if (ok) ok = mbar_wait(bar + ACC_FULL, ga & 1u, abort_flag, p.status, ST_MR_FWD + 3);
          ++ga;
        }
        if (k == 0 || !live) continue;
        tc_fence_after();
        uint32_t y[16];
        tmem_ld_16(tmem + lane_off + F_Y + 16 * w, y);
        tmem_wait_ld();
        const int t = (un.j0 + i) * TILE + r, D = p.slabs * CH;
        if (*bad && t < p.L) {
#pragma unroll 1
          for (int c = 0; c < CH; ++c) {
            float v = 0.f;
#pragma unroll
            for (int q = 0; q < CH; ++q) if (q == c) v = __uint_as_float(y[q]);
            if (finite(v)) continue;
            v = fir_element<-1>(p.feat + (size_t)un.b * p.L * 3 * D, nullptr, h, p.K, p.L, D, t, un.slab * CH + c);
#pragma unroll
            for (int q = 0; q < CH; ++q) if (q == c) y[q] = __float_as_uint(v);
          }
        }
        const uint32_t* xw = reinterpret_cast<const uint32_t*>(x);
        uint32_t zw[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const uint32_t a = xw[3 * q], b = xw[3 * q + 1], c = xw[3 * q + 2];
          zw[q] = pk(lo(a) * (__uint_as_float(y[2 * q]) + sBias[2 * q] * (hi(a) * lo(b))),
                     hi(b) * (__uint_as_float(y[2 * q + 1]) + sBias[2 * q + 1] * (lo(c) * hi(c))));
        }
        if (r == 0) bulk_wait_read<0>();
        bar_sync(2 + w, 128);                          // the tile stored before has been read
        sts128(out + r * 32u, zw[0], zw[1], zw[2], zw[3]);
        sts128(out + r * 32u + 16, zw[4], zw[5], zw[6], zw[7]);
        fence_proxy_async();
        bar_sync(2 + w, 128);
        if (r == 0) { tma_store_3d(&tmZ, out, CH * un.slab, (un.j0 + i) * TILE, un.b); bulk_commit(); }
      }
    }
    if (r == 0) bulk_wait<0>();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 9) { tc_fence_after(); tmem_dealloc(tmem, F_TMEM); }
}

// ------------------------------------------------------------------------------------ backward
// dfeat = (dz y, du v, du x2) interleaved, y formed again, dh, dbias.  The roles work on tiles of 128 rows, each a few tiles ahead of the
// next, over rings of staged rows and of u / g images:
//
//   warps 0-3     T and T' into tensor memory; u and g of a tile (two threads a row: no bank conflicts at 96 bytes a row)
//   warp 13       MMA: y and du of a tile once g of the next one is there, then the tap gradient's products
//   warps 4-11    outputs, a tile per four warps: the gradient replaces the features in place
//   warp 14       TMA store of the tile; hands its buffer back to the loader, warp 12
//
// Tensor memory holds both Toeplitz operands (256 columns), the tap gradient and the accumulators of two tiles, so that no operand but the
// narrow images passes through shared memory.  G U' is taken in halves of 64 rows t against the 192 rows from 128 before the half to its
// end: lags 0 .. 127 lie in 192 columns then, 256 with whole tiles.
constexpr int B_THREADS = 480, B_NRAW = 10, B_NUG = 6;
constexpr uint32_t RAW_B = FEAT_B + DZ_B, B_U = B_NRAW * RAW_B, B_G = B_U + (B_NUG + 1) * IMG, B_MISC = B_G + (B_NUG + 1) * IMG,
                   B_DIAG = B_MISC + 2 * 384 * 4, B_BAR = B_DIAG + 24 * 48 * 4, B_SMEM = B_BAR + 512 + 1024;
constexpr uint32_t B_T = 0, B_TT = 128, B_P = 256, B_ACC = 448;
enum { R_FULL = 0, R_FREE = 80, I_READY = 160, I_FREE = 208, A_FULL = 256, A_FREE = 264, U_DONE = 288, P_FREE = 296,
       O_READY = 304, B_ABORT = 384, B_SLOT = 388, B_BAD = 392 };

__global__ void __launch_bounds__(B_THREADS, 1)
mr_umma_bwd_kernel(const __grid_constant__ CUtensorMap tmF, const __grid_constant__ CUtensorMap tmZ, const __grid_constant__ CUtensorMap tmD,
                   Params p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t bar = base + B_BAR, sU = base + B_U, sG = base + B_G;
  uint32_t* sR = reinterpret_cast<uint32_t*>(gen + B_MISC);     // reversed taps, then the taps in order
  float* sDiag = reinterpret_cast<float*>(gen + B_DIAG);        // [4 quarters][6 blocks][48]: sums along the diagonals of 16 x 32 blocks
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gen + B_BAR + B_ABORT);
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gen + B_BAR + B_SLOT);
  volatile int* bad = reinterpret_cast<volatile int*>(gen + B_BAR + B_BAD);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int i = 0; i < B_NRAW; ++i) { mbar_init(bar + R_FULL + 8 * i, 1); mbar_init(bar + R_FREE + 8 * i, 1); mbar_init(bar + O_READY + 8 * i, 128); }
    for (int i = 0; i < B_NUG; ++i) { mbar_init(bar + I_READY + 8 * i, 128); mbar_init(bar + I_FREE + 8 * i, 1); }
    mbar_init(bar + A_FULL, 1); mbar_init(bar + A_FREE, 256); mbar_init(bar + U_DONE, 1); mbar_init(bar + P_FREE, 256);
    *abort_flag = 0; *bad = 0;
    fence_barrier_init();
    prefetch_tmap(&tmF); prefetch_tmap(&tmZ); prefetch_tmap(&tmD);
  }
  if (warp == 13) { tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  auto wait = [&](uint32_t b, uint32_t phase, uint32_t code) { return mbar_wait(bar + b, phase & 1u, abort_flag, p.status, ST_MR_BWD + code); };

  // Tiles of a run by index i: 0 is the one before it, 1 .. n its own, n + 1 the one behind it.  q counts the tiles of all runs, o the
  // runs' own tiles, v the runs.
  if (warp == 12) {
    if (elect_one()) {
      bool ok = true;
      uint32_t q = 0;
      for (int u = blockIdx.x; u < p.units && ok; u += gridDim.x) {
        const Unit un = unit_of(p, u);
        for (int i = 0; i <= un.n + 1; ++i, ++q) {
          const uint32_t slot = q % B_NRAW, use = q / B_NRAW, full = bar + R_FULL + 8 * slot, dst = base + slot * RAW_B;
          if (use && !(ok = wait(R_FREE + 8 * slot, use - 1, 0))) break;
          const int row = (un.j0 - 1 + i) * TILE;
          mbar_expect_tx(full, RAW_B);
          tma_load_3d(dst, &tmF, 3 * CH * un.slab, row, un.b, full);
          tma_load_3d(dst + FEAT_B, &tmZ, CH * un.slab, row, un.b, full);
        }
      }
      if (!ok) linger();
    }
  } else if (warp == 13) {
    if (elect_one()) {
      const uint32_t id_a = umma_idesc_bf16(128, 32, 0, 1), id_p = umma_idesc_bf16(64, 192, 0, 0);
      uint32_t q = 0, pairs = 0, v = 0;
      bool ok = true;
      for (int u = blockIdx.x; u < p.units && ok; u += gridDim.x, ++v) {
        const Unit un = unit_of(p, u);
        auto img = [&](int i) { return (q + i) % B_NUG; };
        int ready = 0;                                 // tiles whose images are there
        for (int i = 1; i <= un.n && ok; i += 2, ++pairs) {      // outputs of tiles i and i + 1
          const int last = min(i + 2, un.n + 1);
          for (; ready <= last && ok; ++ready) ok = wait(I_READY + 8 * img(ready), (q + ready) / B_NUG, 1);
          if (ok && pairs) ok = wait(A_FREE, pairs - 1, 2);
          if (!ok) break;
          tc_fence_after();
#pragma unroll
          for (int kk = 0; kk < 16; ++kk)              // T1 u(before) + T0 u
            umma_bf16_ts(tmem + B_ACC, tmem + B_T + kk * 8, desc_pair(sU + (kk < 8 ? img(i - 1) : img(i)) * IMG, kk & 7), id_a, kk ? 1u : 0u);
#pragma unroll
          for (int kk = 0; kk < 16; ++kk)              // T1' g(behind) + T0' g
            umma_bf16_ts(tmem + B_ACC + 32, tmem + B_TT + kk * 8, desc_pair(sG + (kk < 8 ? img(i + 1) : img(i)) * IMG, kk & 7), id_a,
                         kk ? 1u : 0u);
          umma_commit(bar + A_FULL);
          if (i == 1 && v && !(ok = wait(P_FREE, v - 1, 3))) break;
          tc_fence_after();
          for (int j = i; j <= min(i + 1, un.n); ++j)
#pragma unroll
            for (int half = 0; half < 2; ++half)
              umma_bf16(tmem + B_P, desc_rows(sG + img(j) * IMG + half * 2048u), desc_rows(sU + img(j - 1) * IMG + half * 2048u), id_p,
                        (j > 1 || half) ? 1u : 0u);
          for (int j = i - 1; j <= (i + 2 > un.n ? un.n + 1 : i); ++j) umma_commit(bar + I_FREE + 8 * img(j));
          if (i + 2 > un.n) umma_commit(bar + U_DONE);
        }
        q += un.n + 2;
      }
    }
  } else if (warp == 14) {
    if (elect_one()) {
      uint32_t q = 0, o = 0, before = 0;
      bool ok = true;
      for (int u = blockIdx.x; u < p.units && ok; u += gridDim.x) {
        const Unit un = unit_of(p, u);
        for (int i = 1; i <= un.n; ++i, ++o) {
          const uint32_t slot = (q + i) % B_NRAW;
          if (!(ok = wait(O_READY + 8 * (o % B_NRAW), o / B_NRAW, 4))) break;
          tma_store_3d(&tmD, base + slot * RAW_B, 3 * CH * un.slab, (un.j0 - 1 + i) * TILE, un.b);
          bulk_commit();
          if (o) { bulk_wait_read<1>(); mbar_arrive(bar + R_FREE + 8 * before); }
          before = slot;
        }
        q += un.n + 2;
      }
      bulk_wait<0>();
    }
  } else if (warp < 4) {
    const int r = tid;
    const uint32_t lane_off = uint32_t(warp * 32) << 16;
    uint32_t q = 0, v = 0;
    int group = -1;
    bool ok = true;
    for (int u = blockIdx.x; u < p.units; u += gridDim.x, ++v) {
      const Unit un = unit_of(p, u);
      const int g = un.slab * CH / p.dg;
      if (v && ok) ok = wait(U_DONE, v - 1, 5);        // all products with the operands of the run before
      if (g != group) {
        const float* h = p.h + (size_t)g * p.K;
        bar_sync(1, 128);
        tap_words(sR, [&](int x) { return x > 255 - p.K && x < 256 ? h[255 - x] : 0.f; }, tid, 128);
        tap_words(sR + 384, [&](int x) { return x > 126 && x < 127 + p.K ? h[x - 127] : 0.f; }, tid, 128);
        bar_sync(1, 128);
        tc_fence_after();
#pragma unroll
        for (int part = 0; part < 2; ++part) {         // T1, T0; T1', T0'
          taps_to_tmem(tmem + lane_off + B_T + part * 32, sR, 127 - r + 64 * part);
          taps_to_tmem(tmem + lane_off + B_T + 64 + part * 32, sR, 255 - r + 64 * part);
          taps_to_tmem(tmem + lane_off + B_TT + part * 32, sR + 384, 255 - r + 64 * part);
          taps_to_tmem(tmem + lane_off + B_TT + 64 + part * 32, sR + 384, 127 - r + 64 * part);
        }
        tmem_wait_st();
        group = g;
      }
      for (int i = 0; i <= un.n + 1; ++i, ++q) {
        const uint32_t slot = q % B_NRAW, img = q % B_NUG, src = base + slot * RAW_B;
        if (ok) ok = wait(R_FULL + 8 * slot, q / B_NRAW, 6);
        __nv_bfloat162 chk = __floats2bfloat162_rn(0.f, 0.f);
        const __nv_bfloat162 zero = chk;
        uint32_t uw[2][4], gw[2][4];
#pragma unroll
        for (int it = 0; it < 2; ++it) {
          const int row = it * 64 + (tid >> 1), half = tid & 1;
          uint32_t xw[12];
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            const uint4 t = lds128(src + row * 96u + half * 48u + k * 16u);
            xw[4 * k] = t.x; xw[4 * k + 1] = t.y; xw[4 * k + 2] = t.z; xw[4 * k + 3] = t.w;
          }
          const uint4 z = lds128(src + FEAT_B + row * 32u + half * 16u);
          const uint32_t zw[4] = {z.x, z.y, z.z, z.w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            uw[it][k] = gate_u(xw[3 * k], xw[3 * k + 1], xw[3 * k + 2]);
            gw[it][k] = gate_g(xw[3 * k], xw[3 * k + 1], zw[k]);
            chk = __hfma2(b2(uw[it][k]), zero, __hfma2(b2(gw[it][k]), zero, chk));
          }
        }
        if (w2(chk) & 0x7fff7fffu) *bad = 1;           // 0 x Inf, 0 x NaN
        if (q >= B_NUG && ok) ok = wait(I_FREE + 8 * img, q / B_NUG - 1, 7);
#pragma unroll
        for (int it = 0; it < 2; ++it) {
          const uint32_t o = img * IMG + img_chunk(it * 64 + (tid >> 1), tid & 1);
          sts128(sU + o, uw[it][0], uw[it][1], uw[it][2], uw[it][3]);
          sts128(sG + o, gw[it][0], gw[it][1], gw[it][2], gw[it][3]);
          if (img == 0) {                              // once more behind the last slot: pairs and windows are contiguous
            sts128(sU + B_NUG * IMG + o, uw[it][0], uw[it][1], uw[it][2], uw[it][3]);
            sts128(sG + B_NUG * IMG + o, gw[it][0], gw[it][1], gw[it][2], gw[it][3]);
          }
        }
        fence_proxy_async();
        tc_fence_before();
        mbar_arrive(bar + I_READY + 8 * img);
        if (i == 0 || i == un.n + 1) {                 // no outputs: nobody else reads these rows
          bar_sync(1, 128);
          if (tid == 0) mbar_arrive(bar + R_FREE + 8 * slot);
        }
      }
    }
  } else {
    const int e = (warp - 4) >> 2, quarter = warp & 3, r = quarter * 32 + lane;
    // Lanes whose row has bit 2 set take the upper eight channels first: rows of 96 bytes then lie in different banks.
    const int first = (r >> 2) & 1;
    const uint32_t lane_off = uint32_t(quarter * 32) << 16;
    uint32_t q = 0, o = 0, v = 0, pairs = 0;
    bool ok = true;
    for (int u = blockIdx.x; u < p.units; u += gridDim.x, ++v) {
      const Unit un = unit_of(p, u);
      const float* bias = p.bias + un.slab * CH;
      float db[2][8];
#pragma unroll
      for (int c = 0; c < 16; ++c) db[c >> 3][c & 7] = 0.f;
      for (int first_i = 1; first_i <= un.n; first_i += 2, ++pairs) {
        const int i = first_i + e;
        if (ok) ok = wait(A_FULL, pairs, 9);
        tc_fence_after();
        uint32_t y[16], d[16];
        tmem_ld_16(tmem + lane_off + B_ACC + e * 16, y);
        tmem_ld_16(tmem + lane_off + B_ACC + 32 + e * 16, d);
        tmem_wait_ld();
        tc_fence_before();
        mbar_arrive(bar + A_FREE);
        if (i > un.n) continue;
        const uint32_t slot = (q + i) % B_NRAW, src = base + slot * RAW_B;
        if (ok) ok = wait(R_FULL + 8 * slot, (q + i) / B_NRAW, 8);
        const int t = (un.j0 - 1 + i) * TILE + r;
        if (*bad && t < p.L) {
          const int D = p.slabs * CH;
          const bf16 *f = p.feat + (size_t)un.b * p.L * 3 * D, *z = p.dz + (size_t)un.b * p.L * D;
          const float* h = p.h + (size_t)(un.slab * CH / p.dg) * p.K;
#pragma unroll 1
          for (int c = 0; c < CH; ++c) {
            float yc = 0.f, dc = 0.f;
#pragma unroll
            for (int k = 0; k < CH; ++k) if (k == c) { yc = __uint_as_float(y[k]); dc = __uint_as_float(d[k]); }
            if (!finite(yc)) yc = fir_element<-1>(f, z, h, p.K, p.L, D, t, un.slab * CH + c);
            if (!finite(dc)) dc = fir_element<1>(f, z, h, p.K, p.L, D, t, un.slab * CH + c);
#pragma unroll
            for (int k = 0; k < CH; ++k) if (k == c) { y[k] = __float_as_uint(yc); d[k] = __float_as_uint(dc); }
          }
        }
        if (first) {
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            uint32_t s = y[k]; y[k] = y[k + 8]; y[k + 8] = s;
            s = d[k]; d[k] = d[k + 8]; d[k + 8] = s;
          }
        }
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          const int half = hh ^ first;
          const uint32_t at = src + r * 96u + half * 48u;
          uint32_t xw[12];
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            const uint4 w = lds128(at + k * 16u);
            xw[4 * k] = w.x; xw[4 * k + 1] = w.y; xw[4 * k + 2] = w.z; xw[4 * k + 3] = w.w;
          }
          const uint4 z = lds128(src + FEAT_B + r * 32u + half * 16u);
          const uint32_t zw[4] = {z.x, z.y, z.z, z.w};
          const float4 ba = __ldg(reinterpret_cast<const float4*>(bias + half * 8)), bb = __ldg(reinterpret_cast<const float4*>(bias + half * 8 + 4));
          const float bs[8] = {ba.x, ba.y, ba.z, ba.w, bb.x, bb.y, bb.z, bb.w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const uint32_t a = xw[3 * k], b = xw[3 * k + 1], c = xw[3 * k + 2], w = zw[k];
            const float u0 = hi(a) * lo(b), u1 = lo(c) * hi(c), g0 = lo(w) * lo(a), g1 = hi(w) * hi(b);
            const float y0 = __uint_as_float(y[8 * hh + 2 * k]) + bs[2 * k] * u0, y1 = __uint_as_float(y[8 * hh + 2 * k + 1]) + bs[2 * k + 1] * u1;
            const float d0 = __uint_as_float(d[8 * hh + 2 * k]) + bs[2 * k] * g0, d1 = __uint_as_float(d[8 * hh + 2 * k + 1]) + bs[2 * k + 1] * g1;
            db[hh][2 * k] += g0 * u0;                  // rows outside the sequence carry dz = 0
            db[hh][2 * k + 1] += g1 * u1;
            xw[3 * k] = pk(lo(w) * y0, d0 * lo(b));
            xw[3 * k + 1] = pk(d0 * hi(a), hi(w) * y1);
            xw[3 * k + 2] = pk(d1 * hi(c), d1 * lo(c));
          }
#pragma unroll
          for (int k = 0; k < 3; ++k) sts128(at + k * 16u, xw[4 * k], xw[4 * k + 1], xw[4 * k + 2], xw[4 * k + 3]);
        }
        fence_proxy_async();
        mbar_arrive(bar + O_READY + 8 * ((o + i - 1) % B_NRAW));
      }
      q += un.n + 2;
      o += un.n;

      // Tap gradient: dh[s] is the sum of G U' along the diagonals row - column = s - 128.  A warp holds 16 rows (the lanes below 16 of
      // its quarter) and three blocks of 32 columns; from column to column the running sum of a diagonal moves one lane up, and leaves
      // at lane 15.
      if (ok) ok = wait(U_DONE, v, 10);
      tc_fence_after();
      bar_sync(2, 256);                                // the sums of the run before have been read
      {
        uint32_t w[3][32];
#pragma unroll
        for (int k = 0; k < 3; ++k) tmem_ld_32x32(tmem + lane_off + B_P + e * 96 + k * 32, w[k]);
        tmem_wait_ld();
        tc_fence_before();
        mbar_arrive(bar + P_FREE);
        float run[3] = {0.f, 0.f, 0.f};
        float* dst = sDiag + (quarter * 6 + e * 3) * 48;
#pragma unroll
        for (int c = 0; c < 32; ++c)
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            const float up = __shfl_up_sync(0xffffffffu, run[k], 1);
            run[k] = (lane ? up : 0.f) + __uint_as_float(w[k][c]);
            if (lane == 15) dst[k * 48 + 46 - c] = run[k];
          }
        if (lane < 15) {
#pragma unroll
          for (int k = 0; k < 3; ++k) dst[k * 48 + lane] = run[k];
        }
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float a = first ? db[1][k] : db[0][k], b = first ? db[0][k] : db[1][k];
        db[0][k] = a; db[1][k] = b;
      }
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        float s = db[c >> 3][c & 7];
#pragma unroll
        for (int m = 16; m; m >>= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
        if (lane == c) atomicAdd(p.dbias + un.slab * CH + c, s);
      }
      bar_sync(2, 256);
      if (r < p.K && e == 0) {
        float sum = 0.f;
        for (int k = 0; k < 24; ++k) {
          const int d = r - 16 * (k / 6) - 128 + 32 * (k % 6);
          if (d >= -31 && d <= 15) sum += sDiag[k * 48 + d + 31];
        }
        if (*bad && !finite(sum)) {
          const int D = p.slabs * CH;
          sum = tap_gradient(p.feat + (size_t)un.b * p.L * 3 * D, p.dz + (size_t)un.b * p.L * D, un.j0 * TILE, min((un.j0 + un.n) * TILE, p.L), D,
                             un.slab * CH, r);
        }
        atomicAdd(p.dh + (size_t)(un.slab * CH / p.dg) * p.K + r, sum);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 13) { tc_fence_after(); tmem_dealloc(tmem, 512); }
}

// ------------------------------------------------------------------------------------ host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);
static EncodeTiledFn get_encode() {
  static EncodeTiledFn fn = [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) ptr = nullptr;
    return reinterpret_cast<EncodeTiledFn>(ptr);
  }();
  return fn;
}
// [B, L, W] bf16, boxes of `cols` columns x 128 rows; rows outside of 0 .. L - 1 read as zeros
static int make_map(CUtensorMap* out, const void* ptr, int B, int L, int W, int cols) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return -6;
  cuuint64_t dims[3] = {(cuuint64_t)W, (cuuint64_t)L, (cuuint64_t)B}, strides[2] = {(cuuint64_t)W * 2, (cuuint64_t)W * 2 * L};
  cuuint32_t box[3] = {(cuuint32_t)cols, TILE, 1}, one[3] = {1, 1, 1};
  return enc(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : -6;
}
// Tiles of a run: the fewest waves x steps (two tiles each, and what a run costs once, in steps).
static int tiles_per_run(int tiles, int columns, int slots, float once) {
  int best = tiles;
  float cost = 1e30f;
  for (int segs = 1; segs <= tiles && segs <= 256; ++segs) {
    const int tps = (tiles + segs - 1) / segs;
    const long long units = (long long)columns * ((tiles + tps - 1) / tps);
    const float c = (float)((units + slots - 1) / slots) * ((tps + 1) / 2 + once);
    if (c < cost) { cost = c; best = tps; }
  }
  return best;
}

}  // namespace mru
}  // namespace sb

using namespace sb;
using namespace sb::mru;

static bool supported(int D, int G, int K) { return G > 0 && D % G == 0 && (D / G) % CH == 0 && K >= 1 && K <= TILE; }

// feat [B, L, 3D], z [B, L, D]: bf16, 16-byte aligned.  h [G, K], bias [D] fp32.
extern "C" int sb_mr_umma_fwd(const void* feat, const float* h, const float* bias, void* z, int B, int L, int D, int G, int K,
                              unsigned int* status, cudaStream_t st) {
  if (!supported(D, G, K) || ((reinterpret_cast<uintptr_t>(feat) | reinterpret_cast<uintptr_t>(z)) & 15)) return -1;
  if (B <= 0 || L <= 0 || D <= 0) return 0;
  if (cudaFuncSetAttribute(mr_umma_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, F_SMEM) != cudaSuccess) return -5;
  CUtensorMap tf, tz;
  int rc = make_map(&tf, feat, B, L, 3 * D, 3 * CH);
  if (!rc) rc = make_map(&tz, z, B, L, D, CH);
  if (rc) return rc;
  const int tiles = (L + TILE - 1) / TILE, slabs = D / CH, slots = 2 * num_sms(), tps = tiles_per_run(tiles, slabs * B, slots, 1.f);
  const int units = slabs * B * ((tiles + tps - 1) / tps);
  mr_umma_fwd_kernel<<<units < slots ? units : slots, THREADS, F_SMEM, st>>>(
      tf, tz, Params{h, bias, nullptr, nullptr, (const bf16*)feat, nullptr, B, L, K, D / G, slabs, tiles, tps, units, status});
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// dz like z, dfeat like feat, bias 16-byte aligned; adds into dh [G, K] and dbias [D], fp32.
extern "C" int sb_mr_umma_bwd(const void* feat, const float* h, const float* bias, const void* dz, void* dfeat, float* dh, float* dbias,
                              int B, int L, int D, int G, int K, unsigned int* status, cudaStream_t st) {
  if (!supported(D, G, K) || ((reinterpret_cast<uintptr_t>(feat) | reinterpret_cast<uintptr_t>(dz) | reinterpret_cast<uintptr_t>(dfeat) |
                               reinterpret_cast<uintptr_t>(bias)) & 15)) return -1;
  if (B <= 0 || L <= 0 || D <= 0) return 0;
  if (cudaFuncSetAttribute(mr_umma_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, B_SMEM) != cudaSuccess) return -5;
  CUtensorMap tf, tz, td;
  int rc = make_map(&tf, feat, B, L, 3 * D, 3 * CH);
  if (!rc) rc = make_map(&tz, dz, B, L, D, CH);
  if (!rc) rc = make_map(&td, dfeat, B, L, 3 * D, 3 * CH);
  if (rc) return rc;
  const int tiles = (L + TILE - 1) / TILE, slabs = D / CH, slots = num_sms(), tps = tiles_per_run(tiles, slabs * B, slots, 2.f);
  const int units = slabs * B * ((tiles + tps - 1) / tps);
  mr_umma_bwd_kernel<<<units < slots ? units : slots, B_THREADS, B_SMEM, st>>>(
      tf, tz, td, Params{h, bias, dh, dbias, (const bf16*)feat, (const bf16*)dz, B, L, K, D / G, slabs, tiles, tps, units, status});
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
