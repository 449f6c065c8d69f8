// Streaming kernels of the short depthwise convolutions (included by conv.cu, which describes the operators).
//
// A warp owns a strip of neighbouring channels and walks down the rows of a run on its own: asynchronous 16-byte copies put the
// next rows into a ring of shared memory that belongs to this warp alone, the filter windows are registers, every fp32 quantity is
// a pair of channels in one 64-bit register.  No block barrier anywhere: a warp waits for its own copies and for nothing else, so
// copies are in flight all the time, which is what the tiled kernels these replace lacked (stage a tile, wait, barrier, compute; 55 to
// 85 % of the copy rate).  KB of copies in flight per SM (blocks of four warps x rows of the ring ahead x bytes of a row): featuriser
// forward 4 x 11 x 512 B, 90 with 3 taps; its backward 2 x 11 x 512 B, 45; Hyena-SE forward 3 x 13 x 768 B, 120 with 7 taps; its
// backward 2 x 6 x 1024 B, 49 with 7 taps, where issue (52 % of the slots) and the serial body bound it more than copies.  The interleaved (x1, x2, v) triples of four channels are 24 bytes,
// read as three 8-byte words at a stride of 24 bytes (no bank conflict); gradients of triples go back into the ring slot their
// row came from and leave with full 16-byte stores.
// Two or three blocks of four warps per SM (one wave; the featuriser's forward, whose runs have two edge rows only, is cut for nine
// blocks per SM, of which four run at a time): the registers of a fourth are worth more to the scheduling of the unrolled bodies - Hyena-SE backward, L = 8192, D = 4096:
// 88 us with two blocks, 97 with three (168 registers), 123 with four (128).  Whole blocks per strip: four blocks too many for the
// wave cost a second one.
#pragma once
#include "device_info.h"
#include "f32x2.cuh"
#include "halo_src.cuh"

namespace sb {
typedef __nv_bfloat16 bf16;

constexpr int CS_WPB = 4;                 // warps per block; they share nothing
constexpr int CS_MIN_ROWS = 16;

__device__ __forceinline__ void cs_copy(uint32_t dst, const void* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cs_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cs_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ uint2 cs_lds8(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint4 cs_lds16(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void cs_sts8(uint32_t a, uint32_t x, uint32_t y) {
  asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(a), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void cs_red4(float* p, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

// filter taps: fp32, or bf16 as the parameter stores them
struct CsTaps { const float* f; const bf16* h; };
__device__ __forceinline__ float cs_tap(const CsTaps& w, size_t i) { return w.h ? __bfloat162float(w.h[i]) : w.f[i]; }

// The run of this warp: batch row b, output rows [ra, rb)
struct CsRun { int b, ra, rb; };
__device__ __forceinline__ bool cs_run(int L, int t_min, int R, int nchunk, int B, CsRun& r) {
  const int i = blockIdx.y * CS_WPB + (threadIdx.x >> 5);
  if (i >= nchunk * B) return false;
  r.b = i / nchunk;
  r.ra = t_min + (i - r.b * nchunk) * R;
  r.rb = min(r.ra + R, L);
  return r.ra < r.rb;
}

// Rows of an unrolled body (a multiple of K, so that window slots are registers with fixed names) and of the ring (a multiple of
// that, so that ring slots are fixed offsets from one or two bases).
template <int K> constexpr int CS_U = K <= 4 ? 12 : K;
template <int K> constexpr int CS_RING = K <= 4 ? 12 : 2 * K;
template <bool V> struct CsBool { static constexpr bool value = V; };

// ------------------------------------------------------------------------------------ featuriser convolution
// Both kernels run most of a run in bodies without any check (the body's own rows, the rows it fetches and the rows it stores all lie
// inside the sequence); the first and last bodies of a run check every row.

// y[t] = sum_j w[j] x[t-(K-1)+j]: a lane owns 8 channels and copies them itself, so the ring needs no warp barrier either.
// wf: when not null the taps are also written there in fp32 (the backward's copy).
template <int K>
__global__ void __launch_bounds__(32 * CS_WPB, K <= 4 ? 3 : 2)
dwconv_fwd_stream_kernel(const bf16* __restrict__ x, const HaloSrc halo, const CsTaps w, float* __restrict__ wf,
                         bf16* __restrict__ y, int B, int L, int C, int R, int nchunk) {
  constexpr int H = K - 1, U = CS_U<K>, RING = CS_RING<K>, P = RING - 1;
  extern __shared__ __align__(16) uint4 cs_smem[];
  const int lane = threadIdx.x & 31, c0 = blockIdx.x * 256 + lane * 8;
  if (c0 >= C) return;
  if (wf && blockIdx.y == 0 && threadIdx.x < 32) {
    for (int i = 0; i < 8 * K; ++i) wf[(size_t)c0 * K + i] = cs_tap(w, (size_t)c0 * K + i);
  }
  CsRun r;
  if (!cs_run(L, 0, R, nchunk, B, r)) return;
  const uint32_t ring = (uint32_t)__cvta_generic_to_shared(cs_smem) + ((threadIdx.x >> 5) * RING * 32 + lane) * 16;
  const int t0 = r.ra - H, n_rows = r.rb - t0;
  const bf16* src = x + ((ptrdiff_t)r.b * L + t0) * C + c0;                 // next row to fetch
  auto fetch = [&](int n, uint32_t dst) {                // checked: row n of the run
    if (n < n_rows) {
      const int t = t0 + n;
      if (t >= 0) cs_copy(dst, src, true);
      else {
        const bf16* h = halo_row(halo, r.b, t + H, H, C);
        cs_copy(dst, h ? h + c0 : x, h != nullptr);
      }
      src += C;
    }
    cs_commit();
  };
#pragma unroll 1
  for (int n = 0; n < P; ++n) fetch(n, ring + n * 512);
  f2 wr[4][K], win[4][K];
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int j = 0; j < K; ++j) {
      wr[q][j] = f2_pack(cs_tap(w, (size_t)(c0 + 2 * q) * K + j), cs_tap(w, (size_t)(c0 + 2 * q + 1) * K + j));
      win[q][j] = 0;
    }
  bf16* out = y + ((size_t)r.b * L + r.ra) * C + c0;
  uint32_t cur = ring, oth = ring + (RING - U) * 512;
  auto body = [&](auto edge, int n0) {
    constexpr bool EDGE = decltype(edge)::value;
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const int n = n0 + k;
      if (EDGE && n >= n_rows) break;
      cs_wait<P - 1>();
      const uint4 v = cs_lds16(cur + k * 512);
      const uint32_t dst = k ? cur + (k - 1) * 512 : oth + (U - 1) * 512;   // row n - 1's slot: that row is in registers
      if (EDGE) fetch(n + P, dst);
      else { cs_copy(dst, src, true); cs_commit(); src += C; }
      win[0][k % K] = f2_bf(v.x); win[1][k % K] = f2_bf(v.y); win[2][k % K] = f2_bf(v.z); win[3][k % K] = f2_bf(v.w);
      if (EDGE && n < H) continue;
      f2 o[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        o[q] = f2_mul(wr[q][0], win[q][(k + 1) % K]);
#pragma unroll
        for (int j = 1; j < K; ++j) o[q] = f2_fma(wr[q][j], win[q][(k + 1 + j) % K], o[q]);
      }
      *reinterpret_cast<uint4*>(out) = make_uint4(pack_bf2(o[0]), pack_bf2(o[1]), pack_bf2(o[2]), pack_bf2(o[3]));
      out += C;
    }
    const uint32_t s = cur; cur = oth; oth = s;
  };
#pragma unroll 1
  for (int n0 = 0; n0 < n_rows; n0 += U) {
    if (n0 > 0 && n0 + U - 1 + P < n_rows) body(CsBool<false>{}, n0);
    else body(CsBool<true>{}, n0);
  }
}

// dx[t] = sum_j w[j] dy[t+(K-1)-j], dw[j] += sum_t dy[t] x[t-(K-1)+j].  A lane owns 4 channels; step n of a run brings row ra + n of dy
// and row ra + n - (K-1) of x, which is the pair of rows that output row ra + n - (K-1) completes with.
template <int K>
__global__ void __launch_bounds__(32 * CS_WPB, 2)
dwconv_bwd_stream_kernel(const bf16* __restrict__ x, const HaloSrc halo, const int has_halo, const float* __restrict__ w,
                         const bf16* __restrict__ dy, bf16* __restrict__ dx, bf16* __restrict__ dhalo, float* __restrict__ dw,
                         int B, int L, int C, int R, int nchunk, const int ahead_mode, const HaloSrc ahead) {
  constexpr int H = K - 1, U = CS_U<K>, RING = CS_RING<K>, P = RING - 1;
  extern __shared__ __align__(16) uint4 cs_smem[];
  const int lane = threadIdx.x & 31, cw = blockIdx.x * 128, c0 = cw + lane * 4;
  CsRun r;
  if (!cs_run(L, has_halo && !ahead_mode ? -H : 0, R, nchunk, B, r)) return;
  const bool live = c0 < C;
  // the copies of a row: lanes 0-15 the 256 bytes of x, lanes 16-31 those of dy
  const bool is_g = lane >= 16;
  const int cc = cw + (lane & 15) * 8;
  const bool cok = cc < C;
  const uint32_t ring = (uint32_t)__cvta_generic_to_shared(cs_smem) + (threadIdx.x >> 5) * RING * 512;
  const int n_rows = r.rb - r.ra + H;
  const bf16* src = (is_g ? dy : x) + ((ptrdiff_t)r.b * L + r.ra - (is_g ? 0 : H)) * C + cc;   // next row to fetch
  auto fetch = [&](int n, uint32_t dst) {
    if (n < n_rows) {
      const int t = r.ra + n - (is_g ? 0 : H);
      const bf16* e = nullptr;
      if (t >= 0 && t < L) e = src;
      else if (!is_g && t < 0 && t >= -H) { e = halo_row(halo, r.b, t + H, H, C); if (e) e += cc; }
      else if (is_g && t >= L && ahead_mode) { e = halo_row(ahead, r.b, t - L, H, C); if (e) e += cc; }
      const bool ok = cok && e;
      cs_copy(dst, ok ? e : x, ok);
      src += C;
    }
    cs_commit();
  };
#pragma unroll 1
  for (int n = 0; n < P; ++n) fetch(n, ring + n * 512 + lane * 16);
  f2 wr[2][K], xw[2][K], gw[2][K], acc[2][K];
#pragma unroll
  for (int q = 0; q < 2; ++q)
#pragma unroll
    for (int j = 0; j < K; ++j) {
      wr[q][j] = live ? f2_pack(w[(size_t)(c0 + 2 * q) * K + j], w[(size_t)(c0 + 2 * q + 1) * K + j]) : 0;
      xw[q][j] = 0; gw[q][j] = 0; acc[q][j] = 0;
    }
  bf16* out = dx + ((ptrdiff_t)r.b * L + r.ra) * C + c0;   // output row of step H
  uint32_t cur = ring, oth = ring + (RING - U) * 512;
  auto body = [&](auto edge, int n0) {
    constexpr bool EDGE = decltype(edge)::value;
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const int n = n0 + k;
      if (EDGE && n >= n_rows) break;
      cs_wait<P - 1>();
      __syncwarp();                                      // every lane's part of the row is there; the previous row is read
      const uint32_t dst = (k ? cur + (k - 1) * 512 : oth + (U - 1) * 512) + lane * 16;
      if (EDGE) fetch(n + P, dst);
      else { if (cok) cs_copy(dst, src, true); cs_commit(); src += C; }
      const uint2 xv = cs_lds8(cur + k * 512 + lane * 8), gv = cs_lds8(cur + k * 512 + lane * 8 + 256);
      xw[0][k % K] = f2_bf(xv.x); xw[1][k % K] = f2_bf(xv.y);
      gw[0][k % K] = f2_bf(gv.x); gw[1][k % K] = f2_bf(gv.y);
      if (EDGE && n < H) continue;
      f2 o[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const f2 g0 = gw[q][(k + 1) % K];
        o[q] = f2_mul(wr[q][0], gw[q][k % K]);
        acc[q][0] = f2_fma(g0, xw[q][(k + 1) % K], acc[q][0]);
#pragma unroll
        for (int j = 1; j < K; ++j) {
          o[q] = f2_fma(wr[q][j], gw[q][(k + K - j) % K], o[q]);
          acc[q][j] = f2_fma(g0, xw[q][(k + 1 + j) % K], acc[q][j]);
        }
      }
      const uint2 ov = make_uint2(pack_bf2(o[0]), pack_bf2(o[1]));
      if (EDGE) {
        const int t = r.ra + n - H;
        bf16* to = t >= 0 ? out : dhalo ? dhalo + ((size_t)r.b * H + (t + H)) * C + c0 : nullptr;
        if (to && live) *reinterpret_cast<uint2*>(to) = ov;
      } else if (live) *reinterpret_cast<uint2*>(out) = ov;
      out += C;
    }
    const uint32_t s = cur; cur = oth; oth = s;
  };
  const int n_fast = min(n_rows, L - r.ra);              // rows of dy inside the sequence
#pragma unroll 1
  for (int n0 = 0; n0 < n_rows; n0 += U) {
    if (n0 > 0 && n0 + U - 1 + P < n_fast && r.ra + n0 >= H) body(CsBool<false>{}, n0);
    else body(CsBool<true>{}, n0);
  }
  if (!live) return;
  float a[4 * K];                                        // taps of the four channels, as dw holds them
#pragma unroll
  for (int q = 0; q < 2; ++q)
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const float2 v = f2_unpack(acc[q][j]);
      a[2 * q * K + j] = v.x; a[(2 * q + 1) * K + j] = v.y;
    }
#pragma unroll
  for (int k = 0; k < K; ++k) cs_red4(dw + (size_t)c0 * K + 4 * k, a[4 * k], a[4 * k + 1], a[4 * k + 2], a[4 * k + 3]);
}

// ------------------------------------------------------------------------------------ Hyena-SE
constexpr int CE_FROW = 768;              // bytes of a staged feature row of 128 channels
constexpr int CE_BROW = 1024;             // and of one with the row of dz behind it
template <int K> constexpr int CE_U = K <= 3 ? 6 : K == 4 ? 8 : K;       // rows of a body of the backward; its ring has twice as many

// Taps of the four channels of a lane.  SHARED: they belong to one filter group.
template <int K, bool SHARED> struct CeTaps {
  f2 w[SHARED ? 1 : 2][K];
  __device__ __forceinline__ void load(const CsTaps& src, int c0, int D, int dg) {
#pragma unroll
    for (int q = 0; q < (SHARED ? 1 : 2); ++q) {
      const int a = min(c0 + 2 * q, D - 1), b = SHARED ? a : min(c0 + 2 * q + 1, D - 1);
#pragma unroll
      for (int j = 0; j < K; ++j) w[q][j] = f2_pack(cs_tap(src, (size_t)(a / dg) * K + j), cs_tap(src, (size_t)(b / dg) * K + j));
    }
  }
  __device__ __forceinline__ f2 operator()(int q, int j) const { return w[SHARED ? 0 : q][j]; }
};

__device__ __forceinline__ void ce_feat(uint32_t a, FeatPair& p, FeatPair& q) {
  const uint2 u = cs_lds8(a), v = cs_lds8(a + 8), w = cs_lds8(a + 16);
  p = feat_pair(u.x, u.y, v.x);
  q = feat_pair(v.y, w.x, w.y);
}

// z[t] = x1[t] * sum_j w[j] u[t-(K-1)+j], u = x2 * v (pre, post: with or without the two gates)
template <int K, bool SHARED>
__global__ void __launch_bounds__(32 * CS_WPB, 3)
se_fwd_stream_kernel(const bf16* __restrict__ feat, const HaloSrc halo, const CsTaps w, float* __restrict__ wf, int G,
                     bf16* __restrict__ z, int B, int L, int D, int dg, int R, int nchunk, const int pre, const int post) {
  constexpr int H = K - 1, U = CS_U<K>, RING = CS_RING<K>, P = RING - 1;
  extern __shared__ __align__(16) uint4 cs_smem[];
  const int lane = threadIdx.x & 31, cw = blockIdx.x * 128, c0 = cw + lane * 4;
  if (wf && blockIdx.y == 0) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < G * K; i += gridDim.x * blockDim.x) wf[i] = cs_tap(w, i);
  }
  CsRun r;
  if (!cs_run(L, 0, R, nchunk, B, r)) return;
  const bool live = c0 < D;
  const int W = 3 * D;
  const int e0 = 3 * cw + lane * 8;                      // this lane's two 16-byte pieces of a row (48 pieces in all)
  const bool ok0 = e0 < W, ok1 = lane < 16 && e0 + 256 < W;
  const uint32_t ring = (uint32_t)__cvta_generic_to_shared(cs_smem) + (threadIdx.x >> 5) * RING * CE_FROW;
  const int t0 = r.ra - H, n_rows = r.rb - t0;
  const bf16* src = feat + ((ptrdiff_t)r.b * L + t0) * W + e0;              // next row to fetch
  auto fetch = [&](int n, uint32_t dst) {
    if (n < n_rows) {
      const int t = t0 + n;
      const bf16* e = src;
      if (t < 0) { e = halo_row(halo, r.b, t + H, H, W); if (e) e += e0; }
      cs_copy(dst, e && ok0 ? e : feat, e && ok0);
      if (lane < 16) cs_copy(dst + 512, e && ok1 ? e + 256 : feat, e && ok1);
      src += W;
    }
    cs_commit();
  };
#pragma unroll 1
  for (int n = 0; n < P; ++n) fetch(n, ring + n * CE_FROW + lane * 16);
  CeTaps<K, SHARED> wr;
  wr.load(w, c0, D, dg);
  f2 uw[2][K];
#pragma unroll
  for (int j = 0; j < K; ++j) { uw[0][j] = 0; uw[1][j] = 0; }
  bf16* out = z + ((size_t)r.b * L + r.ra) * D + c0;
  uint32_t cur = ring, oth = ring + (RING - U) * CE_FROW;
  auto body = [&](auto edge, int n0) {
    constexpr bool EDGE = decltype(edge)::value;
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const int n = n0 + k;
      if (EDGE && n >= n_rows) break;
      cs_wait<P - 1>();
      __syncwarp();
      const uint32_t dst = (k ? cur + (k - 1) * CE_FROW : oth + (U - 1) * CE_FROW) + lane * 16;
      if (EDGE) fetch(n + P, dst);
      else {
        if (ok0) cs_copy(dst, src, true);
        if (ok1) cs_copy(dst + 512, src + 256, true);
        cs_commit();
        src += W;
      }
      FeatPair f[2];
      ce_feat(cur + k * CE_FROW + lane * 24, f[0], f[1]);
#pragma unroll
      for (int q = 0; q < 2; ++q) uw[q][k % K] = pre ? f2_mul(f[q].x2, f[q].v) : f[q].v;
      if (EDGE && n < H) continue;
      f2 o[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        o[q] = f2_mul(wr(q, 0), uw[q][(k + 1) % K]);
#pragma unroll
        for (int j = 1; j < K; ++j) o[q] = f2_fma(wr(q, j), uw[q][(k + 1 + j) % K], o[q]);
        if (post) o[q] = f2_mul(f[q].x1, o[q]);
      }
      if (live) *reinterpret_cast<uint2*>(out) = make_uint2(pack_bf2(o[0]), pack_bf2(o[1]));
      out += D;
    }
    const uint32_t s = cur; cur = oth; oth = s;
  };
#pragma unroll 1
  for (int n0 = 0; n0 < n_rows; n0 += U) {
    if (n0 > 0 && n0 + U - 1 + P < n_rows) body(CsBool<false>{}, n0);
    else body(CsBool<true>{}, n0);
  }
}

// Row s of features and dz arrives with step n = s - ra; the step completes output row s - (K-1), whose features and dz are still
// in the ring:
//   conv[t] = sum_j w[j] u[t-(K-1)+j]            dx1 = dz * conv
//   du[t]   = sum_j w[j] dconv[t+(K-1)-j]        dx2 = du * v, dv = du * x2            (dconv = dz * x1)
//   dw[j]  += dconv[t] u[t-(K-1)+j]
// The results overwrite the row's features in the ring and leave one step later, after the warp barrier, as 16-byte stores.
template <int K, bool SHARED>
__global__ void __launch_bounds__(32 * CS_WPB, 2)
se_bwd_stream_kernel(const bf16* __restrict__ feat, const HaloSrc halo, const int has_halo, const float* __restrict__ w,
                     const bf16* __restrict__ dz, bf16* __restrict__ dfeat, bf16* __restrict__ dhalo, float* __restrict__ dw,
                     int B, int L, int D, int dg, int R, int nchunk, const int pre, const int post, const int ahead_mode,
                     const HaloSrc ahead_f, const HaloSrc ahead_g) {
  constexpr int H = K - 1, U = CE_U<K>, RING = 2 * U, P = RING - K - 1;
  static_assert(U % K == 0 && P >= 1, "window and ring slots of a body are at fixed places");
  extern __shared__ __align__(16) uint4 cs_smem[];
  const int lane = threadIdx.x & 31, cw = blockIdx.x * 128, c0 = cw + lane * 4;
  CsRun r;
  if (!cs_run(L, has_halo && !ahead_mode ? -H : 0, R, nchunk, B, r)) return;
  const bool live = c0 < D;
  const int W = 3 * D;
  // 64 pieces of 16 bytes per row: 48 of the features, 16 of dz; this lane's first is always features
  const bool g2 = lane >= 16;
  const int e0 = 3 * cw + lane * 8, e1 = g2 ? cw + (lane - 16) * 8 : e0 + 256, ld1 = g2 ? D : W;
  const bool ok0 = e0 < W, ok1 = e1 < ld1;
  const uint32_t ring = (uint32_t)__cvta_generic_to_shared(cs_smem) + (threadIdx.x >> 5) * RING * CE_BROW;
  const int t0 = r.ra - H, n_rows = r.rb + H - t0;       // rows ra - H .. rb + H - 1; row q of the run is t0 + q
  const bf16* s0 = feat + ((ptrdiff_t)r.b * L + t0) * W + e0;               // next row to fetch, both pieces
  const bf16* s1 = (g2 ? dz : feat) + ((ptrdiff_t)r.b * L + t0) * ld1 + e1;
  auto fetch = [&](int q, uint32_t dst) {
    if (q < n_rows) {
      const int t = t0 + q;
      const bf16 *a = nullptr, *c = nullptr;
      if (t >= 0 && t < L) { a = s0; c = s1; }
      else {
        const bf16 *ef = nullptr, *eg = nullptr;
        if (t < 0 && t >= -H) ef = halo_row(halo, r.b, t + H, H, W);
        else if (t >= L && ahead_mode) { ef = halo_row(ahead_f, r.b, t - L, H, W); eg = halo_row(ahead_g, r.b, t - L, H, D); }
        if (ef) a = ef + e0;
        if (g2 ? eg : ef) c = (g2 ? eg : ef) + e1;
      }
      cs_copy(dst, a && ok0 ? a : feat, a && ok0);
      cs_copy(dst + 512, c && ok1 ? c : feat, c && ok1);
      s0 += W; s1 += ld1;
    }
    cs_commit();
  };
#pragma unroll 1
  for (int q = 0; q < H + P; ++q) fetch(q, ring + q * CE_BROW + lane * 16);
  CeTaps<K, SHARED> wr;
  wr.load(CsTaps{w, nullptr}, c0, D, dg);
  f2 uw[2][K], gw[2][K], acc[SHARED ? 1 : 2][K];
#pragma unroll
  for (int j = 0; j < K; ++j) {
    uw[0][j] = 0; uw[1][j] = 0; gw[0][j] = 0; gw[1][j] = 0; acc[0][j] = 0;
    if constexpr (!SHARED) acc[1][j] = 0;
  }
  bf16* out = dfeat + ((ptrdiff_t)r.b * L + r.ra) * W + e0;                 // next gradient row to leave
  const bool tail = lane < 16 && ok1;
  auto flush = [&](bf16* to, uint32_t s) {
    if (ok0) *reinterpret_cast<uint4*>(to) = cs_lds16(s + lane * 16);
    if (tail) *reinterpret_cast<uint4*>(to + 256) = cs_lds16(s + 512 + lane * 16);
  };
  auto flush_checked = [&](int t, uint32_t s) {
    if (t >= 0) flush(out, s);
    else if (dhalo) flush(dhalo + ((size_t)r.b * H + (t + H)) * W + e0, s);
    out += W;
  };
  const int n_steps = r.rb - r.ra + H;
  uint32_t cur = ring, oth = ring + U * CE_BROW;
  auto body = [&](auto edge, int n0) {
    constexpr bool EDGE = decltype(edge)::value;
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const int n = n0 + k;                              // new row n + H of the run, output row n
      if (EDGE && n >= n_steps) break;
      cs_wait<P - 1>();
      __syncwarp();                                      // row n + H is complete, the results of row n - 1 too, row n - 2 has left
      const uint32_t dst = (k >= 2 ? cur + (k - 2) * CE_BROW : oth + (U - 2 + k) * CE_BROW) + lane * 16;
      const uint32_t done = k >= 1 ? cur + (k - 1) * CE_BROW : oth + (U - 1) * CE_BROW;
      if (EDGE) {
        fetch(n + H + P, dst);
        if (n > H) flush_checked(t0 + n - 1, done);
      } else {
        if (ok0) cs_copy(dst, s0, true);
        if (ok1) cs_copy(dst + 512, s1, true);
        cs_commit();
        s0 += W; s1 += ld1;
        flush(out, done);
        out += W;
      }
      const uint32_t sn = k + H < U ? cur + (k + H) * CE_BROW : oth + (k + H - U) * CE_BROW, so = cur + k * CE_BROW;
      FeatPair f[2];
      {
        const uint2 gv = cs_lds8(sn + CE_FROW + lane * 8);
        gw[0][k % K] = f2_bf(gv.x); gw[1][k % K] = f2_bf(gv.y);
        if (post) {
          ce_feat(sn + lane * 24, f[0], f[1]);
          gw[0][k % K] = f2_mul(gw[0][k % K], f[0].x1); gw[1][k % K] = f2_mul(gw[1][k % K], f[1].x1);
        }
      }
      ce_feat(so + lane * 24, f[0], f[1]);
#pragma unroll
      for (int q = 0; q < 2; ++q) uw[q][k % K] = pre ? f2_mul(f[q].x2, f[q].v) : f[q].v;
      if (EDGE && n < H) continue;
      const uint2 gv = cs_lds8(so + CE_FROW + lane * 8);
      uint32_t o[6];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const f2 g = f2_bf(q ? gv.y : gv.x), g0 = gw[q][(k + 1) % K];
        f2 conv = f2_mul(wr(q, 0), uw[q][(k + 1) % K]), du = f2_mul(wr(q, 0), gw[q][k % K]);
        f2& a0 = acc[SHARED ? 0 : q][0];
        a0 = f2_fma(g0, uw[q][(k + 1) % K], a0);
#pragma unroll
        for (int j = 1; j < K; ++j) {
          conv = f2_fma(wr(q, j), uw[q][(k + 1 + j) % K], conv);
          du = f2_fma(wr(q, j), gw[q][(k + K - j) % K], du);
          f2& aj = acc[SHARED ? 0 : q][j];
          aj = f2_fma(g0, uw[q][(k + 1 + j) % K], aj);
        }
        const float2 a = f2_unpack(post ? f2_mul(g, conv) : 0), b = f2_unpack(pre ? f2_mul(du, f[q].v) : 0),
                     c = f2_unpack(pre ? f2_mul(du, f[q].x2) : du);
        o[3 * q] = pack_bf2(a.x, b.x); o[3 * q + 1] = pack_bf2(c.x, a.y); o[3 * q + 2] = pack_bf2(b.y, c.y);
      }
#pragma unroll
      for (int k2 = 0; k2 < 3; ++k2) cs_sts8(so + lane * 24 + k2 * 8, o[2 * k2], o[2 * k2 + 1]);
    }
    const uint32_t s = cur; cur = oth; oth = s;
  };
  const int q_fast = min(n_rows, L - t0);                // rows inside the sequence
#pragma unroll 1
  for (int n0 = 0; n0 < n_steps; n0 += U) {
    if (n0 >= K && n0 + U - 1 + H + P < q_fast && t0 + n0 > 0) body(CsBool<false>{}, n0);
    else body(CsBool<true>{}, n0);
  }
  __syncwarp();
  flush_checked(t0 + n_steps - 1, ring + ((n_steps - 1) % RING) * CE_BROW);  // the last row's results
  // filter gradient: over the channels of the lane, then over the lanes of one group, then one atomic per tap
  if constexpr (SHARED) {
    const int lpg = dg >> 2;                             // lanes per group
    const int span = dg % 128 == 0 ? 32 : ((lpg & (lpg - 1)) == 0 && lpg <= 32) ? lpg : 1;
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const float2 v = f2_unpack(acc[0][j]);
      float s = live ? v.x + v.y : 0.f;
      for (int o = span >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (live && (lane & (span - 1)) == 0) atomicAdd(dw + (size_t)(c0 / dg) * K + j, s);
    }
  } else if (live) {
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int j = 0; j < K; ++j) {
        const float2 v = f2_unpack(acc[q][j]);
        atomicAdd(dw + (size_t)((c0 + 2 * q) / dg) * K + j, v.x);
        atomicAdd(dw + (size_t)((c0 + 2 * q + 1) / dg) * K + j, v.y);
      }
  }
}

// Rows per run and runs per batch row for `steps` output rows of B batch rows in `cols` strips, when a wave holds `blocks` blocks per SM.
static inline int cs_rows(int B, int steps, int cols, int blocks, int& nchunk) {
  const long long runs = (long long)sb::num_sms() * blocks / cols * CS_WPB / B;   // whole blocks that fit the wave, per batch row
  long long r = runs > 0 ? (steps + runs - 1) / runs : steps;
  if (r < CS_MIN_ROWS) r = CS_MIN_ROWS;
  nchunk = (int)((steps + r - 1) / r);
  return (int)r;
}

}  // namespace sb
