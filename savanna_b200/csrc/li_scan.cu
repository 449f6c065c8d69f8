// Hyena-LI with the implicit modal filter, evaluated as what it is: an order-O diagonal linear recurrence.
//
//   h[d,t] = sum_o R[d,o] lam[d,o]^t          =>   s_o[t] = lam_o s_o[t-1] + u[t],   y[t] = sum_o R_o s_o[t] + bias u[t]
//   u = x2 * v,  z = x1 * y                        (features interleaved (x1,x2,v), channel-last bf16, fp32 state)
//
// The sequence is cut into chunks of TC steps that run in parallel (chunked scan):
//   1. local   : every chunk runs from a zero state and stores its end state          [B, NC, D, O]
//   2. prefix  : per (b, d, o) a serial pass over the NC chunk states turns them into the state ENTERING each chunk
//   3. apply   : every chunk reruns from its entering state and writes z
// so the cost is two streaming reads of the features and one write of z, instead of the size-2L fp32 FFTs the
// filter's materialised form needs.  The backward pass uses the same structure twice: a forward scan of the state s and its
// sensitivity w = ds/dlam (gradients of R, lam, bias and dx1), and a reverse scan of the adjoint a[t] = R dy[t] + lam a[t+1]
// (gradients of x2 and v).  `state_in` / `state_out` expose the recurrence state at the shard boundaries, which is all context
// parallelism needs to hand over.  O is padded to 16 (lam = 0, R = 0 beyond the real order).
//
// Two sets of kernels: first the per-thread ones (any D, any alignment; also the context-parallel scan at the end of the file), in
// which one thread owns one channel, its O states in registers, and a warp reads 32 channels x 3 features = 192 contiguous bytes
// per time step; then the tiled ones (D % 8 == 0, 16-byte aligned tensors), which are the ones that normally run.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "device_info.h"
#include "entries.h"
#include "f32x2.cuh"
#include "pdl.cuh"

namespace sb {
typedef __nv_bfloat16 bf16;
constexpr int LO = 16;            // padded filter order
constexpr int LI_THREADS = 128;

__device__ __forceinline__ float b2f(const bf16 v) { return __bfloat162float(v); }

struct LiDims { int B, L, D, TC, NC; };

__device__ __forceinline__ void load_vec16(const float* p, float (&r)[LO]) {
  const float4* q = reinterpret_cast<const float4*>(p);
#pragma unroll
  for (int i = 0; i < LO / 4; ++i) { float4 t = q[i]; r[4 * i] = t.x; r[4 * i + 1] = t.y; r[4 * i + 2] = t.z; r[4 * i + 3] = t.w; }
}
__device__ __forceinline__ void store_vec16(float* p, const float (&r)[LO]) {
  float4* q = reinterpret_cast<float4*>(p);
#pragma unroll
  for (int i = 0; i < LO / 4; ++i) q[i] = make_float4(r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
}

// ------------------------------------------------------------------------------------ forward
// pass 1: chunk-local end state from a zero state
__global__ void __launch_bounds__(LI_THREADS)
li_local_kernel(const bf16* __restrict__ feat, const float* __restrict__ loglam, float* __restrict__ Sloc, LiDims d) {
  const int ch = blockIdx.x * LI_THREADS + threadIdx.x;
  if (ch >= d.D) return;
  const int n = blockIdx.y, b = blockIdx.z;
  float lam[LO], s[LO];
  load_vec16(loglam + (size_t)ch * LO, lam);
#pragma unroll
  for (int o = 0; o < LO; ++o) { lam[o] = __expf(lam[o]); s[o] = 0.f; }
  const int t0 = n * d.TC, t1 = min(t0 + d.TC, d.L);
  const bf16* f = feat + ((size_t)b * d.L + t0) * 3 * d.D + 3 * ch;
#pragma unroll 8
  for (int t = t0; t < t1; ++t, f += 3 * d.D) {
    const float u = b2f(f[1]) * b2f(f[2]);
#pragma unroll
    for (int o = 0; o < LO; ++o) s[o] = lam[o] * s[o] + u;
  }
  store_vec16(Sloc + (((size_t)b * d.NC + n) * d.D + ch) * LO, s);
}

// pass 2: exclusive prefix over chunks, in place: S[n] <- state entering chunk n.  One thread per (b, ch, o).
// Chunks are full (TC steps) except possibly the last one, whose end state only feeds state_out.
__global__ void li_prefix_kernel(float* __restrict__ S, const float* __restrict__ loglam, const float* __restrict__ state_in,
                                 float* __restrict__ state_out, LiDims d) {
  const size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  const size_t per_b = (size_t)d.D * LO;
  if (idx >= (size_t)d.B * per_b) return;
  const int b = idx / per_b;
  const size_t r = idx - (size_t)b * per_b;               // ch * LO + o
  const float ll = loglam[r];
  const float step = __expf(ll * d.TC);
  float carry = state_in ? state_in[idx] : 0.f;
  float* p = S + (size_t)b * d.NC * per_b + r;
  // the chunk states are independent loads: fetch eight ahead, then run the serial carry over them
  for (int n0 = 0; n0 < d.NC; n0 += 8) {
    float loc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) loc[j] = n0 + j < d.NC ? p[(size_t)(n0 + j) * per_b] : 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int n = n0 + j;
      if (n < d.NC) {
        p[(size_t)n * per_b] = carry;
        const int len = min(d.TC, d.L - n * d.TC);
        const float st = len == d.TC ? step : __expf(ll * len);
        carry = st * carry + loc[j];
      }
    }
  }
  if (state_out) state_out[idx] = carry;
}

// pass 3: rerun each chunk from its entering state and emit z
__global__ void __launch_bounds__(LI_THREADS)
li_apply_kernel(const bf16* __restrict__ feat, const float* __restrict__ loglam, const float* __restrict__ R,
                const float* __restrict__ bias, const float* __restrict__ Sin, bf16* __restrict__ z, LiDims d) {
  const int ch = blockIdx.x * LI_THREADS + threadIdx.x;
  if (ch >= d.D) return;
  const int n = blockIdx.y, b = blockIdx.z;
  float lam[LO], s[LO], rr[LO];
  load_vec16(loglam + (size_t)ch * LO, lam);
  load_vec16(R + (size_t)ch * LO, rr);
  load_vec16(Sin + (((size_t)b * d.NC + n) * d.D + ch) * LO, s);
#pragma unroll
  for (int o = 0; o < LO; ++o) lam[o] = __expf(lam[o]);
  const float be = bias[ch];
  const int t0 = n * d.TC, t1 = min(t0 + d.TC, d.L);
  const bf16* f = feat + ((size_t)b * d.L + t0) * 3 * d.D + 3 * ch;
  bf16* zo = z + ((size_t)b * d.L + t0) * d.D + ch;
#pragma unroll 8
  for (int t = t0; t < t1; ++t, f += 3 * d.D, zo += d.D) {
    const float x1 = b2f(f[0]);
    const float u = b2f(f[1]) * b2f(f[2]);
    float y = be * u;
#pragma unroll
    for (int o = 0; o < LO; ++o) { s[o] = lam[o] * s[o] + u; y += rr[o] * s[o]; }
    *zo = __float2bfloat16_rn(x1 * y);
  }
}

// ------------------------------------------------------------------------------------ backward
// pass B1: chunk-local quantities from zero states:
//   Sloc  end state;  Wloc end sensitivity (w[t] = s[t-1] + lam w[t-1]);
//   Aloc  adjoint leaving the chunk on its left edge: sum_t lam^(t-t0) R dy[t], dy = dz * x1
__global__ void __launch_bounds__(LI_THREADS)
li_bwd_local_kernel(const bf16* __restrict__ feat, const bf16* __restrict__ dz, const float* __restrict__ loglam,
                    const float* __restrict__ R, float* __restrict__ Sloc, float* __restrict__ Wloc,
                    float* __restrict__ Aloc, LiDims d) {
  const int ch = blockIdx.x * LI_THREADS + threadIdx.x;
  if (ch >= d.D) return;
  const int n = blockIdx.y, b = blockIdx.z;
  float lam[LO], s[LO], w[LO], pw[LO], a[LO];
  load_vec16(loglam + (size_t)ch * LO, lam);
#pragma unroll
  for (int o = 0; o < LO; ++o) { lam[o] = __expf(lam[o]); s[o] = 0.f; w[o] = 0.f; pw[o] = 1.f; a[o] = 0.f; }
  const int t0 = n * d.TC, t1 = min(t0 + d.TC, d.L);
  const bf16* f = feat + ((size_t)b * d.L + t0) * 3 * d.D + 3 * ch;
  const bf16* g = dz + ((size_t)b * d.L + t0) * d.D + ch;
#pragma unroll 4
  for (int t = t0; t < t1; ++t, f += 3 * d.D, g += d.D) {
    const float u = b2f(f[1]) * b2f(f[2]);
    const float dy = b2f(*g) * b2f(f[0]);
#pragma unroll
    for (int o = 0; o < LO; ++o) {
      w[o] = s[o] + lam[o] * w[o];
      s[o] = lam[o] * s[o] + u;
      a[o] += pw[o] * dy;
      pw[o] *= lam[o];
    }
  }
  float rr[LO];
  load_vec16(R + (size_t)ch * LO, rr);
#pragma unroll
  for (int o = 0; o < LO; ++o) a[o] *= rr[o];
  const size_t off = (((size_t)b * d.NC + n) * d.D + ch) * LO;
  store_vec16(Sloc + off, s);
  store_vec16(Wloc + off, w);
  store_vec16(Aloc + off, a);
}

// pass B2: (S, W) exclusive prefix (forward), A exclusive suffix (reverse), in place.
//   S_in[n+1] = lam^len S_in[n] + Sloc[n]
//   W_in[n+1] = lam^len W_in[n] + len lam^(len-1) S_in[n] + Wloc[n]
//   A_in[n-1] = lam^len(n) A_in[n] + Aloc[n]          (A_in[n] = adjoint at the right edge of chunk n)
// Also: w_end (sensitivity of the final state), dstate_in = lam * (adjoint at t = 0).
__global__ void li_bwd_prefix_kernel(float* __restrict__ S, float* __restrict__ W, float* __restrict__ A,
                                     const float* __restrict__ loglam, const float* __restrict__ state_in,
                                     const float* __restrict__ dstate_out, float* __restrict__ w_end,
                                     float* __restrict__ dstate_in, LiDims d) {
  const size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  const size_t per_b = (size_t)d.D * LO;
  if (idx >= (size_t)d.B * per_b) return;
  const int b = idx / per_b;
  const size_t r = idx - (size_t)b * per_b;
  const float ll = loglam[r];
  const size_t base = (size_t)b * d.NC * per_b + r;
  float cs = state_in ? state_in[idx] : 0.f, cw = 0.f;
  const float st_full = __expf(ll * d.TC), stm1_full = __expf(ll * (d.TC - 1));
  // independent loads of eight chunks ahead of the serial carries (forward for S and W, backward for A)
  for (int n0 = 0; n0 < d.NC; n0 += 8) {
    float ls[8], lw[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const size_t o = base + (size_t)(n0 + j) * per_b;
      ls[j] = n0 + j < d.NC ? S[o] : 0.f;
      lw[j] = n0 + j < d.NC ? W[o] : 0.f;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int n = n0 + j;
      if (n < d.NC) {
        const size_t o = base + (size_t)n * per_b;
        S[o] = cs; W[o] = cw;
        const int len = min(d.TC, d.L - n * d.TC);
        const float st = len == d.TC ? st_full : __expf(ll * len);
        const float stm1 = len == d.TC ? stm1_full : __expf(ll * (len - 1));
        cw = st * cw + len * stm1 * cs + lw[j];
        cs = st * cs + ls[j];
      }
    }
  }
  if (w_end) w_end[idx] = cw;
  // The gradient of the returned state, g = dL/ds[L-1], enters the adjoint at the LAST step without a factor lam
  // (a[L-1] = R dy[L-1] + g): the last chunk therefore starts from a zero adjoint, the reverse kernel adds g at its first
  // step, and the carry into the chunk before it picks up lam^(len-1) g.
  const float gout = dstate_out ? dstate_out[idx] : 0.f;
  float ca = 0.f;
  for (int n0 = d.NC - 1; n0 >= 0; n0 -= 8) {
    float la[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) la[j] = n0 - j >= 0 ? A[base + (size_t)(n0 - j) * per_b] : 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int n = n0 - j;
      if (n >= 0) {
        A[base + (size_t)n * per_b] = ca;
        const int len = min(d.TC, d.L - n * d.TC);
        ca = (len == d.TC ? st_full : __expf(ll * len)) * ca + la[j];
        if (n == d.NC - 1 && gout != 0.f) ca += (len == d.TC ? stm1_full : __expf(ll * (len - 1))) * gout;
      }
    }
  }
  if (dstate_in) dstate_in[idx] = __expf(ll) * ca;
}

// pass B3 (forward direction): y, dx1 = dz*y (into tmp), and per-chunk partial sums of dR, dlam, dbias
__global__ void __launch_bounds__(LI_THREADS)
li_bwd_apply_fwd_kernel(const bf16* __restrict__ feat, const bf16* __restrict__ dz, const float* __restrict__ loglam,
                        const float* __restrict__ R, const float* __restrict__ bias, const float* __restrict__ Sin,
                        const float* __restrict__ Win, bf16* __restrict__ dx1, float* __restrict__ dRp,
                        float* __restrict__ dLp, float* __restrict__ dBp, LiDims d) {
  const int ch = blockIdx.x * LI_THREADS + threadIdx.x;
  if (ch >= d.D) return;
  const int n = blockIdx.y, b = blockIdx.z;
  float lam[LO], s[LO], w[LO], rr[LO], dr[LO], dl[LO];
  const size_t off = (((size_t)b * d.NC + n) * d.D + ch) * LO;
  load_vec16(loglam + (size_t)ch * LO, lam);
  load_vec16(R + (size_t)ch * LO, rr);
  load_vec16(Sin + off, s);
  load_vec16(Win + off, w);
#pragma unroll
  for (int o = 0; o < LO; ++o) { lam[o] = __expf(lam[o]); dr[o] = 0.f; dl[o] = 0.f; }
  const float be = bias[ch];
  float db = 0.f;
  const int t0 = n * d.TC, t1 = min(t0 + d.TC, d.L);
  const bf16* f = feat + ((size_t)b * d.L + t0) * 3 * d.D + 3 * ch;
  const bf16* g = dz + ((size_t)b * d.L + t0) * d.D + ch;
  bf16* o1 = dx1 + ((size_t)b * d.L + t0) * d.D + ch;
#pragma unroll 4
  for (int t = t0; t < t1; ++t, f += 3 * d.D, g += d.D, o1 += d.D) {
    const float x1 = b2f(f[0]);
    const float u = b2f(f[1]) * b2f(f[2]);
    const float gz = b2f(*g);
    const float dy = gz * x1;
    float y = be * u;
#pragma unroll
    for (int o = 0; o < LO; ++o) {
      w[o] = s[o] + lam[o] * w[o];
      s[o] = lam[o] * s[o] + u;
      y += rr[o] * s[o];
      dr[o] += dy * s[o];
      dl[o] += dy * w[o];
    }
    db += dy * u;
    *o1 = __float2bfloat16_rn(gz * y);
  }
#pragma unroll
  for (int o = 0; o < LO; ++o) dl[o] *= rr[o];
  store_vec16(dRp + off, dr);
  store_vec16(dLp + off, dl);
  dBp[((size_t)b * d.NC + n) * d.D + ch] = db;
}

// pass R3 (reverse direction): adjoint scan, writes the full interleaved gradient (dx1 from tmp)
__global__ void __launch_bounds__(LI_THREADS)
li_bwd_apply_rev_kernel(const bf16* __restrict__ feat, const bf16* __restrict__ dz, const float* __restrict__ loglam,
                        const float* __restrict__ R, const float* __restrict__ bias, const float* __restrict__ Ain,
                        const bf16* __restrict__ dx1, bf16* __restrict__ dfeat, const float* __restrict__ dstate_out,
                        LiDims d) {
  const int ch = blockIdx.x * LI_THREADS + threadIdx.x;
  if (ch >= d.D) return;
  const int n = blockIdx.y, b = blockIdx.z;
  float lam[LO], a[LO], rr[LO];
  load_vec16(loglam + (size_t)ch * LO, lam);
  load_vec16(R + (size_t)ch * LO, rr);
  load_vec16(Ain + (((size_t)b * d.NC + n) * d.D + ch) * LO, a);
#pragma unroll
  for (int o = 0; o < LO; ++o) lam[o] = __expf(lam[o]);
  const float be = bias[ch];
  const int t0 = n * d.TC, t1 = min(t0 + d.TC, d.L);
  const bf16* f = feat + ((size_t)b * d.L + (t1 - 1)) * 3 * d.D + 3 * ch;
  const bf16* g = dz + ((size_t)b * d.L + (t1 - 1)) * d.D + ch;
  const bf16* i1 = dx1 + ((size_t)b * d.L + (t1 - 1)) * d.D + ch;
  bf16* df = dfeat + ((size_t)b * d.L + (t1 - 1)) * 3 * d.D + 3 * ch;
  const bool tail = dstate_out != nullptr && n == d.NC - 1;       // the chunk that ends the sequence: see li_bwd_prefix_kernel
  float gs[LO];
  if (tail) load_vec16(dstate_out + ((size_t)b * d.D + ch) * LO, gs);
#pragma unroll 8
  for (int t = t1 - 1; t >= t0; --t, f -= 3 * d.D, g -= d.D, i1 -= d.D, df -= 3 * d.D) {
    const float x1 = b2f(f[0]), x2 = b2f(f[1]), v = b2f(f[2]);
    const float dy = b2f(*g) * x1;
    float du = be * dy;
#pragma unroll
    for (int o = 0; o < LO; ++o) { a[o] = rr[o] * dy + lam[o] * a[o]; }
    if (tail && t == t1 - 1) {
#pragma unroll
      for (int o = 0; o < LO; ++o) a[o] += gs[o];
    }
#pragma unroll
    for (int o = 0; o < LO; ++o) du += a[o];
    df[0] = *i1;
    df[1] = __float2bfloat16_rn(du * v);
    df[2] = __float2bfloat16_rn(du * x2);
  }
}

// ------------------------------------------------------------------------------------ tiled kernels
// The kernels above walk the sequence with 2-byte loads at a stride of a whole row: a warp moves 192 useful bytes per
// step with 96 load instructions, and the time loop waits on them.  The tiled kernels below (D % 8 == 0, 16-byte aligned
// tensors) stage rows of the interleaved features in shared memory with 16-byte asynchronous copies and run the
// recurrences out of it.
//
// One thread owns TWO neighbouring channels and carries every fp32 quantity as a (channel, channel + 1) pair in a 64-bit
// register, so each recurrence step is one packed `fma.rn.f32x2`.  With one channel per thread these kernels were bound
// by shared memory: the three 2-byte reads of an interleaved (x1, x2, v) triple hit 16 of the 32 banks twice.  The pair's
// 12 bytes are three 32-bit words at a stride of three words between lanes - every bank once - and the word layout
// (x1 x2 | v x1 | x2 v) unpacks with one shift or mask per value.
//   forward   local / apply: a ring of LV_STAGES tiles of LV_ROWS steps, any chunk length; z leaves straight from
//             registers (a warp stores 128 contiguous bytes per step)
//   backward  chunks of LB_TC steps resident in shared memory.  `li_bwd_local`: two warps run the state forward, two the
//             adjoint backward.  `li_bwd_apply`: three roles of two warps share the staged chunk: (1) y, dx1 and the dR
//             partials, (2) the dlam partials, (3) the adjoint, dx2 and dv.
// The backward carries the adjoint without the residues, ah[t] = dy[t] + lam ah[t+1] (a = R ah; one FMA less per mode and
// step), and takes the pole gradient chunk by chunk from the sensitivity w[t] = ds[t]/dlam WITHIN the chunk (w = 0 at its
// left edge):
//     dlam = R ( sum_t dy[t] w[t] + lam ah(right edge) w(last step) ),
// the second term being what the chunk's end state still does to the rest of the sequence.  So no sensitivity is passed
// between chunks: the prefix pass carries two arrays instead of three.
//
// Measured at B = 1, L = 8192, D = 4096 on a B200 (us; in brackets the one-channel-per-thread kernels these replace):
// forward 43 + 10 + 81 (55 + 29 + 95), backward 80 + 36 + 272 + 18 (143 + 156 + 319 and about ten tensor operations that
// prepared the filter and summed the partials).  Forward and backward with their host side: 849 -> 552.  The recurrences
// need 48 FMA per value forward and 144 backward, 54 and 163 us at the 30 TFMA/s that packed and plain FMA both reach here
// (the packed form only halves the issue slots), so the sweeps sit between that bound and the copy time of their data.
constexpr int LV_CH = 128;               // channels per block
constexpr int LV_PAIRS = LV_CH / 2;      // threads of one role
constexpr int LV_ROWS = 16;              // steps per ring tile (forward)
constexpr int LV_STAGES = 3;
constexpr int LB_TC = 64;                // chunk length of the backward
constexpr int LV_FW = 3 * LV_CH / 2;     // 32-bit words per staged feature row
constexpr int LV_GW = LV_CH / 2;         // 32-bit words per staged row of a [.., D] tensor

// The filter, prepared once per call by li_prep_kernel: log-poles -exp(p) exp(gamma), poles, residues and the correction of
// pole_corr, [D, 16] fp32 (modes beyond the order O: pole 0, residue 0).  The C entries that are handed log-poles (sb_li_fwd,
// sb_li_bwd) have no poles: lam and corr are null there and the kernels form them.
struct LiModal { const float* ll; const float* lam; const float* R; const float* corr; int O; };
static int g_li_tiled = 1;               // sb_li_set_variant

// Rounding the pole to fp32 changes it by a factor 1 + e, e = log(lam) - ll, and what the recurrence makes of the entering state
// over a chunk of T steps by 1 + T e.  In the state itself the prefix pass, which uses exp(ll T), hides that; the sensitivity that
// role (2) of the backward hands on at the chunk's last step, w = .. + T lam^(T-1) s, carries it: T (exp((T-1) ll) - lam^(T-1)) =
// T (T-1) exp((T-1) ll) (ll - log(lam)) times the entering state puts it right.  Relative error of the pole gradients against 64
// bits at L = 8192, D = 4096: 1.9e-6, 2.7e-6 without, 2.5e-6 with the sensitivity carried from chunk to chunk; 1 us of 551.
__device__ __forceinline__ float pole_corr(float ll, float lam) {
  constexpr float T = LB_TC;
  return lam > 0.f ? T * (T - 1.f) * expf((T - 1.f) * ll) * (ll - logf(lam)) : 0.f;
}

__global__ void li_prep_kernel(const float* __restrict__ gamma, const float* __restrict__ p, const float* __restrict__ R,
                               float* __restrict__ out, int D, int O) {
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x, n = (size_t)D * LO;
  let_next_start();
  if (i >= n) return;
  const int o = (int)(i % LO);
  const size_t j = i / LO * O + o;
  const float ll = o < O ? -expf(p[j]) * expf(gamma[j]) : -1.0e30f;
  out[i] = ll;
  const float lam = o < O ? expf(ll) : 0.f;
  out[n + i] = lam;
  out[2 * n + i] = o < O ? R[j] : 0.f;
  out[3 * n + i] = pole_corr(ll, lam);
}

// [.., D, 16] scratch: rows ch and ch + 1 are 32 consecutive floats
__device__ __forceinline__ void load_pairs(const float* p, bool live, f2 (&r)[LO]) {
  float a[LO], b[LO];
#pragma unroll
  for (int o = 0; o < LO; ++o) { a[o] = 0.f; b[o] = 0.f; }
  if (live) { load_vec16(p, a); load_vec16(p + LO, b); }
#pragma unroll
  for (int o = 0; o < LO; ++o) r[o] = f2_pack(a[o], b[o]);
}
__device__ __forceinline__ void store_pairs(float* p, const f2 (&r)[LO]) {
  float a[LO], b[LO];
#pragma unroll
  for (int o = 0; o < LO; ++o) { const float2 t = f2_unpack(r[o]); a[o] = t.x; b[o] = t.y; }
  store_vec16(p, a);
  store_vec16(p + LO, b);
}

__device__ __forceinline__ void li_cp_async16(uint32_t smem_dst, const void* src, int nbytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_dst), "l"(src), "r"(nbytes) : "memory");
}
__device__ __forceinline__ void li_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void li_cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Stage ROWS rows of `src` (row r at src + r * ld elements; rows >= n_rows and 16-byte chunks >= ncv zero-filled) into
// dst[ROWS][CHK chunks] with NT threads: a thread keeps its chunk column and walks down the rows.
template <int ROWS, int CHK, int NT>
__device__ __forceinline__ void li_stage(uint32_t dst, const bf16* src, size_t ld, int n_rows, int ncv, int tid) {
  constexpr int STEP = NT / CHK;                         // rows staged side by side
  const int r0 = tid / CHK, c = tid - r0 * CHK;
  if (r0 >= STEP) return;
  const bf16* p = src + (size_t)r0 * ld + c * 8;
  uint32_t q = dst + (r0 * CHK + c) * 16;
#pragma unroll 8
  for (int r = r0; r < ROWS; r += STEP, p += STEP * ld, q += STEP * CHK * 16) {
    const bool ok = r < n_rows && c < ncv;
    li_cp_async16(q, ok ? p : src, ok ? 16 : 0);
  }
}

__device__ __forceinline__ void load_poles(const LiModal& m, size_t off, bool live, f2 (&lam)[LO]) {
  load_pairs((m.lam ? m.lam : m.ll) + off, live, lam);
  if (m.lam) return;
#pragma unroll
  for (int o = 0; o < LO; ++o) { const float2 t = f2_unpack(lam[o]); lam[o] = f2_pack(expf(t.x), expf(t.y)); }
}

__device__ __forceinline__ void load_corr(const LiModal& m, size_t off, f2 (&c)[LO]) {
  load_pairs((m.corr ? m.corr : m.ll) + off, true, c);
  if (m.corr) return;
#pragma unroll
  for (int o = 0; o < LO; ++o) {
    const float2 t = f2_unpack(c[o]);
    c[o] = f2_pack(pole_corr(t.x, expf(t.x)), pole_corr(t.y, expf(t.y)));
  }
}

__device__ __forceinline__ FeatPair li_feat(const uint32_t* row, int lane3) { return feat_pair(row[lane3], row[lane3 + 1], row[lane3 + 2]); }
__device__ __forceinline__ f2 li_pair(const uint32_t* row, int i) { return f2_bf(row[i]); }

// forward pass 1 (APPLY = false): end state of each chunk from a zero state.
// forward pass 3 (APPLY = true): rerun each chunk from its entering state S and emit z.
template <bool APPLY>
__global__ void __launch_bounds__(LV_PAIRS)
li_fwd_tiled_kernel(const bf16* __restrict__ feat, const LiModal m, const float* __restrict__ bias, float* S, bf16* z, LiDims d) {
  __shared__ __align__(16) uint32_t ring[LV_STAGES][LV_ROWS][LV_FW];
  const int tid = threadIdx.x, c0 = blockIdx.x * LV_CH, ch = c0 + 2 * tid;
  const int n = blockIdx.y, b = blockIdx.z;
  const bool live = ch < d.D;
  const int t0 = n * d.TC, t1 = min(t0 + d.TC, d.L);
  const size_t ld = (size_t)3 * d.D;
  const bf16* src = feat + ((size_t)b * d.L + t0) * ld + 3 * c0;
  const int ncv = min(3 * LV_CH / 8, 3 * (d.D - c0) / 8);
  const int ntile = (t1 - t0 + LV_ROWS - 1) / LV_ROWS;
  const uint32_t ring_a = static_cast<uint32_t>(__cvta_generic_to_shared(&ring[0][0][0]));
  constexpr uint32_t TILE_B = LV_ROWS * LV_FW * 4;
#pragma unroll
  for (int k = 0; k < LV_STAGES - 1; ++k) {
    if (k < ntile)
      li_stage<LV_ROWS, 3 * LV_CH / 8, LV_PAIRS>(ring_a + k * TILE_B, src + (size_t)k * LV_ROWS * ld, ld, t1 - t0 - k * LV_ROWS, ncv, tid);
    li_cp_commit();
  }
  let_next_start();
  wait_for_previous();                   // the features are the call's own inputs; poles and entering states are not
  f2 lam[LO], s[LO], rr[APPLY ? LO : 1], be = 0;
  load_poles(m, (size_t)ch * LO, live, lam);
  float* Sp = S + (((size_t)b * d.NC + n) * d.D + ch) * LO;
  if constexpr (APPLY) {
    load_pairs(m.R + (size_t)ch * LO, live, rr);
    load_pairs(Sp, live, s);
    if (live) be = f2_pack(bias[ch], bias[ch + 1]);
  } else {
#pragma unroll
    for (int o = 0; o < LO; ++o) s[o] = 0;
  }
  uint32_t* zo = APPLY ? reinterpret_cast<uint32_t*>(z + ((size_t)b * d.L + t0) * d.D + ch) : nullptr;
  const size_t zld = d.D / 2;
  for (int k = 0; k < ntile; ++k) {
    li_cp_wait<LV_STAGES - 2>();
    __syncthreads();                     // tile k has landed for everyone; everyone is done with tile k - 1's buffer
    const int kn = k + LV_STAGES - 1;
    if (kn < ntile)
      li_stage<LV_ROWS, 3 * LV_CH / 8, LV_PAIRS>(ring_a + (kn % LV_STAGES) * TILE_B, src + (size_t)kn * LV_ROWS * ld, ld,
                                                 t1 - t0 - kn * LV_ROWS, ncv, tid);
    li_cp_commit();
    const uint32_t (*T)[LV_FW] = ring[k % LV_STAGES];
    const int rows = min(LV_ROWS, t1 - t0 - k * LV_ROWS);
    auto step = [&](int r) {
      const FeatPair f = li_feat(T[r], 3 * tid);
      const f2 u = f2_mul(f.x2, f.v);
      if constexpr (APPLY) {
        f2 y0 = f2_mul(be, u), y1 = 0;
#pragma unroll
        for (int o = 0; o < LO; o += 2) {
          s[o] = f2_fma(lam[o], s[o], u);
          s[o + 1] = f2_fma(lam[o + 1], s[o + 1], u);
          y0 = f2_fma(rr[o], s[o], y0);
          y1 = f2_fma(rr[o + 1], s[o + 1], y1);
        }
        if (live) zo[0] = pack_bf2(f2_mul(f.x1, f2_add(y0, y1)));
        zo += zld;
      } else {
#pragma unroll
        for (int o = 0; o < LO; ++o) s[o] = f2_fma(lam[o], s[o], u);
      }
    };
    if (rows == LV_ROWS) {
#pragma unroll 4
      for (int r = 0; r < LV_ROWS; ++r) step(r);
    } else {
#pragma unroll 1
      for (int r = 0; r < rows; ++r) step(r);
    }
  }
  if constexpr (!APPLY) {
    if (live) store_pairs(Sp, s);
  }
}

// Exclusive prefix of the chunk states over the chunks, in place (see li_prefix_kernel): one thread per (b, ch, o), the
// loads of AHEAD chunks in flight ahead of the serial carry.  REVERSE: exclusive suffix (the adjoint).  `scale`: factor on the
// local terms; `carry`: what enters at the first chunk; `tail`: gradient of the returned state (REVERSE).
// Bound by the latency of one batch of loads after another.  At L = 8192, D = 4096 with 16 and with 32 loads in flight: the
// backward's 128 chunks 54 and 36 us.  The whole forward with 8, 16 and 32: L = 8192, D = 4096 (16 chunks) 137.1, 137.5 and 139.6 us,
// L = 32768 (64 chunks) 424, 414 and 416, L = 1237, D = 1024 (39 chunks, chained launches) 22.6, 20.7 and 25.8.
constexpr int LP_AHEAD_FWD = 16, LP_AHEAD_BWD = 32;
template <bool REVERSE, int AHEAD>
__device__ __forceinline__ float li_carry(float* p, size_t per_b, float ll, float scale, float carry, float tail,
                                          const LiDims& d) {
  const float step = expf(ll * d.TC);
  for (int k0 = 0; k0 < d.NC; k0 += AHEAD) {
    float loc[AHEAD];
#pragma unroll
    for (int j = 0; j < AHEAD; ++j) {
      const int n = REVERSE ? d.NC - 1 - (k0 + j) : k0 + j;
      loc[j] = k0 + j < d.NC ? p[(size_t)n * per_b] : 0.f;
    }
#pragma unroll
    for (int j = 0; j < AHEAD; ++j) {
      if (k0 + j < d.NC) {
        const int n = REVERSE ? d.NC - 1 - (k0 + j) : k0 + j;
        p[(size_t)n * per_b] = carry;
        const int len = min(d.TC, d.L - n * d.TC);
        carry = fmaf(len == d.TC ? step : expf(ll * len), carry, scale * loc[j]);
        // the gradient of the returned state enters at the last step without a factor lam (see li_bwd_prefix_kernel)
        if (REVERSE && n == d.NC - 1 && tail != 0.f) carry += expf(ll * (len - 1)) * tail;
      }
    }
  }
  return carry;
}
__device__ __forceinline__ float state_at(const float* s, int b, int ch, int o, const LiModal& m, int D) {
  return (s && o < m.O) ? s[((size_t)b * D + ch) * m.O + o] : 0.f;
}

__global__ void __launch_bounds__(128)
li_prefix_tiled_kernel(float* S, const LiModal m, const float* __restrict__ state_in, float* __restrict__ state_out, LiDims d) {
  let_next_start();
  wait_for_previous();
  const size_t per_b = (size_t)d.D * LO;
  const size_t r = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  const int b = blockIdx.y;
  if (r >= per_b) return;
  const int ch = (int)(r / LO), o = (int)(r % LO);
  const float ll = m.ll[r];
  const float end = li_carry<false, LP_AHEAD_FWD>(S + (size_t)b * d.NC * per_b + r, per_b, ll, 1.f,
                                                  state_at(state_in, b, ch, o, m, d.D), 0.f, d);
  if (state_out && o < m.O) state_out[((size_t)b * d.D + ch) * m.O + o] = end;
}

// Backward prefixes: blockIdx.z = 0 the states, 1 the adjoints (carrying R, `with_R`, when a state gradient has to ride along or
// the caller wants finished partial sums).
__global__ void __launch_bounds__(128)
li_bwd_prefix_tiled_kernel(float* S, float* A, const LiModal m, const float* __restrict__ state_in, const float* __restrict__ dstate_out,
                           float* __restrict__ dstate_in, int with_R, LiDims d) {
  let_next_start();
  wait_for_previous();
  const size_t per_b = (size_t)d.D * LO;
  const size_t r = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  const int b = blockIdx.y;
  if (r >= per_b) return;
  const int ch = (int)(r / LO), o = (int)(r % LO);
  const bool real = o < m.O;
  const float ll = m.ll[r];
  const size_t base = (size_t)b * d.NC * per_b + r;
  if (blockIdx.z == 0) {
    li_carry<false, LP_AHEAD_BWD>(S + base, per_b, ll, 1.f, state_at(state_in, b, ch, o, m, d.D), 0.f, d);
  } else {
    const float R = m.R[r];
    const float end = li_carry<true, LP_AHEAD_BWD>(A + base, per_b, ll, with_R ? R : 1.f, 0.f,
                                                   state_at(dstate_out, b, ch, o, m, d.D), d);
    if (dstate_in && real) dstate_in[((size_t)b * d.D + ch) * m.O + o] = expf(ll) * (with_R ? end : R * end);
  }
}

// Shared-memory image of a backward chunk: features and dz as they are in memory.
constexpr int LBL_SMEM = LB_TC * (LV_FW + LV_GW) * 4;            // 64 KB
constexpr int LBA_SMEM = LBL_SMEM + LB_TC * LV_FW * 4;           // + the gradient tile: 112 KB, two blocks per SM

// backward pass 1: end state (Sloc, warps 0-1) and adjoint leaving the left edge (Aloc, warps 2-3) of every chunk
__global__ void __launch_bounds__(2 * LV_PAIRS)
li_bwd_local_tiled_kernel(const bf16* __restrict__ feat, const bf16* __restrict__ dz, const LiModal m, float* __restrict__ S,
                          float* __restrict__ A, LiDims d) {
  extern __shared__ __align__(16) uint32_t li_sm[];
  uint32_t (*fS)[LV_FW] = reinterpret_cast<uint32_t (*)[LV_FW]>(li_sm);
  uint32_t (*gS)[LV_GW] = reinterpret_cast<uint32_t (*)[LV_GW]>(li_sm + LB_TC * LV_FW);
  const int tid = threadIdx.x, c0 = blockIdx.x * LV_CH, pair = tid & (LV_PAIRS - 1), ch = c0 + 2 * pair;
  const int n = blockIdx.y, b = blockIdx.z;
  const bool live = ch < d.D;
  const int t0 = n * LB_TC, rows = min(LB_TC, d.L - t0);
  const uint32_t f_a = static_cast<uint32_t>(__cvta_generic_to_shared(fS)), g_a = static_cast<uint32_t>(__cvta_generic_to_shared(gS));
  const int ncf = min(3 * LV_CH / 8, 3 * (d.D - c0) / 8), ncg = min(LV_CH / 8, (d.D - c0) / 8);
  li_stage<LB_TC, 3 * LV_CH / 8, 2 * LV_PAIRS>(f_a, feat + ((size_t)b * d.L + t0) * 3 * d.D + 3 * c0, (size_t)3 * d.D, rows, ncf, tid);
  li_stage<LB_TC, LV_CH / 8, 2 * LV_PAIRS>(g_a, dz + ((size_t)b * d.L + t0) * d.D + c0, d.D, rows, ncg, tid);
  li_cp_commit();
  let_next_start();
  f2 lam[LO], s[LO];
  load_poles(m, (size_t)ch * LO, live, lam);
#pragma unroll
  for (int o = 0; o < LO; ++o) s[o] = 0;
  li_cp_wait<0>();
  __syncthreads();
  float* out;
  if (tid < LV_PAIRS) {
#pragma unroll 4
    for (int r = 0; r < rows; ++r) {
      const FeatPair f = li_feat(fS[r], 3 * pair);
      const f2 u = f2_mul(f.x2, f.v);
#pragma unroll
      for (int o = 0; o < LO; ++o) s[o] = f2_fma(lam[o], s[o], u);
    }
    out = S;
  } else {
#pragma unroll 4
    for (int r = rows - 1; r >= 0; --r) {
      const f2 dy = f2_mul(li_pair(gS[r], pair), f2_pack(lo_f(fS[r][3 * pair]), hi_f(fS[r][3 * pair + 1])));
#pragma unroll
      for (int o = 0; o < LO; ++o) s[o] = f2_fma(lam[o], s[o], dy);
    }
    out = A;
  }
  if (live) store_pairs(out + (((size_t)b * d.NC + n) * d.D + ch) * LO, s);
}

// backward pass 3: see the head of this section.  S and A hold the entering state / adjoint of every chunk; dRp and dLp (which
// may be A) receive the chunk's partial sums of dR and dlam (dlam without the factor R unless GOUT).  GOUT: the adjoint
// carries R, and the gradient of the final state (dstate_out, [B, D, O]) if there is one.
template <bool GOUT>
__global__ void __launch_bounds__(3 * LV_PAIRS, 2)
li_bwd_apply_tiled_kernel(const bf16* __restrict__ feat, const bf16* __restrict__ dz, const LiModal m, const float* __restrict__ bias,
                          const float* S, const float* A, float* dRp, float* dLp, float* __restrict__ dBp, bf16* __restrict__ dfeat,
                          const float* __restrict__ dstate_out, LiDims d) {
  extern __shared__ __align__(16) uint32_t li_sm[];
  uint32_t (*fS)[LV_FW] = reinterpret_cast<uint32_t (*)[LV_FW]>(li_sm);
  uint32_t (*gS)[LV_GW] = reinterpret_cast<uint32_t (*)[LV_GW]>(li_sm + LB_TC * LV_FW);
  uint32_t (*oS)[LV_FW] = reinterpret_cast<uint32_t (*)[LV_FW]>(li_sm + LB_TC * (LV_FW + LV_GW));
  constexpr int NT = 3 * LV_PAIRS;
  const int tid = threadIdx.x, c0 = blockIdx.x * LV_CH, role = tid / LV_PAIRS, pair = tid - role * LV_PAIRS, ch = c0 + 2 * pair;
  const int n = blockIdx.y, b = blockIdx.z;
  const bool live = ch < d.D;
  const int t0 = n * LB_TC, rows = min(LB_TC, d.L - t0);
  const uint32_t f_a = static_cast<uint32_t>(__cvta_generic_to_shared(fS)), g_a = static_cast<uint32_t>(__cvta_generic_to_shared(gS));
  const int ncf = min(3 * LV_CH / 8, 3 * (d.D - c0) / 8), ncg = min(LV_CH / 8, (d.D - c0) / 8);
  li_stage<LB_TC, 3 * LV_CH / 8, NT>(f_a, feat + ((size_t)b * d.L + t0) * 3 * d.D + 3 * c0, (size_t)3 * d.D, rows, ncf, tid);
  li_stage<LB_TC, LV_CH / 8, NT>(g_a, dz + ((size_t)b * d.L + t0) * d.D + c0, d.D, rows, ncg, tid);
  li_cp_commit();
  let_next_start();
  wait_for_previous();
  const size_t off = (((size_t)b * d.NC + n) * d.D + ch) * LO;
  f2 lam[LO], s[LO];                                     // s: state (roles 0, 1) or adjoint (role 2) entering the chunk
  load_poles(m, (size_t)ch * LO, live, lam);
  load_pairs((role == 2 ? A : S) + off, live, s);
  li_cp_wait<0>();
  __syncthreads();                                       // the chunk has landed; S and A of this block have been read
  if (role == 0) {
    f2 rr[LO], dr[LO], be = 0, db = 0;
    load_pairs(m.R + (size_t)ch * LO, live, rr);
    if (live) be = f2_pack(bias[ch], bias[ch + 1]);
#pragma unroll
    for (int o = 0; o < LO; ++o) dr[o] = 0;
#pragma unroll 2
    for (int r = 0; r < rows; ++r) {
      const FeatPair f = li_feat(fS[r], 3 * pair);
      const f2 u = f2_mul(f.x2, f.v), gz = li_pair(gS[r], pair), dy = f2_mul(gz, f.x1);
      f2 y0 = f2_mul(be, u), y1 = 0;
#pragma unroll
      for (int o = 0; o < LO; o += 2) {
        s[o] = f2_fma(lam[o], s[o], u);
        s[o + 1] = f2_fma(lam[o + 1], s[o + 1], u);
        y0 = f2_fma(rr[o], s[o], y0);
        y1 = f2_fma(rr[o + 1], s[o + 1], y1);
        dr[o] = f2_fma(dy, s[o], dr[o]);
        dr[o + 1] = f2_fma(dy, s[o + 1], dr[o + 1]);
      }
      db = f2_fma(dy, u, db);
      const uint32_t w = pack_bf2(f2_mul(gz, f2_add(y0, y1)));
      uint16_t* o16 = reinterpret_cast<uint16_t*>(&oS[r][3 * pair]);
      o16[0] = (uint16_t)w;
      o16[3] = (uint16_t)(w >> 16);
    }
    if (live) {
      store_pairs(dRp + off, dr);
      const float2 t = f2_unpack(db);
      *reinterpret_cast<float2*>(dBp + ((size_t)b * d.NC + n) * d.D + ch) = t;
    }
  } else if (role == 1) {
    f2 w[LO], dl[LO];
#pragma unroll
    for (int o = 0; o < LO; ++o) { w[o] = 0; dl[o] = 0; }
#pragma unroll 2
    for (int r = 0; r < rows; ++r) {
      const FeatPair f = li_feat(fS[r], 3 * pair);
      const f2 u = f2_mul(f.x2, f.v), dy = f2_mul(li_pair(gS[r], pair), f.x1);
#pragma unroll
      for (int o = 0; o < LO; ++o) {
        w[o] = f2_fma(lam[o], w[o], s[o]);
        s[o] = f2_fma(lam[o], s[o], u);
        dl[o] = f2_fma(dy, w[o], dl[o]);
      }
    }
    if (live) {
      f2 a[LO];
      if (rows == LB_TC) {                                 // (a shorter chunk is the last one: nothing enters from its right)
        load_corr(m, (size_t)ch * LO, a);
        load_pairs(S + off, true, s);
#pragma unroll
        for (int o = 0; o < LO; ++o) w[o] = f2_fma(a[o], s[o], w[o]);
      }
      load_pairs(A + off, true, a);
#pragma unroll
      for (int o = 0; o < LO; ++o) {
        f2 e = f2_mul(lam[o], a[o]);
        if constexpr (GOUT) {
          if (n == d.NC - 1)
            e = f2_add(e, f2_pack(state_at(dstate_out, b, ch, o, m, d.D), state_at(dstate_out, b, ch + 1, o, m, d.D)));
          dl[o] = f2_mul(f2_pack(m.R[(size_t)ch * LO + o], m.R[(size_t)(ch + 1) * LO + o]), dl[o]);
        }
        dl[o] = f2_fma(e, w[o], dl[o]);
      }
      store_pairs(dLp + off, dl);
    }
  } else {
    f2 rr[LO], be = 0;
    load_pairs(m.R + (size_t)ch * LO, live, rr);
    if (live) be = f2_pack(bias[ch], bias[ch + 1]);
#pragma unroll 2
    for (int r = rows - 1; r >= 0; --r) {
      const FeatPair f = li_feat(fS[r], 3 * pair);
      const f2 dy = f2_mul(li_pair(gS[r], pair), f.x1);
      f2 d0 = f2_mul(be, dy), d1 = 0;
      if constexpr (GOUT) {
#pragma unroll
        for (int o = 0; o < LO; ++o) s[o] = f2_fma(lam[o], s[o], f2_mul(rr[o], dy));
        if (n == d.NC - 1 && r == rows - 1 && live) {
#pragma unroll
          for (int o = 0; o < LO; ++o)
            s[o] = f2_add(s[o], f2_pack(state_at(dstate_out, b, ch, o, m, d.D), state_at(dstate_out, b, ch + 1, o, m, d.D)));
        }
#pragma unroll
        for (int o = 0; o < LO; o += 2) { d0 = f2_add(d0, s[o]); d1 = f2_add(d1, s[o + 1]); }
      } else {
#pragma unroll
        for (int o = 0; o < LO; o += 2) {
          s[o] = f2_fma(lam[o], s[o], dy);
          s[o + 1] = f2_fma(lam[o + 1], s[o + 1], dy);
          d0 = f2_fma(rr[o], s[o], d0);
          d1 = f2_fma(rr[o + 1], s[o + 1], d1);
        }
      }
      const f2 du = f2_add(d0, d1);
      const float2 dx2 = f2_unpack(f2_mul(du, f.v)), dv = f2_unpack(f2_mul(du, f.x2));
      uint16_t* o16 = reinterpret_cast<uint16_t*>(&oS[r][3 * pair]);
      o16[1] = __bfloat16_as_ushort(__float2bfloat16_rn(dx2.x));
      o16[2] = __bfloat16_as_ushort(__float2bfloat16_rn(dv.x));
      oS[r][3 * pair + 2] = pack_bf2(f2_pack(dx2.y, dv.y));
    }
  }
  __syncthreads();
  bf16* dst = dfeat + ((size_t)b * d.L + t0) * 3 * d.D + 3 * c0;
  constexpr int CHK = 3 * LV_CH / 8;
  for (int idx = tid; idx < rows * CHK; idx += NT) {
    const int r = idx / CHK, c = idx - r * CHK;
    if (c < ncf) *reinterpret_cast<uint4*>(dst + (size_t)r * 3 * d.D + c * 8) = *reinterpret_cast<const uint4*>(&oS[r][c * 4]);
  }
}

// Sums the per-chunk partials over batch and chunks (in a fixed order) and finishes the filter gradients:
//   dR, dgamma = dp = dlam lam log(lam) ([D, O]) and dbias [D].  One thread per (channel, mode) column and row slice.
constexpr int LR_COLS = 32, LR_SLICES = 8;
__global__ void __launch_bounds__(LR_COLS * LR_SLICES)
li_bwd_reduce_kernel(const float* dRp, const float* dLp, const float* dBp, const LiModal m, int scale_by_R, float* dR, float* dll, float* db,
                     int n_rows, int D) {
  __shared__ float red[2][LR_SLICES][LR_COLS];
  const int cx = threadIdx.x % LR_COLS, sl = threadIdx.x / LR_COLS;
  const int n_modal = (D * LO + LR_COLS - 1) / LR_COLS;              // blocks [0, n_modal): dR / dlam; the rest: dbias
  const bool modal = (int)blockIdx.x < n_modal;
  const size_t width = modal ? (size_t)D * LO : (size_t)D;
  const size_t col = (size_t)(modal ? blockIdx.x : blockIdx.x - n_modal) * LR_COLS + cx;
  float a0 = 0.f, a1 = 0.f;
  wait_for_previous();
  if (col < width) {
    if (modal) {
#pragma unroll 4
      for (int i = sl; i < n_rows; i += LR_SLICES) { a0 += dRp[(size_t)i * width + col]; a1 += dLp[(size_t)i * width + col]; }
    } else {
#pragma unroll 4
      for (int i = sl; i < n_rows; i += LR_SLICES) a0 += dBp[(size_t)i * width + col];
    }
  }
  red[0][sl][cx] = a0;
  red[1][sl][cx] = a1;
  __syncthreads();
  if (sl || col >= width) return;
#pragma unroll
  for (int j = 1; j < LR_SLICES; ++j) { a0 += red[0][j][cx]; a1 += red[1][j][cx]; }
  if (!modal) { db[col] = a0; return; }
  const int ch = (int)(col / LO), o = (int)(col % LO);
  if (o >= m.O) return;
  const size_t i = (size_t)ch * m.O + o;
  dR[i] = a0;
  const float g = (scale_by_R ? m.R[col] * a1 : a1) * m.lam[col] * m.ll[col];
  dll[i] = isfinite(g) ? g : 0.f;
}

// ------------------------------------------------------------------------------------ context parallel: all-to-all inside the scan
// Sequence-sharded ranks (zigzag: rank r holds natural chunks r and 2cp-1-r of `chunk_len` rows, [B, l, Dtot] with
// l = 2 chunk_len) switch to a channel-sharded scan over the whole sequence (this rank: d = Dtot / cp channels) and back.
// Only the pre-gated signal u = x2 v travels: every rank writes u into a symmetric staging buffer, and after one
// stream-ordered barrier the scan's first pass reads its channel block of every chunk straight from the owner's
// staging buffer (plain peer loads), keeping a local copy for the second pass.  The second pass stores y straight into
// the owner's staging buffer (plain peer stores); after the second barrier the owner gates it with its own x1.  No
// tensor is permuted or copied by a separate kernel, and a third of the bytes of exchanging (x1, x2, v) and z cross
// NVLink.  `LiCpMap.base[j]`: row 0 of natural chunk j in its owner's staging buffer, already offset to this rank's
// channel block.  The scan chunk length TC must divide chunk_len, so a scan chunk never straddles two owners.
struct LiCpMap {
  void* base[32];
  long long batch_stride;   // elements between batches of a staging buffer (l * Dtot)
  int row_stride;           // elements between rows (Dtot)
  int chunk_len;
  int n_chunks;             // 2 cp
};

__device__ __forceinline__ bf16* cp_row(const LiCpMap& m, int b, int t) {
  const int j = t / m.chunk_len;
  return reinterpret_cast<bf16*>(m.base[j]) + (size_t)b * m.batch_stride + (size_t)(t - j * m.chunk_len) * m.row_stride;
}

// pass 1: pull u from the owners, keep a local copy [B, L, d], chunk-local end state from a zero state
__global__ void __launch_bounds__(LI_THREADS)
li_cp_local_kernel(const LiCpMap u_in, bf16* __restrict__ ufull, const float* __restrict__ loglam, float* __restrict__ Sloc,
                   LiDims d) {
  const int ch = blockIdx.x * LI_THREADS + threadIdx.x;
  if (ch >= d.D) return;
  const int n = blockIdx.y, b = blockIdx.z;
  float lam[LO], s[LO];
  load_vec16(loglam + (size_t)ch * LO, lam);
#pragma unroll
  for (int o = 0; o < LO; ++o) { lam[o] = __expf(lam[o]); s[o] = 0.f; }
  const int t0 = n * d.TC, t1 = min(t0 + d.TC, d.L);
  const bf16* src = cp_row(u_in, b, t0) + ch;
  bf16* dst = ufull + ((size_t)b * d.L + t0) * d.D + ch;
#pragma unroll 8
  for (int t = t0; t < t1; ++t, src += u_in.row_stride, dst += d.D) {
    const bf16 raw = *src;
    *dst = raw;
    const float u = b2f(raw);
#pragma unroll
    for (int o = 0; o < LO; ++o) s[o] = lam[o] * s[o] + u;
  }
  store_vec16(Sloc + (((size_t)b * d.NC + n) * d.D + ch) * LO, s);
}

// pass 3: rerun each chunk from its entering state; y goes to the owner of the rows
__global__ void __launch_bounds__(LI_THREADS)
li_cp_apply_kernel(const bf16* __restrict__ ufull, const float* __restrict__ loglam, const float* __restrict__ R,
                   const float* __restrict__ bias, const float* __restrict__ Sin, const LiCpMap y_out, LiDims d) {
  const int ch = blockIdx.x * LI_THREADS + threadIdx.x;
  if (ch >= d.D) return;
  const int n = blockIdx.y, b = blockIdx.z;
  float lam[LO], s[LO], rr[LO];
  load_vec16(loglam + (size_t)ch * LO, lam);
  load_vec16(R + (size_t)ch * LO, rr);
  load_vec16(Sin + (((size_t)b * d.NC + n) * d.D + ch) * LO, s);
#pragma unroll
  for (int o = 0; o < LO; ++o) lam[o] = __expf(lam[o]);
  const float be = bias[ch];
  const int t0 = n * d.TC, t1 = min(t0 + d.TC, d.L);
  const bf16* f = ufull + ((size_t)b * d.L + t0) * d.D + ch;
  bf16* yo = cp_row(y_out, b, t0) + ch;
#pragma unroll 8
  for (int t = t0; t < t1; ++t, f += d.D, yo += y_out.row_stride) {
    const float u = b2f(*f);
    float y = be * u;
#pragma unroll
    for (int o = 0; o < LO; ++o) { s[o] = lam[o] * s[o] + u; y += rr[o] * s[o]; }
    *yo = __float2bfloat16_rn(y);
  }
}

// backward pass B1: pull dy = dz x1 from the owners (local copy [B, L, d]); Sloc, Wloc, Aloc as in li_bwd_local_kernel
__global__ void __launch_bounds__(LI_THREADS)
li_cp_bwd_local_kernel(const bf16* __restrict__ ufull, const LiCpMap dy_in, bf16* __restrict__ dyfull,
                       const float* __restrict__ loglam, const float* __restrict__ R, float* __restrict__ Sloc,
                       float* __restrict__ Wloc, float* __restrict__ Aloc, LiDims d) {
  const int ch = blockIdx.x * LI_THREADS + threadIdx.x;
  if (ch >= d.D) return;
  const int n = blockIdx.y, b = blockIdx.z;
  float lam[LO], s[LO], w[LO], pw[LO], a[LO];
  load_vec16(loglam + (size_t)ch * LO, lam);
#pragma unroll
  for (int o = 0; o < LO; ++o) { lam[o] = __expf(lam[o]); s[o] = 0.f; w[o] = 0.f; pw[o] = 1.f; a[o] = 0.f; }
  const int t0 = n * d.TC, t1 = min(t0 + d.TC, d.L);
  const bf16* f = ufull + ((size_t)b * d.L + t0) * d.D + ch;
  const bf16* g = cp_row(dy_in, b, t0) + ch;
  bf16* gd = dyfull + ((size_t)b * d.L + t0) * d.D + ch;
#pragma unroll 4
  for (int t = t0; t < t1; ++t, f += d.D, g += dy_in.row_stride, gd += d.D) {
    const float u = b2f(*f);
    const bf16 raw = *g;
    *gd = raw;
    const float dy = b2f(raw);
#pragma unroll
    for (int o = 0; o < LO; ++o) {
      w[o] = s[o] + lam[o] * w[o];
      s[o] = lam[o] * s[o] + u;
      a[o] += pw[o] * dy;
      pw[o] *= lam[o];
    }
  }
  float rr[LO];
  load_vec16(R + (size_t)ch * LO, rr);
#pragma unroll
  for (int o = 0; o < LO; ++o) a[o] *= rr[o];
  const size_t off = (((size_t)b * d.NC + n) * d.D + ch) * LO;
  store_vec16(Sloc + off, s);
  store_vec16(Wloc + off, w);
  store_vec16(Aloc + off, a);
}

// backward pass B3 (forward direction): y back to the owners (for dx1 = dz y), per-chunk partials of dR, dlam, dbias
__global__ void __launch_bounds__(LI_THREADS)
li_cp_bwd_apply_fwd_kernel(const bf16* __restrict__ ufull, const bf16* __restrict__ dyfull, const float* __restrict__ loglam,
                           const float* __restrict__ R, const float* __restrict__ bias, const float* __restrict__ Sin,
                           const float* __restrict__ Win, const LiCpMap y_out, float* __restrict__ dRp,
                           float* __restrict__ dLp, float* __restrict__ dBp, LiDims d) {
  const int ch = blockIdx.x * LI_THREADS + threadIdx.x;
  if (ch >= d.D) return;
  const int n = blockIdx.y, b = blockIdx.z;
  float lam[LO], s[LO], w[LO], rr[LO], dr[LO], dl[LO];
  const size_t off = (((size_t)b * d.NC + n) * d.D + ch) * LO;
  load_vec16(loglam + (size_t)ch * LO, lam);
  load_vec16(R + (size_t)ch * LO, rr);
  load_vec16(Sin + off, s);
  load_vec16(Win + off, w);
#pragma unroll
  for (int o = 0; o < LO; ++o) { lam[o] = __expf(lam[o]); dr[o] = 0.f; dl[o] = 0.f; }
  const float be = bias[ch];
  float db = 0.f;
  const int t0 = n * d.TC, t1 = min(t0 + d.TC, d.L);
  const bf16* f = ufull + ((size_t)b * d.L + t0) * d.D + ch;
  const bf16* g = dyfull + ((size_t)b * d.L + t0) * d.D + ch;
  bf16* yo = cp_row(y_out, b, t0) + ch;
#pragma unroll 4
  for (int t = t0; t < t1; ++t, f += d.D, g += d.D, yo += y_out.row_stride) {
    const float u = b2f(*f);
    const float dy = b2f(*g);
    float y = be * u;
#pragma unroll
    for (int o = 0; o < LO; ++o) {
      w[o] = s[o] + lam[o] * w[o];
      s[o] = lam[o] * s[o] + u;
      y += rr[o] * s[o];
      dr[o] += dy * s[o];
      dl[o] += dy * w[o];
    }
    db += dy * u;
    *yo = __float2bfloat16_rn(y);
  }
#pragma unroll
  for (int o = 0; o < LO; ++o) dl[o] *= rr[o];
  store_vec16(dRp + off, dr);
  store_vec16(dLp + off, dl);
  dBp[((size_t)b * d.NC + n) * d.D + ch] = db;
}

// backward pass R3 (reverse direction): adjoint scan, du back to the owners (for dx2 = du v, dv = du x2)
__global__ void __launch_bounds__(LI_THREADS)
li_cp_bwd_apply_rev_kernel(const bf16* __restrict__ dyfull, const float* __restrict__ loglam, const float* __restrict__ R,
                           const float* __restrict__ bias, const float* __restrict__ Ain, const LiCpMap du_out, LiDims d) {
  const int ch = blockIdx.x * LI_THREADS + threadIdx.x;
  if (ch >= d.D) return;
  const int n = blockIdx.y, b = blockIdx.z;
  float lam[LO], a[LO], rr[LO];
  load_vec16(loglam + (size_t)ch * LO, lam);
  load_vec16(R + (size_t)ch * LO, rr);
  load_vec16(Ain + (((size_t)b * d.NC + n) * d.D + ch) * LO, a);
#pragma unroll
  for (int o = 0; o < LO; ++o) lam[o] = __expf(lam[o]);
  const float be = bias[ch];
  const int t0 = n * d.TC, t1 = min(t0 + d.TC, d.L);
  const bf16* g = dyfull + ((size_t)b * d.L + (t1 - 1)) * d.D + ch;
  bf16* uo = cp_row(du_out, b, t1 - 1) + ch;
#pragma unroll 8
  for (int t = t1 - 1; t >= t0; --t, g -= d.D, uo -= du_out.row_stride) {
    const float dy = b2f(*g);
    float du = be * dy;
#pragma unroll
    for (int o = 0; o < LO; ++o) { a[o] = rr[o] * dy + lam[o] * a[o]; du += a[o]; }
    *uo = __float2bfloat16_rn(du);
  }
}

// Local gate kernels around the exchange, 8 channels per thread (feat rows are 3D interleaved (x1, x2, v)).
// mode 0: out[n, D] = x2 v                     (u, staged before the forward scan)
// mode 1: out[n, D] = x1 a                     (z = x1 y after the forward scan;  dy = dz x1 before the backward scan)
__global__ void li_cp_gate_kernel(const bf16* __restrict__ feat, const bf16* __restrict__ a, bf16* __restrict__ out,
                                  size_t n_vec, int mode) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n_vec; i += (size_t)gridDim.x * blockDim.x) {
    const uint4* fp = reinterpret_cast<const uint4*>(feat) + 3 * i;
    const uint4 q0 = fp[0], q1 = fp[1], q2 = fp[2];
    const uint32_t fw[12] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w, q2.x, q2.y, q2.z, q2.w};
    float all[24];
#pragma unroll
    for (int j = 0; j < 12; ++j) {
      const float2 t = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&fw[j]));
      all[2 * j] = t.x; all[2 * j + 1] = t.y;
    }
    float r[8];
    if (mode == 0) {
#pragma unroll
      for (int j = 0; j < 8; ++j) r[j] = all[3 * j + 1] * all[3 * j + 2];
    } else {
      const uint4 av = reinterpret_cast<const uint4*>(a)[i];
      const uint32_t aw[4] = {av.x, av.y, av.z, av.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 t = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&aw[j]));
        r[2 * j] = all[6 * j] * t.x; r[2 * j + 1] = all[6 * j + 3] * t.y;
      }
    }
    uint4 o;
    __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
    for (int j = 0; j < 4; ++j) o2[j] = __floats2bfloat162_rn(r[2 * j], r[2 * j + 1]);
    reinterpret_cast<uint4*>(out)[i] = o;
  }
}

// dfeat[n, 3D] = (dz y, du v, du x2) from the returned y and du
__global__ void li_cp_finalize_bwd_kernel(const bf16* __restrict__ feat, const bf16* __restrict__ dz, const bf16* __restrict__ y,
                                          const bf16* __restrict__ du, bf16* __restrict__ dfeat, size_t n_vec) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n_vec; i += (size_t)gridDim.x * blockDim.x) {
    const uint4* fp = reinterpret_cast<const uint4*>(feat) + 3 * i;
    const uint4 q0 = fp[0], q1 = fp[1], q2 = fp[2];
    const uint32_t fw[12] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w, q2.x, q2.y, q2.z, q2.w};
    float all[24], gz[8], yy[8], dd[8], o[24];
#pragma unroll
    for (int j = 0; j < 12; ++j) {
      const float2 t = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&fw[j]));
      all[2 * j] = t.x; all[2 * j + 1] = t.y;
    }
    const uint4 a = reinterpret_cast<const uint4*>(dz)[i], bq = reinterpret_cast<const uint4*>(y)[i],
                c = reinterpret_cast<const uint4*>(du)[i];
    const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {bq.x, bq.y, bq.z, bq.w}, cw[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 t = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&aw[j])); gz[2 * j] = t.x; gz[2 * j + 1] = t.y;
      t = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&bw[j])); yy[2 * j] = t.x; yy[2 * j + 1] = t.y;
      t = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&cw[j])); dd[2 * j] = t.x; dd[2 * j + 1] = t.y;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      o[3 * j] = gz[j] * yy[j];
      o[3 * j + 1] = dd[j] * all[3 * j + 2];
      o[3 * j + 2] = dd[j] * all[3 * j + 1];
    }
    uint4 ov[3];
    __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(ov);
#pragma unroll
    for (int j = 0; j < 12; ++j) o2[j] = __floats2bfloat162_rn(o[2 * j], o[2 * j + 1]);
    uint4* dp = reinterpret_cast<uint4*>(dfeat) + 3 * i;
    dp[0] = ov[0]; dp[1] = ov[1]; dp[2] = ov[2];
  }
}

}  // namespace sb

using namespace sb;

static inline LiDims li_dims(int B, int L, int D, int TC) { return LiDims{B, L, D, TC, (L + TC - 1) / TC}; }

// Scratch sizes (floats): S = B*NC*D*16.  Callers allocate and pass them.
extern "C" int sb_li_num_chunks(int L, int TC) { return (L + TC - 1) / TC; }

static inline bool aligned16(const void* a, const void* b, const void* c = nullptr) {
  return (((uintptr_t)a | (uintptr_t)b | (uintptr_t)c) & 15) == 0;
}

// The forward's three passes, as a chain of programmatic dependents for chunks of up to 64 steps; `first`: nothing before them belongs to
// the chain.  Blocks that wait for the pass before them take the slots that it leaves free, unevenly over the SMs, and a block of a longer
// chunk is too much work for that.  Chained / one after the other, us: L = 300, D = 512 12.4 / 20.1, B = 2, L = 1237, D = 1024 30.6 / 33.0
// (chunks of 32), but L = 2048, D = 4096 62 / 52, L = 8192, D = 1024 62 / 54 (128) and D = 4096 183 / 137 (512; 150 with the last pass
// alone left out of the chain).
static int li_fwd_chain(bool first, const bf16* feat, const LiModal& m, const float* bias, const float* state_in, float* state_out, float* S,
                        bf16* z, dim3 grid, const LiDims& d, cudaStream_t st) {
  const dim3 modes((unsigned)(((size_t)d.D * LO + 127) / 128), d.B);
  const bool single = d.TC > 64;
  int rc = launch_chained(first || single, li_fwd_tiled_kernel<false>, grid, LV_PAIRS, 0, st, feat, m, bias, S, (bf16*)nullptr, d);
  if (!rc) rc = launch_chained(single, li_prefix_tiled_kernel, modes, 128, 0, st, S, m, state_in, state_out, d);
  if (!rc) rc = launch_chained(single, li_fwd_tiled_kernel<true>, grid, LV_PAIRS, 0, st, feat, m, bias, S, z, d);
  return rc;
}

// The backward's passes up to the chunks' partial sums (chunks of 64 steps); the reduction behind them is chained as well.  The apply pass
// has one block of 112 KB per chunk and 128 channels: launched while the prefix pass still runs, two of them share an SM beside idle ones,
// unless there is a block for every SM anyway, or the blocks of all three passes find an SM each.  In between it waits for the prefix pass
// to end.  us with the reduction, one after the other / all chained / all but the apply pass (* the one chosen here):
//   L = 64, D = 256 30.8 / *26.6 / 27.8        L = 1237, D = 1024 46.2 / *40.6 / 43.0        L = 200, D = 512 32.6 / 34.9 / *28.7
//   L = 300, D = 256 31.8 / *26.7 / 28.7       L = 1024, D = 2048 49.2 / *43.1 / 45.2        L = 300, D = 1024 32.9 / 36.8 / *30.0
//   L = 2048, D = 4096 121 / *115 / 118        L = 8192, D = 4096 401 / *396 / 401           L = 64, D = 3072 34.9 / 36.7 / *33.6
// The rule gives away 2 us at L <= 128 where the prefix pass's own blocks (512, 1024) happen to occupy the SMs evenly: L = 64,
// D = 4096 39.0 / 32.9 / *34.9.
template <bool GOUT>
static int li_bwd_chain(const bf16* feat, const bf16* dz, const LiModal& m, const float* bias, const float* state_in, const float* dstate_out,
                        float* dstate_in, int with_R, float* S, float* A, float* dRp, float* dLp, float* dBp, bf16* dfeat, const LiDims& d,
                        cudaStream_t st) {
  const dim3 grid((d.D + LV_CH - 1) / LV_CH, d.NC, d.B), modes((unsigned)(((size_t)d.D * LO + 127) / 128), d.B, 2);
  const long long blocks = (long long)grid.x * grid.y * grid.z, sms = sb::num_sms();
  const bool own_sms = 2 * blocks + (long long)modes.x * modes.y * modes.z <= sms;
  int rc = launch_chained(true, li_bwd_local_tiled_kernel, grid, 2 * LV_PAIRS, LBL_SMEM, st, feat, dz, m, S, A, d);
  if (!rc) rc = launch_chained(false, li_bwd_prefix_tiled_kernel, modes, 128, 0, st, S, A, m, state_in, dstate_out, dstate_in, with_R, d);
  if (!rc)
    rc = launch_chained(blocks < sms && !own_sms, li_bwd_apply_tiled_kernel<GOUT>, grid, 3 * LV_PAIRS, LBA_SMEM, st, feat, dz, m, bias, (const float*)S,
                        (const float*)A, dRp, dLp, dBp, dfeat, dstate_out, d);
  return rc;
}

// The forward scan on prepared log-poles and residues ([D, 16]): the tiled kernels for D % 8 == 0 and 16-byte aligned features and
// output, else the per-thread ones (L = 8192, D = 4096: 0.14 and 0.28 ms).
static int li_forward(const void* feat, const float* loglam, const float* R, const float* bias, const float* state_in,
                      float* state_out, float* S, void* z, const LiDims& d, cudaStream_t st) {
  const size_t n = (size_t)d.D * LO;
  if (g_li_tiled && d.D % 8 == 0 && aligned16(feat, z)) {
    const LiModal m{loglam, nullptr, R, nullptr, LO};
    const dim3 grid((d.D + LV_CH - 1) / LV_CH, d.NC, d.B);
    return li_fwd_chain(true, (const bf16*)feat, m, bias, state_in, state_out, S, (bf16*)z, grid, d, st);
  } else {
    const dim3 grid((d.D + LI_THREADS - 1) / LI_THREADS, d.NC, d.B);
    li_local_kernel<<<grid, LI_THREADS, 0, st>>>((const bf16*)feat, loglam, S, d);
    li_prefix_kernel<<<(unsigned)((d.B * n + 255) / 256), 256, 0, st>>>(S, loglam, state_in, state_out, d);
    li_apply_kernel<<<grid, LI_THREADS, 0, st>>>((const bf16*)feat, loglam, R, bias, S, (bf16*)z, d);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int sb_li_fwd(const void* feat, const float* loglam, const float* R, const float* bias, const float* state_in,
                         float* state_out, float* S_scratch, void* z, int B, int L, int D, int TC, cudaStream_t st) {
  if (B * L == 0) return 0;
  return li_forward(feat, loglam, R, bias, state_in, state_out, S_scratch, z, li_dims(B, L, D, TC), st);
}

// 1 (default): shared-memory tiled scan kernels where the shape allows; 0: the per-thread streaming kernels
extern "C" int sb_li_set_variant(int tiled) { sb::g_li_tiled = tiled ? 1 : 0; return 0; }
// Chunk length with which sb_li_bwd takes the tiled kernels, which keep a whole chunk in shared memory, for a given choice of
// the caller; the scratch arrays are sized with the value returned here.
extern "C" int sb_li_bwd_chunk(int D, int TC) { return (sb::g_li_tiled && D % 8 == 0) ? sb::LB_TC : TC; }

// Tiled forward: gamma, p, R [D, O] fp32 (O <= 16), state_in / state_out [B, D, O] or null.  Scratch: modal 4*D*16 floats
// (the prepared filter, which the backward takes over), S B*NC*D*16 floats.  D % 8 == 0, feat and z 16-byte aligned.
extern "C" int sb_li_fwd_tiled(const void* feat, const float* gamma, const float* p, const float* R, const float* bias,
                               const float* state_in, float* state_out, float* modal, float* S, void* z, int B, int L, int D, int O,
                               int TC, cudaStream_t st) {
  if ((D % 8) || O < 1 || O > LO || TC < 1 || ((uintptr_t)feat % 16) || ((uintptr_t)z % 16)) return -1;
  if ((long long)B * L * D == 0) return 0;
  LiDims d = li_dims(B, L, D, TC);
  const size_t n = (size_t)D * LO;
  const LiModal m{modal, modal + n, modal + 2 * n, modal + 3 * n, O};
  dim3 grid((D + LV_CH - 1) / LV_CH, d.NC, B);
  li_prep_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(gamma, p, R, modal, D, O);
  if (cudaGetLastError() != cudaSuccess) return -2;
  return li_fwd_chain(false, (const bf16*)feat, m, bias, state_in, state_out, S, (bf16*)z, grid, d, st);
}

extern "C" int sb_li_bwd_tiled_chunk() { return LB_TC; }

// function attributes belong to the current device's context: set on every call (they cost a lookup)
static bool li_bwd_tiled_ready() {
  return cudaFuncSetAttribute(li_bwd_local_tiled_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, LBL_SMEM) == cudaSuccess &&
         cudaFuncSetAttribute(li_bwd_apply_tiled_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, LBA_SMEM) == cudaSuccess &&
         cudaFuncSetAttribute(li_bwd_apply_tiled_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, LBA_SMEM) == cudaSuccess;
}

// Tiled backward, chunk length sb_li_bwd_tiled_chunk().  modal: as the forward left it.  Scratch: S, A, dRp B*NC*D*16 floats,
// dBp B*NC*D floats.  Outputs: dfeat, dR and dll = dgamma = dp [D, O], db [D], dstate_in [B, D, O] or null.
extern "C" int sb_li_bwd_tiled(const void* feat, const void* dz, const float* modal, const float* bias, const float* state_in,
                               const float* dstate_out, float* S, float* A, float* dRp, float* dBp, void* dfeat, float* dR,
                               float* dll, float* db, float* dstate_in, int B, int L, int D, int O, cudaStream_t st) {
  if ((D % 8) || O < 1 || O > LO || ((uintptr_t)feat % 16) || ((uintptr_t)dz % 16) || ((uintptr_t)dfeat % 16)) return -1;
  if ((long long)B * L * D == 0) return 0;
  if (!li_bwd_tiled_ready()) return -5;
  LiDims d = li_dims(B, L, D, LB_TC);
  const size_t n = (size_t)D * LO;
  const LiModal m{modal, modal + n, modal + 2 * n, modal + 3 * n, O};
  const int rc = dstate_out ? li_bwd_chain<true>((const bf16*)feat, (const bf16*)dz, m, bias, state_in, dstate_out, dstate_in, 1, S, A, dRp, A,
                                                dBp, (bf16*)dfeat, d, st)
                            : li_bwd_chain<false>((const bf16*)feat, (const bf16*)dz, m, bias, state_in, nullptr, dstate_in, 0, S, A, dRp, A,
                                                 dBp, (bf16*)dfeat, d, st);
  if (rc) return rc;
  const unsigned blocks = (unsigned)((n + LR_COLS - 1) / LR_COLS + (D + LR_COLS - 1) / LR_COLS);
  return launch_chained(false, li_bwd_reduce_kernel, dim3(blocks), LR_COLS * LR_SLICES, 0, st, (const float*)dRp, (const float*)A,
                        (const float*)dBp, m, dstate_out ? 0 : 1, dR, dll, db, B * d.NC, D);
}

// Scratch: S, W, A, dRp, dLp each B*NC*D*16 floats; dBp B*NC*D floats; dx1_tmp B*L*D bf16.
// Outputs: dfeat; per-chunk partials dRp/dLp/dBp (the caller sums over B and NC); w_end, dstate_in optional.  The tiled kernels
// run for chunks of sb_li_bwd_chunk(D, TC) steps; with a gradient of the final state, whose share of dlam the caller forms from
// w_end, the per-thread ones do.
extern "C" int sb_li_bwd(const void* feat, const void* dz, const float* loglam, const float* R, const float* bias,
                         const float* state_in, const float* dstate_out, float* S, float* W, float* A, float* dRp,
                         float* dLp, float* dBp, void* dx1_tmp, void* dfeat, float* w_end, float* dstate_in, int B, int L,
                         int D, int TC, cudaStream_t st) {
  if (B * L == 0) return 0;
  LiDims d = li_dims(B, L, D, TC);
  if (g_li_tiled && D % 8 == 0 && TC == LB_TC && !dstate_out && !w_end && aligned16(feat, dz, dfeat)) {
    if (!li_bwd_tiled_ready()) return -5;
    const LiModal m{loglam, nullptr, R, nullptr, LO};
    return li_bwd_chain<true>((const bf16*)feat, (const bf16*)dz, m, bias, state_in, nullptr, dstate_in, 1, S, A, dRp, dLp, dBp, (bf16*)dfeat, d,
                              st);
  }
  if (!dx1_tmp || !W) return -1;
  dim3 grid((D + LI_THREADS - 1) / LI_THREADS, d.NC, B);
  const size_t n = (size_t)B * D * LO;
  li_bwd_local_kernel<<<grid, LI_THREADS, 0, st>>>((const bf16*)feat, (const bf16*)dz, loglam, R, S, W, A, d);
  li_bwd_prefix_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(S, W, A, loglam, state_in, dstate_out, w_end, dstate_in, d);
  li_bwd_apply_fwd_kernel<<<grid, LI_THREADS, 0, st>>>((const bf16*)feat, (const bf16*)dz, loglam, R, bias, S, W,
                                                      (bf16*)dx1_tmp, dRp, dLp, dBp, d);
  li_bwd_apply_rev_kernel<<<grid, LI_THREADS, 0, st>>>((const bf16*)feat, (const bf16*)dz, loglam, R, bias, A,
                                                      (const bf16*)dx1_tmp, (bf16*)dfeat, dstate_out, d);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

static inline unsigned li_gate_grid(size_t n_vec) {
  size_t g = (n_vec + 255) / 256;
  const size_t cap = 2048;
  return (unsigned)(g > cap ? cap : (g < 1 ? 1 : g));
}

// out[n, D] = x2 v (mode 0) or x1 a (mode 1) for feat [n, 3D]; D % 8 == 0, 16-byte aligned rows.
extern "C" int sb_li_cp_gate(const void* feat, const void* a, void* out, long long n_rows, int D, int mode, cudaStream_t st) {
  if ((D % 8) || (mode == 1 && !a)) return -1;
  const size_t n_vec = (size_t)n_rows * (D / 8);
  if (n_vec == 0) return 0;
  li_cp_gate_kernel<<<li_gate_grid(n_vec), 256, 0, st>>>((const bf16*)feat, (const bf16*)a, (bf16*)out, n_vec, mode);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

extern "C" int sb_li_cp_finalize_bwd(const void* feat, const void* dz, const void* y, const void* du, void* dfeat,
                                     long long n_rows, int D, cudaStream_t st) {
  if (D % 8) return -1;
  const size_t n_vec = (size_t)n_rows * (D / 8);
  if (n_vec == 0) return 0;
  li_cp_finalize_bwd_kernel<<<li_gate_grid(n_vec), 256, 0, st>>>((const bf16*)feat, (const bf16*)dz, (const bf16*)y,
                                                                (const bf16*)du, (bf16*)dfeat, n_vec);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

static inline bool li_cp_map_ok(const LiCpMap* m, int L, int TC) {
  return m && m->n_chunks >= 1 && m->n_chunks <= 32 && m->chunk_len > 0 && (long long)m->chunk_len * m->n_chunks == L &&
         (m->chunk_len % TC) == 0;
}

// Channel-sharded forward scan of this rank (d channels, whole sequence L) with the exchange inside: u pulled from the
// owners' staging (u_in) into ufull [B, L, d], y stored into the owners' staging (y_out).  S: B*NC*d*16 floats.
extern "C" int sb_li_cp_fwd(const LiCpMap* u_in, const LiCpMap* y_out, const float* loglam, const float* R, const float* bias,
                            float* S, void* ufull, int B, int L, int d, int TC, cudaStream_t st) {
  if (B * L == 0) return 0;
  if (!li_cp_map_ok(u_in, L, TC) || !li_cp_map_ok(y_out, L, TC)) return -9;
  LiDims dm = li_dims(B, L, d, TC);
  dim3 grid((d + LI_THREADS - 1) / LI_THREADS, dm.NC, B);
  li_cp_local_kernel<<<grid, LI_THREADS, 0, st>>>(*u_in, (bf16*)ufull, loglam, S, dm);
  const size_t n = (size_t)B * d * LO;
  li_prefix_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(S, loglam, nullptr, nullptr, dm);
  li_cp_apply_kernel<<<grid, LI_THREADS, 0, st>>>((const bf16*)ufull, loglam, R, bias, S, *y_out, dm);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// Backward of the above: dy pulled from the owners (dy_in) into dyfull, y and du stored into the owners' staging.
// Scratch S, W, A, dRp, dLp: B*NC*d*16 floats each; dBp: B*NC*d floats (the caller sums the partials over B and NC).
extern "C" int sb_li_cp_bwd(const LiCpMap* dy_in, const LiCpMap* y_out, const LiCpMap* du_out, const void* ufull, void* dyfull,
                            const float* loglam, const float* R, const float* bias, float* S, float* W, float* A, float* dRp,
                            float* dLp, float* dBp, int B, int L, int d, int TC, cudaStream_t st) {
  if (B * L == 0) return 0;
  if (!li_cp_map_ok(dy_in, L, TC) || !li_cp_map_ok(y_out, L, TC) || !li_cp_map_ok(du_out, L, TC)) return -9;
  LiDims dm = li_dims(B, L, d, TC);
  dim3 grid((d + LI_THREADS - 1) / LI_THREADS, dm.NC, B);
  li_cp_bwd_local_kernel<<<grid, LI_THREADS, 0, st>>>((const bf16*)ufull, *dy_in, (bf16*)dyfull, loglam, R, S, W, A, dm);
  const size_t n = (size_t)B * d * LO;
  li_bwd_prefix_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(S, W, A, loglam, nullptr, nullptr, nullptr, nullptr, dm);
  li_cp_bwd_apply_fwd_kernel<<<grid, LI_THREADS, 0, st>>>((const bf16*)ufull, (const bf16*)dyfull, loglam, R, bias, S, W, *y_out,
                                                         dRp, dLp, dBp, dm);
  li_cp_bwd_apply_rev_kernel<<<grid, LI_THREADS, 0, st>>>((const bf16*)dyfull, loglam, R, bias, A, *du_out, dm);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// ------------------------------------------------------------------------------------ allocation-free variant
// See li_scan_noalloc.h for who needs this and for the contract.
#include <stdio.h>

#include "li_scan_noalloc.h"

// The chunk-state scratch of the forward scan, resident in the library's device image (one copy per GPU).
static __device__ __align__(256) float g_li_noalloc_scratch[SB_LI_NOALLOC_SCRATCH_BYTES / sizeof(float)];

// In host code the symbol above is only a handle; the kernels need its device address, looked up once per device.
static float* g_li_noalloc_ptr[64] = {nullptr};

extern "C" int sb_li_fwd_noalloc(const void* feat, const float* loglam, const float* R, const float* bias,
                                 const float* state_in, float* state_out, void* z, int B, int L, int D, int TC,
                                 cudaStream_t st) {
  if (B <= 0 || L <= 0 || D <= 0 || TC <= 0) return 0;
  LiDims d = li_dims(B, L, D, TC);
  const unsigned long long need = (unsigned long long)B * d.NC * D * LO * sizeof(float);
  if (need > SB_LI_NOALLOC_SCRATCH_BYTES) {
    fprintf(stderr,
            "sb_li_fwd_noalloc: B=%d L=%d D=%d TC=%d needs %llu bytes of chunk-state scratch, the built-in buffer holds "
            "%u; use sb_li_fwd with a caller-provided buffer\n", B, L, D, TC, need, SB_LI_NOALLOC_SCRATCH_BYTES);
    return SB_LI_NOALLOC_TOO_LARGE;
  }
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return SB_LI_NOALLOC_SETUP_FAILED;
  if (g_li_noalloc_ptr[dev] == nullptr) {
    float* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress((void**)&p, g_li_noalloc_scratch);
    if (e != cudaSuccess || p == nullptr) {
      fprintf(stderr, "sb_li_fwd_noalloc: cudaGetSymbolAddress failed on device %d: %s\n", dev, cudaGetErrorString(e));
      return SB_LI_NOALLOC_SETUP_FAILED;
    }
    g_li_noalloc_ptr[dev] = p;
  }
  return li_forward(feat, loglam, R, bias, state_in, state_out, g_li_noalloc_ptr[dev], z, d, st);
}
