// One decode step of a multi-hybrid model: every layer advances by one token from its cached state.
//
// A step is matrix-vector work: at batch <= 8 the time is the read of the weights and, on small models, the launches.  A
// layer is five kernels - norm + in-projection, state update, out-projection + residual, norm + w1|w2, gate + w3 +
// residual - issued by one host call for the whole model, where the operator-by-operator form takes about fifty.
//
//   dec_linear   out[b, n] = act_in(x)[b, :] . W[n, :] (+ bias) (+ residual): one warp per two output rows streams the bf16
//                weights in 16-byte loads against the inputs of all batch rows, which every block prepares in shared
//                memory (as they are, RMS-normalised, or gated); fp32 accumulation, one rounding of the result
//   dec_hyena    featuriser taps, gate and the recurrent form of the operator: a ring of past u for the FIR filters, the
//                modal states for the long filter.  Filters are read as their parameters are stored (decay window, poles
//                from gamma and p), so a step never works from an older copy of them
//   dec_attn     rotary embedding, append to the key / value cache, attention over the cache: the keys of one head are
//                split over a cluster of eight blocks that merge their partial softmax through distributed shared memory
//
// Rings are indexed by position: the row of time t lives in slot t mod n.
//
// Measured on a B200: four layers (one of each operator), width 1024, two sequences, a prompt of 517 tokens and 16 steps:
// 50.2 ms operator by operator (3 ms a step, all of it launches; the key / value cache was copied and converted to fp32 on
// every step), 3.6 ms with these kernels one after the other, 3.2 ms as programmatic dependents (with one scan less per Hyena-LI layer
// in the prefill).  Two rows per warp keep 3072 outputs on 192 blocks while every lane has eight 16-byte weight loads in flight.  By
// itself a matrix-vector kernel takes 6 us, a Hyena step 5 to 6, attention over 525 keys 9: launch gap, the first loads' latency and
// the reductions, not bandwidth, which is why a kernel is under way before the one in front of it has finished.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "pdl.cuh"

namespace sb {
namespace dec {
namespace cg = cooperative_groups;
typedef __nv_bfloat16 bf16;

constexpr int MAX_B = 8;
constexpr int THREADS = 256;
constexpr int ROWS_PER_WARP = 2;
constexpr int ROWS_PER_BLOCK = THREADS / 32 * ROWS_PER_WARP;
constexpr int AHEAD = 4;               // 16-byte weight loads per row and lane before the inputs are there: rows of up to 1024
constexpr int HD = 128;                // head dimension of dec_attn
constexpr int SPLIT = 8;               // blocks per head
constexpr int ATT_THREADS = 128;

enum { IN_PLAIN = 0, IN_NORM = 1, IN_GATE = 2 };
enum { OP_SE = 0, OP_MR = 1, OP_LI = 2, OP_ATTN = 3 };

// Bits of Layer::f32: the filter parameters stored in fp32 (the others are bf16).
enum { F_CONV = 1, F_TAPS = 2, F_DECAY = 4, F_BIAS = 8, F_GAMMA = 16, F_P = 32, F_R = 64 };

// Mirrors `_DecLayer` of inference/cached.py.
struct Layer {
  int kind, H, F, kf, K, G, O, heads, rd, act, pregate, postgate, form1, form2, norm2, cap;
  int f32, conv_g, tap_ld, newest_first;   // conv_g: groups of the featuriser; taps [G, tap_ld], of which K are used
  float eps1, eps2, pos_scale;
  const bf16 *norm1_w, *w_in, *w_out, *b_out, *norm2_w, *w12, *w3, *b3;
  const void *conv_w, *taps, *decay, *bias, *gamma, *p, *R;    // [conv_g, kf], [G, tap_ld] x2, [H], [G, O] x3
  const float* inv_freq;
  bf16* proj_ring;                     // [B, kf - 1, 3H]
  float* u_ring;                       // [B, K - 1, H]
  float* state;                        // [B, H, O]
  bf16 *kc, *vc;                       // [B, cap, heads, 128]
};

__device__ __forceinline__ float2 bf2(uint32_t w) { return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); }
__device__ __forceinline__ float rbf(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
__device__ __forceinline__ uint32_t pk(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float activation(float x, int act) {
  if (act == 0) return x / (1.f + expf(-x));
  if (act == 1) return 0.5f * x * (1.f + erff(x * 0.70710678118654752f));
  if (act == 2) return fmaxf(x, 0.f);
  return x;
}

// Type of a filter parameter: known at compile time (AS_BF16, AS_F32) or by its bit of Layer::f32 (AS_STORED).
enum { AS_STORED = 0, AS_BF16 = 1, AS_F32 = 2 };
template <int AS>
__device__ __forceinline__ float param(const void* p, size_t i, int bit) {
  const bool f32 = AS == AS_F32 || (AS == AS_STORED && bit);
  return f32 ? reinterpret_cast<const float*>(p)[i] : __bfloat162float(reinterpret_cast<const bf16*>(p)[i]);
}
// The taps of one channel, j = 0 the one of the oldest value.  With a decay window a tap is their product, which is rounded as
// the parameters' own type rounds it.
template <int AS>
struct Taps {
  const void *t, *d;
  size_t first;
  ptrdiff_t step;
  int f32;
  __device__ __forceinline__ Taps(const Layer& l, int ch)
      : t(l.taps), d(l.decay), first((size_t)(ch / (l.H / l.G)) * l.tap_ld + (l.newest_first ? l.K - 1 : 0)),
        step(l.newest_first ? -1 : 1), f32(l.f32) {}
  template <bool DECAY>
  __device__ __forceinline__ float at(int j) const {
    const size_t i = first + step * j;
    const float v = param<AS>(t, i, f32 & F_TAPS);
    if (!DECAY) return v;
    const float w = v * param<AS>(d, i, f32 & F_DECAY);
    return AS == AS_F32 || (f32 & (F_TAPS | F_DECAY)) ? w : rbf(w);
  }
};

// The kernels of a step are a chain of programmatic dependents (pdl.cuh): weights, filters, caches and states, which earlier steps left,
// are loaded ahead.
struct LinArgs {
  const bf16* x;          // [B, K] (IN_GATE: [B, 2K] = [a | b])
  const bf16* norm_w;
  const bf16* W;          // [N, K]
  const bf16* bias;       // [N] or null
  const bf16* res;        // [B, N] or null
  void* out;              // [B, N] bf16, or fp32 (out_f32)
  int B, K, N, mode, act, form, out_f32;
  float eps;
};

template <int BT>
__global__ void __launch_bounds__(THREADS)
dec_linear_kernel(LinArgs a) {
  extern __shared__ __align__(16) uint32_t xs[];          // [BT][K / 2] packed bf16
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, kv = a.K / 8;
  uint4* xv = reinterpret_cast<uint4*>(xs);
  let_next_start();
  const int n0 = (blockIdx.x * (THREADS / 32) + warp) * ROWS_PER_WARP;
  const uint4* wr[ROWS_PER_WARP];
#pragma unroll
  for (int r = 0; r < ROWS_PER_WARP; ++r) wr[r] = reinterpret_cast<const uint4*>(a.W + (size_t)min(n0 + r, a.N - 1) * a.K);
  // the first weights are on their way while the kernel before this one runs
  uint4 ahead[AHEAD][ROWS_PER_WARP];
#pragma unroll
  for (int k = 0; k < AHEAD; ++k)
#pragma unroll
    for (int r = 0; r < ROWS_PER_WARP; ++r)
      ahead[k][r] = lane + 32 * k < kv ? __ldg(wr[r] + lane + 32 * k) : make_uint4(0, 0, 0, 0);
  wait_for_previous();
  if (a.mode == IN_NORM) {
    if (warp < BT) {
      const int b = warp;
      if (b < a.B) {
        const uint4* src = reinterpret_cast<const uint4*>(a.x + (size_t)b * a.K);
        float ss = 0.f;
        for (int i = lane; i < kv; i += 32) {
          const uint4 q = src[i];
          const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) { const float2 f = bf2(w[j]); ss += f.x * f.x + f.y * f.y; }
        }
        ss = warp_sum(ss);
        const float r = a.form == 0 ? rsqrtf(ss / a.K + a.eps) : 1.f / (sqrtf(ss / a.K) + a.eps);
        const uint4* nw = reinterpret_cast<const uint4*>(a.norm_w);
        for (int i = lane; i < kv; i += 32) {
          const uint4 q = src[i], g = nw[i];
          const uint32_t w[4] = {q.x, q.y, q.z, q.w}, gw[4] = {g.x, g.y, g.z, g.w};
          uint32_t o[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) { const float2 f = bf2(w[j]), s = bf2(gw[j]); o[j] = pk(f.x * r * s.x, f.y * r * s.y); }
          xv[b * kv + i] = make_uint4(o[0], o[1], o[2], o[3]);
        }
      } else {
        for (int i = lane; i < kv; i += 32) xv[b * kv + i] = make_uint4(0, 0, 0, 0);
      }
    }
  } else {
    for (int i = tid; i < BT * kv; i += THREADS) {
      const int b = i / kv, c = i - b * kv;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (b < a.B) {
        if (a.mode == IN_PLAIN) {
          v = reinterpret_cast<const uint4*>(a.x + (size_t)b * a.K)[c];
        } else {
          const uint4 q = reinterpret_cast<const uint4*>(a.x + (size_t)b * 2 * a.K)[c];
          const uint4 g = reinterpret_cast<const uint4*>(a.x + (size_t)b * 2 * a.K + a.K)[c];
          const uint32_t w[4] = {q.x, q.y, q.z, q.w}, gw[4] = {g.x, g.y, g.z, g.w};
          uint32_t o[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 f = bf2(w[j]), s = bf2(gw[j]);
            o[j] = pk(activation(f.x, a.act) * s.x, activation(f.y, a.act) * s.y);
          }
          v = make_uint4(o[0], o[1], o[2], o[3]);
        }
      }
      xv[i] = v;
    }
  }
  __syncthreads();
  if (n0 >= a.N) return;
  float acc[ROWS_PER_WARP][BT];
#pragma unroll
  for (int r = 0; r < ROWS_PER_WARP; ++r)
#pragma unroll
    for (int b = 0; b < BT; ++b) acc[r][b] = 0.f;
  auto use = [&](const uint4 (&w)[ROWS_PER_WARP], int i) {
#pragma unroll
    for (int b = 0; b < BT; ++b) {
      const uint4 x = xv[b * kv + i];
      const uint32_t xw[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int r = 0; r < ROWS_PER_WARP; ++r) {
        const uint32_t ww[4] = {w[r].x, w[r].y, w[r].z, w[r].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = bf2(xw[j]), s = bf2(ww[j]);
          acc[r][b] = fmaf(f.x, s.x, acc[r][b]);
          acc[r][b] = fmaf(f.y, s.y, acc[r][b]);
        }
      }
    }
  };
#pragma unroll
  for (int k = 0; k < AHEAD; ++k)
    if (lane + 32 * k < kv) use(ahead[k], lane + 32 * k);
#pragma unroll 4
  for (int i = lane + 32 * AHEAD; i < kv; i += 32) {
    uint4 w[ROWS_PER_WARP];
#pragma unroll
    for (int r = 0; r < ROWS_PER_WARP; ++r) w[r] = __ldg(wr[r] + i);
    use(w, i);
  }
#pragma unroll
  for (int r = 0; r < ROWS_PER_WARP; ++r) {
    const int n = n0 + r;
    float mine = 0.f;
#pragma unroll
    for (int b = 0; b < BT; ++b) { const float s = warp_sum(acc[r][b]); if (lane == b) mine = s; }
    if (lane < a.B && lane < BT && n < a.N) {
      if (a.bias) mine += __bfloat162float(a.bias[n]);
      if (a.res) mine += __bfloat162float(a.res[(size_t)lane * a.N + n]);
      if (a.out_f32) reinterpret_cast<float*>(a.out)[(size_t)lane * a.N + n] = mine;
      else reinterpret_cast<bf16*>(a.out)[(size_t)lane * a.N + n] = __float2bfloat16_rn(mine);
    }
  }
}

// ------------------------------------------------------------------------------------ Hyena operators
// 32 channels of one batch row per block; eight slices share the filter taps (or modes) of a channel.
// The types of the parameters as they usually are (featuriser bf16, filter all bf16 or all fp32) are compiled in, and what does
// not need the new u comes before the first barrier, while one warp forms u: 6.1 us a launch for the medium and long filters at
// width 1024, two sequences, against 8.3 (average of all three) with a test of Layer::f32 at every load, which keeps the loads
// from being issued together, and everything after the barrier.
constexpr int HY_SLICES = 8;
__device__ __forceinline__ float tap_at(const float (&t)[4], int j) { return j == 0 ? t[0] : j == 1 ? t[1] : j == 2 ? t[2] : t[3]; }
template <int CONV, int FILT>
__global__ void __launch_bounds__(32 * HY_SLICES)
dec_hyena_kernel(Layer l, const bf16* proj, bf16* z, int pos) {
  __shared__ float su[32], sx1[32], sb[32], part[HY_SLICES][32];
  const int cx = threadIdx.x & 31, sl = threadIdx.x >> 5, ch = blockIdx.x * 32 + cx, b = blockIdx.y;
  const bool live = ch < l.H;
  let_next_start();
  if (sl == 0 && live) {
    float f[3];
    const int n = l.kf - 1;
    constexpr int TAPS = 4;                                // featuriser taps loaded ahead, with the past rows they multiply
    float past[3][TAPS], tap[3][TAPS];
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      const int c = 3 * ch + p;
      const size_t w = (size_t)(c / (3 * l.H / l.conv_g)) * l.kf;
      const bf16* ring = l.proj_ring + (size_t)b * n * 3 * l.H + c;
#pragma unroll
      for (int j = 0; j < TAPS; ++j) {
        tap[p][j] = j <= n ? param<CONV>(l.conv_w, w + j, l.f32 & F_CONV) : 0.f;
        past[p][j] = j < n ? __bfloat162float(ring[(size_t)((pos + j) % n) * 3 * l.H]) : 0.f;
      }
    }
    const float bias = l.kind == OP_SE ? 0.f : param<FILT>(l.bias, ch, l.f32 & F_BIAS);
    wait_for_previous();
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      const int c = 3 * ch + p;
      const size_t w = (size_t)(c / (3 * l.H / l.conv_g)) * l.kf;
      const int wf = l.f32 & F_CONV;
      const bf16 cur = proj[(size_t)b * 3 * l.H + c];
      bf16* ring = l.proj_ring + (size_t)b * n * 3 * l.H + c;
      float acc = (n < TAPS ? tap_at(tap[p], n) : param<CONV>(l.conv_w, w + n, wf)) * __bfloat162float(cur);
#pragma unroll
      for (int j = 0; j < TAPS; ++j)
        if (j < n) acc += tap[p][j] * past[p][j];
      for (int j = TAPS; j < n; ++j) acc += param<CONV>(l.conv_w, w + j, wf) * __bfloat162float(ring[(size_t)((pos + j) % n) * 3 * l.H]);
      if (n > 0) ring[(size_t)(pos % n) * 3 * l.H] = cur;
      f[p] = rbf(acc);                                     // the parallel path rounds the featuriser output
    }
    const float u = f[1] * f[2];
    sx1[cx] = f[0];
    su[cx] = (l.kind == OP_SE && !l.pregate) ? f[2] : u;
    sb[cx] = l.kind == OP_SE ? 0.f : bias * u;             // no bias, and without its pre-gate u may be what it likes
  }
  // what does not need the new u: the past of the FIR filters, the parameters and states of the first modes
  float y = 0.f;
  constexpr int MODES = 2;                                 // of this slice, held over the barrier: orders up to 16
  float lam[MODES], st[MODES], R[MODES];
  const size_t mode0 = live ? (size_t)(ch / (l.H / l.G)) * l.O : 0, st0 = ((size_t)b * l.H + ch) * l.O;
  auto mode = [&](int o, float& lm, float& s, float& r) {
    const size_t i = mode0 + o;
    s = l.state[st0 + o];
    r = param<FILT>(l.R, i, l.f32 & F_R);
    lm = expf(-expf(param<FILT>(l.p, i, l.f32 & F_P)) * expf(param<FILT>(l.gamma, i, l.f32 & F_GAMMA)));
  };
  if (live && l.kind == OP_LI) {
#pragma unroll
    for (int k = 0; k < MODES; ++k)
      if (sl + k * HY_SLICES < l.O) mode(sl + k * HY_SLICES, lam[k], st[k], R[k]);
  } else if (live) {
    const int n = l.K - 1, now = n > 0 ? pos % n : 0;
    const Taps<FILT> taps(l, ch);
    const float* ring = l.u_ring + (size_t)b * n * l.H + ch;
    auto past = [&](auto decay) {
#pragma unroll 8
      for (int j = sl; j < n; j += HY_SLICES) {
        int slot = now + j;
        if (slot >= n) slot -= n;
        y += taps.template at<decay.value>(j) * ring[(size_t)slot * l.H];
      }
    };
    if (l.decay) past(std::true_type{}); else past(std::false_type{});
  }
  __syncthreads();
  if (live && l.kind == OP_LI) {
    const float u = su[cx];
    auto advance = [&](int o, float lm, float s, float r) {
      s = lm * s + u;
      l.state[st0 + o] = s;
      y += r * s;
    };
#pragma unroll
    for (int k = 0; k < MODES; ++k)
      if (sl + k * HY_SLICES < l.O) advance(sl + k * HY_SLICES, lam[k], st[k], R[k]);
    for (int o = sl + MODES * HY_SLICES; o < l.O; o += HY_SLICES) {
      float lm, s, r;
      mode(o, lm, s, r);
      advance(o, lm, s, r);
    }
  }
  part[sl][cx] = y;
  __syncthreads();
  if (sl || !live) return;
#pragma unroll
  for (int j = 1; j < HY_SLICES; ++j) y += part[j][cx];
  if (l.kind != OP_LI) {
    const int n = l.K - 1;
    const Taps<FILT> taps(l, ch);
    y += (l.decay ? taps.template at<true>(n) : taps.template at<false>(n)) * su[cx];
    if (n > 0) l.u_ring[((size_t)b * n + pos % n) * l.H + ch] = su[cx];
  }
  y += sb[cx];
  z[(size_t)b * l.H + ch] = __float2bfloat16_rn((l.kind != OP_SE || l.postgate) ? sx1[cx] * y : y);
}

// ------------------------------------------------------------------------------------ attention
__global__ void __cluster_dims__(SPLIT, 1, 1) __launch_bounds__(ATT_THREADS)
dec_attn_kernel(Layer l, const bf16* proj, bf16* z, int pos) {
  __shared__ float raw[3][HD], sq[HD], sk[HD];
  __shared__ float wm[4], wl[4], wo[4][HD];
  __shared__ float cm, cl, co[HD];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int h = blockIdx.x / SPLIT, b = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bf16* row = proj + ((size_t)b * l.heads + h) * 3 * HD;
  const size_t ld = (size_t)l.heads * HD, base = ((size_t)b * l.cap * l.heads + h) * HD;
  const int chunk = (pos + SPLIT - 1) / SPLIT, j0 = rank * chunk, j1 = min(pos, j0 + chunk);
  let_next_start();
  for (int j = j0 + (tid >> 1); j < j1; j += ATT_THREADS / 2) {      // this block's keys and values: two 128-byte lines a row each
    const size_t off = base + (size_t)j * ld + (tid & 1) * 64;
    asm volatile("prefetch.global.L2 [%0];" ::"l"(l.kc + off));
    asm volatile("prefetch.global.L2 [%0];" ::"l"(l.vc + off));
  }
  wait_for_previous();
#pragma unroll
  for (int p = 0; p < 3; ++p) raw[p][tid] = __bfloat162float(row[p * HD + tid]);
  __syncthreads();
  {
    float q = raw[0][tid], k = raw[1][tid];
    if (tid < l.rd) {
      const int half = l.rd / 2, i = tid % half, o = tid < half ? tid + half : tid - half;
      const float ang = (float)pos / l.pos_scale * l.inv_freq[i], c = cosf(ang), s = sinf(ang), sg = tid < half ? -1.f : 1.f;
      q = q * c + sg * raw[0][o] * s;
      k = k * c + sg * raw[1][o] * s;
    }
    sq[tid] = rbf(q);
    sk[tid] = rbf(k);
  }
  if (rank == 0) {                                         // append the new token
    l.kc[base + (size_t)pos * ld + tid] = __float2bfloat16_rn(sk[tid]);
    l.vc[base + (size_t)pos * ld + tid] = row[2 * HD + tid];
  }
  __syncthreads();
  const float scale = 0.08838834764831845f;                // 1 / sqrt(128)
  float qf[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) qf[i] = sq[4 * lane + i];
  float m = -INFINITY, lsum = 0.f, o4[4] = {0.f, 0.f, 0.f, 0.f};
  constexpr int U = 4;
  for (int j = j0 + warp * U; j < j1; j += 4 * U) {
    uint2 kq[U], vq[U];
#pragma unroll
    for (int i = 0; i < U; ++i) {
      const size_t off = base + (size_t)min(j + i, j1 - 1) * ld + 4 * lane;
      kq[i] = *reinterpret_cast<const uint2*>(l.kc + off);
      vq[i] = *reinterpret_cast<const uint2*>(l.vc + off);
    }
    float s[U], mx = m;
#pragma unroll
    for (int i = 0; i < U; ++i) {
      const float2 a = bf2(kq[i].x), c = bf2(kq[i].y);
      s[i] = warp_sum(qf[0] * a.x + qf[1] * a.y + qf[2] * c.x + qf[3] * c.y) * scale;
      if (j + i >= j1) s[i] = -INFINITY;
      mx = fmaxf(mx, s[i]);
    }
    const float al = m == -INFINITY ? 0.f : expf(m - mx);
    m = mx;
    lsum *= al;
#pragma unroll
    for (int i = 0; i < 4; ++i) o4[i] *= al;
#pragma unroll
    for (int i = 0; i < U; ++i) {
      const float p = s[i] == -INFINITY ? 0.f : expf(s[i] - mx);
      const float2 a = bf2(vq[i].x), c = bf2(vq[i].y);
      lsum += p;
      o4[0] += p * a.x; o4[1] += p * a.y; o4[2] += p * c.x; o4[3] += p * c.y;
    }
  }
  if (rank == 0 && warp == 0) {                            // the new token's own key
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) s += qf[i] * sk[4 * lane + i];
    s = warp_sum(s) * scale;
    const float mx = fmaxf(m, s), al = m == -INFINITY ? 0.f : expf(m - mx), p = expf(s - mx);
    m = mx;
    lsum = lsum * al + p;
#pragma unroll
    for (int i = 0; i < 4; ++i) o4[i] = o4[i] * al + p * raw[2][4 * lane + i];
  }
  if (lane == 0) { wm[warp] = m; wl[warp] = lsum; }
#pragma unroll
  for (int i = 0; i < 4; ++i) wo[warp][4 * lane + i] = o4[i];
  __syncthreads();
  {
    float M = fmaxf(fmaxf(wm[0], wm[1]), fmaxf(wm[2], wm[3])), L = 0.f, O = 0.f;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const float e = wm[w] == -INFINITY ? 0.f : expf(wm[w] - M);
      L += e * wl[w];
      O += e * wo[w][tid];
    }
    co[tid] = O;
    if (tid == 0) { cm = M; cl = L; }
  }
  cluster.sync();
  if (rank == 0) {
    float M = -INFINITY, L = 0.f, O = 0.f;
    for (int r = 0; r < SPLIT; ++r) M = fmaxf(M, *cluster.map_shared_rank(&cm, r));
    for (int r = 0; r < SPLIT; ++r) {
      const float pm = *cluster.map_shared_rank(&cm, r), e = pm == -INFINITY ? 0.f : expf(pm - M);
      L += e * *cluster.map_shared_rank(&cl, r);
      O += e * *cluster.map_shared_rank(&co[tid], r);
    }
    z[((size_t)b * l.heads + h) * HD + tid] = __float2bfloat16_rn(O / L);
  }
  cluster.sync();                                          // peers' shared memory stays until it has been read
}

static int launch_hyena(const Layer& l, const bf16* proj, bf16* z, int B, int pos, cudaStream_t st) {
  const int used = l.kind == OP_SE ? F_TAPS : l.kind == OP_MR ? F_TAPS | F_BIAS | (l.decay ? F_DECAY : 0) : F_BIAS | F_GAMMA | F_P | F_R;
  const dim3 grid((l.H + 31) / 32, B);
  const int threads = 32 * HY_SLICES;
  auto* kernel = (l.f32 & F_CONV)            ? dec_hyena_kernel<AS_F32, AS_STORED>
                 : (l.f32 & used) == used    ? dec_hyena_kernel<AS_BF16, AS_F32>
                 : !(l.f32 & used)           ? dec_hyena_kernel<AS_BF16, AS_BF16>
                                             : dec_hyena_kernel<AS_BF16, AS_STORED>;
  return launch_chained(false, kernel, grid, threads, 0, st, l, proj, z, pos);
}

static int launch_linear(const LinArgs& a, cudaStream_t st, bool first = false) {
  const int blocks = (a.N + ROWS_PER_BLOCK - 1) / ROWS_PER_BLOCK;
  const int bt = a.B <= 1 ? 1 : a.B <= 2 ? 2 : a.B <= 4 ? 4 : 8;
  const size_t sm = (size_t)bt * a.K * 2;
  auto* kernel = bt == 1 ? dec_linear_kernel<1> : bt == 2 ? dec_linear_kernel<2> : bt == 4 ? dec_linear_kernel<4> : dec_linear_kernel<8>;
  if (sm > 48 * 1024 && cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm) != cudaSuccess) return -5;
  return launch_chained(first, kernel, dim3(blocks), THREADS, sm, st, a);
}

}  // namespace dec
}  // namespace sb

using namespace sb::dec;
using sb::launch_chained;

// Largest input width of a projection at batch B (its inputs have to fit in shared memory).
extern "C" int sb_decode_max_width(int B) { return B < 1 || B > MAX_B ? 0 : 200 * 1024 / 2 / (B <= 1 ? 1 : B <= 2 ? 2 : B <= 4 ? 4 : 8) / 8 * 8; }
extern "C" int sb_decode_layer_bytes() { return (int)sizeof(Layer); }

// Advances `n_layers` layers by the token at position `pos` (0-based: the caches hold `pos` earlier tokens).  x [B, D] bf16:
// the embedding of the token on entry, the residual stream on exit.  Scratch: proj [B, max 3H], z [B, max H], a [B, D],
// ab [B, max 2F], all bf16.  logits [B, V] fp32 through the final norm and w_head [V, D] unless w_head is null.
extern "C" int sb_decode_step(const Layer* layers, int n_layers, void* x, void* proj, void* z, void* a, void* ab, int B, int D, int pos,
                              const void* final_norm, float final_eps, int final_form, const void* w_head, int V, float* logits,
                              cudaStream_t st) {
  if (B < 1 || B > MAX_B || (D % 8) || pos < 0) return -1;
  bf16 *xb = (bf16*)x, *pb = (bf16*)proj, *zb = (bf16*)z, *abuf = (bf16*)a, *abb = (bf16*)ab;
  int rc = 0;
  for (int i = 0; i < n_layers && !rc; ++i) {
    const Layer& l = layers[i];
    if ((l.H % 8) || (l.F % 8) || (l.kind == OP_ATTN && pos >= l.cap)) return -1;
    rc = launch_linear(LinArgs{xb, l.norm1_w, l.w_in, nullptr, nullptr, pb, B, D, 3 * l.H, IN_NORM, 0, l.form1, 0, l.eps1}, st, i == 0);
    if (rc) return rc;
    rc = l.kind == OP_ATTN ? launch_chained(false, dec_attn_kernel, dim3(l.heads * SPLIT, B), ATT_THREADS, 0, st, l, (const bf16*)pb, zb, pos)
                           : launch_hyena(l, pb, zb, B, pos, st);
    if (rc) return rc;
    rc = launch_linear(LinArgs{zb, nullptr, l.w_out, l.b_out, xb, abuf, B, l.H, D, IN_PLAIN, 0, 0, 0, 0.f}, st);
    if (rc) return rc;
    rc = launch_linear(LinArgs{abuf, l.norm2_w, l.w12, nullptr, nullptr, abb, B, D, 2 * l.F, l.norm2 ? IN_NORM : IN_PLAIN, 0, l.form2, 0,
                               l.eps2}, st);
    if (rc) return rc;
    rc = launch_linear(LinArgs{abb, nullptr, l.w3, l.b3, abuf, xb, B, l.F, D, IN_GATE, l.act, 0, 0, 0.f}, st);
  }
  if (!rc && w_head)
    rc = launch_linear(LinArgs{xb, (const bf16*)final_norm, (const bf16*)w_head, nullptr, nullptr, logits, B, D, V, IN_NORM, 0, final_form,
                               1, final_eps}, st);
  if (rc) return rc;
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}
