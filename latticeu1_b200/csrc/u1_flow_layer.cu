// Fused coupling layers of the 2D U(1) flow: one kernel per layer and
// direction for proposals, one for its backward.  The reference has no flow;
// the method is that of Kanwar et al., arXiv:2003.06413.
//
// theta[b][mu][x1][x0] on an L x L lattice, layer (mu, off):
//   P(x) = th_0(x) + th_1(x+e0) - th_0(x+e1) - th_1(x);
//   context = (cos P, sin P) on the frozen plaquettes, 0 elsewhere;
//   hidden = LeakyReLU(conv3x3(context; W1, B1)), circular padding;
//   params = conv3x3(hidden; W2, B2) at the active plaquettes;
//   the mixture transform (u1_ncp.cuh) moves each active plaquette, its updated
//   link absorbs the change, and logdet[b] = sum of log H' over the active ones.
// Weights are rounded to bfloat16 on load, everything else is FP32.
//
// Stripe coordinates.  Let v run along nu = 1 - mu and u along the stripes.
// Within a period of four the active plaquettes are one row of v, s = 0, and
// (counting v downwards from it for mu = 1) the frozen ones are s = 1 and 2;
// s = 3 is neither.  So of conv2's inputs only the hidden rows s = -1, 0, 1
// are ever read, and of conv1's nine taps only those that land on a frozen
// row are not multiplied by zero:
//   s = -1: row 2 of the stripe below (dv = -1);  s = 0: row 1 (dv = +1);
//   s = +1: row 1 (dv = 0) and row 2 (dv = +1),
// 12 of 36 tap rows.  Both directions mu use this one picture: a pixel (j, u, s)
// is (x1, x0) = (off + 4j + s, u) for mu = 0 and (u, off - 1 - 4j - s) for mu = 1,
// and the weights are staged in (dv, du) order.
//
// Work split.  A pair of neighbouring active plaquettes (u, u + 1) of one
// configuration belongs to two threads, each of which sums all 2K + 1 parameters
// of both over half of the hidden channels, in registers; they exchange the
// halves and each takes one plaquette through the transform.  Per hidden channel
// and row a thread reads four hidden values and the 3 (2K + 2) weights, which all
// its warp shares, for 12 (K + 1) multiply-adds, issued in pairs (fma.rn.f32x2).
// A block holds as many configurations as balance the SMs best (flow_nc).
//
// B200, 32 hidden channels, K = 6, batch 1024: forward 295 -> 109 us at L = 32
// and 85 -> 34 us at L = 16, backward 2255 -> 366 us and about 550 -> 117 us,
// against one configuration per 512-thread block, a shared read per multiply-add
// operand and all nine taps.  Both are now bound about evenly by the
// multiply-add pipe (47 % and 41 % of its cycles) and shared-memory wavefronts
// (52 % and 67 %) at 16 warps per SM, which the registers of the sums allow.
#include <cuda_bf16.h>

#include <algorithm>
#include <string>

#include "u1_internal.h"
#include "u1_ncp.cuh"

namespace {

int flfail(int code, const std::string &msg) {
  u1i::set_error(msg);
  return code;
}

constexpr int kFwdThreads = 512;
constexpr int kBwdThreads = 256;
constexpr int kChunk = 8;  // hidden channels held in shared memory at a time, half of them per thread of a pair

using F2 = unsigned long long;  // two packed floats

__device__ __forceinline__ F2 pack2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 unpack2(F2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ void fma2(F2 &acc, F2 a, F2 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float bf16_round(float v) { return __bfloat162float(__float2bfloat16(v)); }
__device__ __forceinline__ float lrelu(float v, float slope) { return v > 0.f ? v : slope * v; }

struct FlowK {
  const float *th_in;
  int batch, L, mu, off, H;
  const float *W1, *B1, *W2, *B2;
  float slope;
  int nc;     // configurations per block
  int lp;     // row pitch: u = -1 .. L at columns 1 .. L + 2
  int rp;     // pitch of one hidden row class (all rows of the block), = 2 mod 32
  int cp;     // pitch of one context plane, in (cos, sin) pairs
  // forward
  float *th_out, *logdet;
  // backward
  const float *gth_out, *gld;
  float *gth_in, *wpart;
  int nw;     // weight-gradient entries
  u1b::FastDivK dL, dLL2, dact, dtp, dhp;  // divisions by L, 2 L^2, L^2/4, L^2/8, L/2
};
__device__ __forceinline__ int div_by(int n, u1b::FastDivK d) { return (int)u1b::fast_div((uint32_t)n, d); }

// Floats between the weights of consecutive (channel, row) pairs: three taps
// of 2 NP outputs, whole 16-byte words.
template <int NP>
struct FlowDims {
  static constexpr int K = NP - 1, C2 = 2 * K + 1;
  static constexpr int WS = (6 * NP + 3) & ~3;
  static constexpr int NG = (2 * NP + 3) / 4;   // groups of four outputs
  static constexpr int GP = 4 * (NG | 1);       // pitch of a plaquette's parameter gradients (an odd number of groups)
};

// Pixel (x1 * L + x0) of stripe coordinates (v = 4 j + s >= -1, u).
__device__ __forceinline__ int flow_pixel(const FlowK &f, int v, int u) {
  if (f.mu == 0) {
    int x1 = f.off + v;
    x1 = x1 < 0 ? x1 + f.L : x1 >= f.L ? x1 - f.L : x1;
    return x1 * f.L + u;
  }
  int x0 = f.off - 1 - v;
  x0 = x0 < 0 ? x0 + f.L : x0;
  x0 = x0 < 0 ? x0 + f.L : x0;
  return u * f.L + x0;
}
// Weight offset ky * 3 + kx of tap (dv, du) = (dvi - 1, dui - 1).
__device__ __forceinline__ int flow_tap(int mu, int dvi, int dui) { return mu == 0 ? dvi * 3 + dui : dui * 3 + 2 - dvi; }

__device__ __forceinline__ float plaq_angle(const FlowK &f, const float *__restrict__ th, int p) {
  const int L = f.L, LL = L * L, x1 = div_by(p, f.dL), x0 = p - x1 * L;
  const int x0p = x0 + 1 == L ? 0 : x0 + 1, x1p = x1 + 1 == L ? 0 : x1 + 1;
  return th[p] + th[LL + x1 * L + x0p] - th[x1p * L + x0] - th[LL + p];
}

// The thread's pair of active plaquettes and its half of the channels.
struct FlowSite {
  int g;          // which half; also the plaquette of the pair it transforms
  int peer;       // thread holding the other half
  int cfg, j, u;  // configuration within the block, stripe, first u
  int at;         // row * lp + u + 2 (row = cfg * stripes + j)
  int up, dn;     // the same in the next / previous stripe
  bool live;
};
__device__ __forceinline__ FlowSite flow_site(const FlowK &f) {
  FlowSite s;
  const int hp = f.L / 2, ns = f.L / 4, tp = hp * ns, pairs = f.nc * tp, t = (int)threadIdx.x;
  s.g = t >= pairs ? 1 : 0;
  const int pair = t - s.g * pairs;
  s.peer = s.g ? pair : pair + pairs;
  s.cfg = div_by(pair, f.dtp);
  const int r = pair - s.cfg * tp;
  s.j = div_by(r, f.dhp);
  s.u = 2 * (r - s.j * hp);
  s.live = pair < pairs && (int)blockIdx.x * f.nc + s.cfg < f.batch;
  const int row = s.cfg * ns, jn = s.j + 1 == ns ? 0 : s.j + 1, jp = s.j == 0 ? ns - 1 : s.j - 1;
  s.at = (row + s.j) * f.lp + s.u + 2;
  s.up = (row + jn) * f.lp + s.u + 2;
  s.dn = (row + jp) * f.lp + s.u + 2;
  return s;
}

// A pair's two values at s.at of a padded plane, with the copies beyond the row's ends.
__device__ __forceinline__ void store_pair(float *plane, const FlowK &f, const FlowSite &s, float a, float b) {
  *reinterpret_cast<float2 *>(plane + s.at) = make_float2(a, b);
  if (s.u == 0) plane[s.at + f.L] = a;
  if (s.u == f.L - 2) plane[s.at - f.L + 1] = b;
}
// Values at u - 1 .. u + 2 of a padded plane.
__device__ __forceinline__ void load_window(const float *plane, int at, float (&w)[4]) {
  w[0] = plane[at - 1];
  const float2 m = *reinterpret_cast<const float2 *>(plane + at);
  w[1] = m.x;
  w[2] = m.y;
  w[3] = plane[at + 2];
}

// Weights in (dv, du) order: w1[c][20] = ([dv][du][ci], bias), w2[(c * 3 + dv) * WS + du * 2 NP + o], b2[2 NP].
template <int NP>
__device__ __forceinline__ void stage_weights(const FlowK &f, float *w1, float *w2, float *b2) {
  constexpr int WS = FlowDims<NP>::WS, C2 = FlowDims<NP>::C2;
  const int nt = (int)blockDim.x, H = f.H;
  for (int t = (int)threadIdx.x; t < 20 * H; t += nt) {
    const int c = t / 20, r = t - 20 * c;
    const int ci = r & 1, k = r >> 1;
    w1[t] = r < 18 ? bf16_round(f.W1[c * 18 + ci * 9 + flow_tap(f.mu, k / 3, k % 3)]) : r == 18 ? bf16_round(f.B1[c]) : 0.f;
  }
  constexpr int PADS = WS - 3 * C2;  // entries of a (channel, row) that hold no weight
  for (int t = (int)threadIdx.x; t < 3 * H * PADS; t += nt) {
    const int r = t / PADS, e = t - r * PADS;
    w2[r * WS + (e < 3 ? e * 2 * NP + C2 : 6 * NP + e - 3)] = 0.f;
  }
#pragma unroll 8
  for (int t = (int)threadIdx.x; t < C2 * H * 9; t += nt) {  // in memory order: o, channel, ky, kx
    const int oc = t / 9, k = t - 9 * oc, ky = k / 3, kx = k - 3 * ky;
    const int o = oc / H, c = oc - o * H;
    const int dvi = f.mu == 0 ? ky : 2 - kx, dui = f.mu == 0 ? kx : ky;
    w2[(c * 3 + dvi) * WS + dui * 2 * NP + o] = bf16_round(f.W2[t]);
  }
  for (int t = (int)threadIdx.x; t < 2 * NP; t += nt) b2[t] = t < C2 ? bf16_round(f.B2[t]) : 0.f;
}

// (cos P, sin P) of the frozen plaquettes: planes ctx[row * cp].
__device__ __forceinline__ void fill_context(const FlowK &f, float2 *ctx) {
  const int L = f.L, nact = L * L / 4, n = f.nc * 2 * nact;
  for (int t = (int)threadIdx.x; t < n; t += (int)blockDim.x) {
    const int q = div_by(t, f.dact), cfg = q >> 1, row = q & 1;
    const int a = t - q * nact, j = div_by(a, f.dL), u = a - j * L;
    const int b = (int)blockIdx.x * f.nc + cfg;
    float2 v = make_float2(0.f, 0.f);
    if (b < f.batch)
      sincosf(plaq_angle(f, f.th_in + (size_t)b * 2 * L * L, flow_pixel(f, 4 * j + 1 + row, u)), &v.y, &v.x);
    float2 *c = ctx + row * f.cp + (cfg * (L / 4) + j) * f.lp;
    c[u + 2] = v;
    if (u == 0) c[L + 2] = v;
    if (u == L - 1) c[1] = v;
  }
}

// The context a pair's hidden values read: rows 2 (stripe below), 1 and 2 (own), u - 1 .. u + 2.
struct CtxWindow {
  F2 a[4], b[4], c[4];  // (cos, sin) pairs
};
__device__ __forceinline__ void load_window2(const float2 *plane, int at, F2 (&w)[4]) {
  w[0] = *reinterpret_cast<const F2 *>(plane + at - 1);
  const ulonglong2 m = *reinterpret_cast<const ulonglong2 *>(plane + at);
  w[1] = m.x;
  w[2] = m.y;
  w[3] = *reinterpret_cast<const F2 *>(plane + at + 2);
}
__device__ __forceinline__ void load_context(const FlowK &f, const FlowSite &s, const float2 *ctx, CtxWindow &x) {
  load_window2(ctx + f.cp, s.dn, x.a);
  load_window2(ctx, s.at, x.b);
  load_window2(ctx + f.cp, s.at, x.c);
}
// One channel's conv1 weights: pairs over ci of tap (dv, du), and the bias.
struct W1Row {
  F2 w[9];
  float bias;
};
__device__ __forceinline__ W1Row load_w1(const float *w1c) {
  W1Row r;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const ulonglong2 v = reinterpret_cast<const ulonglong2 *>(w1c)[q];
    r.w[2 * q] = v.x;
    r.w[2 * q + 1] = v.y;
  }
  const ulonglong2 v = reinterpret_cast<const ulonglong2 *>(w1c)[4];
  r.w[8] = v.x;
  r.bias = unpack2(v.y).x;
  return r;
}
// conv1 pre-activations of one channel: pre[row s = -1, 0, 1][pixel].
__device__ __forceinline__ void conv1_pair(const W1Row &r, const CtxWindow &x, float (&pre)[3][2]) {
#pragma unroll
  for (int px = 0; px < 2; ++px) {
    F2 p0 = pack2(r.bias, 0.f), p1 = p0, p2 = p0;
#pragma unroll
    for (int du = 0; du < 3; ++du) {
      fma2(p0, r.w[du], x.a[px + du]);
      fma2(p1, r.w[6 + du], x.b[px + du]);
      fma2(p2, r.w[3 + du], x.b[px + du]);
      fma2(p2, r.w[6 + du], x.c[px + du]);
    }
    const float2 e0 = unpack2(p0), e1 = unpack2(p1), e2 = unpack2(p2);
    pre[0][px] = e0.x + e0.y;
    pre[1][px] = e1.x + e1.y;
    pre[2][px] = e2.x + e2.y;
  }
}

// acc[pixel][output pair] += conv2 taps of one (channel, row) pair.
template <int NP>
__device__ __forceinline__ void conv2_pair(const float *w2, const float (&h)[4], F2 (&acc)[2][NP]) {
  constexpr int NW = FlowDims<NP>::WS / 4;
  F2 w[2 * NW], hh[4];
#pragma unroll
  for (int q = 0; q < NW; ++q) {
    const ulonglong2 v = reinterpret_cast<const ulonglong2 *>(w2)[q];
    w[2 * q] = v.x;
    w[2 * q + 1] = v.y;
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) hh[k] = pack2(h[k], h[k]);
#pragma unroll
  for (int du = 0; du < 3; ++du)
#pragma unroll
    for (int n = 0; n < NP; ++n) {
      fma2(acc[0][n], w[du * NP + n], hh[du]);
      fma2(acc[1][n], w[du * NP + n], hh[du + 1]);
    }
}

// Parameters (a_0..a_{K-1}, logit_0..logit_{K-1}, shift) of plaquette u + g of the
// pair; every thread of the block must call it.  hid is free on return.
template <int NP>
__device__ __forceinline__ void layer_params(const FlowK &f, const FlowSite &s, const float2 *ctx, const float *w1,
                                             const float *w2, const float *b2, float *hid, float (&prm)[2 * NP]) {
  F2 acc[2][NP];
#pragma unroll
  for (int n = 0; n < NP; ++n)
    acc[0][n] = acc[1][n] = s.g ? pack2(0.f, 0.f) : pack2(b2[2 * n], b2[2 * n + 1]);
  CtxWindow x;
  if (s.live) load_context(f, s, ctx, x);
  for (int c0 = 0; c0 < f.H; c0 += kChunk) {
    const int half = min(kChunk, f.H - c0) / 2, first = s.g * half;  // H is a multiple of 4
    if (s.live)
      for (int cl = first; cl < first + half; ++cl) {
        float pre[3][2];
        conv1_pair(load_w1(w1 + 20 * (c0 + cl)), x, pre);
#pragma unroll
        for (int r = 0; r < 3; ++r)
          store_pair(hid + (cl * 3 + r) * f.rp, f, s, lrelu(pre[r][0], f.slope), lrelu(pre[r][1], f.slope));
      }
    __syncthreads();
    if (s.live)
#pragma unroll 2
      for (int q = 3 * first; q < 3 * (first + half); ++q) {
        float h[4];
        load_window(hid + q * f.rp, s.at, h);
        conv2_pair<NP>(w2 + (3 * c0 + q) * FlowDims<NP>::WS, h, acc);
      }
    __syncthreads();
  }
  // the two halves: each thread hands over its sums of the other's plaquette
  F2 *swap = reinterpret_cast<F2 *>(hid);
  const int nt = (int)blockDim.x;
#pragma unroll
  for (int n = 0; n < NP; ++n) swap[n * nt + threadIdx.x] = s.g ? acc[0][n] : acc[1][n];
  __syncthreads();
#pragma unroll
  for (int n = 0; n < NP; ++n) {
    const float2 a = unpack2(s.g ? acc[1][n] : acc[0][n]);
    const float2 b = unpack2(s.live ? swap[n * nt + s.peer] : 0ull);
    prm[2 * n] = a.x + b.x;
    prm[2 * n + 1] = a.y + b.y;
  }
  __syncthreads();
}

// Shared memory: w1[20 H], w2[3 H WS], b2[20], ctx[4 cp], hid[max(3 kChunk rp, 2 NP threads)].
template <int NP, bool INV>
__global__ void __launch_bounds__(kFwdThreads, 1) k_flow_forward(const FlowK f) {
  constexpr int K = FlowDims<NP>::K;
  extern __shared__ float4 flow_sm[];
  float *w1 = reinterpret_cast<float *>(flow_sm);
  float *w2 = w1 + 20 * f.H;
  float *b2 = w2 + 3 * f.H * FlowDims<NP>::WS;
  float2 *ctx = reinterpret_cast<float2 *>(b2 + 20);
  float *hid = reinterpret_cast<float *>(ctx + 2 * f.cp);
  __shared__ double ld[kFwdThreads];
  const FlowSite s = flow_site(f);
  const int L = f.L, LL = L * L, b0 = (int)blockIdx.x * f.nc;
  const int ncfg = min(f.nc, f.batch - b0);
  stage_weights<NP>(f, w1, w2, b2);
  fill_context(f, ctx);
  // links the layer leaves unchanged
  for (int t = (int)threadIdx.x; t < ncfg * 2 * LL; t += (int)blockDim.x) {
    const int e = t - div_by(t, f.dLL2) * 2 * LL, comp = e >= LL ? 1 : 0, p = e - comp * LL;
    const int x1 = div_by(p, f.dL);
    const bool updated = comp == f.mu && (((f.mu == 0 ? x1 : p - x1 * L) - f.off) & 3) == 0;
    if (!updated) f.th_out[(size_t)b0 * 2 * LL + t] = f.th_in[(size_t)b0 * 2 * LL + t];
  }
  __syncthreads();
  float prm[2 * NP];
  layer_params<NP>(f, s, ctx, w1, w2, b2, hid, prm);
  float lg = 0.f;
  if (s.live) {
    const float *th = f.th_in + (size_t)(b0 + s.cfg) * 2 * LL;
    const int p = flow_pixel(f, 4 * s.j, s.u + s.g);
    const float dy = u1b::ncp_transform<K, INV>(plaq_angle(f, th, p), prm, lg);
    const int x1 = div_by(p, f.dL), x0 = p - x1 * L;
    const int link = f.mu == 0 ? p : LL + x1 * L + (x0 + 1 == L ? 0 : x0 + 1);
    f.th_out[(size_t)(b0 + s.cfg) * 2 * LL + link] = th[link] + dy;
  }
  ld[threadIdx.x] = (double)lg;
  __syncthreads();
  // log-det of each configuration: eight threads add strided shares, in order
  const int tp = LL / 8, pairs = f.nc * tp, grp = (int)threadIdx.x & 7;
  for (int c = (int)threadIdx.x >> 3; c < ncfg; c += (int)blockDim.x / 8) {
    double v = 0.0;
    for (int t = grp; t < tp; t += 8) v += ld[c * tp + t] + ld[pairs + c * tp + t];
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) v += __shfl_xor_sync(0xffu << (threadIdx.x & 24), v, o);
    if (grp == 0) f.logdet[b0 + c] = (float)v;
  }
}

// Backward of k_flow_forward<INV>: the parameters are recomputed, then, given
// gth_out (dL/dtheta_out) and gld (dL/dlogdet), the adjoint runs back through
// the transform, conv2, the LeakyReLU, conv1, the context and the plaquettes:
//   gth_in = gth_out + plaquette-adjoint(gP),
//   gP = [active] d/dP of the transform + [frozen] (-sin P, cos P) . g_context.
// kChunk hidden channels are in shared memory at a time (their values and the
// gradients of their pre-activations).  Per (channel, row) a thread forms the
// two gradients of its pair from the parameter gradients of the four
// neighbouring plaquettes, which it keeps in registers.  Weight gradients are
// sums over plaquettes: a lane owns one channel and four outputs (W2) or one
// channel and input (W1) and walks along stripes with a sliding window, so a
// step of u costs one shared read per row; lanes and warps are then added in a
// fixed order and each block stores one partial row, summed over blocks in
// order by k_flow_wgrad_reduce.  No atomics.
// Shared memory (floats): w1[20 H], w2[3 H WS], b2[20], ctx[4 cp],
// gprm[nc nact GP], work[max(6 kChunk rp, warps kChunk (9 GP + 20), 2 NP threads, nc LL)]:
// the chunk's hidden values and gradients, then the warps' weight-gradient
// sums; at the end gP.
template <int NP, bool INV>
__global__ void __launch_bounds__(kBwdThreads, 2) k_flow_backward(const FlowK f) {
  using Dm = FlowDims<NP>;
  constexpr int K = Dm::K, C2 = Dm::C2, GP = Dm::GP, WS = Dm::WS, NG = Dm::NG;
  constexpr int NGP = NG <= 1 ? 1 : NG <= 2 ? 2 : 4;  // output groups taken at once (five in two goes)
  constexpr int AS2 = 32 / (kChunk * NGP);            // stripe shares of a warp (W2)
  extern __shared__ float4 flow_sm[];
  const int L = f.L, LL = L * L, ns = L / 4, nact = LL / 4;
  const int nt = (int)blockDim.x, tid = (int)threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = nt >> 5;
  float *w1 = reinterpret_cast<float *>(flow_sm);
  float *w2 = w1 + 20 * f.H;
  float *b2 = w2 + 3 * f.H * WS;
  float2 *ctx = reinterpret_cast<float2 *>(b2 + 20);
  float *gprm = reinterpret_cast<float *>(ctx + 2 * f.cp);
  float *hid = gprm + f.nc * nact * GP;
  float *ghid = hid + 3 * kChunk * f.rp;
  float *red2 = hid, *red1 = red2 + nwarps * kChunk * 9 * GP, *gP = hid;
  const FlowSite s = flow_site(f);
  const int b0 = (int)blockIdx.x * f.nc, ncfg = min(f.nc, f.batch - b0), nrows = ncfg * ns;
  stage_weights<NP>(f, w1, w2, b2);
  fill_context(f, ctx);
  __syncthreads();
  float g_active = 0.f;  // dL/dP of the thread's active plaquette
  {
    float prm[2 * NP];
    layer_params<NP>(f, s, ctx, w1, w2, b2, hid, prm);
    // ---- transform adjoint: parameter gradients and the active plaquettes' gP
    if (s.live) {
      const float *th = f.th_in + (size_t)(b0 + s.cfg) * 2 * LL, *go = f.gth_out + (size_t)(b0 + s.cfg) * 2 * LL;
      const int p = flow_pixel(f, 4 * s.j, s.u + s.g);
      const int x1 = div_by(p, f.dL), x0 = p - x1 * L;
      const int link = f.mu == 0 ? p : LL + x1 * L + (x0 + 1 == L ? 0 : x0 + 1);
      float gq[2 * NP];
      u1b::ncp_transform_backward<K, INV>(plaq_angle(f, th, p), prm, go[link], f.gld ? f.gld[b0 + s.cfg] : 0.f,
                                          g_active, gq);
      gq[2 * NP - 1] = 0.f;
      float *dst = gprm + ((s.cfg * ns + s.j) * L + s.u + s.g) * GP;
#pragma unroll
      for (int o = 0; o < GP; ++o) dst[o] = o < 2 * NP ? gq[o < 2 * NP ? o : 0] : 0.f;
    }
  }
  __syncthreads();
  float *wp = f.wpart + (size_t)blockIdx.x * f.nw;
  // a row of partial sums, in (dv, du) order: W1[c][dv][du][ci], B1[c], W2[c][dv][du][o], B2[o]
  float *gW1 = wp, *gB1 = wp + f.H * 18, *gW2 = gB1 + f.H, *gB2 = gW2 + C2 * f.H * 9;
  for (int o = warp; o < C2; o += nwarps) {  // gB2[o] = sum of the parameter gradients
    float v = 0.f;
    for (int a = lane; a < ncfg * nact; a += 32) v += gprm[a * GP + o];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    if (lane == 0) gB2[o] = v;
  }
  // parameter gradients of the plaquettes u - 1 .. u + 2 of the thread's stripe
  F2 gq[4][NP];
  if (s.live) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      int u = s.u + k - 1;
      u = u < 0 ? u + L : u >= L ? u - L : u;
      const float2 *src = reinterpret_cast<const float2 *>(gprm + ((s.cfg * ns + s.j) * L + u) * GP);
#pragma unroll
      for (int n = 0; n < NP; ++n) {
        const float2 v = src[n];
        gq[k][n] = pack2(v.x, v.y);
      }
    }
  }
  F2 gc[2][2];  // context gradients [frozen row][pixel], pairs over ci, over the thread's channels
#pragma unroll
  for (int q = 0; q < 4; ++q) gc[q >> 1][q & 1] = pack2(0.f, 0.f);
  for (int c0 = 0; c0 < f.H; c0 += kChunk) {
    const int nch = min(kChunk, f.H - c0), first = s.g * (nch / 2);
    if (s.live) {
      CtxWindow x;
      load_context(f, s, ctx, x);
      for (int cl = first; cl < first + nch / 2; ++cl) {
        float pre[3][2];
        conv1_pair(load_w1(w1 + 20 * (c0 + cl)), x, pre);
#pragma unroll
        for (int r = 0; r < 3; ++r) {
          // dL/dh(u) = sum_du sum_o W2[o][c][r][du] gprm[u - du][o]
          F2 a0 = pack2(0.f, 0.f), a1 = a0;
          const ulonglong2 *wr = reinterpret_cast<const ulonglong2 *>(w2 + (3 * (c0 + cl) + r) * WS);
#pragma unroll
          for (int q = 0; q < (3 * NP + 1) / 2; ++q) {
            const ulonglong2 w = wr[q];
            const int du = (2 * q) / NP, n = 2 * q - du * NP, du1 = (2 * q + 1) / NP, n1 = 2 * q + 1 - du1 * NP;
            fma2(a0, w.x, gq[2 - du][n]);
            fma2(a1, w.x, gq[3 - du][n]);
            if (2 * q + 1 < 3 * NP) {
              fma2(a0, w.y, gq[2 - (du1 < 3 ? du1 : 0)][n1]);
              fma2(a1, w.y, gq[3 - (du1 < 3 ? du1 : 0)][n1]);
            }
          }
          const float2 e0 = unpack2(a0), e1 = unpack2(a1);
          const float d0 = e0.x + e0.y, d1 = e1.x + e1.y;
          store_pair(hid + (cl * 3 + r) * f.rp, f, s, lrelu(pre[r][0], f.slope), lrelu(pre[r][1], f.slope));
          store_pair(ghid + (cl * 3 + r) * f.rp, f, s, pre[r][0] > 0.f ? d0 : f.slope * d0,
                     pre[r][1] > 0.f ? d1 : f.slope * d1);
        }
      }
    }
    __syncthreads();
    // ---- gW2[o][c][dv][du] = sum_a gprm[a][o] h[c][dv](u + du), by half rows
    constexpr int GO = (NG + NGP - 1) / NGP;  // goes
    const int half = L / 2;
    const int cl2 = (lane / NGP) % kChunk, as2 = lane / (NGP * kChunk);
    F2 acc2[GO][9][2];
#pragma unroll
    for (int go = 0; go < GO; ++go) {
      const int og = go * NGP + lane % NGP;
#pragma unroll
      for (int k = 0; k < 9; ++k) acc2[go][k][0] = acc2[go][k][1] = pack2(0.f, 0.f);
      if (og < NG && cl2 < nch)
        for (int it = warp * AS2 + as2; it < 2 * nrows; it += nwarps * AS2) {
          const int row = it >> 1, u0 = (it & 1) * half;
          const float *h0 = hid + cl2 * 3 * f.rp + row * f.lp + u0 + 1;  // u0 - 1
          F2 w[3][3];
#pragma unroll
          for (int r = 0; r < 3; ++r) {
            const float *hr = h0 + r * f.rp;
            w[r][1] = pack2(hr[0], hr[0]);
            w[r][2] = pack2(hr[1], hr[1]);
          }
          const ulonglong2 *gr = reinterpret_cast<const ulonglong2 *>(gprm + (row * L + u0) * GP + 4 * og);
#pragma unroll 4
          for (int u = 0; u < half; ++u) {
            const ulonglong2 g = gr[u * (GP / 4)];
#pragma unroll
            for (int r = 0; r < 3; ++r) {
              const float v = h0[r * f.rp + u + 2];
              w[r][0] = w[r][1];
              w[r][1] = w[r][2];
              w[r][2] = pack2(v, v);
#pragma unroll
              for (int du = 0; du < 3; ++du) {
                fma2(acc2[go][r * 3 + du][0], g.x, w[r][du]);
                fma2(acc2[go][r * 3 + du][1], g.y, w[r][du]);
              }
            }
          }
        }
    }
    // ---- gW1[c][ci][dv][du] = sum over hidden pixels of dL/dpre ctx (pairs over ci), gB1[c] = sum of
    // dL/dpre, by quarter rows
    const int quarter = L / 4, cl1 = lane & 7, as1 = lane >> 3;
    F2 acc1[9];
    float accb = 0.f;
#pragma unroll
    for (int k = 0; k < 9; ++k) acc1[k] = pack2(0.f, 0.f);
    if (cl1 < nch)
      for (int it = warp * 4 + as1; it < 4 * nrows; it += nwarps * 4) {
        const int row = it >> 2, u0 = (it & 3) * quarter, cfg = div_by(row * L, f.dact);
        const int below = row == cfg * ns ? row + ns - 1 : row - 1;
        const float *g0 = ghid + cl1 * 3 * f.rp + row * f.lp + 2;
        const F2 *cb = reinterpret_cast<const F2 *>(ctx) + row * f.lp + 2, *cc = cb + f.cp;
        const F2 *ca = reinterpret_cast<const F2 *>(ctx) + f.cp + below * f.lp + 2;
        F2 wa[3] = {0ull, ca[u0 - 1], ca[u0]}, wb[3] = {0ull, cb[u0 - 1], cb[u0]}, wc[3] = {0ull, cc[u0 - 1], cc[u0]};
#pragma unroll 4
        for (int u = u0; u < u0 + quarter; ++u) {
          wa[0] = wa[1], wa[1] = wa[2], wa[2] = ca[u + 1];
          wb[0] = wb[1], wb[1] = wb[2], wb[2] = cb[u + 1];
          wc[0] = wc[1], wc[1] = wc[2], wc[2] = cc[u + 1];
          const float gm = g0[u], g = g0[f.rp + u], gp = g0[2 * f.rp + u];
          const F2 gm2 = pack2(gm, gm), g2 = pack2(g, g), gp2 = pack2(gp, gp);
          accb += gm + g + gp;
#pragma unroll
          for (int du = 0; du < 3; ++du) {
            fma2(acc1[du], gm2, wa[du]);
            fma2(acc1[3 + du], gp2, wb[du]);
            fma2(acc1[6 + du], g2, wb[du]);
            fma2(acc1[6 + du], gp2, wc[du]);
          }
        }
      }
    // ---- context gradients: frozen row 1 from s = 0, 1; row 2 from s = 1 and, a stripe up, s = -1
    if (s.live)
      for (int cl = first; cl < first + nch / 2; ++cl) {
        const float *g = ghid + cl * 3 * f.rp;
        float gm[4], g0[4], gp[4];
        load_window(g, s.up, gm);
        load_window(g + f.rp, s.at, g0);
        load_window(g + 2 * f.rp, s.at, gp);
        const W1Row w = load_w1(w1 + 20 * (c0 + cl));
        F2 m2[4], z2[4], p2[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          m2[k] = pack2(gm[k], gm[k]);
          z2[k] = pack2(g0[k], g0[k]);
          p2[k] = pack2(gp[k], gp[k]);
        }
#pragma unroll
        for (int du = 0; du < 3; ++du)
#pragma unroll
          for (int px = 0; px < 2; ++px) {
            fma2(gc[0][px], w.w[6 + du], z2[px + 2 - du]);
            fma2(gc[0][px], w.w[3 + du], p2[px + 2 - du]);
            fma2(gc[1][px], w.w[6 + du], p2[px + 2 - du]);
            fma2(gc[1][px], w.w[du], m2[px + 2 - du]);
          }
      }
    __syncthreads();
    // ---- lanes, then warps, added in order
#pragma unroll
    for (int go = 0; go < GO; ++go) {
      const int og = go * NGP + lane % NGP;
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        const float2 p = unpack2(acc2[go][k][0]), q = unpack2(acc2[go][k][1]);
        float v[4] = {p.x, p.y, q.x, q.y};
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
          for (int d = NGP * kChunk; d < 32; d <<= 1) v[e] += __shfl_xor_sync(0xffffffffu, v[e], d);
        if (as2 == 0 && og < NG)
          *reinterpret_cast<float4 *>(red2 + ((warp * kChunk + cl2) * 9 + k) * GP + 4 * og) =
              make_float4(v[0], v[1], v[2], v[3]);
      }
    }
#pragma unroll
    for (int k = 0; k < 10; ++k) {
      float2 v = k < 9 ? unpack2(acc1[k < 9 ? k : 0]) : make_float2(accb, 0.f);
#pragma unroll
      for (int d = 8; d < 32; d <<= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, d);
        if (k < 9) v.y += __shfl_xor_sync(0xffffffffu, v.y, d);
      }
      if (as1 == 0) *reinterpret_cast<float2 *>(red1 + (warp * kChunk + cl1) * 20 + 2 * k) = v;
    }
    __syncthreads();
    for (int t = tid; t < nch * 9 * C2; t += nt) {
      const int ck = t / C2, o = t - ck * C2;
      float v = 0.f;
      for (int w = 0; w < nwarps; ++w) v += red2[(w * kChunk * 9 + ck) * GP + o];
      gW2[c0 * 9 * C2 + t] = v;
    }
    for (int t = tid; t < nch * 20; t += nt) {
      const int cl = t / 20, r = t - 20 * cl;
      float v = 0.f;
      for (int w = 0; w < nwarps; ++w) v += red1[(w * kChunk + cl) * 20 + r];
      if (r < 18)
        gW1[(c0 + cl) * 18 + r] = v;
      else if (r == 18)
        gB1[c0 + cl] = v;
    }
    __syncthreads();
  }
  // the halves of the context gradients: thread g finishes frozen row g
  F2 *swap = reinterpret_cast<F2 *>(hid);
#pragma unroll
  for (int px = 0; px < 2; ++px) swap[px * nt + tid] = s.g ? gc[0][px] : gc[1][px];
  __syncthreads();
  float gf[2] = {0.f, 0.f};  // dL/dP of the pair's plaquettes in frozen row g: ctx = (cos P, sin P)
  if (s.live) {
    const float2 *c0 = ctx + s.g * f.cp + s.at;
#pragma unroll
    for (int px = 0; px < 2; ++px) {
      const float2 a = unpack2(s.g ? gc[1][px] : gc[0][px]), b = unpack2(swap[px * nt + s.peer]);
      gf[px] = fmaf(c0[px].x, a.y + b.y, -(c0[px].y * (a.x + b.x)));
    }
  }
  __syncthreads();
  for (int t = tid; t < f.nc * LL; t += nt) gP[t] = 0.f;
  __syncthreads();
  if (s.live) {
    float *g = gP + s.cfg * LL;
    g[flow_pixel(f, 4 * s.j, s.u + s.g)] = g_active;
#pragma unroll
    for (int px = 0; px < 2; ++px) g[flow_pixel(f, 4 * s.j + 1 + s.g, s.u + px)] = gf[px];
  }
  __syncthreads();
  // plaquette adjoint: P(x) = th0(x) + th1(x+e0) - th0(x+e1) - th1(x)
  for (int t = tid; t < ncfg * LL; t += nt) {
    const int cfg = div_by(t, f.dact) >> 2, p = t - cfg * LL, x1 = div_by(p, f.dL), x0 = p - x1 * L;
    const int x0m = x0 == 0 ? L - 1 : x0 - 1, x1m = x1 == 0 ? L - 1 : x1 - 1;
    const float *g = gP + cfg * LL, *go = f.gth_out + (size_t)(b0 + cfg) * 2 * LL;
    float *dst = f.gth_in + (size_t)(b0 + cfg) * 2 * LL;
    dst[p] = go[p] + g[p] - g[x1m * L + x0];
    dst[LL + p] = go[LL + p] + g[x1 * L + x0m] - g[p];
  }
}

// Sums over rows b of wpart[b][j], to their place in (dW1[c][ci][ky][kx],
// dB1[c], dW2[o][c][ky][kx], dB2[o]).  32 entries per block; thread group g of
// 32 adds rows g, g + 32, ... in order, then the groups are added in order.
__global__ void __launch_bounds__(1024) k_flow_wgrad_reduce(const float *__restrict__ wpart, int nb, int nw, int H,
                                                            int C2, int mu, float *__restrict__ out) {
  __shared__ float sm[32][33];
  const int e = threadIdx.x & 31, g = threadIdx.x >> 5, j = blockIdx.x * 32 + e;
  float acc = 0.f;
  if (j < nw)
#pragma unroll 4
    for (int b = g; b < nb; b += 32) acc += wpart[(size_t)b * nw + j];
  sm[g][e] = acc;
  __syncthreads();
  if (g != 0 || j >= nw) return;
  float v = 0.f;
#pragma unroll
  for (int k = 0; k < 32; ++k) v += sm[k][e];
  int to = j;
  const int n1 = 18 * H, n2 = n1 + H, n3 = n2 + 9 * H * C2;
  if (j < n1) {
    const int c = j / 18, r = j - 18 * c, k = r >> 1;
    to = c * 18 + (r & 1) * 9 + flow_tap(mu, k / 3, k % 3);
  } else if (j >= n2 && j < n3) {
    const int r = j - n2, ck = r / C2, o = r - ck * C2, c = ck / 9, k = ck - 9 * c;
    to = n2 + (o * H + c) * 9 + flow_tap(mu, k / 3, k % 3);
  }
  out[to] = v;
}

int device_sms() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1)
    return 148;
  return n;
}

// Configurations per block, at most `pairs` plaquette pairs: the fewest pairs
// on the busiest SM, a block's weight staging counted as 12 (batch 1024: one
// configuration per block at L = 32, 7 blocks on the busiest SM; seven at L = 16,
// one block per SM).
int flow_nc(int L, int batch, int pairs, int sms) {
  const int tp = L * L / 8;
  int best = 1;
  long long cost = -1;
  for (int nc = 1; nc <= std::max(1, pairs / tp) && nc <= batch; ++nc) {
    const int blocks = (batch + nc - 1) / nc;
    const long long c = (long long)((blocks + sms - 1) / sms) * (nc * tp + 12);
    if (cost < 0 || c < cost) {
      cost = c;
      best = nc;
    }
  }
  return best;
}

void flow_pitches(FlowK &f) {
  const int L = f.L;
  f.lp = L + 4;
  const int plane = f.nc * (L / 4) * f.lp;
  f.cp = plane + (plane & 1);
  f.rp = plane + ((2 - plane) & 31);  // = 2 mod 32: lanes of consecutive channels (3 rp apart) hit different banks
  f.dL = u1b::make_fastdiv((uint32_t)L);
  f.dLL2 = u1b::make_fastdiv((uint32_t)(2 * L * L));
  f.dact = u1b::make_fastdiv((uint32_t)(L * L / 4));
  f.dtp = u1b::make_fastdiv((uint32_t)(L * L / 8));
  f.dhp = u1b::make_fastdiv((uint32_t)(L / 2));
}

// Two threads per pair, and at least `least`: the others help to stage the weights
// and the context, which one warp alone takes longer over than over the sums (four
// layers of 8^2, batch 126, a block of 16 threads' sums: 145 us with 32 threads).
int flow_threads(const FlowK &f, int least) {
  return std::max(least, (2 * f.nc * (f.L * f.L / 8) + 31) / 32 * 32);
}

template <int NP>
size_t flow_weights_floats(int H) {
  return (size_t)20 * H + (size_t)3 * H * FlowDims<NP>::WS + 20;
}

// The largest shared memory of any legal shape, for a block of `pairs` plaquette
// pairs, two threads each (kernels' comments: the parts): (L / 4)(L + 4) floats of
// a plane hold L^2 / 8 pairs, so a plane is at most 4 pairs (L = 4).  Each launch
// sets its kernel's limit to this, the same value whatever its own shape, so
// that threads with other shapes cannot lower it between the setting and the launch.
template <int NP>
size_t flow_forward_smem_most() {
  const size_t pairs = kFwdThreads / 2, plane = 4 * pairs;
  return sizeof(float) * (flow_weights_floats<NP>(32) + 4 * (plane + 1) +
                          std::max(3 * kChunk * (plane + 32), (size_t)2 * NP * kFwdThreads));
}
template <int NP>
size_t flow_backward_smem_most() {
  using Dm = FlowDims<NP>;
  const size_t pairs = kBwdThreads / 2, plane = 4 * pairs;
  return sizeof(float) * (flow_weights_floats<NP>(32) + 4 * (plane + 1) + 2 * pairs * Dm::GP +
                          std::max({6 * kChunk * (plane + 32), (size_t)(kBwdThreads / 32) * kChunk * (9 * Dm::GP + 20),
                                    (size_t)2 * NP * kBwdThreads, 8 * pairs}));
}

template <int NP, bool INV>
int launch_forward(FlowK f, const char *name, cudaStream_t st) {
  const int sms = device_sms();
  f.nc = flow_nc(f.L, f.batch, kFwdThreads / 2, sms);
  flow_pitches(f);
  const int nb = (f.batch + f.nc - 1) / f.nc;
  const int threads = flow_threads(f, nb <= sms ? kFwdThreads : kFwdThreads / 2);
  const size_t work = std::max((size_t)3 * kChunk * f.rp, (size_t)2 * NP * threads);
  const size_t smem = sizeof(float) * (flow_weights_floats<NP>(f.H) + 4 * (size_t)f.cp + work);
  const cudaError_t e =
      cudaFuncSetAttribute(k_flow_forward<NP, INV>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)flow_forward_smem_most<NP>());
  if (e != cudaSuccess) return u1i::cuda_fail(e, name);
  k_flow_forward<NP, INV><<<nb, threads, smem, st>>>(f);
  U1_LAUNCH_CHECK(name);
  return U1_OK;
}

template <int NP, bool INV>
int launch_backward(FlowK f, const char *name, float *wgrad, cudaStream_t st) {
  using Dm = FlowDims<NP>;
  f.nc = flow_nc(f.L, f.batch, kBwdThreads / 2, device_sms());
  flow_pitches(f);
  const int LL = f.L * f.L, threads = flow_threads(f, kBwdThreads), nwarps = threads / 32;
  const size_t work = std::max({6 * (size_t)kChunk * f.rp, (size_t)nwarps * kChunk * (9 * Dm::GP + 20),
                                (size_t)2 * NP * threads, (size_t)f.nc * LL});
  const size_t smem = sizeof(float) * (flow_weights_floats<NP>(f.H) + 4 * (size_t)f.cp +
                                       (size_t)f.nc * (LL / 4) * Dm::GP + work);
  const cudaError_t e =
      cudaFuncSetAttribute(k_flow_backward<NP, INV>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)flow_backward_smem_most<NP>());
  if (e != cudaSuccess) return u1i::cuda_fail(e, name);
  const int nb = (f.batch + f.nc - 1) / f.nc;
  k_flow_backward<NP, INV><<<nb, threads, smem, st>>>(f);
  U1_LAUNCH_CHECK(name);
  k_flow_wgrad_reduce<<<(f.nw + 31) / 32, 1024, 0, st>>>(f.wpart, nb, f.nw, f.H, Dm::C2, f.mu, wgrad);
  U1_LAUNCH_CHECK("k_flow_wgrad_reduce");
  return U1_OK;
}

bool bad_shape(int batch, int L, int mu, int off, int K, int hidden) {
  return batch < 1 || L < 4 || L > 32 || L % 4 || (mu != 0 && mu != 1) || off < 0 || off > 3 || K < 1 ||
         K > u1b::kMaxK || hidden < 4 || hidden > 32 || hidden % 4;
}
const char *const kShapeText = ": bad shape (L a multiple of 4 up to 32, K <= 8, hidden a multiple of 4 up to 32)";

template <bool INV>
int flow_layer_fwd(const char *name, const float *theta_in, float *theta_out, float *logdet, int batch, int L, int mu,
                   int off, int K, int hidden, const float *W1, const float *B1, const float *W2, const float *B2,
                   float slope, void *stream) {
  if (!theta_in || !theta_out || !logdet || !W1 || !B1 || !W2 || !B2)
    return flfail(U1_ERR_INVALID, std::string(name) + ": null pointer");
  if (theta_in == theta_out) return flfail(U1_ERR_INVALID, std::string(name) + ": in and out must not alias");
  if (bad_shape(batch, L, mu, off, K, hidden)) return flfail(U1_ERR_INVALID, std::string(name) + kShapeText);
  FlowK f{};
  f.th_in = theta_in;
  f.batch = batch;
  f.L = L;
  f.mu = mu;
  f.off = off;
  f.H = hidden;
  f.W1 = W1;
  f.B1 = B1;
  f.W2 = W2;
  f.B2 = B2;
  f.slope = slope;
  f.th_out = theta_out;
  f.logdet = logdet;
  cudaStream_t s = (cudaStream_t)stream;
  switch (K) {
    case 1: return launch_forward<2, INV>(f, name, s);
    case 2: return launch_forward<3, INV>(f, name, s);
    case 3: return launch_forward<4, INV>(f, name, s);
    case 4: return launch_forward<5, INV>(f, name, s);
    case 5: return launch_forward<6, INV>(f, name, s);
    case 6: return launch_forward<7, INV>(f, name, s);
    case 7: return launch_forward<8, INV>(f, name, s);
    default: return launch_forward<9, INV>(f, name, s);
  }
}

template <bool INV>
int flow_layer_bwd(const char *name, const float *theta_in, const float *grad_theta_out, const float *grad_logdet,
                   float *grad_theta_in, float *wgrad_partials, float *wgrad, int batch, int L, int mu, int off, int K,
                   int hidden, const float *W1, const float *B1, const float *W2, const float *B2, float slope,
                   void *stream) {
  if (!theta_in || !grad_theta_out || !grad_theta_in || !wgrad_partials || !wgrad || !W1 || !B1 || !W2 || !B2)
    return flfail(U1_ERR_INVALID, std::string(name) + ": null pointer");
  if (bad_shape(batch, L, mu, off, K, hidden)) return flfail(U1_ERR_INVALID, std::string(name) + kShapeText);
  FlowK f{};
  f.th_in = theta_in;
  f.batch = batch;
  f.L = L;
  f.mu = mu;
  f.off = off;
  f.H = hidden;
  f.W1 = W1;
  f.B1 = B1;
  f.W2 = W2;
  f.B2 = B2;
  f.slope = slope;
  f.gth_out = grad_theta_out;
  f.gld = grad_logdet;
  f.gth_in = grad_theta_in;
  f.wpart = wgrad_partials;
  f.nw = hidden * 18 + hidden + (2 * K + 1) * hidden * 9 + (2 * K + 1);
  cudaStream_t s = (cudaStream_t)stream;
  switch (K) {
    case 1: return launch_backward<2, INV>(f, name, wgrad, s);
    case 2: return launch_backward<3, INV>(f, name, wgrad, s);
    case 3: return launch_backward<4, INV>(f, name, wgrad, s);
    case 4: return launch_backward<5, INV>(f, name, wgrad, s);
    case 5: return launch_backward<6, INV>(f, name, wgrad, s);
    case 6: return launch_backward<7, INV>(f, name, wgrad, s);
    case 7: return launch_backward<8, INV>(f, name, wgrad, s);
    default: return launch_backward<9, INV>(f, name, wgrad, s);
  }
}

}  // namespace

extern "C" int u1_flow_layer_forward(const float *theta_in, float *theta_out, float *logdet, int batch, int L,
                                     int mu, int off, int K, int hidden, const float *W1, const float *B1,
                                     const float *W2, const float *B2, float slope, void *stream) {
  return flow_layer_fwd<false>("u1_flow_layer_forward", theta_in, theta_out, logdet, batch, L, mu, off, K, hidden,
                               W1, B1, W2, B2, slope, stream);
}

extern "C" int u1_flow_layer_inverse(const float *theta_in, float *theta_out, float *logdet, int batch, int L,
                                     int mu, int off, int K, int hidden, const float *W1, const float *B1,
                                     const float *W2, const float *B2, float slope, void *stream) {
  return flow_layer_fwd<true>("u1_flow_layer_inverse", theta_in, theta_out, logdet, batch, L, mu, off, K, hidden, W1,
                              B1, W2, B2, slope, stream);
}

extern "C" int u1_flow_layer_backward(const float *theta_in, const float *grad_theta_out, const float *grad_logdet,
                                      float *grad_theta_in, float *wgrad_partials, float *wgrad, int batch, int L,
                                      int mu, int off, int K, int hidden, const float *W1, const float *B1,
                                      const float *W2, const float *B2, float slope, void *stream) {
  return flow_layer_bwd<false>("u1_flow_layer_backward", theta_in, grad_theta_out, grad_logdet, grad_theta_in,
                               wgrad_partials, wgrad, batch, L, mu, off, K, hidden, W1, B1, W2, B2, slope, stream);
}

extern "C" int u1_flow_layer_inverse_backward(const float *theta_in, const float *grad_theta_out,
                                              const float *grad_logdet, float *grad_theta_in, float *wgrad_partials,
                                              float *wgrad, int batch, int L, int mu, int off, int K, int hidden,
                                              const float *W1, const float *B1, const float *W2, const float *B2,
                                              float slope, void *stream) {
  return flow_layer_bwd<true>("u1_flow_layer_inverse_backward", theta_in, grad_theta_out, grad_logdet, grad_theta_in,
                              wgrad_partials, wgrad, batch, L, mu, off, K, hidden, W1, B1, W2, B2, slope, stream);
}
