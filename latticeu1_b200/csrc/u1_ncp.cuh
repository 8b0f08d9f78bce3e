// The circular mixture transform with its parameters in registers (K known at
// compile time), for the fused coupling layers; formulas and parameter order
// as in u1_flow.cu.
#pragma once
#include <cuda_runtime.h>

namespace u1b {

constexpr int kMaxK = 8;

template <int K>
struct NcpMix {
  float w[K], al[K];  // softmax weights, alpha = exp(a) (a clamped to [-8, 8])
};

template <int K, int N>
__device__ __forceinline__ void ncp_mix(const float (&p)[N], NcpMix<K> &m) {
  float mx = p[K];
#pragma unroll
  for (int k = 1; k < K; ++k) mx = fmaxf(mx, p[K + k]);
  float z = 0.f;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    m.w[k] = expf(p[K + k] - mx);
    z += m.w[k];
  }
  const float iz = 1.f / z;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    m.w[k] *= iz;
    m.al[k] = expf(fminf(fmaxf(p[k], -8.f), 8.f));
  }
}

// H = sum_k w_k g_k and H' at x; g, gp: the terms; s, c = sin, cos(x/2).
template <int K>
__device__ __forceinline__ void ncp_values(float x, const NcpMix<K> &m, float &H, float &Hp, float (&g)[K],
                                           float (&gp)[K], float &s, float &c) {
  sincosf(0.5f * x, &s, &c);
  H = 0.f;
  Hp = 0.f;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const float a = m.al[k];
    g[k] = 2.f * atan2f(a * s, c);
    gp[k] = a / (c * c + a * a * s * s);
    H += m.w[k] * g[k];
    Hp += m.w[k] * gp[k];
  }
}

// The solution of H(x) = z on [-pi, pi]; H is monotone and fixes both ends.
// Newton steps inside a bracket.  A computed H is within kNcpNoise of the exact
// one: 3 ulp of the arctangent and 2 + 2 of sine and cosine (1.3e-6 on an angle
// up to pi), the products and sums of up to 8 terms (1.1e-6).  So
//  * an end of the bracket moves only to a point where |H - z| is beyond that,
//    which makes its sign certain, and the next point lies strictly inside: no
//    point is tried twice and the solution never leaves the bracket;
//  * a Newton step is taken only where the residual has halved over the last two
//    evaluations, else the bracket is: near a steep term (alpha up to e^8) H is
//    almost a step, and Newton from either side of it jumps to the other;
//  * within the noise the sign says nothing: the step from there is the answer,
//    once it is too short for the slope to change along it (kNcpStep).
// The error is the rounding of one H over H'.  A bisection to the last bit ends
// at the worst of the crossings that the rounding makes, and the residual is
// summed here without rounding (two-sum), so the error is below that of 40 FP32
// halvings: largest of 600000, logs of alpha of standard deviation 3,
// 1.9e-6 / 1.3e-5; spread over [-8, 8], 9.5e-5 / 1.5e-4 (H' down to 3e-4).
// From evaluation kNcpNewton on only halvings, so kNcpNewton + 40 end every
// search: 2 pi 2^-40 of the steepest H (2981) is far below the noise.
// Evaluations, mean of the longest of 32 (a warp): 3 to 4 for logs of standard
// deviation up to 0.3, 5.6 at 1, 14 at 3, 23 over [-8, 8].  The inverse layer at
// 32^2, 6 terms, batch 1024 (B200): 108 us, 241 us at deviation 3; steps that
// could cycle between the bracket's ends 289 us at either, and wrong.
constexpr float kNcpNoise = 4e-6f;
constexpr float kNcpStep = 1e-5f;
constexpr int kNcpNewton = 24;

template <int K>
__device__ __forceinline__ float ncp_solve(float z, const NcpMix<K> &m) {
  float lo = -3.14159265358979f, hi = 3.14159265358979f;
  float x = fminf(fmaxf(z, lo), hi), r1 = 1e30f, r2 = 1e30f;  // |H - z| of the last two evaluations
  float g[K], gp[K], s, c, H, Hp;
  int fine = 0;  // evaluations within the noise
  for (int it = 0; it < kNcpNewton + 40; ++it) {
    ncp_values<K>(x, m, H, Hp, g, gp, s, c);
    float r = -z, e = 0.f;
#pragma unroll
    for (int k = 0; k < K; ++k) {  // r + e = sum w_k g_k - z, products and sums without rounding
      const float p = m.w[k] * g[k], t = r + p, b = t - r;
      e += ((r - (t - b)) + (p - b)) + fmaf(m.w[k], g[k], -p);
      r = t;
    }
    r += e;
    float xn = x - r / Hp;
    if (fabsf(r) > kNcpNoise) {
      if (r < 0.f)
        lo = x;
      else
        hi = x;
      const float mid = 0.5f * (lo + hi);
      if (!(mid > lo && mid < hi)) return fminf(fmaxf(xn, lo), hi);  // neighbouring floats
      if (!(xn > lo && xn < hi) || fabsf(r) > 0.5f * r2 || it >= kNcpNewton) xn = mid;
      r2 = r1;
      r1 = fabsf(r);
      x = xn;
      continue;
    }
    xn = fminf(fmaxf(xn, lo), hi);
    const float step = fabsf(xn - x);
    x = xn;
    if (step <= kNcpStep || ++fine == 4) break;
  }
  return x;
}

// The change of the updated link that a plaquette angle P brings and log H'
// there: forward H(xc) + shift - xc; INV: the change that undoes a forward step.
template <int K, bool INV, int N>
__device__ __forceinline__ float ncp_transform(float P, const float (&p)[N], float &logd) {
  constexpr float kTwoPi = 6.28318530717958647692f;
  NcpMix<K> m;
  ncp_mix<K>(p, m);
  float g[K], gp[K], s, c, H, Hp;
  if (!INV) {
    const float xc = remainderf(P, kTwoPi);
    ncp_values<K>(xc, m, H, Hp, g, gp, s, c);
    logd = logf(Hp);
    return H + p[2 * K] - xc;
  }
  const float shift = p[2 * K];
  const float z = remainderf(P - shift, kTwoPi);
  const float xs = ncp_solve<K>(z, m);
  ncp_values<K>(xs, m, H, Hp, g, gp, s, c);
  logd = logf(Hp);
  return xs - z - shift;
}

// Its adjoint: from gout = dL/d(change) and gl = dL/dlogd, the gradient gP with
// respect to P (the change's own -P or the solution's included) and gq with
// respect to the parameters.
template <int K, bool INV, int N>
__device__ __forceinline__ void ncp_transform_backward(float P, const float (&p)[N], float gout, float gl, float &gP,
                                                       float (&gq)[N]) {
  constexpr float kTwoPi = 6.28318530717958647692f;
  NcpMix<K> m;
  ncp_mix<K>(p, m);
  float g[K], gp[K], s, c, H, Hp;
  const float x = INV ? ncp_solve<K>(remainderf(P - p[2 * K], kTwoPi), m) : remainderf(P, kTwoPi);
  ncp_values<K>(x, m, H, Hp, g, gp, s, c);
  float dHp_dx = 0.f;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const float a = m.al[k], den = c * c + a * a * s * s;
    dHp_dx += m.w[k] * (-a * s * c * (a * a - 1.f)) / (den * den);
  }
  // gH multiplies dH/d(parameter), gHp multiplies dH'/d(parameter); for the
  // inverse by implicit differentiation at the solution
  const float gHp = gl / Hp;
  const float r = INV ? (gout + gl * dHp_dx / Hp) / Hp : 0.f;
  const float gH = INV ? -r : gout;
  gP = INV ? r - gout : gout * Hp + gHp * dHp_dx - gout;
  gq[2 * K] = gH;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const float a = m.al[k], den = c * c + a * a * s * s, iden2 = 1.f / (den * den);
    const float dg_da = 2.f * s * c / den, dgp_da = (c * c - a * a * s * s) * iden2;
    gq[k] = fabsf(p[k]) > 8.f ? 0.f : (gH * m.w[k] * dg_da + gHp * m.w[k] * dgp_da) * a;
    gq[K + k] = gH * m.w[k] * (g[k] - H) + gHp * m.w[k] * (gp[k] - Hp);
  }
}

}  // namespace u1b
