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

// The solution of H(x) = z on [-pi, pi] (H is monotone and fixes both ends):
// Newton steps kept inside the bracket that the signs seen so far leave, by
// bisection where a step leaves it, until the step is below the float
// resolution of x or 40 evaluations (as many halvings reach it too).
// Newton converges in 4 to 8 evaluations of the K arctangents where the
// bisection alone always takes 40.
template <int K>
__device__ __forceinline__ float ncp_solve(float z, const NcpMix<K> &m) {
  float lo = -3.14159265358979f, hi = 3.14159265358979f;
  float x = fminf(fmaxf(z, lo), hi);
  float g[K], gp[K], s, c, H, Hp;
  for (int it = 0; it < 40; ++it) {
    ncp_values<K>(x, m, H, Hp, g, gp, s, c);
    if (H < z)
      lo = x;
    else
      hi = x;
    float xn = x - (H - z) / Hp;
    if (!(xn >= lo && xn <= hi)) xn = 0.5f * (lo + hi);
    const float step = fabsf(xn - x);
    x = xn;
    if (step <= 1.2e-7f * fmaxf(fabsf(x), 0.25f)) break;
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
