// Two consecutive phases, (p, A) and (p, A + 1), in one launch, one site per
// thread, for lattices that fill the SMs about once.
//
// Within a half-pass only links of parity-p sites change, and a plaquette holds
// two of them: two links that leave one site or two that arrive at one.  So the
// phase (p, B), B = A + 1, needs from the phase (p, A) just before it the new
// links U_A(x) and U_A(x + e_B - e_A), nothing else: sites x + n (e_B - e_A)
// form chains that do not touch one another.  A block that owns whole chains runs
// both phases with a block barrier between them, in place, and without a grid-wide
// one.  For A = 0 it owns (x0, x1)-planes, which are contiguous; for A = 2 the
// chain is a diagonal of the (x2, x3)-plane, lcm(N2, N3) sites long, and the block
// takes `span` consecutive sites of (x0, x1) at each of its positions.
//
// A phase of such a lattice is launch boundary, one round of L2 loads and a chain
// of arithmetic (1.3 us at 8^4, 1.6 at 16^4).  The loads of both phases are issued
// before the first, so the second costs only its arithmetic and a barrier.  Per
// phase, overrelaxation, against the one-site kernel (B200): 16^4 1.61 -> 1.04 us,
// 12^2 x 14 x 16 1.48 -> 1.23, 20^4 2.14 -> 1.61, 22 x 18 x 14 x 30 (only A = 0)
// 2.13 -> 1.87.  The tuner chooses it by timing; at 24^3 x 32 the four-site kernel
// wins (3.15 against 3.47).
#pragma once
#include <algorithm>

#include "u1_internal.h"
#include "u1_update.cuh"

namespace u1b {

template <int D, int A>
struct DuoSite {
  int x[4], k, i, peer;
  bool in;
};

template <int D, int A>
__device__ __forceinline__ DuoSite<D, A> duo_site(const GeomK &g, const DuoK &d, int p, int block) {
  DuoSite<D, A> s;
  const int t = (int)threadIdx.x;
  s.in = t < d.rows;
  if (A == 0) {
    s.i = block * d.rows + t;
    s.in = s.in && s.i < g.Vh;
    if (!s.in) s.i = 0;
    eo_decode_fast<D>(g, s.i, p, s.x, s.k);
    s.peer = s.x[1] == g.N[1] - 1 ? t - (g.N[1] - 1) * g.hN0 : t + g.hN0;
  } else {
    const int tt = s.in ? t : 0;
    const int n = (int)fast_div((uint32_t)tt, d.fspan), c = tt - n * d.span;
    const int diag = (int)fast_div((uint32_t)block, d.fgroups), u = (block - diag * d.groups) * d.span + c;
    s.x[1] = (int)fast_div((uint32_t)u, g.fd[0]);
    s.k = u - s.x[1] * g.hN0;
    s.x[3] = n - (int)fast_div((uint32_t)n, d.fn3) * g.N[3];
    s.x[2] = diag - (n - (int)fast_div((uint32_t)n, d.fn2) * g.N[2]);
    if (s.x[2] < 0) s.x[2] += g.N[2];
    s.x[0] = 2 * s.k + ((s.x[1] + s.x[2] + s.x[3] + p) & 1);
    s.i = s.k + s.x[1] * g.es[1] + s.x[2] * g.es[2] + s.x[3] * g.es[3];
    s.peer = n == d.len - 1 ? t - (d.len - 1) * d.span : t + d.span;
  }
  return s;
}

template <int D, int A, bool MET, int SRC>
__device__ __forceinline__ void update_duo_body(const UpdArgs &a, const DuoK &d, int block, float2 *sm) {
  constexpr int B = A + 1;
  const GeomK &g = a.g;
  const int t = (int)threadIdx.x, p = a.p, q = 1 - p;
  const DuoSite<D, A> s = duo_site<D, A>(g, d, p, block);
  int fwd[4], bwd[4];
  eo_steps<D>(g, s.x, s.k, fwd, bwd);
  int peer = s.peer;
  if (A == 0 && bwd[0] != 0) peer += bwd[0];  // x + e1 - e0
  const Chk ck = make_chk(a);
  phase_entry<MET>(a);
  const int i = s.i;
  const bool frozen = a.ml > 0 && (s.x[D - 1] & (a.ml - 1)) == 0;
  const bool goA = s.in && !(frozen && A != 3), goB = s.in && !(frozen && B != 3);
  const float2 zero = make_float2(0.f, 0.f);
  float2 UA = zero, UB = zero;
  float2 *slabA = a.lat + A * g.V + p * g.Vh, *slabB = a.lat + B * g.V + p * g.Vh;
  // the six links of each staple term of both phases; those this launch stores
  // (directions A and B, parity p) go through the coherent path
  float2 ld[2][D][6];
  if (s.in) {
    UA = ld_live(slabA, i, ck);
    UB = ld_live(slabB, i, ck);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int MU = h ? B : A;
#pragma unroll
      for (int nu = 0; nu < D; ++nu) {
        if (nu == MU) continue;
        const float2 *Lp = a.lat + nu * g.V + p * g.Vh, *Lq = a.lat + nu * g.V + q * g.Vh, *Lm = a.lat + MU * g.V + q * g.Vh;
        ld[h][nu][0] = ld1(Lq, i + fwd[MU], ck);
        ld[h][nu][1] = ld1(Lm, i + fwd[nu], ck);
        ld[h][nu][4] = ld1(Lm, i + bwd[nu], ck);
        ld[h][nu][5] = ld1(Lq, i + bwd[nu], ck);
        if (h == 0 && nu == B) {
          ld[h][nu][2] = UB;
          ld[h][nu][3] = ld_live(Lp, i + fwd[MU] + bwd[nu], ck);
        } else if (!(h == 1 && nu == A)) {
          ld[h][nu][2] = ld1(Lp, i, ck);
          ld[h][nu][3] = ld1(Lp, i + fwd[MU] + bwd[nu], ck);
        }
      }
    }
  }
  // the same operations in the same order as staple_steps (bit-identical links)
  auto staple = [&](const float2 (&l)[D][6], int MU) {
    float2 ss = zero, st = zero;
#pragma unroll
    for (int nu = 0; nu < D; ++nu) {
      if (nu == MU) continue;
      const float2 sum = cadd(cmulc(cmulc(l[nu][0], l[nu][1]), l[nu][2]), cmul(cconjmul(l[nu][3], l[nu][4]), l[nu][5]));
      if (MU == D - 1 || nu == D - 1)
        st = cadd(st, sum);
      else
        ss = cadd(ss, sum);
    }
    return cweigh(ss, a.c.w_ss, st, a.c.w_st);
  };
  const unsigned long long pass = MET ? *a.pass_dev + (unsigned long long)a.hit : 0ull;
  float2 NA = UA;
  if (goA) {
    NA = update_link<D, A, MET, SRC>(a, p, i, staple(ld[0], A), UA, pass);
    if (chk<1, CHK_WRITE>(ck, slabA, i)) slabA[i] = NA;
  }
  sm[t] = NA;
  __syncthreads();
  if (goB) {
    ld[1][A][2] = NA;
    ld[1][A][3] = sm[peer];
    const float2 NB = update_link<D, B, MET, SRC>(a, p, i, staple(ld[1], B), UB, pass);
    if (chk<1, CHK_WRITE>(ck, slabB, i)) slabB[i] = NB;
  }
  pdl_release_dependents();
}

constexpr int kDuoThreads = 512;
constexpr int kDuoSpan = 8;  // fewest consecutive sites of a diagonal's positions: below it loads touch too many lines

template <int D, int A, bool MET, int SRC>
__global__ void __launch_bounds__(kDuoThreads) k_update_duo(const UpdArgs a, const DuoK d) {
  extern __shared__ float2 duo_sm[];
  update_duo_body<D, A, MET, SRC>(a, d, (int)blockIdx.x, duo_sm);
}

__host__ inline int duo_gcd(int a, int b) { return b ? duo_gcd(b, a % b) : a; }

// Layout of phases (p, A), (p, A + 1) in blocks of about `target` threads; false
// where the chains do not fit: a plane of more than kDuoThreads sites, or diagonals
// of which fewer than kDuoSpan fit 256 threads (16 x 18 x 14 x 22, two of 154: 1.80
// us a phase against 1.74 for the one-site kernel).
__host__ inline bool duo_layout(const GeomK &g, int A, int target, DuoK &d) {
  d = DuoK{};
  d.fspan = d.fgroups = d.fn2 = d.fn3 = make_fastdiv(1);
  if (A == 0) {
    const long long plane = (long long)g.hN0 * g.N[1];
    if (plane > kDuoThreads) return false;
    const int planes = (int)(g.Vh / plane), per = std::max(1, std::min(target / (int)plane, planes));
    d.rows = per * (int)plane;
    d.blocks = (planes + per - 1) / per;
  } else {
    const int G = duo_gcd(g.N[2], g.N[3]);
    const long long len = (long long)(g.N[2] / G) * g.N[3], line = (long long)g.hN0 * g.N[1];
    if (len * kDuoSpan > 256 || line < kDuoSpan) return false;
    d.len = (int)len;
    const int most = std::max(256, target);
    for (int s = kDuoSpan; s <= line && s * d.len <= most; ++s)  // even shares of the sites of (x0, x1)
      if (line % s == 0 && (d.span == 0 || s * d.len <= target)) d.span = s;
    if (d.span == 0) return false;
    d.groups = (int)(line / d.span);
    d.rows = d.span * d.len;
    d.blocks = d.groups * G;
    d.fspan = make_fastdiv((uint32_t)d.span);
    d.fgroups = make_fastdiv((uint32_t)d.groups);
    d.fn2 = make_fastdiv((uint32_t)g.N[2]);
    d.fn3 = make_fastdiv((uint32_t)g.N[3]);
  }
  d.threads = (d.rows + 31) / 32 * 32;
  return true;
}

}  // namespace u1b
