// Measurement kernels: fused plaquette (SS/ST) + Polyakov loop, the
// Polyakov-loop field (plain or analytic multihit) and its correlator.
//
// Reference algorithm being replaced:
//   plaquette        src/plaquette.cu:93-118, norms :156-165
//   Polyakov loop    src/polyakov.cu:60-77, :124-139
//   P(x) field       src/polyakov.cu:415-440 (kernel_polyakov_volume<multihit>)
//   correlator       src/polyakov.cu:514-535, norm :568
//   multihit mean    include/lattice_functions.h:92-105
// Reductions: per-thread values are summed in FP64 with xor-shuffle warp
// reductions, block totals go to a per-block partials array, and the last
// block to finish (ticket counter) sums the partials in block order, so
// every result is deterministic run to run.  The reference instead folds
// shared memory serially in thread 0 and uses FP64 atomicAdd
// (include/reduce_block_1d.h:41-64).
#pragma once
#include "u1_cplx.cuh"
#include "u1_geom.cuh"
#include "u1_update.cuh"

namespace u1b {

constexpr int kRedThreads = 256;
constexpr int kRedWarps = kRedThreads / 32;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Block-wide sum of NV values per thread; the totals are valid in threads
// 0..NV-1 (thread k holds value k).  smem must hold kRedWarps*NV doubles.
template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV], double *smem) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    double w = warp_sum(v[k]);
    if (lane == 0) smem[warp * NV + k] = w;
  }
  __syncthreads();
  if (threadIdx.x < NV) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += smem[w * NV + threadIdx.x];
    v[0] = t;  // caller reads v[0] in thread k as total k
  }
  __syncthreads();
}

// Per-thread sum of partials[b * stride + k] over b = threadIdx.x,
// threadIdx.x + blockDim.x, ... < n, added in that order, with kUnroll loads
// in flight (a plain strided loop would wait for every load in turn).
__device__ __forceinline__ double strided_partial_sum(const double *partials, unsigned n, int stride, int k) {
  constexpr int kUnroll = 8;
  double w = 0.0;
  for (unsigned b0 = threadIdx.x; b0 < n; b0 += kUnroll * blockDim.x) {
    double t[kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const unsigned b = b0 + u * blockDim.x;
      t[u] = (b < n) ? __ldcg(partials + (size_t)b * stride + k) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) w += t[u];
  }
  return w;
}

// Block totals already reduced (thread k < NV holds total k in tot): store
// them as this block's partials, take a ticket; the last block sums all
// partials in block order and writes out[k] = scale[k] * total_k, then
// resets `counter` to 0.
template <int NV>
__device__ __forceinline__ void finish_block_totals(double tot, double *smem, double *partials,
                                                    unsigned int *counter, double *out,
                                                    const double (&scale)[NV]) {
  __shared__ bool am_last;
  if (threadIdx.x < NV) {
    partials[(size_t)blockIdx.x * NV + threadIdx.x] = tot;
    __threadfence();  // the writers order their partials before the ticket
  }
  __syncthreads();
  if (threadIdx.x == 0) am_last = (atomicAdd(counter, 1u) == gridDim.x - 1);
  __syncthreads();
  if (!am_last) return;
  __threadfence();
  // Thread j sums partials of blocks j, j + blockDim, j + 2 blockDim, ... in
  // that order.  The loads of kUnroll blocks are issued together before they
  // are added, so the pass costs about one L2 round trip per kUnroll * blockDim
  // blocks (a plain strided loop would wait for every load in turn).
  constexpr int kUnroll = 4;
  double w[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) w[k] = 0.0;
  for (unsigned b0 = threadIdx.x; b0 < gridDim.x; b0 += kUnroll * blockDim.x) {
    double t[kUnroll][NV];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const unsigned b = b0 + u * blockDim.x;
#pragma unroll
      for (int k = 0; k < NV; ++k) t[u][k] = (b < gridDim.x) ? __ldcg(partials + (size_t)b * NV + k) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < kUnroll; ++u)
#pragma unroll
      for (int k = 0; k < NV; ++k) w[k] += t[u][k];
  }
  block_sum<NV>(w, smem);
  if (threadIdx.x < NV) out[threadIdx.x] = w[0] * scale[threadIdx.x];
  if (threadIdx.x == 0) *counter = 0u;
}

// Launch layout of the plaquette + Polyakov measurement.
//  * blocks [0, nb_plaq): plaquettes.  pair != 0 (N0/2 even): thread t
//    takes EO sites i = 2t, 2t+1 of both parities, whose neighbours along
//    x1..x3 sit side by side (128-bit loads); else thread i takes EO site i.
//  * blocks [nb_plaq, nb_plaq + nb_poly): Polyakov loops.  A block holds
//    kRedThreads/chunks spatial sites x `chunks` time chunks; each thread
//    multiplies the Nt/chunks temporal links of its chunk, and the chunk
//    products of a site are combined in shared memory in chunk order.
struct MeasK {
  int nb_plaq;
  int nb_poly;
  int pair;
  int chunks;
};

__host__ inline MeasK measure_layout(const GeomK &g) {
  MeasK m{};
  m.pair = (g.hN0 & 1) == 0;
  const int plaq_threads = m.pair ? g.Vh / 2 : g.Vh;
  m.nb_plaq = (plaq_threads + kRedThreads - 1) / kRedThreads;
  // largest of 8, 4, 2 dividing Nt with at least eight links per chunk (a
  // thread's loads are independent; fewer, fuller blocks cut the per-block
  // reduction cost), else one chunk
  const int Nt = g.N[g.dims - 1];
  m.chunks = 1;
  for (int c = 8; c > 1; c >>= 1)
    if (Nt % c == 0 && Nt / c >= 8) {
      m.chunks = c;
      break;
    }
  m.nb_poly = (g.Vs * m.chunks + kRedThreads - 1) / kRedThreads;
  return m;
}

// Plaquettes (mu < nu) at one site: U_mu(x) U_nu(x+mu) conj(U_mu(x+nu)) conj(U_nu(x)),
// accumulated as (1 - Re P, -Im P) into vs[0..1] (spatial) or vs[2..3] (temporal nu).
__device__ __forceinline__ void plaq_accum(float2 umu, float2 a, float2 b, float2 unu, bool temporal,
                                           float (&vs)[6]) {
  const float2 P = cmulc(cmulc(cmul(umu, a), b), unu);
  const int o = temporal ? 2 : 0;
  vs[o] += 1.f - P.x;
  vs[o + 1] -= P.y;
}

template <int D>
__device__ __forceinline__ void plaq_sites_pair(const float2 *__restrict__ lat, const GeomK &g, int i,
                                                float (&vs)[6]) {
  int x[4], k;
  eo_decode_fast<D>(g, i, 0, x, k);
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    if (p == 1) x[0] = 2 * k + ((x[1] + x[2] + x[3] + 1) & 1);
    int fwd[4], bwd[4];
    eo_steps<D>(g, x, k, fwd, bwd);
    // x0 steps of the second site (x0 + 2): as the first unless it wraps
    const int odd = x[0] & 1;
    const int f0b = odd ? ((k + 1 == g.hN0 - 1) ? g.wrapf[0] : 1) : 0;
    const int q = 1 - p;
    Pair2 U[D];
#pragma unroll
    for (int mu = 0; mu < D; ++mu) U[mu] = ld_vec2(lat + mu * g.V + p * g.Vh, i, no_chk());
#pragma unroll
    for (int mu = 0; mu < D - 1; ++mu) {
#pragma unroll
      for (int nu = mu + 1; nu < D; ++nu) {
        const float2 *Lq_nu = lat + nu * g.V + q * g.Vh;
        const Pair2 a = (mu == 0) ? ld_two(Lq_nu, i + fwd[0], i + 1 + f0b, no_chk()) : ld_vec2(Lq_nu, i + fwd[mu], no_chk());
        const Pair2 b = ld_vec2(lat + mu * g.V + q * g.Vh, i + fwd[nu], no_chk());  // U_mu(x+nu), nu >= 1
        plaq_accum(U[mu].s0, a.s0, b.s0, U[nu].s0, nu == D - 1, vs);
        plaq_accum(U[mu].s1, a.s1, b.s1, U[nu].s1, nu == D - 1, vs);
      }
    }
  }
}

template <int D>
__device__ __forceinline__ void plaq_site(const float2 *__restrict__ lat, const GeomK &g, int i,
                                          float (&vs)[6]) {
  int x[4], k;
  eo_decode_fast<D>(g, i, 0, x, k);
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    if (p == 1) x[0] = 2 * k + ((x[1] + x[2] + x[3] + 1) & 1);
    int fwd[4], bwd[4];
    eo_steps<D>(g, x, k, fwd, bwd);
    const int q = 1 - p;
    float2 U[D];
#pragma unroll
    for (int mu = 0; mu < D; ++mu) U[mu] = __ldg(lat + mu * g.V + p * g.Vh + i);
#pragma unroll
    for (int mu = 0; mu < D - 1; ++mu) {
#pragma unroll
      for (int nu = mu + 1; nu < D; ++nu) {
        const float2 a = __ldg(lat + nu * g.V + q * g.Vh + i + fwd[mu]);  // U_nu(x+mu)
        const float2 b = __ldg(lat + mu * g.V + q * g.Vh + i + fwd[nu]);  // U_mu(x+nu)
        plaq_accum(U[mu], a, b, U[nu], nu == D - 1, vs);
      }
    }
  }
}

// Per-thread terms of measurement block `block` (layout MeasK): vs[0..3] +=
// (1 - Re P, -Im P) of the SS and ST plaquettes, vs[4..5] += the Polyakov
// loop.  lp: kRedThreads float2 of shared memory.  Every thread of the
// block must call it (the Polyakov blocks synchronise).  Shared by the
// single-lattice and batched measurements.
template <int D>
__device__ __forceinline__ void measure_block_values(const float2 *__restrict__ lat, const GeomK &g, int block,
                                                     const MeasK &m, float (&vs)[6], float2 *lp) {
  if (block < m.nb_plaq) {
    const int t = block * blockDim.x + threadIdx.x;
    if (m.pair) {
      if (2 * t < g.Vh) plaq_sites_pair<D>(lat, g, 2 * t, vs);
    } else if (t < g.Vh) {
      plaq_site<D>(lat, g, t, vs);
    }
    return;
  }
  const int per_block = blockDim.x / m.chunks;
  const int sl = threadIdx.x % per_block, c = threadIdx.x / per_block;
  const int j = (block - m.nb_plaq) * per_block + sl;  // spatial site (EO order on the t = 0 slice)
  float2 L = make_float2(1.f, 0.f);
  if (j < g.Vs) {
    const int hs = g.Vs / 2;
    const int p = j >= hs ? 1 : 0;
    const int i = j - p * hs;
    const int Lc = g.N[D - 1] / m.chunks;
    const int est = g.es[D - 1];
    const float2 *base = lat + (D - 1) * g.V + i;
    const int t0 = c * Lc;
    // eight loads in flight, then their products in time order (a padded
    // factor is 1 + 0i, which leaves the product bit for bit unchanged)
    for (int tb = t0; tb < t0 + Lc; tb += 8) {
      float2 u[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int t = tb + k;
        u[k] = (t < t0 + Lc) ? __ldg(base + ((p + t) & 1) * g.Vh + t * est) : make_float2(1.f, 0.f);
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) L = cmul(L, u[k]);
    }
  }
  lp[threadIdx.x] = L;
  __syncthreads();
  if (c == 0 && j < g.Vs) {
    float2 P = lp[sl];
    for (int cc = 1; cc < m.chunks; ++cc) P = cmul(P, lp[cc * per_block + sl]);
    vs[4] += P.x;
    vs[5] += P.y;
  }
}

// FP64 block totals of the measurement terms: only the values this block
// kind produces (plaquette blocks: 0..3, Polyakov blocks: 4..5) go through
// the warp shuffles.  Thread k < 6 returns total k.
__device__ __forceinline__ double measure_block_total(const float (&vs)[6], bool plaq_block, double *smem) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int k0 = plaq_block ? 0 : 4, k1 = plaq_block ? 4 : 6;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    if (k < k0 || k >= k1) continue;
    const double w = warp_sum((double)vs[k]);
    if (lane == 0) smem[warp * 6 + k] = w;
  }
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x >= k0 && threadIdx.x < k1)
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += smem[w * 6 + threadIdx.x];
  __syncthreads();
  return t;
}

// Fused plaquette + Polyakov loop, one launch of m.nb_plaq + m.nb_poly blocks
// (layout MeasK).  out = {SS re, SS im, ST re, ST im, L re, L im}: mean of
// (1 - e^{i theta_P}) per class and (1/V_s) sum_x prod_t U_t.
template <int D>
static __global__ void __launch_bounds__(kRedThreads)
    k_measure(const float2 *__restrict__ lat, GeomK g, MeasK m, double *partials, unsigned int *counter,
              double *out, double normSS, double normST, double normL) {
  __shared__ double smem[kRedWarps * 6];
  __shared__ float2 lp[kRedThreads];
  float vs[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};  // per-thread partial sums of a few terms
  measure_block_values<D>(lat, g, (int)blockIdx.x, m, vs, lp);
  const double tot = measure_block_total(vs, (int)blockIdx.x < m.nb_plaq, smem);
  const double scale[6] = {normSS, normSS, normST, normST, normL, normL};
  finish_block_totals<6>(tot, smem, partials, counter, out, scale);
}

// I1(x)/I0(x) by backward evaluation of the Gauss continued fraction
// r_k = I_k/I_{k-1} = x / (2k + x r_{k+1}) (from the recurrence
// I_{k-1} - I_{k+1} = (2k/x) I_k), truncated at depth ceil(x)+16 where the
// remaining tail is below float precision.  Replaces CUDA's
// cyl_bessel_i1/cyl_bessel_i0 used by the reference
// (include/lattice_functions.h:101).
__device__ __forceinline__ float bessel_ratio_i1_i0(float x) {
  const int K = (int)x + 16;
  float r = 0.0f;
  for (int k = K; k >= 1; --k) r = __fdividef(x, fmaf(x, r, 2.0f * (float)k));
  return r;
}

// Analytic multihit mean of the temporal link whose staple is S:
// conj(S) * I1(beta|S|) / (|S| I0(beta|S|)).
__device__ __forceinline__ float2 multihit_mean(const CoupK &c, float2 S) {
  const float alpha = sqrtf(fmaf(S.x, S.x, S.y * S.y));
  if (!(alpha > 0.f)) return make_float2(0.f, 0.f);
  const float t = bessel_ratio_i1_i0(c.beta * alpha) / alpha;
  return make_float2(t * S.x, -t * S.y);
}

// One spatial site's column of temporal links.  The two spatial sites 2k and
// 2k + 1 of a row share the EO index i0 on the t = 0 slice; the one of parity q
// sits at EO index i0 + t es of parity (q + t) mod 2, and its spatial neighbour
// steps are those of t = 0 throughout.  Threads with consecutive i0 and one q
// read consecutive links.
template <int D>
struct TimeColumn {
  int i0, q;
  int s;  // spatial lexicographic index
  int fwd[4], bwd[4];
};
template <int D>
__device__ __forceinline__ TimeColumn<D> time_column(const GeomK &g, int col) {  // col < Vs
  TimeColumn<D> tc;
  const int hs = g.Vs / 2;
  tc.q = col >= hs ? 1 : 0;
  tc.i0 = col - tc.q * hs;
  int x[4], k;
  eo_decode_fast<D>(g, tc.i0, tc.q, x, k);
  eo_steps<D>(g, x, k, tc.fwd, tc.bwd);
  tc.s = 2 * tc.i0 + (x[0] & 1);  // rows of N0 sites are rows of N0/2 EO indices
  return tc;
}
// The temporal link (MH: its multihit mean) of the column at time t.
template <int D, bool MH>
__device__ __forceinline__ float2 column_link(const float2 *__restrict__ lat, const GeomK &g, const CoupK &c,
                                              const TimeColumn<D> &tc, int t) {
  const int p = (tc.q + t) & 1, i = tc.i0 + t * g.es[D - 1];
  if (!MH) return __ldg(lat + (size_t)(D - 1) * g.V + (size_t)p * g.Vh + i);
  int fwd[4], bwd[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    fwd[k] = tc.fwd[k];
    bwd[k] = tc.bwd[k];
  }
  fwd[D - 1] = t == g.N[D - 1] - 1 ? g.wrapf[D - 1] : g.es[D - 1];
  bwd[D - 1] = t == 0 ? g.wrapb[D - 1] : -g.es[D - 1];
  return multihit_mean(c, staple_steps<D, D - 1>(lat, g, c, i, p, fwd, bwd, no_chk()));
}

// P(x) = prod_t U_t(x,t) (or of the multihit means) for every spatial site,
// stored in spatial lexicographic order; products in FP64.  A block takes 32
// columns and splits time over its 16 warps, whose products are then multiplied
// in time order.  A multihit link is a chain of about 20 dependent divisions
// after its staple, so the kernel lives on threads in flight: at 24^3 x 32 one
// thread per column (54 blocks) took 89 us.
constexpr int kPolyWarps = 16;
template <int D, bool MH>
static __global__ void __launch_bounds__(32 * kPolyWarps)
    k_poly_field(const float2 *__restrict__ lat, GeomK g, CoupK c, double2 *P) {
  __shared__ double2 part[kPolyWarps][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int col = blockIdx.x * 32 + lane;
  const int Nt = g.N[D - 1], per = (Nt + kPolyWarps - 1) / kPolyWarps;
  const TimeColumn<D> tc = time_column<D>(g, min(col, g.Vs - 1));
  double2 prod = make_double2(1.0, 0.0);
  for (int t = w * per; t < min(Nt, (w + 1) * per); ++t) {
    const float2 u = column_link<D, MH>(lat, g, c, tc, t);
    prod = zmul(prod, make_double2((double)u.x, (double)u.y));
  }
  part[w][lane] = prod;
#pragma unroll
  for (int o = 1; o < kPolyWarps; o <<= 1) {
    __syncthreads();
    if ((w & (2 * o - 1)) == 0) part[w][lane] = prod = zmul(prod, part[w + o][lane]);
  }
  if (w == 0 && col < g.Vs) P[tc.s] = prod;
}

// Sums of partials[b * n + k] over blocks b < nb, a warp per k: out[k] = norm * sum.
// Called by every thread of the last block to finish.
__device__ __forceinline__ void finish_columns(const double *partials, int nb, int n, double *out, double norm) {
  const int lane = threadIdx.x & 31;
  for (int k = threadIdx.x >> 5; k < n; k += (int)(blockDim.x >> 5)) {
    double v = 0.0;
#pragma unroll 4
    for (int b = lane; b < nb; b += 32) v += __ldcg(partials + (size_t)b * n + k);
    v = warp_sum(v);
    if (lane == 0) out[k] = v * norm;
  }
}

// Whether this block is the last of `blocks` to get here; its threads then see
// every block's partials.
__device__ __forceinline__ bool last_block(unsigned int *counter, unsigned int blocks) {
  __shared__ bool am_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) am_last = (atomicAdd(counter, 1u) == blocks - 1);
  __syncthreads();
  if (am_last) __threadfence();
  return am_last;
}

// C(r) = norm * sum_x sum_{i<d-1} P(x) conj(P(x + r e_i)), r = 1..R.  A block
// takes kCorrSites sites, a warp one r at a time (no block-wide reduction per
// r: with one, 54 blocks of 256 sites took 36 us at 24^3 x 32).
// partials: gridDim.x * 2R doubles; out: 2R doubles.
constexpr int kCorrSites = 64;
static __global__ void __launch_bounds__(kRedThreads)
    k_poly_corr(const double2 *__restrict__ P, GeomK g, int R, double *partials,
                unsigned int *counter, double *out, double norm) {
  const int lane = threadIdx.x & 31;
  int x[2][3], s[2];
  double2 P0[2];
  int step[3] = {1, g.N[0], g.N[0] * g.N[1]};
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    s[e] = blockIdx.x * kCorrSites + 32 * e + lane;
    const bool in = s[e] < g.Vs;
    int r = in ? s[e] : 0;
    P0[e] = in ? P[r] : make_double2(0.0, 0.0);
    s[e] = r;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      x[e][k] = k < g.tdir ? r % g.N[k] : 0;
      r = k < g.tdir ? r / g.N[k] : r;
    }
  }
  for (int r = 1 + (int)(threadIdx.x >> 5); r <= R; r += kRedWarps) {
    double2 v = make_double2(0.0, 0.0);
#pragma unroll
    for (int k = 0; k < 3; ++k)
      if (k < g.tdir) {
        const int rk = r % g.N[k];  // r may exceed the extent of a direction other than x0
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int xk = x[e][k] + rk, d = xk >= g.N[k] ? rk - g.N[k] : rk;
          v = zadd(v, zmulc(P0[e], P[s[e] + d * step[k]]));
        }
      }
    v.x = warp_sum(v.x);
    v.y = warp_sum(v.y);
    if (lane == 0) *reinterpret_cast<double2 *>(partials + (size_t)blockIdx.x * 2 * R + 2 * (r - 1)) = v;
  }
  if (!last_block(counter, gridDim.x)) return;
  finish_columns(partials, (int)gridDim.x, 2 * R, out, norm);
  if (threadIdx.x == 0) *counter = 0u;
}

}  // namespace u1b
