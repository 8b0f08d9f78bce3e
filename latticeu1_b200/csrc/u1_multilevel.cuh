// Two-level (Luscher-Weisz style) Polyakov-loop correlator kernels.
//
// Reference algorithm being replaced (src/multilevel.cu):
//   multihit field      kernel_l2_multilevel_0<true>   :239-258 (k_ml_slab2)
//   level-2 tensor T2   kernel_l2_multilevel_1         :331-360 (layout :354)
//   level-4 tensor T4   kernel_l2avg_l4_multilevel     :439-456
//   final C(r)          kernel_l4avg_Final_multilevel  :532-553
// Tensor layout (as the reference): element (x, r, i, slab) at
//   x + Vs*(r-1) + Vs*R*i + Vs*R*(d-1)*slab,   x spatial lexicographic.
// Multihit links are formed in FP32 from the float2 links; every slab
// product and the T2/T4 accumulation are FP64 complex.  The multihit links
// of each level-2 slab are multiplied once per (site, slab) (k_ml_slab2), and
// k_ml_T2 adds the sub-updates to T2 a batch at a time.
#pragma once
#include <algorithm>

#include "u1_measure.cuh"

namespace u1b {

// Extents of the multilevel tensors (4D lattices: three spatial directions).
struct MlDims {
  int N0, N1, N2;  // spatial extents
  int Vs;          // N0 * N1 * N2
  int R;           // distances r = 1..R
  int nl2, nl4;    // level-2 and level-4 slabs
};

// Level-2 slab products of the multihit temporal links:
//   P2[x + Vs*l] = mh(x, 2l) * mh(x, 2l+1)   (FP64 complex), x spatial lexicographic.
// Each product is formed once here and read by all R*(d-1) partners of x in
// k_ml_T2 (reference kernel_l2_multilevel_0<true>, src/multilevel.cu:239-258,
// computes the multihit links; its kernel_l2_multilevel_1 re-forms both slab
// products per (x, r, i)).  One thread per link: warps 2j and 2j + 1 of a block
// take the two times of a slab and the first multiplies (one thread per product
// and lexicographic order took 19.8 us at 24^3 x 32).
constexpr int kSlabWarps = 8;
static __global__ void __launch_bounds__(32 * kSlabWarps)
    k_ml_slab2(const float2 *__restrict__ lat, GeomK g, CoupK c, const MlDims m, double2 *__restrict__ P2) {
  constexpr int D = 4;
  __shared__ float2 second[kSlabWarps / 2][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int ncol = (m.Vs + 31) / 32, bt = blockIdx.x / ncol;
  const int col = (blockIdx.x - bt * ncol) * 32 + lane, t = bt * kSlabWarps + w;
  const bool in = col < m.Vs && t < 2 * m.nl2;
  const TimeColumn<D> tc = time_column<D>(g, min(col, m.Vs - 1));
  const float2 u = in ? column_link<D, true>(lat, g, c, tc, t) : make_float2(0.f, 0.f);
  if (w & 1) second[w >> 1][lane] = u;
  __syncthreads();
  if ((w & 1) || !in) return;
  const float2 v = second[w >> 1][lane];
  P2[tc.s + (size_t)m.Vs * (t >> 1)] = zmul(make_double2((double)u.x, (double)u.y), make_double2((double)v.x, (double)v.y));
}

// Two consecutive double2 (32 bytes, 32-byte aligned) in one access.  The
// T2 / T4 tensors are streamed once per launch (no reuse): evict-first
// (.cs) keeps the L2-resident slab products and links in L2.
struct Z2 {
  double2 a, b;
};
__device__ __forceinline__ Z2 ld_z2_stream(const double2 *p) {
  Z2 v;
  asm volatile("ld.global.cs.v4.f64 {%0,%1,%2,%3}, [%4];"
               : "=d"(v.a.x), "=d"(v.a.y), "=d"(v.b.x), "=d"(v.b.y)
               : "l"(p));
  return v;
}
__device__ __forceinline__ void st_z2_stream(double2 *p, Z2 v) {
  asm volatile("st.global.cs.v4.f64 [%0], {%1,%2,%3,%4};" ::"l"(p), "d"(v.a.x), "d"(v.a.y), "d"(v.b.x), "d"(v.b.y)
               : "memory");
}

// T2[x, r, i, slab] += sum over k < nk of P2_k[x, slab] * conj(P2_k[x + r e_i, slab])
// for the level-2 slabs of thickness 2 (reference kernel_l2_multilevel_1,
// src/multilevel.cu:331-360; tensor layout :354), in the order of k; P2_k, the
// slab products of sub-update k, lie `stride` apart.  fresh: T2 starts at zero.
// T2 (127 MB at 24^3 x 32) is HBM-bound to read and write, 39 us, so it is kept
// in registers over a batch of sub-updates instead of going through memory for
// each: a block takes the lines along direction i of a few sites and one range of
// kT2R distances; a thread owns a site, stages its slab product of each k in shared
// memory (two buffers, one barrier per k) and multiplies it with the partners on
// its line.  Blocks: line bundles, fastest, then 3 * ranges of r, then slabs.
constexpr int kT2R = 6;
constexpr int kT2Threads = 512;
struct MlLines {
  int bundle[3];  // lines per block
  int blocks;     // line bundles of the direction with the most (not fits: blocks of sites)
  int threads;
  bool fits;      // every line fits a block
};
__host__ inline MlLines ml_lines(const MlDims &m) {
  MlLines b{};
  const int n[3] = {m.N0, m.N1, m.N2};
  b.fits = std::max({m.N0, m.N1, m.N2}) <= kT2Threads;
  if (!b.fits) {
    b.blocks = (m.Vs + 255) / 256;
    b.threads = 256;
    return b;
  }
  for (int d = 0; d < 3; ++d) {
    const int lines = m.Vs / n[d];
    b.bundle[d] = std::max(1, std::min(lines, 256 / n[d]));
    b.blocks = std::max(b.blocks, (lines + b.bundle[d] - 1) / b.bundle[d]);
    b.threads = std::max(b.threads, (b.bundle[d] * n[d] + 31) / 32 * 32);
  }
  return b;
}
// LONG: a line does not fit a block; sites are taken in order and partners read
// from memory.
template <bool LONG>
static __global__ void __launch_bounds__(kT2Threads)
    k_ml_T2(const double2 *__restrict__ P2, size_t stride, int nk, const MlDims m, const MlLines b, int fresh,
            double2 *__restrict__ T2) {
  __shared__ double2 sm[2][LONG ? 1 : kT2Threads];
  const int ranges = (m.R + kT2R - 1) / kT2R;
  const int bz = blockIdx.x / b.blocks, bx = blockIdx.x - bz * b.blocks;
  const int l = bz / (3 * ranges), y = bz - l * 3 * ranges, dir = y / ranges, r0 = (y - dir * ranges) * kT2R + 1;
  const int n = dir == 0 ? m.N0 : dir == 1 ? m.N1 : m.N2;
  const int t = (int)threadIdx.x;
  int site, pos, self = 0, step;  // self + ((pos + r) % n) * step: the partner's place in shared memory (LONG: site)
  bool in;
  if (LONG) {
    site = bx * (int)blockDim.x + t;
    in = site < m.Vs;
    site = in ? site : 0;
    step = dir == 0 ? 1 : dir == 1 ? m.N0 : m.N0 * m.N1;
    pos = (site / step) % n;
    self = site - pos * step;
  } else {
    const int lb = dir == 0 ? b.bundle[0] : dir == 1 ? b.bundle[1] : b.bundle[2];
    const int lines = m.Vs / n;
    if (bx * lb >= lines) return;
    // consecutive threads take consecutive sites of a row: along the line for direction 0, else across lines
    const int ln = dir == 0 ? t / n : t % lb;
    pos = dir == 0 ? t - ln * n : t / lb;
    const int line = bx * lb + ln, x2 = line / m.N0;
    in = ln < lb && pos < n && line < lines;
    site = dir == 0   ? pos + m.N0 * line
           : dir == 1 ? (line - x2 * m.N0) + m.N0 * (pos + m.N1 * x2)
                      : line + m.N0 * m.N1 * pos;
    site = in ? site : 0;
    step = dir == 0 ? 1 : lb;
    self = dir == 0 ? ln * n : ln;
  }
  int partner[kT2R];
  double2 acc[kT2R];
  double2 *dst = T2 + (size_t)m.Vs * m.R * (dir + 3 * l) + site;
#pragma unroll
  for (int e = 0; e < kT2R; ++e) {
    partner[e] = in ? self + ((pos + r0 + e) % n) * step : 0;  // r may exceed the extent of a direction other than x0
    acc[e] = make_double2(0.0, 0.0);
    if (!fresh && in && r0 + e <= m.R) acc[e] = __ldcs(dst + (size_t)m.Vs * (r0 + e - 1));
  }
  const double2 *src = P2 + (size_t)m.Vs * l;
  double2 pa = in ? __ldg(src + site) : make_double2(0.0, 0.0);
  for (int k = 0; k < nk; ++k) {
    if (!LONG) sm[k & 1][t] = pa;
    const double2 next = (in && k + 1 < nk) ? __ldg(src + (size_t)(k + 1) * stride + site) : make_double2(0.0, 0.0);
    if (!LONG) __syncthreads();
#pragma unroll
    for (int e = 0; e < kT2R; ++e)
      acc[e] = zadd(acc[e], zmulc(pa, LONG ? __ldg(src + (size_t)k * stride + partner[e]) : sm[k & 1][LONG ? 0 : partner[e]]));
    pa = next;
  }
#pragma unroll
  for (int e = 0; e < kT2R; ++e)
    if (in && r0 + e <= m.R) __stcs(dst + (size_t)m.Vs * (r0 + e - 1), acc[e]);
}

// T4[., slab4] += prod_{two level-2 slabs} (T2 * l2norm) (reference
// kernel_l2avg_l4_multilevel, src/multilevel.cu:439-456).  One thread per
// pair of consecutive tensor elements and level-4 slab: 32-byte accesses.
// fresh: T4 starts at zero.
static __global__ void __launch_bounds__(256)
    k_ml_T4(const double2 *__restrict__ T2, const MlDims m, double l2norm, int fresh, double2 *__restrict__ T4) {
  const long long half = (long long)m.Vs * m.R * 3 / 2;  // element pairs per slab
  const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= half * m.nl4) return;
  const long long e2 = id % half;
  const int l4 = (int)(id / half);
  const size_t size = 2 * (size_t)half;
  const Z2 a = ld_z2_stream(T2 + 2 * e2 + size * (2 * l4));
  const Z2 b = ld_z2_stream(T2 + 2 * e2 + size * (2 * l4 + 1));
  double2 *dst = T4 + 2 * e2 + size * l4;
  Z2 t = Z2{make_double2(0.0, 0.0), make_double2(0.0, 0.0)};
  if (!fresh) t = ld_z2_stream(dst);
  t.a = zadd(t.a, zmul(zscale(a.a, l2norm), zscale(b.a, l2norm)));
  t.b = zadd(t.b, zmul(zscale(a.b, l2norm), zscale(b.b, l2norm)));
  st_z2_stream(dst, t);
}

// C(r) = norm * sum_x sum_i prod_{slab4} (T4 * l4norm), r = 1..R.  A block per
// 256 sites and r (gridDim.y = R): T4 is read once, with every load of a thread
// independent (one block per 256 sites for all r took 164 us at 24^3 x 32).
static __global__ void __launch_bounds__(kRedThreads)
    k_ml_final(const double2 *__restrict__ T4, GeomK g, int R, double l4norm, double *partials,
               unsigned int *counter, double *out, double norm) {
  __shared__ double smem[kRedWarps * 2];
  const int s = blockIdx.x * blockDim.x + threadIdx.x, r = blockIdx.y;
  const size_t size = (size_t)g.Vs * R * g.tdir;
  const int nl4 = g.N[g.tdir] / 4;
  double v[2] = {0.0, 0.0};
  if (s < g.Vs) {
    double2 pl[3];
#pragma unroll
    for (int dir = 0; dir < 3; ++dir) pl[dir] = make_double2(1.0, 0.0);
#pragma unroll 4
    for (int l4 = 0; l4 < nl4; ++l4)
#pragma unroll
      for (int dir = 0; dir < 3; ++dir)
        pl[dir] = zmul(pl[dir], zscale(__ldcs(T4 + s + (size_t)g.Vs * r + (size_t)g.Vs * R * dir + size * l4), l4norm));
#pragma unroll
    for (int dir = 0; dir < 3; ++dir) {
      v[0] += pl[dir].x;
      v[1] += pl[dir].y;
    }
  }
  block_sum<2>(v, smem);
  if (threadIdx.x < 2) partials[(size_t)blockIdx.x * 2 * R + 2 * r + threadIdx.x] = v[0];
  if (!last_block(counter, gridDim.x * gridDim.y)) return;
  finish_columns(partials, (int)gridDim.x, 2 * R, out, norm);
  if (threadIdx.x == 0) *counter = 0u;
}

}  // namespace u1b
