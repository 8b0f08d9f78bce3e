// A whole sweep of a small lattice as one launch of one thread-block cluster,
// the links held in the cluster's distributed shared memory.
//
// A phase of the per-phase kernels cannot take less than about 2.2 us (launch
// boundary, three dependent L2 round trips, store), so the 40 phases of a
// sweep of an 8^4 lattice spend their time waiting.  Here block c of the
// cluster keeps the links of EO sites [c hs, (c+1) hs) of both parities
// (2 D hs links, 64 B per site pair in 4D) in its shared memory from the first
// phase to the last, a thread owns one EO site of each parity, neighbours in
// other blocks are read through distributed shared memory, and a phase ends
// with a cluster barrier.  DRAM and L2 are touched once at each end.
// The arithmetic is that of the other bodies in the same order, so the links
// are bit-identical to theirs.
//
// Reference loop replaced: src/update.cu:301-316 (Metropolis) and :379-394
// (overrelaxation): parity x direction, one launch each.
#pragma once
#include "u1_internal.h"
#include "u1_update.cuh"

namespace u1b {

constexpr int kClusterThreads = 1024;  // sites of each parity a block can hold
constexpr int kClusterBlocks = 16;     // blocks of the largest cluster

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ uint32_t cluster_map(uint32_t addr, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// ONE: the cluster is a single block (plain shared memory and block barrier).
template <bool ONE>
__device__ __forceinline__ float2 ld_cluster(uint32_t addr) {
  float2 v;
  if (ONE)
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
  else
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ float2 ld_block(uint32_t addr) { return ld_cluster<true>(addr); }
__device__ __forceinline__ void st_block(uint32_t addr, float2 v) {
  asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(v.x), "f"(v.y) : "memory");
}
template <bool ONE>
__device__ __forceinline__ void cluster_barrier() {
  if (ONE)
    __syncthreads();
  else
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}

// Where a thread finds the rows around its own: shared-memory addresses of
// link k = 0 of direction 0, parity 0.
template <int D>
struct ClusterSite {
  uint32_t own;              // the thread's own link (offset k included)
  uint32_t row;              // its row
  uint32_t up[4], dn[4];     // rows x + e_nu, x - e_nu (nu >= 1), offset k included
  uint32_t diag[4][4];       // rows x + e_mu - e_nu (mu, nu >= 1), offset k included
  int df[2], db[2];          // byte steps along the row to x + e0, x - e0 for the site of parity 0, 1
  int ko;                    // byte offset of k
  int i;                     // EO index
  bool live;
  int xt;                    // time coordinate
};

template <int D, int MU, bool MET, int SRC, bool ONE>
__device__ __forceinline__ void cluster_phase(const UpdArgs &a, const ClusterSite<D> &s, int slab, int p,
                                              unsigned long long pass) {
  const int q = 1 - p;
  if (s.live && (MU == 3 || a.ml == 0 || (s.xt & (a.ml - 1)) != 0)) {
    const int f0 = p ? s.df[1] : s.df[0], b0 = p ? s.db[1] : s.db[0];
    const uint32_t mq = (uint32_t)((2 * MU + q) * slab);
    float2 ss = make_float2(0.f, 0.f), st = make_float2(0.f, 0.f);
#pragma unroll
    for (int nu = 0; nu < D; ++nu) {
      if (nu == MU) continue;
      const uint32_t np = (uint32_t)((2 * nu + p) * slab), nq = (uint32_t)((2 * nu + q) * slab);
      const uint32_t own = s.row + (uint32_t)s.ko;
      const float2 A = ld_cluster<ONE>((MU == 0 ? own + f0 : s.up[MU]) + nq);
      const float2 B = ld_cluster<ONE>((nu == 0 ? own + f0 : s.up[nu]) + mq);
      const float2 C = ld_block(s.own + np);
      const float2 Dd = ld_cluster<ONE>((MU == 0 ? s.dn[nu] + f0 : nu == 0 ? s.up[MU] + b0 : s.diag[MU][nu]) + np);
      const uint32_t back = nu == 0 ? own + b0 : s.dn[nu];
      const float2 E = ld_cluster<ONE>(back + mq);
      const float2 F = ld_cluster<ONE>(back + nq);
      const float2 sum = cadd(cmulc(cmulc(A, B), C), cmul(cconjmul(Dd, E), F));
      if (MU == D - 1 || nu == D - 1)
        st = cadd(st, sum);
      else
        ss = cadd(ss, sum);
    }
    const uint32_t self = s.own + (uint32_t)((2 * MU + p) * slab);
    const float2 S = cweigh(ss, a.c.w_ss, st, a.c.w_st);
    st_block(self, update_link<D, MU, MET, SRC>(a, p, s.i, S, ld_block(self), pass));
  }
  cluster_barrier<ONE>();
}

template <int D, bool MET, int SRC, bool ONE>
__device__ __forceinline__ void cluster_pass(const UpdArgs &a, const ClusterSite<D> &s, int slab,
                                             unsigned long long pass) {
#pragma unroll 1
  for (int p = 0; p < 2; ++p) {
    cluster_phase<D, 0, MET, SRC, ONE>(a, s, slab, p, pass);
    cluster_phase<D, 1, MET, SRC, ONE>(a, s, slab, p, pass);
    if constexpr (D > 2) cluster_phase<D, 2, MET, SRC, ONE>(a, s, slab, p, pass);
    if constexpr (D > 3) cluster_phase<D, 3, MET, SRC, ONE>(a, s, slab, p, pass);
  }
}

// Checked build: whether r0 + step is the first site of one of the lattice's rows
// (which cluster_layout gives a block and a place in it), and whether the four
// steps along x0 stay in the row.  A violation is counted and not followed; with
// the thread's own link these are all the addresses of a sweep.
__device__ __forceinline__ bool chk_row(const Chk &c, int r0, int step, int hN0) {
#ifdef U1_BOUNDS_CHECK
  const int r = r0 + step;
  return chk_count(c, r >= 0 && r < c.Vh && r % hN0 == 0, r);
#else
  return true;
#endif
}
__device__ __forceinline__ bool chk_in_row(const Chk &c, int ko, const int (&df)[2], const int (&db)[2], int bytes) {
#ifdef U1_BOUNDS_CHECK
  bool ok = true;
  for (int p = 0; p < 2; ++p)
    ok = ok && ko + df[p] >= 0 && ko + df[p] < bytes && ko + db[p] >= 0 && ko + db[p] < bytes;
  return chk_count(c, ok, ko / 8);
#else
  return true;
#endif
}

template <int D, int SRC, bool ONE>
__global__ void __launch_bounds__(kClusterThreads, 1)
    k_sweep_cluster(const UpdArgs a, const ClusterK c, int metrop, int ovrn, unsigned long long *pass_rw) {
  extern __shared__ float2 cl_links[];
  const GeomK &g = a.g;
  const int t = (int)threadIdx.x, rank = (int)blockIdx.x;
  const uint32_t base = smem_u32(cl_links);
  const int slab = c.hs * (int)sizeof(float2);
  ClusterSite<D> s;
  s.i = rank * c.hs + t;
  s.live = t < c.hs && s.i < g.Vh;
  {
    int x[4], k, fwd[4], bwd[4];
    eo_decode_fast<D>(g, s.live ? s.i : 0, 0, x, k);
    eo_steps<D>(g, x, k, fwd, bwd);
    s.xt = x[D - 1];
    s.ko = k * 8;
    const int odd0 = x[0] & 1;
    const int kf = (k == g.hN0 - 1 ? 1 - g.hN0 : 1) * 8, kb = (k == 0 ? g.hN0 - 1 : -1) * 8;
    s.df[0] = odd0 ? kf : 0;
    s.df[1] = odd0 ? 0 : kf;
    s.db[0] = odd0 ? 0 : kb;
    s.db[1] = odd0 ? kb : 0;
    const int r0 = (s.live ? s.i : 0) - k;  // EO index of the row's first site
    const Chk ck = make_chk(a);
    auto at = [&](int step) -> uint32_t {   // address of the row r0 + step
      const uint32_t row = chk_row(ck, r0, step, g.hN0) ? fast_div((uint32_t)(r0 + step), g.fd[0]) : 0u;
      const uint32_t owner = ONE ? 0u : fast_div(row, c.fr);
      const uint32_t off = (row - owner * (uint32_t)c.rows) * (uint32_t)(g.hN0 * 8);
      return ONE ? base + off : cluster_map(base + off, (int)owner);
    };
    s.row = at(0);
    s.own = base + (uint32_t)t * 8u;
    if (!chk_in_row(ck, s.ko, s.df, s.db, g.hN0 * 8)) s.df[0] = s.df[1] = s.db[0] = s.db[1] = 0;
#pragma unroll
    for (int mu = 1; mu < D; ++mu) {
      s.up[mu] = at(fwd[mu]) + (uint32_t)s.ko;
      s.dn[mu] = at(bwd[mu]) + (uint32_t)s.ko;
#pragma unroll
      for (int nu = 1; nu < D; ++nu)
        if (nu != mu) s.diag[mu][nu] = at(fwd[mu] + bwd[nu]) + (uint32_t)s.ko;
    }
  }
  pdl_wait_prior_grid();
  const unsigned long long pass0 = metrop ? *a.pass_dev : 0ull;
  if (s.live)
#pragma unroll
    for (int mu = 0; mu < D; ++mu)
#pragma unroll
      for (int p = 0; p < 2; ++p)
        st_block(s.own + (uint32_t)((2 * mu + p) * slab), __ldcg(a.lat + (size_t)mu * g.V + (size_t)p * g.Vh + s.i));
  cluster_barrier<ONE>();
  for (int m = 0; m < metrop; ++m) cluster_pass<D, true, SRC, ONE>(a, s, slab, pass0 + (unsigned long long)m);
  for (int o = 0; o < ovrn; ++o) cluster_pass<D, false, SRC_PHILOX, ONE>(a, s, slab, 0ull);
  if (s.live)
#pragma unroll
    for (int mu = 0; mu < D; ++mu)
#pragma unroll
      for (int p = 0; p < 2; ++p)
        a.lat[(size_t)mu * g.V + (size_t)p * g.Vh + s.i] = ld_block(s.own + (uint32_t)((2 * mu + p) * slab));
  if (rank == 0 && t == 0 && metrop) *pass_rw = pass0 + (unsigned long long)metrop;
}

// Layout of `blocks` blocks; false when a block's share does not fit.
__host__ inline bool cluster_layout(const GeomK &g, int blocks, ClusterK &c) {
  const int rows = g.Vh / g.hN0;
  c.rows = (rows + blocks - 1) / blocks;
  c.blocks = (rows + c.rows - 1) / c.rows;
  if ((long long)c.rows * g.hN0 > kClusterThreads) return false;
  c.hs = c.rows * g.hN0;
  c.threads = (c.hs + 31) / 32 * 32;
  c.fr = make_fastdiv((uint32_t)c.rows);
  return true;
}

}  // namespace u1b
