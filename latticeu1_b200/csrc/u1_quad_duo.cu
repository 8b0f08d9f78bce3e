// Phases (p, 0) and (p, 1) in one launch, four sites per thread.
//
// The second phase needs of the first only the new links U_0(x) and
// U_0(x + e1 - e0) (u1_duo.cuh), which lie in x's (x0, x1)-plane.  A block owns
// whole planes, keeps the new U_0 in shared memory and runs both phases with a
// block barrier between them: one launch boundary less in four phases, and two of
// the second phase's 17 quad loads (U_0 at x and at x + e1 - e0, with the row edge
// of the latter) become shared-memory reads.  A phase of a large lattice is bound
// by those loads (L1 wavefronts in cache, DRAM beyond it), one that fits the L2 by
// the launch boundary as well.  Unlike u1_duo.cuh the loads of the second phase
// are not issued before the first: 35 quad loads a thread do not fit the
// registers.  In a batch, whose second lane already covers the boundaries, the
// same made no difference (7.6 ms a sweep of 512 chains with and without).
//
// The register bound decides how many threads an SM holds, so there are three:
// 96 registers where the grid is then still one wave, 72 where that makes it one
// or holds as many threads as 64 do, 64 elsewhere (a plane of 512 threads at
// 64^4: two blocks an SM instead of one).  Mean over the four phases of a
// half-pass, us, overrelaxation, one phase a launch / this (B200): 24^3 x 32
// (216 threads, 96 registers) 3.28 / 3.04, 24^3 x 48 (288, 96) 4.18 / 3.73
// (a whole sweep 162 -> 152 us), 32^4 (128, 72) 5.27 / 4.95, 48^4 (288, 72) 27.7 /
// 27.5 (Metropolis 34.2 / 31.9), 64^4 (512, 64) 101.0 / 95.7.  40^4 (224 threads of
// which 200 hold sites) is slower, 12.9 / 13.1: the tuner chooses by timing.
#include "u1_internal.h"
#include "u1_update.cuh"

namespace u1b {

__device__ __forceinline__ Quad2 quad_of(const float4 &lo, const float4 &hi) {
  Quad2 q;
  q.s[0] = make_float2(lo.x, lo.y);
  q.s[1] = make_float2(lo.z, lo.w);
  q.s[2] = make_float2(hi.x, hi.y);
  q.s[3] = make_float2(hi.z, hi.w);
  return q;
}

struct QuadSite {
  int k, x1, fwd[4], bwd[4];
  Row4 row;
  bool active;
};
template <int D>
__device__ __forceinline__ QuadSite quad_site(const UpdArgs &a, int i, bool in) {
  QuadSite s;
  int x[4];
  eo_decode_fast<D>(a.g, i, a.p, x, s.k);
  eo_steps<D>(a.g, x, s.k, s.fwd, s.bwd);
  s.x1 = x[1];
  s.row = row4(a.g, x[0], s.k);
  s.active = in && (a.ml == 0 || (x[D - 1] & (a.ml - 1)) != 0);  // planes lie in one time slice
  s.row.mask = __ballot_sync(0xffffffffu, s.active);
  s.row.any = __any_sync(0xffffffffu, s.row.out);
  return s;
}

template <int D, bool MET, int SRC, int THREADS, int CTAS>
__global__ void __launch_bounds__(THREADS, CTAS) k_update_quad_duo(const UpdArgs a, int rows) {
  extern __shared__ float4 quad_sm[];  // new U_0 of the block's sites: first halves of the quads, then second
  float4 *lo = quad_sm, *hi = quad_sm + blockDim.x;
  const int t = (int)threadIdx.x;
  const int b = a.rev ? rev_block(a, (int)blockIdx.x, (int)gridDim.x) : sm_local_block((int)blockIdx.x, a.order);
  int i = 4 * (b * rows + t);
  const bool in = t < rows && i < a.g.Vh;
  if (!in) i = 0;
  const Chk ck = make_chk(a);
  {
    const QuadSite s = quad_site<D>(a, i, in);
    phase_entry<MET>(a);
    if (s.active) {
      const QuadSums o = quad_staples<D, 0, false, -1, 1>(a, i, s.fwd, s.bwd, s.row, ck);
      float2 N[4];
      quad_links<D, 0, MET, SRC>(a, i, o, ck, N);
      lo[t] = make_float4(N[0].x, N[0].y, N[1].x, N[1].y);
      hi[t] = make_float4(N[2].x, N[2].y, N[3].x, N[3].y);
    }
  }
  __syncthreads();
  asm volatile("" : "+r"(i));  // the steps are computed again rather than held in registers meanwhile
  const QuadSite s = quad_site<D>(a, i, in);
  if (s.active) {
    const int m = a.g.hN0 >> 2;  // quads of a row
    const int peer = s.x1 == a.g.N[1] - 1 ? t - (a.g.N[1] - 1) * m : t + m;  // x + e1
    Quad2 up = quad_of(lo[peer], hi[peer]);
    if (!s.row.odd) {  // x + e1 - e0: one site back in the row
      const float4 e = hi[s.k == 0 ? peer + m - 1 : peer - 1];
      up.s[3] = up.s[2];
      up.s[2] = up.s[1];
      up.s[1] = up.s[0];
      up.s[0] = make_float2(e.z, e.w);
    }
    const QuadSums o = quad_staples<D, 1, false, 0>(a, i, s.fwd, s.bwd, s.row, ck, quad_of(lo[t], hi[t]), up);
    float2 N[4];
    quad_links<D, 1, MET, SRC>(a, i, o, ck, N);
  }
  pdl_release_dependents();
}

template <int D, int THREADS, int CTAS>
static cudaError_t launch(const cudaLaunchConfig_t &cfg, const UpdArgs &a, int rows, bool met, int src) {
  if (!met) return cudaLaunchKernelEx(&cfg, k_update_quad_duo<D, false, SRC_PHILOX, THREADS, CTAS>, a, rows);
  if (src == SRC_WINDOW) return cudaLaunchKernelEx(&cfg, k_update_quad_duo<D, true, SRC_WINDOW, THREADS, CTAS>, a, rows);
  return cudaLaunchKernelEx(&cfg, k_update_quad_duo<D, true, SRC_PHILOX, THREADS, CTAS>, a, rows);
}
template <int D>
static cudaError_t launch(const cudaLaunchConfig_t &cfg, const UpdArgs &a, const QuadDuoK &d, bool met, int src) {
  if (d.regs == 96) return launch<D, 288, 2>(cfg, a, d.rows, met, src);
  if (d.regs == 72) return launch<D, 896, 1>(cfg, a, d.rows, met, src);
  return launch<D, 1024, 1>(cfg, a, d.rows, met, src);
}

int launch_quad_duo(const UpdArgs &a, const QuadDuoK &d, cudaStream_t s, bool met, int src) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)d.blocks);
  cfg.blockDim = dim3((unsigned)d.threads);
  cfg.dynamicSmemBytes = (size_t)d.threads * 2 * sizeof(float4);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = a.g.dims == 3 ? launch<3>(cfg, a, d, met, src) : launch<4>(cfg, a, d, met, src);
  u1i::g_launches.fetch_add(1, std::memory_order_relaxed);
  if (e != cudaSuccess) return u1i::cuda_fail(e, "k_update_quad_duo");
  return U1_OK;
}

bool quad_duo_layout(const GeomK &g, int target, int sms, QuadDuoK &d) {
  d = QuadDuoK{};
  if (g.dims < 3 || (g.hN0 & 3) != 0) return false;
  const long long plane = (long long)(g.hN0 / 4) * g.N[1];
  if (plane > 1024) return false;
  if (target >= 256) target = 288;  // the largest block of the kernel with 96 registers
  const int planes = (int)(g.Vh / 4 / plane), per = std::max(1, std::min(target / (int)plane, planes));
  d.rows = per * (int)plane;
  d.threads = (d.rows + 31) / 32 * 32;
  d.blocks = (planes + per - 1) / per;
  const int per72 = 896 / d.threads, per64 = 1024 / d.threads;
  if (d.threads <= 288 && d.blocks <= (long long)sms * (576 / d.threads))
    d.regs = 96;
  else
    d.regs = per72 > 0 && (d.blocks <= (long long)sms * per72 || per72 == per64) ? 72 : 64;
  const int resident = d.regs == 96 ? 576 / d.threads : d.regs == 72 ? per72 : per64;
  d.one_wave = d.blocks <= (long long)sms * resident;
  return true;
}

}  // namespace u1b
