// sac_step1d.cuh -- a whole RK4 step of a small 1D grid in one launch.
//
// A cluster of 8 CTAs holds the grid's stencil fields in shared memory, a segment of
// the cells (and three to either side) each, and runs the four stages of 'fourstep'
// (src/vac.t:439-455) one after another, each as k_face, k_nu, k_update and k_bound do,
// with cluster barriers between them instead of launches (c_tot's maximum crosses by
// distributed shared memory, the stage's output through L2): the same device functions
// in the same order, so the results are theirs bit for bit.
//
// A step of 800 cells was 20 launches whose blocks fill 4 of 148 SMs: their latency
// and the gaps between them, not their work, were its time (182 us per step, 49 us of
// it in k_update's dependent divisions, 34 us in k_bound, which resolved a ghost cell's
// variables one after another).  In one CTA of 1024 threads the kernel took 75 us, one
// SM's FP64 units and its barriers.
#pragma once
#include <cooperative_groups.h>

#include <algorithm>

#include "sac_stage.cuh"

namespace sacgpu {

constexpr int kStep1dThreads = 1024;  // at most; a thread per cell of the segment where they suffice

// shared fields: rho', m_1, rho'+rhob, v_1, the "173" energy, the fluxes (none of b_1),
// the quotients of the three setnu pairs; then a byte per cell (out_of_range)
template <int NDIR>
__host__ __device__ constexpr int step1d_fields() {
  return 5 + (2 * NDIR + 2 - 1) + 3;
}

// the block's maximum of non-negative values in every thread (sh: 33 doubles); NaN when
// any is NaN, as block_max_to
__device__ __forceinline__ double block_max_all(double v, double* sh) {
  const bool anynan = __syncthreads_or(v != v);
  v = warp_max(v != v ? 0.0 : v);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    v = warp_max(threadIdx.x < blockDim.x / 32 ? sh[threadIdx.x] : 0.0);
    if (threadIdx.x == 0) sh[32] = v;
  }
  __syncthreads();
  return anynan ? __longlong_as_double(0x7ff8000000000000ll) : sh[32];
}

template <int NDIR, typename S>
__global__ void __cluster_dims__(kStep1dCtas, 1, 1) __launch_bounds__(kStep1dThreads, 1)
    k_step1d(const __grid_constant__ Step1dArgs p) {
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ double sh[33];
  __shared__ double ct_part[kStep1dCtas];  // each CTA's part of c_tot
  auto cluster = cooperative_groups::this_cluster();
  constexpr int NP = 2 * NDIR + 2, B0 = NDIR + 1;
  const Geom g = p.st[0].g;
  const int lo = g.lo[0], hi = g.hi[0], tid = threadIdx.x, nt = blockDim.x;
  // this CTA's cells c0..c1-1, and with their stencils cb..ce-1
  const int seg = step1d_segment(g.n[0]), rank = (int)cluster.block_rank();
  const int c0 = min(rank * seg, g.n[0]), c1 = min(c0 + seg, g.n[0]);
  const int u0 = max(c0, lo), u1 = min(c1 - 1, hi);  // its mesh cells (none: u0 > u1)
  const int cb = max(c0 - 3, 0), ce = min(c1 + 3, g.n[0]), n = seg + 6;
  S* sm = reinterpret_cast<S*>(smraw) - cb;  // indexed by the grid's cell
  S *rho = sm, *m1 = sm + n, *rt = sm + 2 * n, *v1 = sm + 3 * n, *e173 = sm + 4 * n, *fl = sm + 5 * n;
  S* qn = fl + (NP - 1) * n;
  unsigned char* bad = smraw + (long)step1d_fields<NDIR>() * n * sizeof(S) - cb;
  auto slot = [](int iw) { return iw < B0 + 1 ? iw : iw - 1; };  // b_1 (variable B0 + 1) has no flux
  long ns[3];
  ghost_slabs(g, ns);
  // a CTA's shared memory may be written by the others only once it is known to have
  // started: arrive here, wait before the first write (stage 0), behind its k_face
  cluster.barrier_arrive();
#pragma unroll 1
  for (int s = 0; s < 4; ++s) {
    const Stage2Args& a = p.st[s];
    // ---- k_face ----
    double cm = 0.0;
    for (int c = cb + tid; c < ce; c += nt) {
      const bool mesh = a.visc_on && c >= lo && c <= hi;
      double cc = 0.0;
      const bool b = face_eval<1, NDIR, S>(
          a, Offs{}, c, mesh, a.gamma, &cc, 1u, true,
          [&](int i, S x) {
            if (i == 0) rt[c] = x;
            else if (i == 1) v1[c] = x;
            else if (i == NDIR + 1) e173[c] = x;
          },
          [&](int, int iw, S x) { fl[slot(iw) * n + c] = x; });
      bad[c] = b;
      rho[c] = ((const S*)a.fW[0])[c];
      m1[c] = ((const S*)a.fW[1])[c];
      if (mesh) cm = (cc != cc || cm != cm) ? __longlong_as_double(0x7ff8000000000000ll) : fmax(cm, cc);
    }
    double ct = 0.0;
    if (s == 0) cluster.barrier_wait();
    if (a.visc_on) {
      cm = block_max_all(cm, sh);
      if (tid < kStep1dCtas) *cluster.map_shared_rank(&ct_part[rank], tid) = cm;
      cluster.sync();  // and the fields of this CTA
      for (int r = 0; r < kStep1dCtas; ++r) {
        const double q = ct_part[r];
        ct = (ct != ct || q != q) ? __longlong_as_double(0x7ff8000000000000ll) : fmax(ct, q);
      }
      if (rank == 0 && tid == 0) *(unsigned long long*)a.ctot = (unsigned long long)__double_as_longlong(ct);
    } else {
      __syncthreads();
    }
    // ---- k_nu ----
    if (a.visc_on) {
      const S p04 = (S)(ct * 0.04), p4 = (S)(ct * 0.4);
      for (int c = u0 - 1 + tid; u0 <= u1 && c <= u1; c += nt) {
        int off[6];
        face_offsets(c, 1, c, lo, hi, off);
        S md3, md1;
        face_maxima<true>((const S*)rho, off, md3, md1);
        qn[c] = face_ratio(p04, md3, md1);
        face_maxima<true>((const S*)e173, off, md3, md1);
        qn[n + c] = face_ratio(p04, md3, md1);
        face_maxima<true>((const S*)v1, off, md3, md1);
        qn[2 * n + c] = face_ratio(p4, md3, md1);
      }
      __syncthreads();
    }
    // ---- k_update ----
    double numax = 0.0;
    const bool ct_bad = sizeof(S) == 8 && a.visc_on && ctot_out_of_range((unsigned long long)__double_as_longlong(ct));
    for (int u = u0; u <= u1; u += nt) {  // whole warps, for the vote
      const int c = u + tid;
      const bool in = c <= u1;
      bool slow = a.general || ct_bad;
      if (sizeof(S) == 8 && in)
        for (int q = max(c - 3, cb); q <= min(c + 3, ce - 1); ++q) slow = slow || bad[q];
      slow = __any_sync(0xffffffffu, slow);
      if (!in) continue;
      TileView<S> tv;
      tv.W[0] = rho;
      tv.W[1] = m1;
      tv.D[0] = rt;
      tv.D[1] = v1;
      tv.D[NDIR + 1] = e173;
#pragma unroll
      for (int iw = 0; iw < NP; ++iw)
        if (iw != B0 + 1) tv.F[0][iw] = fl + slot(iw) * n;
      tv.Q[0] = qn;
      tv.Q[1] = qn + n;
      tv.Q[2] = qn + 2 * n;
      tv.st1 = 0;
      tv.c = c;
      tv.cg = c;
      const int pos[3] = {c, 0, 0};
      double nm = 0.0;
      if (slow)
        update_cell<1, NDIR, S, 0, false, true>(a, g, Offs{}, pos, a.qdt, a.qdt2, a.tdep, a.drvA, nm, &tv);
      else
        update_cell<1, NDIR, S, 0, true, true>(a, g, Offs{}, pos, a.qdt, a.qdt2, a.tdep, a.drvA, nm, &tv);
      numax = fmax(numax, nm);
    }
    if (a.visc_on) {
      const double m = block_max_all(numax, sh);
      if (tid == 0) atomic_max_nonneg(a.maxnu, m);
    }
    cluster.sync();  // the stage's output, which the fill and the next stage read
    // ---- k_bound: a thread per ghost cell and variable ----
    if (rank == 0)
      for (int t = tid; t < (int)ns[0] * NP; t += nt)
        bound_cell<S>(p.bc[s], t / NP, ns, t % NP, t % NP + 1);
    cluster.sync();
  }
}

template <typename S>
cudaError_t launch_step1d(const Step1dArgs& p0, cudaStream_t st) {
  Step1dArgs p = p0;
  for (int s = 0; s < 4; ++s) fill_field_ptrs(p.st[s], sizeof(S));
  const Geom& g = p.st[0].g;
  const int m = step1d_segment(g.n[0]) + 6, smem = step1d_smem(g.np, g.n[0], sizeof(S));
  const unsigned nt = (unsigned)std::min(kStep1dThreads, (m + 31) / 32 * 32);
  auto go = [&](auto NR) -> cudaError_t {
    auto* k = k_step1d<decltype(NR)::value, S>;
    // the kernel's own limit, not this grid's size: host threads with grids of other
    // sizes share the attribute
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kStep1dSmem);
    if (e != cudaSuccess) return e;
    k<<<kStep1dCtas, nt, smem, st>>>(p);
    return cudaGetLastError();
  };
  if (g.ndir == 1) return go(std::integral_constant<int, 1>{});
  if (g.ndir == 2) return go(std::integral_constant<int, 2>{});
  return go(std::integral_constant<int, 3>{});
}

}  // namespace sacgpu
