// fno_wgrad.cuh -- a 32-channel layer's weight and bias gradients in one pass.
//
//   gw[o][c] += sum_{b,p} dz[b][o][p] in[b][c][p],   gb[o] += sum_{b,p} dz[b][o][p]
//
// Bound by reading dz and in once.  Four rows of pixels are stacked: A holds their 32
// channels of dz each (128 x 128 pixels, K-major, as they lie in memory), B their C
// channels of in and a row of ones, so that one tcgen05.mma per 16 pixels fills the
// tile's 128 rows; the four diagonal 32 x C blocks and the column of the ones are the
// result (the products between different rows are not read).  A GEMM on one row's 32
// channels filled a quarter of its tile, and the bias was another pass over dz.
//
// Persistent CTAs take four rows at a time, 128 pixels per stage by cp.async, two of
// the three stages in flight.  TMEM accumulates over one task's pixels (at most 1024
// products into each sum); the tasks' sums are added in registers, and each CTA adds
// its own to memory once.  Every mbarrier wait is bounded; on time-out the CTA sets
// bit 0 of the error word, drains its copies and MMAs, frees its TMEM and returns.
#pragma once
#include "fno_row.cuh"

namespace fno {

struct WgradArgs {
  const bf16* dz;  // [B][32][S][F]
  const bf16* in;  // [B][C][S][F]
  float* gw;       // [32][C]
  float* gb;       // [32]
  int B, S, F;
  int* err;
  int wait_tries;
};

constexpr int kWgThreads = 256, kWgPix = 128, kWgStages = 3;

template <int C>
struct WgradSmem {
  static constexpr int A = 4 * kRowN * kWgPix * 2, B = (4 * C + 16) * kWgPix * 2;
  static constexpr int STAGE = A + B, BYTES = kWgStages * STAGE;
};

template <int C>
__global__ void __launch_bounds__(kWgThreads, 1) k_wgrad(const __grid_constant__ WgradArgs a) {
  using L = WgradSmem<C>;
  constexpr int NCH = kWgPix / 8;                      // chunks of 8 pixels in a stage's row
  constexpr int NN = 4 * C + 16;                       // columns: four blocks, the ones (and 15 of zeros)
  constexpr int NA = 4 * kRowN * NCH / kWgThreads, NB = 4 * C * NCH / kWgThreads;
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ uint64_t bar[kWgStages];
  __shared__ uint32_t tmem_sh;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int F = a.F, S = a.S;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_sh)),
                 "r"(256));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int s = 0; s < kWgStages; ++s) mbar_init(&bar[s], 1);
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  // rows 4C .. 4C+15 of every B: a row of ones, then zeros
  for (int i = tid; i < kWgStages * 16 * NCH; i += kWgThreads) {
    const int s = i / (16 * NCH), r = i / NCH % 16, c = i % NCH;
    const uint32_t v = r == 0 ? 0x3f803f80u : 0u;
    *reinterpret_cast<uint4*>(smem + s * L::STAGE + L::A + (((4 * C + r) / 8) * NCH + c) * 128 + (r % 8) * 16) =
        make_uint4(v, v, v, v);
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_sh;
  const int tries = a.wait_tries == 0 ? kWaitTries : (a.wait_tries < 0 ? 0 : a.wait_tries);

  const int S4 = S / 4, ntask = a.B * S4, nck = (F + kWgPix - 1) / kWgPix;
  const int mine = (int)blockIdx.x < ntask ? (ntask - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
  const int n = mine * nck;
  const long plane = (long)S * F;
  int lb = (int)blockIdx.x / S4, ls = (int)blockIdx.x % S4, lc = 0;  // the next stage to load
  const int ch = tid % NCH, row0 = tid / NCH;  // this thread's chunk of rows row0, + 16, ...
  auto load = [&](int i) {  // one cp.async group per call
    if (i < n) {
      uint8_t* st = smem + (i % kWgStages) * L::STAGE;
      const bool in_row = lc * kWgPix + ch * 8 < F;
      const long px = (long)ls * 4 * F + lc * kWgPix + ch * 8;
      const bf16 *pd = a.dz + (long)lb * kRowN * plane + px, *pi = a.in + (long)lb * C * plane + px;
#pragma unroll
      for (int u = 0; u < NA; ++u) {  // row m = r * 32 + o
        const int m = row0 + u * (kWgThreads / NCH);
        uint8_t* d = st + ((m / 8) * NCH + ch) * 128 + (m % 8) * 16;
        if (in_row) cp_async16(d, pd + (m % kRowN) * plane + (long)(m / kRowN) * F);
        else *reinterpret_cast<uint4*>(d) = make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int u = 0; u < NB; ++u) {  // row m = r * C + c
        const int m = row0 + u * (kWgThreads / NCH);
        uint8_t* d = st + L::A + ((m / 8) * NCH + ch) * 128 + (m % 8) * 16;
        if (in_row) cp_async16(d, pi + (m % C) * plane + (long)(m / C) * F);
        else *reinterpret_cast<uint4*>(d) = make_uint4(0, 0, 0, 0);
      }
      if (++lc == nck) {
        lc = 0;
        ls += gridDim.x;
        while (ls >= S4) ls -= S4, ++lb;
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  float sum[C + 1];  // row (r, o) of this thread's block; the last is the ones' column
#pragma unroll
  for (int c = 0; c <= C; ++c) sum[c] = 0.f;
  bool ok = true;
  int issued = 0, ck = 0;  // stages whose products were issued; the stage's place in its task
  load(0);
  load(1);
  for (int i = 0; i < n; ++i) {
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;");
    if (__syncthreads_or(!ok)) {  // stage i has arrived; the sums of a finished task were read
      ok = false;
      break;
    }
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;");
      const uint32_t st = smem_u32(smem + (i % kWgStages) * L::STAGE);
#pragma unroll
      for (int kk = 0; kk < kWgPix / 16; ++kk)
        row_mma(tmem, umma_sdesc(st + kk * 256, 128, NCH * 128), umma_sdesc(st + L::A + kk * 256, 128, NCH * 128),
                umma_idesc(NN, 0, 0), ck > 0 || kk > 0);
      row_commit(&bar[i % kWgStages]);
    }
    issued = i + 1;
    // the stage before has been read: its buffer takes stage i + 2
    if (i > 0 && !mbar_wait(&bar[(i - 1) % kWgStages], (uint32_t)((i - 1) / kWgStages & 1), tries)) ok = false;
    if (ok) load(i + 2);
    if (++ck == nck) {  // the task's sums
      ck = 0;
      if (ok && !mbar_wait(&bar[i % kWgStages], (uint32_t)(i / kWgStages & 1), tries)) ok = false;
      if (__all_sync(0xffffffffu, ok) && warp < 4) {
        asm volatile("tcgen05.fence::after_thread_sync;");
        const uint32_t t0 = tmem + ((uint32_t)(warp * 32) << 16);
#pragma unroll
        for (int q = 0; q < C / 16; ++q) {
          uint32_t v[16];
          asm volatile(
              "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
              : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
              : "r"(t0 + (uint32_t)(warp * C + 16 * q)));
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int e = 0; e < 16; ++e) sum[16 * q + e] += __uint_as_float(v[e]);
        }
        uint32_t v1;
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(v1) : "r"(t0 + (uint32_t)(4 * C)));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        sum[C] += __uint_as_float(v1);
      }
    }
  }
  if (__syncthreads_or(!ok)) {
    if (tid == 0 && a.err) atomicOr(a.err, 1);
    // the MMAs complete in order: let the last issued drain (bounded)
    if (issued > 0) mbar_wait(&bar[(issued - 1) % kWgStages], (uint32_t)((issued - 1) / kWgStages & 1));
  } else if (warp < 4 && n > 0) {
#pragma unroll
    for (int c = 0; c < C; ++c) atomicAdd(a.gw + lane * C + c, sum[c]);
    atomicAdd(a.gb + lane, sum[C]);
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256));
}

}  // namespace fno
