// fno_wgrad.cuh -- a layer's weight and bias gradients in one pass.
//
//   gw[o][c] += sum_{b,p} d[b][o][p] in[b][c][p],   gb[o] += sum_{b,p} d[b][o][p]
//
// for R = 32 or 128 rows o and C columns c.  Bound by reading d and in once.  128 / R
// rows of pixels are stacked: A holds their R channels of d each (128 x 128 pixels,
// K-major, as they lie in memory), B their C channels of in and a row of ones, so that
// one tcgen05.mma per 16 pixels fills the tile's 128 rows; the diagonal R x C blocks
// and the column of the ones are the result (the products between different rows are
// not read).  A GEMM on one row's 32 channels filled a quarter of its tile, and the
// bias was another pass over d.  The projection's second layer has 8 rows of d and
// takes its 128 input channels as A (TR: the result is stored transposed).
//
// Persistent CTAs take 128 / R rows at a time, 128 pixels per stage by cp.async, two of
// the three stages in flight.  TMEM accumulates at most 1024 products into each sum,
// which are then added in registers; each CTA adds its own to memory once.  Every
// mbarrier wait is bounded; on time-out the CTA sets bit 0 of the error word, drains
// its copies and MMAs, frees its TMEM and returns.
//
// Measured (B200, training step of 6 minibatches of 16 samples of 256 x 256): 28.5 ->
// 22.9 ms for the layers' and the lift's gradients (their GEMMs took 173 us each for
// 268 MB, the bias passes 17), 23.1 -> 22.0 for the projection's.
#pragma once
#include "fno_row.cuh"

namespace fno {

struct WgradArgs {
  const bf16* d;   // [B][R][S][F]
  const bf16* in;  // [B][C][S][F]
  float* gw;       // [R][C], or [C][R] (TR)
  float* gb;       // [R], or nullptr
  int B, S, F;
  int* err;
  int wait_tries;
};

constexpr int kWgThreads = 256, kWgPix = 128, kWgStages = 3;

template <int R, int C>
struct WgradSmem {
  static constexpr int ROWS = 128 / R;                      // rows of pixels side by side
  static constexpr int NN = (ROWS * C + 1 + 15) / 16 * 16;  // columns: the blocks, the ones, zeros
  static constexpr int A = 128 * kWgPix * 2, B = NN * kWgPix * 2;
  static constexpr int STAGE = A + B, BYTES = kWgStages * STAGE;
};

template <int R, int C, bool TR>
__global__ void __launch_bounds__(kWgThreads, 1) k_wgrad(const __grid_constant__ WgradArgs a) {
  using L = WgradSmem<R, C>;
  constexpr int NCH = kWgPix / 8;  // chunks of 8 pixels in a stage's row
  constexpr int NN = L::NN, ROWS = L::ROWS, ONES = ROWS * C;
  constexpr int STEP = kWgThreads / NCH, NA = 128 / STEP, NB = (ONES + STEP - 1) / STEP;
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
  // the rows of every B past the input's: a row of ones, then zeros
  for (int i = tid; i < kWgStages * (NN - ONES) * NCH; i += kWgThreads) {
    const int s = i / ((NN - ONES) * NCH), r = ONES + i / NCH % (NN - ONES), c = i % NCH;
    const uint32_t v = r == ONES ? 0x3f803f80u : 0u;
    *reinterpret_cast<uint4*>(smem + s * L::STAGE + L::A + ((r / 8) * NCH + c) * 128 + (r % 8) * 16) =
        make_uint4(v, v, v, v);
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_sh;
  const int tries = a.wait_tries == 0 ? kWaitTries : (a.wait_tries < 0 ? 0 : a.wait_tries);

  const int S4 = S / ROWS, ntask = a.B * S4, nck = (F + kWgPix - 1) / kWgPix;
  const int mine = (int)blockIdx.x < ntask ? (ntask - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
  const int n = mine * nck, per_sum = nck * (4 / ROWS);  // stages; those between readings of the sums
  const long plane = (long)S * F;
  int lb = (int)blockIdx.x / S4, ls = (int)blockIdx.x % S4, lc = 0;  // the next stage to load
  const int ch = tid % NCH, row0 = tid / NCH;  // this thread's chunk of rows row0, + 16, ...
  auto load = [&](int i) {  // one cp.async group per call
    if (i < n) {
      uint8_t* st = smem + (i % kWgStages) * L::STAGE;
      const bool in_row = lc * kWgPix + ch * 8 < F;
      const long px = (long)ls * ROWS * F + lc * kWgPix + ch * 8;
      const bf16 *pd = a.d + (long)lb * R * plane + px, *pi = a.in + (long)lb * C * plane + px;
#pragma unroll
      for (int u = 0; u < NA; ++u) {  // row m = r * R + o
        const int m = row0 + u * STEP;
        uint8_t* d = st + ((m / 8) * NCH + ch) * 128 + (m % 8) * 16;
        if (in_row) cp_async16(d, pd + (m % R) * plane + (long)(m / R) * F);
        else *reinterpret_cast<uint4*>(d) = make_uint4(0, 0, 0, 0);
      }
#pragma unroll
      for (int u = 0; u < NB; ++u) {  // row m = r * C + c
        const int m = row0 + u * STEP;
        if (ONES % STEP != 0 && m >= ONES) break;
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
  int issued = 0, ck = 0;  // stages whose products were issued; the stage's place in its sums
  load(0);
  load(1);
  for (int i = 0; i < n; ++i) {
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;");
    if (__syncthreads_or(!ok)) {  // stage i has arrived; the sums before were read
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
    if (++ck == per_sum || i == n - 1) {
      ck = 0;
      if (ok && !mbar_wait(&bar[i % kWgStages], (uint32_t)(i / kWgStages & 1), tries)) ok = false;
      if (__all_sync(0xffffffffu, ok) && warp < 4) {
        asm volatile("tcgen05.fence::after_thread_sync;");
        const uint32_t t0 = tmem + ((uint32_t)(warp * 32) << 16), tb = t0 + (uint32_t)(warp * 32 / R * C);
#pragma unroll
        for (int q = 0; q < (C + 15) / 16; ++q) {  // (C = 8: the columns past it are not used)
          uint32_t v[16];
          asm volatile(
              "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
              : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
              : "r"(tb + (uint32_t)(16 * q)));
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int e = 0; e < 16; ++e)
            if (16 * q + e < C) sum[16 * q + e] += __uint_as_float(v[e]);
        }
        uint32_t v1;
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(v1) : "r"(t0 + (uint32_t)ONES));
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
    const int o = (warp * 32 + lane) % R;
#pragma unroll
    for (int c = 0; c < C; ++c) atomicAdd(a.gw + (TR ? c * R + o : o * C + c), sum[c]);
    if (a.gb) atomicAdd(a.gb + o, sum[C]);
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256));
}

}  // namespace fno
