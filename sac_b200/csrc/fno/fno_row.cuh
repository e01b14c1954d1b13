// fno_row.cuh -- a Fourier layer's pixel stage, row by row, in one kernel.
//
// For every row (b, s) of F <= 256 pixels and its 32 output channels n
//
//   z[n][f] = bias[n] + sum_k W[n][k] in[b][k][s][f] + sum_j H[f][j] Y[(b,n)][s][j]
//   out     = z | GELU(z) | z * GELU'(pre)           (BF16; pre keeps z if asked)
//   T[b][s][n][j] = sum_f out[n][f] G[j][f]           (the next layer's first DFT)
//
// which serves the lift (no Y, no activation), the forward layers (H = Hy, G = Fy)
// and the backward ones (W transposed, H = FyT, G = HyT).  Against one GEMM launch
// per product it reads each activation once instead of twice, writes no FP32
// intermediate, and its loads run ahead of the products.
//
// Persistent CTAs of 512 threads take 4 rows of one sample at a time, two rows per
// turn, 8 warps to a row.  A pair's input (k x 256 pixels each, MN-major) and its Y
// blocks arrive by cp.async a turn ahead (two stages); one thread issues the pair's
// tcgen05.mma (two tiles of 128 pixels per row, N = 32) into one of two sets of TMEM
// accumulators while all threads run the epilogue of the pair before: tcgen05.ld,
// bias, activation, the BF16 outputs to memory (64-byte runs per channel) and, eight
// channels at a time, into shared memory as the MN-major operand of the product with
// G: after four rows that block is its 128 x 256 A (rows (s, n)), and the accumulator
// (N = 48) is stored as T during the next turn.
//
// Measured (B200, 64 samples of 256 x 256; a middle layer moves 268 MB in, 268 MB out
// and 50 MB of T): 225 us, against 454 + 139 for its GEMMs before; the lift 156 us, the
// last layer 159 (333 each).  It is bound by the epilogue's issue slots and the
// latency of its turn (43 % of the slots used, 38 % at 16 samples); 8 warps per SM took 293 us, and 487
// with 64-bit divisions in the row's indices, which are now stepped.
// Every mbarrier wait is bounded; on time-out the CTA sets bit 0 of the error word,
// drains its copies and MMAs, frees its TMEM and returns.
#pragma once
#include "fno_gemm.cuh"

namespace fno {

struct RowArgs {
  const bf16* in;       // [B][K1][S][F]
  const bf16* w;        // W[n][k] (w_n, w_k strides)
  int w_n, w_k;
  const bf16* h;        // [F][48] or nullptr
  const bf16* y;        // [(b,n)][S][48]
  const float* bias;    // [32] or nullptr
  bf16* out;            // [B][32][S][F]
  bf16* pre;            // forward: z is stored (nullptr: not); ACT_GELU_GRAD: read
  const bf16* g;        // [48][F] (T is computed) or nullptr
  bf16* t;              // [B][S][32][48]
  int B, S, F;
  int* err;
  int wait_tries;
  int t_wait_tries;  // of the wait for the product with G alone (the same meaning)
};

constexpr int kRowN = 32, kRowJ = 48, kRowF = 256, kRowThreads = 512;

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// shared-memory offsets (bytes): W, H, G, the outputs of 4 rows, the input stages
template <int K1, bool SPEC, bool NEXT>
struct RowSmem {
  static constexpr int W = 0;                                    // 32 x 64 K-major
  static constexpr int H = W + kRowN * 64 * 2;                   // 256 x 64 K-major
  static constexpr int G = H + (SPEC ? kRowF * 64 * 2 : 0);      // 48 x 256 K-major
  static constexpr int OUT = G + (NEXT ? kRowJ * kRowF * 2 : 0);  // 128 x 256 MN-major
  static constexpr int STG = OUT + (NEXT ? 4 * kRowN * kRowF * 2 : 0);
  static constexpr int IN_BYTES = K1 * kRowF * 2, Y_BYTES = SPEC ? kRowN * 64 * 2 : 0;
  static constexpr int STAGE = IN_BYTES + Y_BYTES;
  static constexpr int BYTES = STG + 4 * STAGE;  // two stages of two rows
};

__device__ __forceinline__ void row_mma(uint32_t tmem, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n}\n" ::"r"(tmem),
      "l"(da), "l"(db), "r"(idesc), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
}
__device__ __forceinline__ void row_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

template <int K1, bool SPEC, int ACT, bool NEXT, bool PRE>
__global__ void __launch_bounds__(kRowThreads, 1) k_row(const __grid_constant__ RowArgs a) {
  using L = RowSmem<K1, SPEC, NEXT>;
  constexpr bool STORE_PRE = PRE && ACT != ACT_GELU_GRAD;
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ uint64_t bar[2], bar_t;
  __shared__ uint32_t tmem_sh;
  __shared__ float bias_sh[kRowN];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int F = a.F, S = a.S, nch = F / 8;  // chunks of 8 pixels in a row

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_sh)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    mbar_init(&bar_t, 1);
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  // zero everything once (rows, columns and pixels past the sizes stay zero), then
  // the constant operands
  for (int i = tid; i < L::BYTES / 16; i += kRowThreads) reinterpret_cast<uint4*>(smem)[i] = make_uint4(0, 0, 0, 0);
  __syncthreads();
  for (int i = tid; i < kRowN * K1; i += kRowThreads) {  // W: (n/8*8 + k/8)*128 + n%8*16 + k%8*2
    const int n = i / K1, k = i % K1;
    *reinterpret_cast<bf16*>(smem + L::W + ((n / 8) * 8 + k / 8) * 128 + (n % 8) * 16 + (k % 8) * 2) =
        a.w[(long)n * a.w_n + (long)k * a.w_k];
  }
  if constexpr (SPEC) {
    for (int i = tid; i < F * 6; i += kRowThreads) {  // H rows of 6 chunks
      const int f = i / 6, c = i % 6;
      *reinterpret_cast<uint4*>(smem + L::H + ((f / 8) * 8 + c) * 128 + (f % 8) * 16) =
          __ldg(reinterpret_cast<const uint4*>(a.h + (long)f * kRowJ) + c);
    }
  }
  if constexpr (NEXT) {
    for (int i = tid; i < kRowJ * nch; i += kRowThreads) {  // G rows of F/8 chunks
      const int j = i / nch, c = i % nch;
      *reinterpret_cast<uint4*>(smem + L::G + ((j / 8) * 32 + c) * 128 + (j % 8) * 16) =
          __ldg(reinterpret_cast<const uint4*>(a.g + (long)j * F) + c);
    }
  }
  if (tid < kRowN) bias_sh[tid] = a.bias ? a.bias[tid] : 0.0f;
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_sh;
  const uint32_t id1 = umma_idesc(kRowN, 1, 0), id2 = umma_idesc(kRowN, 0, 0), idt = umma_idesc(kRowJ, 1, 0);
  const int tries = a.wait_tries == 0 ? kWaitTries : (a.wait_tries < 0 ? 0 : a.wait_tries);
  const int t_tries = a.t_wait_tries == 0 ? tries : (a.t_wait_tries < 0 ? 0 : a.t_wait_tries);

  // this CTA's rows: tasks of 4 rows, blockIdx.x, + gridDim.x, ...
  const int S4 = S / 4, ntask = a.B * S4;
  const int mine = (int)blockIdx.x < ntask ? (ntask - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
  const int npair = 2 * mine;
  // the sample and row of a position in that sequence, stepped pair by pair
  struct Pos {
    int b, s4, r;
  };
  auto step = [&](Pos& q) {
    q.r ^= 2;
    if (q.r) return;
    q.s4 += gridDim.x;
    while (q.s4 >= S4) q.s4 -= S4, ++q.b;
  };
  Pos pl{(int)blockIdx.x / S4, (int)blockIdx.x % S4, 0};  // the next pair to load
  Pos pe = pl, pt = pl;                                  // the epilogue's pair; the task of the next T
  const long plane = (long)S * F;
  // this thread's chunks of a pair: pixel chunk c of channel k of row w, one Y chunk
  constexpr int NL = 2 * K1 * kRowF / 8 / kRowThreads;
  long lsrc[NL];
  int ldst[NL];
#pragma unroll
  for (int u = 0; u < NL; ++u) {
    const int q = tid + u * kRowThreads, w = q / (K1 * nch), q1 = q - w * K1 * nch, k = q1 / nch, c = q1 % nch;
    lsrc[u] = w < 2 ? k * plane + (long)w * F + c * 8 : -1;
    ldst[u] = w * L::STAGE + ((k / 8) * 32 + c) * 128 + (k % 8) * 16;
  }
  const int yw = tid / (kRowN * 6), yn = tid % (kRowN * 6) / 6, yc = tid % 6;
  const int ydst = yw * L::STAGE + L::IN_BYTES + ((yn / 8) * 8 + yc) * 128 + (yn % 8) * 16;
  auto load_pair = [&](int i) {  // cp.async of pair i into its stage; one group per call
    if (i < npair) {
      const int sr = pl.s4 * 4 + pl.r;
      uint8_t* st = smem + L::STG + (i & 1) * 2 * L::STAGE;
      const bf16* src = a.in + (long)pl.b * K1 * plane + (long)sr * F;
#pragma unroll
      for (int u = 0; u < NL; ++u)
        if (lsrc[u] >= 0) cp_async16(st + ldst[u], src + lsrc[u]);
      if constexpr (SPEC)
        if (yw < 2) cp_async16(st + ydst, a.y + (((long)pl.b * kRowN + yn) * S + sr + yw) * kRowJ + yc * 8);
      step(pl);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto issue_pair = [&](int i) {  // by one thread: the products of pair i
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t w0 = smem_u32(smem + L::W), h0 = smem_u32(smem + L::H);
    for (int w = 0; w < 2; ++w) {
      const uint32_t st = smem_u32(smem + L::STG + ((i & 1) * 2 + w) * L::STAGE);
      for (int tile = 0; tile < (F + 127) / 128; ++tile) {
        const uint32_t acc = tmem + (uint32_t)((i & 1) * 128 + w * 64 + tile * 32);
#pragma unroll
        for (int kk = 0; kk < K1 / 16; ++kk)
          row_mma(acc, umma_sdesc(st + kk * 2 * kRowF * 16 + tile * 2048, kRowF * 16, 128),
                  umma_sdesc(w0 + kk * 256, 128, 1024), id1, kk > 0);
        if constexpr (SPEC) {
#pragma unroll
          for (int kk = 0; kk < kRowJ / 16; ++kk)
            row_mma(acc, umma_sdesc(h0 + tile * 16384 + kk * 256, 128, 1024),
                    umma_sdesc(st + L::IN_BYTES + kk * 256, 128, 1024), id2, 1u);
        }
      }
    }
    row_commit(&bar[i & 1]);
  };

  bool ok = true;
  int issued = 0;    // pairs whose products were issued
  int t_issued = 0;  // products with G issued
  int t_done = 0;    // ... and stored
  // T of the task whose product was issued last: row m = (s, n) of the accumulator
  auto store_t = [&]() {
    // one outcome per warp: the loads below need all its lanes, together
    if (!__all_sync(0xffffffffu, mbar_wait(&bar_t, (uint32_t)(t_done & 1), t_tries))) {
      ok = false;
      return;
    }
    ++t_done;
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (warp < 4) {
      uint4* dst = reinterpret_cast<uint4*>(a.t + (((long)pt.b * S + pt.s4 * 4 + warp) * kRowN + lane) * kRowJ);
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        uint32_t v[16];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
              "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
            : "r"(tmem + ((uint32_t)(warp * 32) << 16) + 256u + 16u * q));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        uint32_t p[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const __nv_bfloat162 x = __floats2bfloat162_rn(__uint_as_float(v[2 * e]), __uint_as_float(v[2 * e + 1]));
          p[e] = *reinterpret_cast<const uint32_t*>(&x);
        }
        dst[2 * q] = make_uint4(p[0], p[1], p[2], p[3]);
        dst[2 * q + 1] = make_uint4(p[4], p[5], p[6], p[7]);
      }
    }
    pt.r = 2;
    step(pt);
  };

  load_pair(0);
  load_pair(1);
  if (npair > 0) {
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (tid == 0) issue_pair(0);
    issued = 1;
  }
  const int w = warp >> 3, tile = (warp >> 2) & 1, f = tile * 128 + (warp & 3) * 32 + lane;  // this thread's pixel
  for (int i = 0; i < npair; ++i) {
    if (!mbar_wait(&bar[i & 1], (uint32_t)((i >> 1) & 1), tries)) ok = false;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;");
    // pair i is done, pair i + 1 has arrived; pair i - 1 was read from its accumulators
    // and staged
    if (__syncthreads_or(!ok)) {
      ok = false;
      break;
    }
    if (i + 1 < npair) {
      if (tid == 0) issue_pair(i + 1);
      issued = i + 2;
    }
    load_pair(i + 2);  // into the stage of pair i
    asm volatile("tcgen05.fence::after_thread_sync;");
    uint32_t o[kRowN / 2];  // the row's outputs, channel pairs
    const bool live = ok && f < F;
    if (ok && tile * 128 < F) {
      uint32_t v[32];
#pragma unroll
      for (int q = 0; q < 2; ++q)
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
            : "=r"(v[16 * q]), "=r"(v[16 * q + 1]), "=r"(v[16 * q + 2]), "=r"(v[16 * q + 3]), "=r"(v[16 * q + 4]),
              "=r"(v[16 * q + 5]), "=r"(v[16 * q + 6]), "=r"(v[16 * q + 7]), "=r"(v[16 * q + 8]), "=r"(v[16 * q + 9]),
              "=r"(v[16 * q + 10]), "=r"(v[16 * q + 11]), "=r"(v[16 * q + 12]), "=r"(v[16 * q + 13]),
              "=r"(v[16 * q + 14]), "=r"(v[16 * q + 15])
            : "r"(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)((i & 1) * 128 + w * 64 + tile * 32 + 16 * q)));
      const long off = (long)pe.b * kRowN * plane + (long)(pe.s4 * 4 + pe.r + w) * F + f;
      bf16 pr[kRowN];
      if constexpr (ACT == ACT_GELU_GRAD) {
#pragma unroll
        for (int n = 0; n < kRowN; ++n) pr[n] = live ? a.pre[off + n * plane] : __float2bfloat16(0.f);
      }
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int n = 0; n < kRowN; n += 2) {
        float z[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          z[e] = __uint_as_float(v[n + e]) + bias_sh[n + e];
          if constexpr (STORE_PRE)
            if (live) a.pre[off + (n + e) * plane] = __float2bfloat16(z[e]);
          if constexpr (ACT == ACT_GELU_GRAD) z[e] *= gelu_grad_f(__bfloat162float(pr[n + e]));
        }
        if constexpr (ACT == ACT_GELU) gelu_2(z[0], z[1]);
        const __nv_bfloat162 x = __floats2bfloat162_rn(z[0], z[1]);
        o[n / 2] = *reinterpret_cast<const uint32_t*>(&x);
        if (live) {
          a.out[off + n * plane] = x.x;
          a.out[off + (n + 1) * plane] = x.y;
        }
      }
    }
    if constexpr (NEXT) {
      // the product of the task before has read the staged rows, and its accumulator is
      // free for the next one
      if (pe.r == 0 && t_issued > t_done && ok) store_t();
      if (live && ok) {  // (f/8 * 16 + (r*4 + n/8))*128 + f%8*16
        uint8_t* d = smem + L::OUT + ((f >> 3) * 16 + (pe.r + w) * 4) * 128 + (f & 7) * 16;
#pragma unroll
        for (int q = 0; q < 4; ++q)
          *reinterpret_cast<uint4*>(d + q * 128) = make_uint4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
      }
      if (pe.r == 2) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;");
        if (__syncthreads_or(!ok)) {
          ok = false;
          break;
        }
        if (tid == 0) {
          asm volatile("tcgen05.fence::after_thread_sync;");
          const uint32_t a0 = smem_u32(smem + L::OUT), g0 = smem_u32(smem + L::G);
          for (int kk = 0; kk < (F + 15) / 16; ++kk)
            row_mma(tmem + 256u, umma_sdesc(a0 + kk * 4096, 2048, 128), umma_sdesc(g0 + kk * 256, 128, 4096), idt, kk > 0);
          row_commit(&bar_t);
        }
        ++t_issued;
      }
    }
    step(pe);
  }
  if (ok && NEXT && t_issued > t_done) store_t();
  if (__syncthreads_or(!ok)) {
    if (tid == 0 && a.err) atomicOr(a.err, 1);
    // let the MMAs in flight drain (bounded) before the memory is released
    if (issued > 0) mbar_wait(&bar[(issued - 1) & 1], (uint32_t)(((issued - 1) >> 1) & 1));
    if (issued > 1) mbar_wait(&bar[(issued - 2) & 1], (uint32_t)(((issued - 2) >> 1) & 1));
    if (t_issued > 0) mbar_wait(&bar_t, (uint32_t)((t_issued - 1) & 1));
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
}

}  // namespace fno
