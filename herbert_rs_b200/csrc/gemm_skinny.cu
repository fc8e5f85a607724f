// Skinny matrix product for decoding: few activation rows against a whole weight matrix.
//   C[M,N] (op)= A[M,K] * W[N,K]^T,  M <= 64, bfloat16 operands, float accumulation.
//
// A decode step reads every weight once and is bound by that stream, so the kernel is laid out
// around the weight bytes (the reference's matvec has the same premise: one pass over W per
// token, backends/backend_bf16_avx512/src/avx512_bf16_matvec.S:1-60).  The weight rows are the
// M operand of the tensor-core instruction ("swapped" roles): one CTA owns 16 weight rows, its 8
// warps share K, and every lane fetches 16 contiguous bytes of a weight row straight from global
// memory into the registers mma.sync.m16n8k16 wants.  The k index inside one instruction is
// permuted the same way for both operands (a lane's 8 consecutive elements serve k-slots
// {2t,2t+1,2t+8,2t+9} of two instructions), which leaves the dot products unchanged.  Up to 32 rows a lane's pieces wait between memory and
// registers in shared memory of its own (cp.async, read back by the lane that asked: no barrier), so that what a CTA has under
// way is not bound by its registers: six batches where the grid gives an SM one CTA, three where it gives two and a batch and the sums
// leave room, else two (see `depth` below; a batch is 32 KB, from 17 rows on 16 KB).  What an SM has under way is its rate: with two batches
// in registers (32 KB a CTA) the products of 2,048 rows, one CTA an SM, ran at 2.7 TB/s.  And with the SM's shared memory taken, the next
// kernel's CTAs (they start early, see common.cuh) find one place where one of these has left, so they spread over the SMs; kernels
// without that crowded on the SMs that were done first, which made early starts slower than none.  Measured on a B200 with both (before -> now, us
// a pass): the 0.6B-sized decoder's two steps of one sequence 1,806 -> 1,505, four steps of eight sequences on eight 8B-sized layers 4,142 -> 3,994,
// four of 17 and 32 on the 0.6B-sized one 4,744 -> 3,970 and 4,980 -> 4,395, turns of the designs 1.03 to 1.08 times faster; the ring without early
// starts 1,690 and 4,141, early starts without the ring 1,992 and 6,015.
// From 33 rows on every CTA reads so many activations that what the ring takes from L1 costs more than it gives (64 x 3,072 on 1,024 rows
// alone 13.4 us without, 13.9 with it; four 0.6B-sized steps of 63 sequences 7,500 without early starts, 8,210 with ring and early starts,
// 7,000 as it is now): there a batch waits in registers, and the next kernel is let start when a CTA's last weights are in.
// The activation rows (at most 64 x K) come through L1/L2.  Partial sums of the 8 warps meet in
// shared memory; the epilogue stores, adds into the float residual stream, or applies SwiGLU to
// rows stored as 8 gate rows followed by the 8 up rows of the same channels.
#include <stdlib.h>

#include "api.h"
#include "common.cuh"
#include "per_device.h"

#define SK_WARPS 8
#define SK_THREADS (SK_WARPS * 32)
#define SK_NORM_ROWS 16
#define SK_RING(NT) ((NT) < 8)      // up to 32 rows; see above

__device__ __forceinline__ void sk_copy16(unsigned dst, const void* src, bool there) {      // zeros where there is nothing
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(there ? 16 : 0) : "memory");
}
__device__ __forceinline__ uint4 sk_read16(unsigned src) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(src) : "memory");
  return v;
}
__device__ __forceinline__ uint4 ld_stream16(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void mma_bf16_16816(float* d, unsigned a0, unsigned a1, unsigned a2, unsigned a3,
                                               unsigned b0, unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// A norm shared between two products.  RMSNorm is y = x * w / rms(x): the product that last adds
// into the residual stream x can also write x * w (bfloat16) and, per group of its output columns,
// the sum of x^2; the product that reads y takes x * w as its activation and multiplies its results
// by 1 / rms, which it gets from those partial sums.  No kernel between the two, no pass over x.
struct SkinnyNorm {
  const float* in_sumsq;   // consumer: [in_parts][SK_NORM_ROWS] partial sums of x^2 of the activation rows, or null
  int in_parts;
  float in_eps;            // 1/rms = rsqrt(sum / K + eps)
  const float* out_w;      // producer (residual epilogue): the next norm's weight [N], or null
  bf16* out_xw;            // [M, out_ld] = residual * out_w
  int out_ld;
  float* out_sumsq;        // [units][SK_NORM_ROWS]
  // SwiGLU epilogue only (with and without a norm).  > 0: the clamped form with this limit (HB_ACT_SWISH_CLAMP)
  float glu_limit;
};

// NT: 8-token tiles (M <= 8 * NT).  RG: groups of 16 weight rows per CTA; a warp multiplies each
// activation fragment it loads with RG weight fragments, so the activation traffic per weight byte
// falls with RG (with 16 rows per CTA and 8 tokens it is half the weight traffic).  UNROLL: k steps
// of 32 per batch of loads; `depth` batches (2, 3 or 6) are in flight.
template <int NT, int RG, int UNROLL, int EPI, bool NORM>
__global__ void __launch_bounds__(SK_THREADS, (NT * RG <= 2) ? 3 : 2)
gemm_skinny_kernel(const bf16* A, int lda, const bf16* __restrict__ W, int ldw, void* Cv, int ldc,
                   int M, int N, int K, int units_per_cta, int depth, SkinnyNorm nm) {
  // A unit is 16 * RG weight rows.  A CTA walks units_per_cta consecutive units, so that the grid is
  // no larger than what the GPU holds at once (no partly filled last wave) and every CTA streams
  // the same number of bytes.
  __shared__ float red[SK_WARPS][16 * RG][NT * 8 + 1];
  __shared__ float inv_rms[NORM ? SK_NORM_ROWS : 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int n_units = (N + 16 * RG - 1) / (16 * RG);
  int unit = blockIdx.x * units_per_cta;
  constexpr bool RING = SK_RING(NT);
  const int ksteps = (K + 31) >> 5, batches = ksteps > warp ? (ksteps - warp + SK_WARPS * UNROLL - 1) / (SK_WARPS * UNROLL) : 0;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  // The ring: `depth` batches of UNROLL steps, of every step 2 RG pieces of 16 bytes a lane.  The next batch to ask for is batch
  // ab of unit au; the sequence runs on over the units' ends, so the next unit's first batches are under way while this
  // one's sums are combined.  Pieces beyond K or N are zeros.
  extern __shared__ __align__(16) unsigned char sk_ring[];
  constexpr unsigned BATCH = UNROLL * RG * 2 * 512;
  const unsigned ring = (unsigned)__cvta_generic_to_shared(sk_ring) + warp * depth * BATCH + lane * 16;
  const int unit_end = min(unit + units_per_cta, n_units);
  int au = unit, ab = 0, aslot = 0;
  const bf16* w_at = W;
  unsigned w_ok = 0;                       // bit 2 rg + (0: row g, 1: row g + 8)
  auto ask_unit = [&]() {
    w_ok = 0;
    const int r0 = au * RG * 16 + g;
    w_at = W + (size_t)min(r0, N - 1) * ldw + 8 * t;
#pragma unroll
    for (int i = 0; i < 2 * RG; ++i) w_ok |= (r0 + 8 * i < N ? 1u : 0u) << i;
  };
  auto ask = [&]() {
    if (au < unit_end && batches > 0) {
      const int ks0 = warp + ab * SK_WARPS * UNROLL;
      const unsigned dst = ring + aslot * BATCH;
#pragma unroll
      for (int u = 0; u < UNROLL; ++u) {
        const int k = (ks0 + u * SK_WARPS) * 32;
        const bool ok = k + 8 * t < K;     // K is a multiple of 8: a lane's 8 elements are all inside or all outside
#pragma unroll
        for (int i = 0; i < 2 * RG; ++i) {
          const bool there = ok && ((w_ok >> i) & 1u);
          sk_copy16(dst + (u * 2 * RG + i) * 512, there ? w_at + (size_t)(8 * i) * ldw + k : W, there);
        }
      }
      if (++ab == batches) {
        ab = 0;
        ++au;
        ask_unit();
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (++aslot == depth) aslot = 0;
  };
  // Without a ring: a batch in registers and the next one on its way into others.
  uint4 wa[RING ? 1 : UNROLL][2 * RG], wb[RING ? 1 : UNROLL][2 * RG];
  auto fetch = [&](int b, uint4 (&d)[RING ? 1 : UNROLL][2 * RG]) {      // batch b of unit au
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      const int k = (warp + (b * UNROLL + u) * SK_WARPS) * 32;
#pragma unroll
      for (int i = 0; i < 2 * RG; ++i) d[RING ? 0 : u][i] = k + 8 * t < K && ((w_ok >> i) & 1u) ? ld_stream16(w_at + (size_t)(8 * i) * ldw + k) : zero;
    }
  };
  // Weights never depend on the previous kernel: the first batches are asked for before the wait on it.  With the ring the next kernel
  // may start as soon as that is done; it finds room on an SM when one of this kernel's CTAs has left (see `depth` below), so
  // its CTAs come to stand where there is one free place, not several on the SMs that are done first.
  ask_unit();
  if constexpr (RING) {
    for (int i = 0; i < depth; ++i) ask();
    pdl_launch();
  } else fetch(0, wa);
  pdl_wait();
  if (NORM) {
    // 1 / rms of the activation rows from the producer's partial sums: warp w sums rows w and w + 8
    // in a fixed order; the first __syncthreads() before an epilogue publishes them
    for (int m = warp; m < NT * 8; m += SK_WARPS) {
      float sum = 0.0f;
      if (nm.in_sumsq != nullptr && m < M)
        for (int i = lane; i < nm.in_parts; i += 32) sum += nm.in_sumsq[(size_t)i * SK_NORM_ROWS + m];
      sum = warp_sum(sum);
      if (lane == 0) inv_rms[m] = nm.in_sumsq != nullptr ? rsqrtf(sum / (float)K + nm.in_eps) : 1.0f;
    }
  }
  // Activations of a batch are asked for together (up to 16 rows), a batch ahead (up to 8).
  constexpr bool AHEAD = NT == 1, WHOLE = NT <= 2;
  uint4 xs[AHEAD ? 2 : 1][UNROLL][WHOLE ? NT : 1];
  auto load_x = [&](int b, int nt, uint4 (&d)[UNROLL][WHOLE ? NT : 1]) {
    const int m = nt * 8 + g;
    const bf16* row = A + (size_t)(m < M ? m : 0) * lda + 8 * t;
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      const int k = (warp + (b * UNROLL + u) * SK_WARPS) * 32;
      d[u][WHOLE ? nt : 0] = m < M && k + 8 * t < K ? *reinterpret_cast<const uint4*>(row + k) : zero;
    }
  };
  int slot = 0;
  for (; unit < unit_end; ++unit) {
    const int row0 = unit * 16 * RG;
    float acc[RG][NT][4];
#pragma unroll
    for (int rg = 0; rg < RG; ++rg)
#pragma unroll
      for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[rg][i][j] = 0.0f;

    auto batch = [&](int b, uint4 (&x)[UNROLL][WHOLE ? NT : 1], uint4 (&xn)[UNROLL][WHOLE ? NT : 1]) {
      if constexpr (WHOLE) {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) load_x(AHEAD ? b + 1 : b, nt, AHEAD ? xn : x);
      }
      if (depth == 2) asm volatile("cp.async.wait_group 1;" ::: "memory");
      else if (depth == 3) asm volatile("cp.async.wait_group 2;" ::: "memory");
      else asm volatile("cp.async.wait_group 5;" ::: "memory");
      const unsigned src = ring + slot * BATCH;
      uint4 w[WHOLE ? 1 : UNROLL][2 * RG];
      if constexpr (WHOLE) {
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
#pragma unroll
          for (int i = 0; i < 2 * RG; ++i) w[0][i] = sk_read16(src + (u * 2 * RG + i) * 512);
#pragma unroll
          for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int rg = 0; rg < RG; ++rg) {
              const uint4 lo = w[0][2 * rg], hi = w[0][2 * rg + 1], v = x[u][nt];
              mma_bf16_16816(acc[rg][nt], lo.x, hi.x, lo.y, hi.y, v.x, v.y);
              mma_bf16_16816(acc[rg][nt], lo.z, hi.z, lo.w, hi.w, v.z, v.w);
            }
        }
      } else {
#pragma unroll
        for (int u = 0; u < UNROLL; ++u)
#pragma unroll
          for (int i = 0; i < 2 * RG; ++i) w[u][i] = sk_read16(src + (u * 2 * RG + i) * 512);
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          load_x(b, nt, x);
#pragma unroll
          for (int u = 0; u < UNROLL; ++u)
#pragma unroll
            for (int rg = 0; rg < RG; ++rg) {
              const uint4 lo = w[u][2 * rg], hi = w[u][2 * rg + 1], v = x[u][0];
              mma_bf16_16816(acc[rg][nt], lo.x, hi.x, lo.y, hi.y, v.x, v.y);
              mma_bf16_16816(acc[rg][nt], lo.z, hi.z, lo.w, hi.w, v.z, v.w);
            }
        }
      }
      ask();                               // into the slot just read: behind the instructions that took its values
      if (++slot == depth) slot = 0;
    };
    if constexpr (!RING) {
      for (int b = 0; b < batches; ++b) {
        fetch(b + 1, wb);
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
          const int k = (warp + (b * UNROLL + u) * SK_WARPS) * 32 + 8 * t;
#pragma unroll
          for (int n0 = 0; n0 < NT; n0 += 4) {             // four groups of rows are asked for together
            uint4 x[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const int m = (n0 + j) * 8 + g;
              x[j] = m < M && k < K ? *reinterpret_cast<const uint4*>(A + (size_t)m * lda + k) : zero;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
              for (int rg = 0; rg < RG; ++rg) {
                const uint4 lo = wa[RING ? 0 : u][2 * rg], hi = wa[RING ? 0 : u][2 * rg + 1];
                mma_bf16_16816(acc[rg][n0 + j], lo.x, hi.x, lo.y, hi.y, x[j].x, x[j].y);
                mma_bf16_16816(acc[rg][n0 + j], lo.z, hi.z, lo.w, hi.w, x[j].z, x[j].w);
              }
          }
        }
#pragma unroll
        for (int u = 0; u < UNROLL; ++u)
#pragma unroll
          for (int i = 0; i < 2 * RG; ++i) wa[RING ? 0 : u][i] = wb[RING ? 0 : u][i];
      }
      if (unit + 1 < unit_end) {           // the next unit's first batch, under this unit's sums
        ++au;
        ask_unit();
        fetch(0, wa);
      } else pdl_launch();
    } else if constexpr (AHEAD) {
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) load_x(0, nt, xs[0]);
      for (int b = 0; b < batches; b += 2) {
        batch(b, xs[0], xs[1]);
        if (b + 1 < batches) batch(b + 1, xs[1], xs[0]);
      }
    } else {
      for (int b = 0; b < batches; ++b) batch(b, xs[0], xs[0]);
    }
    // accumulator layout: acc[..][nt][0..1] = (weight row g, tokens nt*8 + 2t, 2t+1); [2..3] = row g+8
#pragma unroll
    for (int rg = 0; rg < RG; ++rg)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        red[warp][rg * 16 + g][nt * 8 + 2 * t] = acc[rg][nt][0];
        red[warp][rg * 16 + g][nt * 8 + 2 * t + 1] = acc[rg][nt][1];
        red[warp][rg * 16 + g + 8][nt * 8 + 2 * t] = acc[rg][nt][2];
        red[warp][rg * 16 + g + 8][nt * 8 + 2 * t + 1] = acc[rg][nt][3];
      }
    __syncthreads();
    if (EPI == HB_EPI_SWIGLU) {
      // per group of 16 rows: 8 channels x (NT*8) tokens; output column = (row group) * 8 + channel
      for (int idx = threadIdx.x; idx < RG * 8 * NT * 8; idx += SK_THREADS) {
        const int ch = idx & 7, rg = (idx >> 3) % RG, m = idx / (8 * RG);
        if (m >= M) continue;
        float gate = 0.0f, up = 0.0f;
#pragma unroll
        for (int w = 0; w < SK_WARPS; ++w) {
          gate += red[w][rg * 16 + ch][m];
          up += red[w][rg * 16 + ch + 8][m];
        }
        if (NORM) {
          gate *= inv_rms[m];
          up *= inv_rms[m];
        }
        const int col = (unit * RG + rg) * 8 + ch;
        float slope = 1.0f;
        if (nm.glu_limit > 0.0f) {
          gate = fminf(gate, nm.glu_limit);
          up = fminf(fmaxf(up, -nm.glu_limit), nm.glu_limit) + 1.0f;
          slope = HB_SWISH_CLAMP_SLOPE;
        }
        if (row0 + rg * 16 + ch + 8 < N) ((bf16*)Cv)[(size_t)m * ldc + col] = __float2bfloat16_rn((gate / (1.0f + expf(-slope * gate))) * up);
      }
    } else {
      // 16 * RG * NT * 8 is a multiple of 128: whole warps enter an iteration, and the 16 * RG
      // consecutive lanes that share a token row can sum over their columns with shuffles
      for (int idx = threadIdx.x; idx < 16 * RG * NT * 8; idx += SK_THREADS) {
        const int r = idx % (16 * RG), m = idx / (16 * RG);
        const int n = row0 + r;
        const bool ok = m < M && n < N;
        float s = 0.0f;
#pragma unroll
        for (int w = 0; w < SK_WARPS; ++w) s += red[w][r][m];
        if (NORM) s *= inv_rms[m];
        const size_t o = (size_t)m * ldc + n;
        float sq = 0.0f;
        if (ok) {
          if (EPI == HB_EPI_STORE) ((bf16*)Cv)[o] = __float2bfloat16_rn(s);
          else if (EPI == HB_EPI_STORE_F32) ((float*)Cv)[o] = s;
          else {
            const float v = ((float*)Cv)[o] + s;
            ((float*)Cv)[o] = v;
            if (NORM && nm.out_w != nullptr) {
              nm.out_xw[(size_t)m * nm.out_ld + n] = __float2bfloat16_rn(v * nm.out_w[n]);
              sq = v * v;
            }
          }
        }
        if (NORM && EPI == HB_EPI_RESIDUAL && nm.out_w != nullptr) {
#pragma unroll
          for (int d = 1; d < 16 * RG; d <<= 1) sq += __shfl_xor_sync(0xffffffffu, sq, d);
          if (r == 0 && m < SK_NORM_ROWS) nm.out_sumsq[(size_t)unit * SK_NORM_ROWS + m] = sq;
        }
      }
    }
    __syncthreads();   // the partial sums are read: the next unit may overwrite them
  }
}

template <int NT, int RG, int UNROLL, bool NORM = false>
static int skinny_launch(const bf16* A, int lda, const bf16* W, int ldw, void* C, int ldc, int M, int N, int K,
                         int epi, cudaStream_t s, SkinnyNorm nm = SkinnyNorm{}) {
  // as many CTAs as the GPU holds at once, each with an equal run of units
  constexpr int PER_SM = NT * RG <= 2 ? 3 : 2, BATCH = SK_WARPS * UNROLL * RG * 1024;
  static HbPerDevice kept;
  int dev = 0;
  cudaGetDevice(&dev);
  const int sms = hb_per_device(kept, dev, [&]() {
    const void* kernels[4] = {(const void*)gemm_skinny_kernel<NT, RG, UNROLL, HB_EPI_STORE, NORM>, (const void*)gemm_skinny_kernel<NT, RG, UNROLL, HB_EPI_STORE_F32, NORM>,
                              (const void*)gemm_skinny_kernel<NT, RG, UNROLL, HB_EPI_RESIDUAL, NORM>, (const void*)gemm_skinny_kernel<NT, RG, UNROLL, HB_EPI_SWIGLU, NORM>};
    for (const void* k : kernels) {
      const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 6 * BATCH);
      if (e != cudaSuccess) {
        hb_set_error("gemm_skinny: cannot reserve %d bytes of shared memory: %s", 6 * BATCH, cudaGetErrorString(e));
        return -1;
      }
    }
    int n = 0;
    return cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && n > 0 ? n : 148;
  });
  if (sms < 0) return 3;
  const int n_units = ceil_div(N, 16 * RG), slots = PER_SM * sms;
  // fewer than one and a half waves: one unit per CTA keeps more loads in flight than halving the grid
  const int upc = (2 * n_units > 3 * slots) ? ceil_div(n_units, slots) : 1;
  const unsigned grid = (unsigned)ceil_div(n_units, upc);
  // What an SM's CTAs have under way together fills its shared memory.  (Three batches where the grid gives an SM one CTA, so that the
  // next product's first batches fit beside them: 0.6B-sized steps 1,551 instead of 1,505 us, the 2,048-wide designs 1 to 2 % slower.)
  const int depth = !SK_RING(NT) ? 0 : (int)grid <= sms ? 6 : (int)grid <= 2 * sms && NT * RG <= 2 ? 3 : 2;
  const size_t smem = (size_t)depth * BATCH;
  switch (epi) {
    case HB_EPI_STORE: hb_launch_pdl(gemm_skinny_kernel<NT, RG, UNROLL, HB_EPI_STORE, NORM>, dim3(grid), dim3(SK_THREADS), smem, s, A, lda, W, ldw, C, ldc, M, N, K, upc, depth, nm); break;
    case HB_EPI_STORE_F32: hb_launch_pdl(gemm_skinny_kernel<NT, RG, UNROLL, HB_EPI_STORE_F32, NORM>, dim3(grid), dim3(SK_THREADS), smem, s, A, lda, W, ldw, C, ldc, M, N, K, upc, depth, nm); break;
    case HB_EPI_RESIDUAL: hb_launch_pdl(gemm_skinny_kernel<NT, RG, UNROLL, HB_EPI_RESIDUAL, NORM>, dim3(grid), dim3(SK_THREADS), smem, s, A, lda, W, ldw, C, ldc, M, N, K, upc, depth, nm); break;
    case HB_EPI_SWIGLU: hb_launch_pdl(gemm_skinny_kernel<NT, RG, UNROLL, HB_EPI_SWIGLU, NORM>, dim3(grid), dim3(SK_THREADS), smem, s, A, lda, W, ldw, C, ldc, M, N, K, upc, depth, nm); break;
    default: HB_FAIL(2, "gemm_skinny: unknown epilogue %d", epi);
  }
  HB_CHECK_LAUNCH("gemm_skinny");
  return 0;
}

// epi HB_EPI_SWIGLU: W holds 2I rows in groups of 16 (8 gate, 8 up); C is [M, I] bfloat16.
// Two row groups per CTA halve the activation traffic and double the loads a CTA has in flight;
// worth it where there are enough rows that the grid still fills the GPU (gate/up at one row:
// 38.7 -> 34.3 us).
static bool skinny_two_groups(int M, int N) { return M <= 16 && N >= 8192; }

extern "C" int hb_gemm_skinny_bf16(const void* A, int lda, const void* W, int ldw, void* C, int ldc, int M, int N,
                                   int K, int epi, float glu_limit, void* stream) {
  HB_REQUIRE(M > 0 && N > 0 && K > 0, "gemm_skinny: sizes must be positive");
  HB_REQUIRE(M <= 64, "gemm_skinny: at most 64 activation rows, got %d", M);
  HB_REQUIRE(K % 8 == 0 && lda % 8 == 0 && ldw % 8 == 0, "gemm_skinny: K (%d) and the leading dimensions (%d, %d) must be multiples of 8", K, lda, ldw);
  HB_REQUIRE(((uintptr_t)A & 15) == 0 && ((uintptr_t)W & 15) == 0, "gemm_skinny: operands must be 16-byte aligned");
  HB_REQUIRE(epi != HB_EPI_SWIGLU || N % 16 == 0, "gemm_skinny: SwiGLU rows come in groups of 16, N=%d", N);
  cudaStream_t s = (cudaStream_t)stream;
  const bf16* a = (const bf16*)A;
  const bf16* w = (const bf16*)W;
  const bool two = skinny_two_groups(M, N);
  SkinnyNorm nm{};
  nm.glu_limit = epi == HB_EPI_SWIGLU ? glu_limit : 0.0f;
  if (M <= 8) return two ? skinny_launch<1, 2, 2>(a, lda, w, ldw, C, ldc, M, N, K, epi, s, nm)
                         : skinny_launch<1, 1, 4>(a, lda, w, ldw, C, ldc, M, N, K, epi, s, nm);
  if (M <= 16) return two ? skinny_launch<2, 2, 2>(a, lda, w, ldw, C, ldc, M, N, K, epi, s, nm)
                          : skinny_launch<2, 1, 4>(a, lda, w, ldw, C, ldc, M, N, K, epi, s, nm);
  if (M <= 32) return skinny_launch<4, 1, 2>(a, lda, w, ldw, C, ldc, M, N, K, epi, s, nm);
  return skinny_launch<8, 1, 2>(a, lda, w, ldw, C, ldc, M, N, K, epi, s, nm);
}

// How many groups of output columns the product of an [M, K] activation with an [N, K] matrix
// writes partial sums for (the first dimension of out_sumsq).
extern "C" int hb_gemm_skinny_norm_parts(int M, int N) {
  return ceil_div(N, skinny_two_groups(M, N) ? 32 : 16);
}

// The same product with a shared norm on either side (M <= 16):
//   in_sumsq != null: A holds x * w of a norm over K; results are multiplied by 1 / rms of the rows,
//     rms^2 = sum over in_parts partial sums / K + in_eps;
//   out_w != null (epi HB_EPI_RESIDUAL): besides C += ..., out_xw = C * out_w (bfloat16) and
//     out_sumsq[hb_gemm_skinny_norm_parts(M, N)][16] = partial sums of C^2.
extern "C" int hb_gemm_skinny_norm_bf16(const void* A, int lda, const void* W, int ldw, void* C, int ldc, int M,
                                        int N, int K, int epi, const float* in_sumsq, int in_parts, float in_eps,
                                        const float* out_w, void* out_xw, int out_ld, float* out_sumsq,
                                        void* stream) {
  HB_REQUIRE(M > 0 && N > 0 && K > 0, "gemm_skinny_norm: sizes must be positive");
  HB_REQUIRE(M <= SK_NORM_ROWS, "gemm_skinny_norm: at most %d activation rows, got %d", SK_NORM_ROWS, M);
  HB_REQUIRE(K % 8 == 0 && lda % 8 == 0 && ldw % 8 == 0, "gemm_skinny_norm: K (%d) and the leading dimensions (%d, %d) must be multiples of 8", K, lda, ldw);
  HB_REQUIRE(((uintptr_t)A & 15) == 0 && ((uintptr_t)W & 15) == 0, "gemm_skinny_norm: operands must be 16-byte aligned");
  HB_REQUIRE(epi != HB_EPI_SWIGLU || N % 16 == 0, "gemm_skinny_norm: SwiGLU rows come in groups of 16, N=%d", N);
  HB_REQUIRE(in_sumsq == nullptr || in_parts > 0, "gemm_skinny_norm: partial sums without a count");
  HB_REQUIRE(out_w == nullptr || (epi == HB_EPI_RESIDUAL && out_xw != nullptr && out_sumsq != nullptr),
             "gemm_skinny_norm: the next norm's input is written by the residual epilogue and needs both outputs");
  SkinnyNorm nm{in_sumsq, in_parts, in_eps, out_w, (bf16*)out_xw, out_ld, out_sumsq};
  cudaStream_t s = (cudaStream_t)stream;
  const bf16* a = (const bf16*)A;
  const bf16* w = (const bf16*)W;
  const bool two = skinny_two_groups(M, N);
  if (M <= 8) return two ? skinny_launch<1, 2, 2, true>(a, lda, w, ldw, C, ldc, M, N, K, epi, s, nm)
                         : skinny_launch<1, 1, 4, true>(a, lda, w, ldw, C, ldc, M, N, K, epi, s, nm);
  return two ? skinny_launch<2, 2, 2, true>(a, lda, w, ldw, C, ldc, M, N, K, epi, s, nm)
             : skinny_launch<2, 1, 4, true>(a, lda, w, ldw, C, ldc, M, N, K, epi, s, nm);
}
