// The routed feed-forward of steps with few tokens (decode batches), bfloat16: every chosen expert's matrices are read
// once, however many of the step's tokens chose it.
//
//   mid[u] = act(Up_e h[t])   (gated: act(Gate_e h[t]) * (Up_e h[t])),   u = t * top + r, e = ids[u]
//   y[t] (+)= sum_r weights[u] * Down_e mid[u]
//
// Bound by the stream of the chosen experts' weights.  A warp per output number, as before, read every weight row once
// per token that chose its expert and kept two loads of a lane under way.  Here 16 weight rows are the M operand of
// mma.sync (as in gemm_skinny.cu: 16-byte streaming loads, two batches ahead, k permuted inside the instruction) and the
// tokens that chose the expert its columns.  The choice lies in device memory, so every CTA first sorts the pairs by expert for itself.
//   first product    the rows of all chosen experts, 16 at a time, are one list that persistent CTAs share evenly; the eight
//                    warps of a CTA share K
//   second product   a cluster of S CTAs owns 16 rows of every expert; its warps share the (expert, K) ranges evenly, multiply
//                    what they summed by the pairs' weights when the expert changes, and the parts are added in order
// Measured on a B200 (first + second product, inside a step, 4 of 32 experts of 1,408 over 2,048): 8 tokens 49 + 35 -> 41 + 31 us, 16
// tokens 91 + 59 -> 58 + 40 us (5.5 TB/s in the first product).
#include <cooperative_groups.h>

#include "api.h"
#include "common.cuh"
#include "mma_utils.cuh"
#include "moe_act.cuh"

namespace cg = cooperative_groups;

#define FW_WARPS 8
#define FW_THREADS (FW_WARPS * 32)
#define FW_UNROLL 4
#define FW_MAX_TOKENS 32
#define FW_MAX_PAIRS 512
#define FW_MAX_EXPERTS 1024

__device__ __forceinline__ uint4 fw_stream16(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

// The chosen experts in order of their index, and their pairs.  An entry has at most `cap` pairs: an expert that a
// token names twice may need two entries (a router's choices are distinct, so from it every expert has one).
struct FwSorted {
  int n;                                 // entries
  int expert[FW_MAX_PAIRS];
  int first[FW_MAX_PAIRS + 1];           // pairs first[i] .. first[i + 1] - 1 of `pair` chose expert[i]
  int pair[FW_MAX_PAIRS];
};

// Every thread of the CTA; cnt: n_experts ints of shared memory.  An index outside the experts is left out.
__device__ __forceinline__ void fw_sort(FwSorted& o, int* cnt, const int* ids, int n_pairs, int E, int cap) {
  const int tid = threadIdx.x, lane = tid & 31;
  for (int e = tid; e < E; e += FW_THREADS) cnt[e] = 0;
  __syncthreads();
  for (int u = tid; u < n_pairs; u += FW_THREADS)
    if ((unsigned)ids[u] < (unsigned)E) atomicAdd(&cnt[ids[u]], 1);
  __syncthreads();
  if (tid < 32) {
    int n = 0, at = 0;
    for (int e0 = 0; e0 < E; e0 += 32) {
      const int e = e0 + lane, c = e < E ? cnt[e] : 0, m = (c + cap - 1) / cap;
      int incl = c, mi = m;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, d), w = __shfl_up_sync(0xffffffffu, mi, d);
        if (lane >= d) { incl += v; mi += w; }
      }
      for (int j = 0; j < m; ++j) {
        o.expert[n + mi - m + j] = e;
        o.first[n + mi - m + j] = at + incl - c + j * cap;
      }
      if (e < E) cnt[e] = at + incl - c;       // where the expert's next pair goes
      n += __shfl_sync(0xffffffffu, mi, 31);
      at += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) { o.n = n; o.first[n] = at; }
  }
  __syncthreads();
  for (int u = tid; u < n_pairs; u += FW_THREADS)
    if ((unsigned)ids[u] < (unsigned)E) o.pair[atomicAdd(&cnt[ids[u]], 1)] = u;
  __syncthreads();
}

// NT: groups of 8 tokens (no expert has more than NT * 8 pairs).  GLU: the 16 rows are 8 gate rows and the up rows of the
// same channels.
template <int NT, bool GLU>
__global__ void __launch_bounds__(FW_THREADS, 2)
moe_few_up_kernel(const bf16* h, int ld, const bf16* __restrict__ up, const int* ids, const float* in_w,
                  bf16* __restrict__ mid, int n_pairs, int top, int E, int D, int F, int act, float limit) {
  extern __shared__ int cnt[];
  __shared__ FwSorted so;
  __shared__ float red[FW_WARPS][16][NT * 8 + 1];
  pdl_wait();
  pdl_launch();
  fw_sort(so, cnt, ids, n_pairs, E, NT * 8);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int N = GLU ? 2 * F : F, per = (N + 15) >> 4;                     // units of 16 rows of an expert
  const int total = so.n * per;
  int unit = (int)((long long)total * blockIdx.x / gridDim.x);
  const int end = (int)((long long)total * (blockIdx.x + 1) / gridDim.x);
  if (unit >= end) return;
  const int ksteps = (D + 31) >> 5;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  uint4 wa[FW_UNROLL], wb[FW_UNROLL], na[FW_UNROLL], nb[FW_UNROLL];
  const bf16 *w_lo, *w_hi;
  bool lo_ok, hi_ok;
  auto set_unit = [&](int u) {
    const int x = u / per, r_lo = (u - x * per) * 16 + g, r_hi = r_lo + 8;
    lo_ok = r_lo < N;
    hi_ok = r_hi < N;
    const bf16* base = up + (size_t)so.expert[x] * N * D;
    w_lo = base + (size_t)(lo_ok ? r_lo : 0) * D;
    w_hi = base + (size_t)(hi_ok ? r_hi : 0) * D;
  };
  auto load = [&](int ks0, uint4* ra, uint4* rb) {
#pragma unroll
    for (int u = 0; u < FW_UNROLL; ++u) {
      const int k = (ks0 + u * FW_WARPS) * 32 + 8 * t;
      const bool ok = k < D;                                             // D is a multiple of 8
      ra[u] = ok && lo_ok ? fw_stream16(w_lo + k) : zero;
      rb[u] = ok && hi_ok ? fw_stream16(w_hi + k) : zero;
    }
  };
  int x = -1, pairs = 0, p0 = 0;
  const bf16* hr[NT];
  set_unit(unit);
  load(warp, wa, wb);
  for (; unit < end; ++unit) {
    const int xu = unit / per;
    if (xu != x) {                                                       // another expert: its pairs are the columns
      x = xu;
      p0 = so.first[x];
      pairs = so.first[x + 1] - p0;
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) hr[nt] = nt * 8 + g < pairs ? h + (size_t)(so.pair[p0 + nt * 8 + g] / top) * ld : nullptr;
    }
    float acc[NT][4];
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
    for (int ks0 = warp; ks0 < ksteps; ks0 += FW_WARPS * FW_UNROLL) {
      load(ks0 + FW_WARPS * FW_UNROLL, na, nb);
      auto multiply = [&](int nt) {
        uint4 v[FW_UNROLL];                                              // asked for together: one way to L1 or L2 per batch
#pragma unroll
        for (int u = 0; u < FW_UNROLL; ++u) {
          const int k = (ks0 + u * FW_WARPS) * 32 + 8 * t;
          v[u] = k < D && hr[nt] != nullptr ? *reinterpret_cast<const uint4*>(hr[nt] + k) : zero;
        }
#pragma unroll
        for (int u = 0; u < FW_UNROLL; ++u) {
          mma16816(acc[nt], wa[u].x, wb[u].x, wa[u].y, wb[u].y, v[u].x, v[u].y);
          mma16816(acc[nt], wa[u].z, wb[u].z, wa[u].w, wb[u].w, v[u].z, v[u].w);
        }
      };
      multiply(0);
#pragma unroll
      for (int nt = 1; nt < NT; ++nt)
        if (nt * 8 < pairs) multiply(nt);
#pragma unroll
      for (int u = 0; u < FW_UNROLL; ++u) { wa[u] = na[u]; wb[u] = nb[u]; }
    }
    if (unit + 1 < end) {                                                // the next unit's first batch, under this unit's sums
      set_unit(unit + 1);
      load(warp, wa, wb);
    }
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      red[warp][g][nt * 8 + 2 * t] = acc[nt][0];
      red[warp][g][nt * 8 + 2 * t + 1] = acc[nt][1];
      red[warp][g + 8][nt * 8 + 2 * t] = acc[nt][2];
      red[warp][g + 8][nt * 8 + 2 * t + 1] = acc[nt][3];
    }
    __syncthreads();
    const int row0 = (unit - x * per) * 16;
    for (int i = tid; i < (GLU ? 8 : 16) * pairs; i += FW_THREADS) {
      const int r = GLU ? i & 7 : i & 15, c = GLU ? i >> 3 : i >> 4, u = so.pair[p0 + c];
      if (row0 + r >= N) continue;
      float a = 0.0f, b = 0.0f;
#pragma unroll
      for (int w = 0; w < FW_WARPS; ++w) {
        a += red[w][r][c];
        if (GLU) b += red[w][r + 8][c];
      }
      if (GLU && in_w) { a *= in_w[u]; b *= in_w[u]; }
      mid[(size_t)u * F + (GLU ? (row0 >> 1) + r : row0 + r)] = __float2bfloat16_rn(GLU ? moe_glu(a, b, act, limit) : moe_act(a, act));
    }
    __syncthreads();                                                     // the sums are read: the next unit may overwrite them
  }
}

template <int NT>
__global__ void __launch_bounds__(FW_THREADS, 2)
moe_few_down_kernel(const bf16* mid, const bf16* __restrict__ down, const int* ids, const float* wts,
                    float* y, int ldy, int n_tokens, int top, int E, int D, int F, int accumulate) {
  extern __shared__ int cnt[];
  __shared__ FwSorted so;
  __shared__ float ys[FW_WARPS][16][NT * 8 + 1];                          // a warp's sums per row and token
  __shared__ float mine[16][NT * 8];
  pdl_wait();
  pdl_launch();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  for (int i = lane; i < 16 * (NT * 8 + 1); i += 32) (&ys[warp][0][0])[i] = 0.0f;
  fw_sort(so, cnt, ids, n_tokens * top, E, NT * 8);
  const int S = gridDim.x, part = blockIdx.x, row0 = blockIdx.y * 16;
  const int ksteps = (F + 31) >> 5, total = so.n * ksteps, share = S * FW_WARPS, me = part * FW_WARPS + warp;
  const int q0 = (int)((long long)total * me / share), q1 = (int)((long long)total * (me + 1) / share);
  const bool lo_ok = row0 + g < D, hi_ok = row0 + g + 8 < D;
  const size_t o_lo = (size_t)(lo_ok ? row0 + g : 0) * F + 8 * t, o_hi = (size_t)(hi_ok ? row0 + g + 8 : 0) * F + 8 * t;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  uint4 wa[FW_UNROLL], wb[FW_UNROLL], na[FW_UNROLL], nb[FW_UNROLL];
  // A batch is at most FW_UNROLL steps of one expert; loads and products walk the same batches, the loads one ahead.
  int lx = q0 / ksteps, lk = q0 - lx * ksteps, lq = q0;                   // where the loads are
  auto load = [&](uint4* ra, uint4* rb) {
    int n = min(FW_UNROLL, min(ksteps - lk, q1 - lq));
    const bf16* base = down + (n > 0 ? (size_t)so.expert[lx] * D * F + lk * 32 : 0);
#pragma unroll
    for (int u = 0; u < FW_UNROLL; ++u) {
      const bool ok = u < n && (lk + u) * 32 + 8 * t < F;                 // F is a multiple of 8
      ra[u] = ok && lo_ok ? fw_stream16(base + o_lo + u * 32) : zero;
      rb[u] = ok && hi_ok ? fw_stream16(base + o_hi + u * 32) : zero;
    }
    lq += n;
    lk += n;
    if (lk == ksteps) { lk = 0; ++lx; }
  };
  float acc[NT][4];
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
  int x = q0 / ksteps, k0 = q0 - x * ksteps, p0 = 0, pairs = 0;
  const bf16* mr[NT];
  auto open = [&]() {
    p0 = so.first[x];
    pairs = so.first[x + 1] - p0;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) mr[nt] = nt * 8 + g < pairs ? mid + (size_t)so.pair[p0 + nt * 8 + g] * F + 8 * t : nullptr;
  };
  auto fold = [&]() {                                                     // this expert's sums, weighted, to their tokens
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int col = nt * 8 + 2 * t + c;
        if (col < pairs) {
          const int u = so.pair[p0 + col], tok = u / top;
          const float w = wts ? wts[u] : 1.0f;
          atomicAdd(&ys[warp][g][tok], w * acc[nt][c]);                   // atomic for a token that names the expert twice
          atomicAdd(&ys[warp][g + 8][tok], w * acc[nt][2 + c]);
        }
        acc[nt][c] = 0.0f;
        acc[nt][2 + c] = 0.0f;
      }
  };
  if (q0 < q1) {
    open();
    load(wa, wb);
    for (int q = q0; q < q1;) {
      load(na, nb);
      const int n = min(FW_UNROLL, min(ksteps - k0, q1 - q));
      auto multiply = [&](int nt) {
        uint4 v[FW_UNROLL];                                               // asked for together: one way to L2 per batch
#pragma unroll
        for (int u = 0; u < FW_UNROLL; ++u) {
          const int k = (k0 + u) * 32;
          v[u] = u < n && k + 8 * t < F && mr[nt] != nullptr ? *reinterpret_cast<const uint4*>(mr[nt] + k) : zero;
        }
#pragma unroll
        for (int u = 0; u < FW_UNROLL; ++u) {
          mma16816(acc[nt], wa[u].x, wb[u].x, wa[u].y, wb[u].y, v[u].x, v[u].y);
          mma16816(acc[nt], wa[u].z, wb[u].z, wa[u].w, wb[u].w, v[u].z, v[u].w);
        }
      };
      multiply(0);
#pragma unroll
      for (int nt = 1; nt < NT; ++nt)
        if (nt * 8 < pairs) multiply(nt);
      q += n;
      k0 += n;
      if (k0 == ksteps) {
        k0 = 0;
        fold();
        ++x;
        if (q < q1) open();
      }
#pragma unroll
      for (int u = 0; u < FW_UNROLL; ++u) { wa[u] = na[u]; wb[u] = nb[u]; }
    }
    if (k0 != 0) fold();
  }
  __syncthreads();
  for (int i = tid; i < 16 * n_tokens; i += FW_THREADS) {
    const int r = i & 15, tok = i >> 4;
    float s = ys[0][r][tok];
#pragma unroll
    for (int w = 1; w < FW_WARPS; ++w) s += ys[w][r][tok];
    mine[r][tok] = s;
  }
  cg::cluster_group cluster = cg::this_cluster();
  if (S > 1) cluster.sync(); else __syncthreads();
  if (part == 0)
    for (int i = tid; i < 16 * n_tokens; i += FW_THREADS) {
      const int r = i & 15, tok = i >> 4;
      if (row0 + r >= D) continue;
      float s = mine[r][tok];
      for (int p = 1; p < S; ++p) s += *cluster.map_shared_rank(&mine[r][tok], p);
      float* o = y + (size_t)tok * ldy + row0 + r;
      *o = accumulate ? *o + s : s;
    }
  if (S > 1) cluster.sync();                                              // nobody leaves while its part is still read
}

// Whether a step takes these kernels: few tokens, every row of the operands on 16 bytes, a gated expert's gate and up rows in
// groups of 8.
extern "C" int hb_moe_experts_few_ok(const void* h, int ld, const void* up, const void* down, const void* mid, int n_tokens, int top,
                                     int E, int D, int F, int gated) {
  return n_tokens > 0 && top > 0 && n_tokens <= FW_MAX_TOKENS && (long long)n_tokens * top <= FW_MAX_PAIRS && E > 0 && E <= FW_MAX_EXPERTS &&
         (gated == 0 || gated == 2) && D > 0 && F > 0 && D % 8 == 0 && F % 8 == 0 && ld % 8 == 0 && ceil_div(D, 16) <= 65535 &&
         (((uintptr_t)h | (uintptr_t)up | (uintptr_t)down | (uintptr_t)mid) & 15) == 0;
}

template <int NT>
static int few_launch(const bf16* h, int ld, const bf16* up, const bf16* down, const int* ids, const float* in_w, const float* out_w, bf16* mid,
                      float* y, int ldy, int n_tokens, int D, int E, int F, int top, int act, int gated, float limit, int accumulate, cudaStream_t s) {
  int sms = 0, dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int n_pairs = n_tokens * top;
  const size_t smem = (size_t)E * sizeof(int);
  // two CTAs an SM, fewer where there are not that many units
  const long long units = (long long)(n_pairs < E ? n_pairs : E) * ceil_div(gated ? 2 * F : F, 16);
  const unsigned grid = (unsigned)(units < 2LL * sms ? units : 2LL * sms);
  if (gated) hb_launch(moe_few_up_kernel<NT, true>, dim3(grid), dim3(FW_THREADS), smem, s, h, ld, up, ids, in_w, mid, n_pairs, top, E, D, F, act, limit);
  else hb_launch(moe_few_up_kernel<NT, false>, dim3(grid), dim3(FW_THREADS), smem, s, h, ld, up, ids, in_w, mid, n_pairs, top, E, D, F, act, limit);
  const int tiles = ceil_div(D, 16);
  int S = 1;
  while (S < 8 && tiles * S * 3 < 4 * sms) S <<= 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(S, tiles);
  cfg.blockDim = dim3(FW_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = S;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = hb_pdl_enabled() == 1 ? 2 : 1;
  cudaLaunchKernelEx(&cfg, moe_few_down_kernel<NT>, (const bf16*)mid, down, ids, out_w, y, ldy, n_tokens, top, E, D, F, accumulate);
  return 0;
}

extern "C" int hb_moe_experts_few_bf16(const void* h, int ld, const void* up, const void* down, const int* ids,
                                       const float* weights, void* mid, float* y, int ldy, int n_tokens, int D, int E, int F, int top,
                                       int act, int gated, float act_limit, int weigh_input, int accumulate, void* stream) {
  HB_REQUIRE(hb_moe_experts_few_ok(h, ld, up, down, mid, n_tokens, top, E, D, F, gated),
             "moe_experts_few: at most %d tokens and %d pairs, widths in multiples of 8, 16-byte aligned rows", FW_MAX_TOKENS, FW_MAX_PAIRS);
  HB_REQUIRE(!weigh_input || gated, "moe_experts_few: the weight multiplies the input of gated experts only");
  HB_REQUIRE(act != HB_ACT_SWISH_CLAMP || gated, "moe_experts_few: the clamped activation is a gated expert's");
  const float* in_w = weigh_input ? weights : nullptr;
  const float* out_w = weigh_input ? nullptr : weights;
#define FW_GO(NT) few_launch<NT>((const bf16*)h, ld, (const bf16*)up, (const bf16*)down, ids, in_w, out_w, (bf16*)mid, y, ldy, n_tokens, D, E, F, top, act, gated, act_limit, accumulate, (cudaStream_t)stream)
  if (n_tokens <= 8) FW_GO(1);
  else if (n_tokens <= 16) FW_GO(2);
  else FW_GO(4);
#undef FW_GO
  HB_CHECK_LAUNCH("moe_experts_few");
  return 0;
}
