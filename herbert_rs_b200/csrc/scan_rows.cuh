// The recurrences over a matrix of state per head, token by token, with a register tile per thread: what the four
// mixers' scans (linear_scan.cu, general_delta.cu, gla.cu) share.  Per head, S [dk][dv] in float:
//
//   SCAN_GLA      S <- diag(a) S + k v^T;                          o = scale * S^T q     vectors q, k, a
//   SCAN_DECAY    S <- d S + k v^T;                                o = S^T q             vectors q, k; d per head
//   SCAN_DELTA    S <- g S; u = beta (v - S^T k); S <- S + k u^T;   o = S^T q             vectors q, k; g, beta per token and head
//   SCAN_GENERAL  S <- diag(w) S - p (u^T S) + k v^T;               o = S^T r             vectors r, k, w, u, p (both terms read the old S)
//
// A thread holds 8 rows x CPT columns of the state; the dk = 8 R rows of a column lie in R neighbouring lanes.  A float4 of a
// key-side vector that it loads from shared memory then serves 4 CPT entries: with one column a thread, as the other kernels
// of these files have it, the loads from shared memory (128 bytes a cycle and SM into registers, however many lanes read the same
// ones) take longer than the multiply-adds.  The sums over the key channels that the next token waits for end with log2 R
// exchanges; a token's other vectors are asked for before them and the next token's first one under its update.  Rows go two at a
// time through packed multiply-adds (each half rounds as fmaf does).  The read-outs belong to no chain: every lane leaves
// its part of them in shared memory, and a chunk's are added afterwards.  The vectors of CH tokens are copied ahead
// asynchronously by address arithmetic alone.  The CTAs of a sequence are neighbours in the grid, so that an SM's second CTA
// comes from another sequence; the kernel starts after the one before it has ended, since CTAs that come in beside its last
// ones crowd on the SMs that are free first (2.5 times the time where there is one CTA an SM).
// Bound by the token's chain (sum, exchange, update) where sequences and heads are few, else by multiply-adds and
// shared memory alike.  Measured on a B200 inside a prompt's step, heads of 128 x 128 (GLA: 4 heads of 256 x 512), the other kernels of these
// files -> this one: 16 heads x 2,048 tokens of the delta rule 1,014 -> 351 us, with constant decays 353 -> 245; two sequences of 1,301
// and 700 tokens of the generalised rule 1,315 -> 425; GLA over four of up to 1,500 855 -> 407.  One token a sequence, 16 heads of
// 128 x 128, 1, 8 and 64 sequences: the delta rule 4.5 / 10.7 / 63 -> 4.1 / 8.6 / 51, the generalised rule 5.3 / 26 / 194 -> 4.3 / 8.7 / 53
// (GLA keeps the other kernel there: gla.cu).
#pragma once
#include "common.cuh"

#define SR_THREADS 128
enum { SCAN_GLA = 0, SCAN_DECAY = 1, SCAN_DELTA = 2, SCAN_GENERAL = 3 };

struct ScanRows {
  const float* vec[5]; long long ldvec[5];   // vector j of token t and query/key head g: vec[j] + t * ldvec[j] + g * dk (SCAN_GENERAL: + 5 dk g)
  const float* v; long long ldv;             // v + t * ldv + h * dv + c
  const float* gates;                        // SCAN_DELTA: [tokens][2 H]: g, then beta
  const float* decay;                        // SCAN_DECAY: [H]
  float* state;                              // [slots][H][dk][dv]
  const int* seq_slot;
  const int* seq_start;
  float* out; long long ldo;
  int H, G, dv;
  float scale;                               // SCAN_GLA
};

__device__ __forceinline__ unsigned long long sr_pack(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float sr_hsum(unsigned long long v) {
  float a, b;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
  return a + b;
}
__device__ __forceinline__ unsigned long long sr_fma(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long sr_mul(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ unsigned long long sr_add(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// Columns of the state per CTA, and its shared memory in floats
template <int KIND, int R, int CPT> struct SrShape {
  static constexpr int NV = KIND == SCAN_GENERAL ? 5 : KIND == SCAN_GLA ? 3 : 2;
  static constexpr int DK = 8 * R, NG = SR_THREADS / R, COLS = NG * CPT;      // NG groups of lanes, CPT columns each
  static constexpr int CH = KIND == SCAN_GENERAL || KIND == SCAN_GLA ? 8 : 16; // tokens per stage
  static constexpr int TOKEN = NV * DK, STAGE = CH * (TOKEN + COLS + (KIND == SCAN_DELTA ? 4 : 0));
  static constexpr int PART = R * CPT + 4;                                    // a group's parts of a token's read-out; 4 floats on, the next group's lie in other banks
  static constexpr size_t SMEM = (size_t)(2 * STAGE + 2 * CH * NG * PART) * sizeof(float);
};
// N neighbouring floats: shared or global memory that starts on 4 N bytes, 16 at most
template <int N> __device__ __forceinline__ void sr_get(float* d, const float* p) {
#pragma unroll
  for (int i = 0; i < N; i += (N < 4 ? N : 4)) {
    if constexpr (N >= 4) {
      const float4 x = *reinterpret_cast<const float4*>(p + i);
      d[i] = x.x; d[i + 1] = x.y; d[i + 2] = x.z; d[i + 3] = x.w;
    } else {
      const float2 x = *reinterpret_cast<const float2*>(p);
      d[0] = x.x; d[1] = x.y;
    }
  }
}
template <int N> __device__ __forceinline__ void sr_put(float* p, const float* d) {
#pragma unroll
  for (int i = 0; i < N; i += (N < 4 ? N : 4)) {
    if constexpr (N >= 4) *reinterpret_cast<float4*>(p + i) = make_float4(d[i], d[i + 1], d[i + 2], d[i + 3]);
    else *reinterpret_cast<float2*>(p) = make_float2(d[0], d[1]);
  }
}

template <int KIND, int R, int CPT>
__global__ void __launch_bounds__(SR_THREADS) scan_rows_kernel(ScanRows a) {
  using SH = SrShape<KIND, R, CPT>;
  constexpr int NV = SH::NV, DK = SH::DK, NG = SH::NG, COLS = SH::COLS, TOKEN = SH::TOKEN, STAGE = SH::STAGE, PART = SH::PART, CH = SH::CH;
  constexpr int VW = CPT < 4 ? CPT : 4;
  constexpr bool FEEDBACK = KIND == SCAN_DELTA || KIND == SCAN_GENERAL;
  constexpr int FIRST = KIND == SCAN_DELTA ? 1 : 3;               // the vector of the sum that the next token waits for
  typedef unsigned long long u64;
  extern __shared__ __align__(16) float sh[];
  float* parts = sh + 2 * STAGE;                                  // [2][CH][NG][PART]
  pdl_wait();
  const int b = blockIdx.z, h = blockIdx.y, tid = threadIdx.x;
  const int rg = tid % R, cg = tid / R;                           // rows 4 (rg + R i) .. + 3 for i < 2; columns cg CPT ..
  const int col = blockIdx.x * COLS + cg * CPT;
  const int qh = h / (a.H / a.G);
  const int t0 = a.seq_start[b], t1 = a.seq_start[b + 1];
  float* S = a.state + ((size_t)a.seq_slot[b] * a.H + h) * DK * (size_t)a.dv + col;
  // dv is a multiple of 4: runs of VW columns are inside or outside together
  u64 s[CPT][4];                                                  // row pairs
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = 4 * (rg + R * (i >> 1)) + 2 * (i & 1);
    float lo[CPT], hi[CPT];
#pragma unroll
    for (int c = 0; c < CPT; ++c) lo[c] = hi[c] = 0.0f;
#pragma unroll
    for (int c = 0; c < CPT; c += VW)
      if (col + c < a.dv) {
        sr_get<VW>(lo + c, S + (size_t)r * a.dv + c);
        sr_get<VW>(hi + c, S + (size_t)(r + 1) * a.dv + c);
      }
#pragma unroll
    for (int c = 0; c < CPT; ++c) s[c][i] = sr_pack(lo[c], hi[c]);
  }
  u64 dd = 0;
  if (KIND == SCAN_DECAY) dd = sr_pack(a.decay[h], a.decay[h]);

  const size_t hoff = KIND == SCAN_GENERAL ? (size_t)h * 5 * DK : (size_t)qh * DK;
  auto copy16 = [](float* d, const float* g) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(d)), "l"(g));
  };
  auto copy4 = [](float* d, const float* g) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(d)), "l"(g));
  };
  auto stage = [&](int buf, int c0) {
    float* vs = sh + buf * STAGE;
    const int n = t1 - c0 < CH ? t1 - c0 : CH;
    constexpr int PER = DK / 4;                                   // pieces of a vector: a power of two
#pragma unroll
    for (int j = 0; j < NV; ++j)
      for (int i = tid; i < n * PER; i += SR_THREADS) {
        const int tt = i / PER, r = (i % PER) * 4;
        copy16(vs + tt * TOKEN + j * DK + r, a.vec[j] + (c0 + tt) * a.ldvec[j] + hoff + r);
      }
    float* xs = vs + CH * TOKEN;
    for (int i = tid; i < n * COLS; i += SR_THREADS) {
      const int tt = i / COLS, c = blockIdx.x * COLS + i % COLS;
      if (c < a.dv) copy4(xs + i, a.v + (c0 + tt) * a.ldv + (size_t)h * a.dv + c);
    }
    if (KIND == SCAN_DELTA)
      for (int i = tid; i < 2 * n; i += SR_THREADS)
        copy4(xs + CH * COLS + i, a.gates + (size_t)(c0 + (i >> 1)) * 2 * a.H + (i & 1) * a.H + h);
    asm volatile("cp.async.commit_group;");
  };

  // a chunk's read-outs: VW columns a thread, the lanes' parts in order
  auto sum_up = [&](int buf, int c0, int n) {
    for (int i = tid; i < n * (COLS / VW); i += SR_THREADS) {
      const int tt = i / (COLS / VW), c = (i % (COLS / VW)) * VW, cc = blockIdx.x * COLS + c;
      if (cc >= a.dv) continue;
      const float* p = parts + ((buf * CH + tt) * NG + c / CPT) * PART + c % CPT;
      float y[4][VW], sum[VW];                                    // four sums side by side, added in pairs
#pragma unroll
      for (int r = 0; r < R; ++r) {
        float x[VW];
        sr_get<VW>(x, p + r * CPT);
#pragma unroll
        for (int e = 0; e < VW; ++e) y[r & 3][e] = r < 4 ? x[e] : y[r & 3][e] + x[e];
      }
#pragma unroll
      for (int e = 0; e < VW; ++e) sum[e] = (y[0][e] + y[1][e]) + (y[2][e] + y[3][e]);
      if (KIND == SCAN_GLA)
#pragma unroll
        for (int e = 0; e < VW; ++e) sum[e] *= a.scale;
      sr_put<VW>(a.out + (c0 + tt) * a.ldo + (size_t)h * a.dv + cc, sum);
    }
  };

  // One barrier a chunk: behind it this chunk's vectors are there, nobody reads the last chunk's any more (the next ones may
  // overwrite them) and the last chunk's parts are complete.
  if (t0 < t1) stage(0, t0);
  int buf = 0;
  for (int c0 = t0; c0 < t1; c0 += CH, buf ^= 1) {
    const int n = t1 - c0 < CH ? t1 - c0 : CH;
    asm volatile("cp.async.wait_group 0;");
    __syncthreads();
    if (c0 + CH < t1) stage(buf ^ 1, c0 + CH);
    if (c0 > t0) sum_up(buf ^ 1, c0 - CH, CH);
    const float* ks = sh + buf * STAGE;
    const float* xs = ks + CH * TOKEN;
    float* ps = parts + buf * CH * NG * PART + cg * PART + rg * CPT;
    auto vec = [&](int tt, int j, u64* d) {                       // this thread's rows of vector j as four pairs
      const ulonglong2* p = reinterpret_cast<const ulonglong2*>(ks + tt * TOKEN + j * DK) + rg;
      const ulonglong2 x = p[0], y = p[R];
      d[0] = x.x; d[1] = x.y; d[2] = y.x; d[3] = y.y;
    };
    u64 first[4] = {0, 0, 0, 0};
    if constexpr (FEEDBACK) vec(0, FIRST, first);
    auto token = [&](int tt) {
      float x[CPT];
      sr_get<CPT>(x, xs + tt * COLS + cg * CPT);
      u64 o[CPT];
      if constexpr (!FEEDBACK) {
        u64 q[4], k[4], w[4];
        vec(tt, 0, q);
        vec(tt, 1, k);
        if constexpr (KIND == SCAN_GLA) vec(tt, 2, w);
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          const u64 xx = sr_pack(x[c], x[c]);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            s[c][i] = sr_fma(KIND == SCAN_GLA ? w[i] : dd, s[c][i], sr_mul(k[i], xx));
            o[c] = i == 0 ? sr_mul(s[c][i], q[i]) : sr_fma(s[c][i], q[i], o[c]);
          }
        }
      } else {
        float g = 0.0f, beta = 0.0f;
        if constexpr (KIND == SCAN_DELTA) { g = xs[CH * COLS + 2 * tt]; beta = xs[CH * COLS + 2 * tt + 1]; }
        u64 q[4], k[4], w[4], p[4];
        vec(tt, 0, q);
        if constexpr (KIND == SCAN_GENERAL) {
          vec(tt, 1, k);
          vec(tt, 2, w);
          vec(tt, 4, p);
        }
        float seen[CPT];
#pragma unroll
        for (int c = 0; c < CPT; ++c)
          seen[c] = sr_hsum(sr_add(sr_fma(s[c][1], first[1], sr_mul(s[c][0], first[0])), sr_fma(s[c][3], first[3], sr_mul(s[c][2], first[2]))));
#pragma unroll
        for (int e = R >> 1; e > 0; e >>= 1)
#pragma unroll
          for (int c = 0; c < CPT; ++c) seen[c] += __shfl_xor_sync(0xffffffffu, seen[c], e);
        if constexpr (KIND == SCAN_DELTA) {
#pragma unroll
          for (int i = 0; i < 4; ++i) k[i] = first[i];
        }
        vec(tt + 1 < CH ? tt + 1 : 0, FIRST, first);        // past a short chunk's tokens: read and not used
        const u64 gg = sr_pack(g, g);
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          const float f = KIND == SCAN_DELTA ? beta * fmaf(-g, seen[c], x[c]) : x[c];
          const u64 xx = sr_pack(f, f), nn = sr_pack(-seen[c], -seen[c]);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if constexpr (KIND == SCAN_DELTA) s[c][i] = sr_fma(k[i], xx, sr_mul(s[c][i], gg));
            else s[c][i] = sr_fma(w[i], s[c][i], sr_fma(p[i], nn, sr_mul(k[i], xx)));
            o[c] = i == 0 ? sr_mul(s[c][i], q[i]) : sr_fma(s[c][i], q[i], o[c]);
          }
        }
      }
      float of[CPT];
#pragma unroll
      for (int c = 0; c < CPT; ++c) of[c] = sr_hsum(o[c]);
      sr_put<CPT>(ps + tt * NG * PART, of);
    };
    if (n == CH) {
#pragma unroll 4
      for (int tt = 0; tt < CH; ++tt) token(tt);
    } else {
      for (int tt = 0; tt < n; ++tt) token(tt);
    }
  }
  if (t0 < t1) {
    __syncthreads();
    const int n = (t1 - t0 - 1) % CH + 1;
    sum_up(buf ^ 1, t1 - n, n);
  }
  pdl_launch();      // not before: CTAs that wait take issue slots
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = 4 * (rg + R * (i >> 1)) + 2 * (i & 1);
    float lo[CPT], hi[CPT];
#pragma unroll
    for (int c = 0; c < CPT; ++c) asm("mov.b64 {%0, %1}, %2;" : "=f"(lo[c]), "=f"(hi[c]) : "l"(s[c][i]));
#pragma unroll
    for (int c = 0; c < CPT; c += VW)
      if (col + c < a.dv) {
        sr_put<VW>(S + (size_t)r * a.dv + c, lo + c);
        sr_put<VW>(S + (size_t)(r + 1) * a.dv + c, hi + c);
      }
  }
}

template <int KIND, int R, int CPT>
static void scan_rows_go(const ScanRows& a, int n_seqs, cudaStream_t s) {
  using SH = SrShape<KIND, R, CPT>;
  if (SH::SMEM > 48 * 1024) cudaFuncSetAttribute(scan_rows_kernel<KIND, R, CPT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SH::SMEM);
  hb_launch_after(scan_rows_kernel<KIND, R, CPT>, dim3(ceil_div(a.dv, SH::COLS), a.H, n_seqs), dim3(SR_THREADS), SH::SMEM, s, a);
}

// Runs the recurrence with these kernels if its sizes allow it: dk of 64, 128 or 256, columns in groups of 4, every row of
// a vector, of the results and of the state on 16 bytes.
template <int KIND>
static bool scan_rows(const ScanRows& a, int n_seqs, int dk, cudaStream_t s) {
  if ((dk != 64 && dk != 128 && dk != 256) || a.dv % 4 != 0 || a.H > 65535 || a.ldo % 4 != 0 || (((uintptr_t)a.state | (uintptr_t)a.out) & 15) != 0) return false;
  for (int j = 0; j < SrShape<KIND, 8, 2>::NV; ++j)
    if (((uintptr_t)a.vec[j] & 15) != 0 || a.ldvec[j] % 4 != 0) return false;
  int sms = 0, dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // Four columns a thread take fewer loads from shared memory per entry, two make twice the CTAs: four as soon as every
  // SM has one.  (us with 2 and 4: 16 heads x 2,048 tokens of the delta rule, 128 or 64 CTAs, 359 and 544; 32 heads x up to 1,301
  // tokens of the generalised one, 256 or 128, 395 and 432; 256 heads x up to 600, 2,048 or 1,024, 589 and 486.)
  const int groups = SR_THREADS * 8 / dk;
  const int cpt = (long long)n_seqs * a.H * ceil_div(a.dv, groups * 4) >= sms ? 4 : 2;
  if (n_seqs > 65535) return false;
#define SR_GO(R)                                            \
  do {                                                      \
    if (cpt == 4) scan_rows_go<KIND, R, 4>(a, n_seqs, s);   \
    else scan_rows_go<KIND, R, 2>(a, n_seqs, s);            \
  } while (0)
  if (dk == 64) SR_GO(8); else if (dk == 128) SR_GO(16); else SR_GO(32);
#undef SR_GO
  return true;
}
