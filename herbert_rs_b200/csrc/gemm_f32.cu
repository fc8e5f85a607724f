// Matrix products of the true 32-bit path:  C[M,N] (op)= A[M,K] * W[N,K]^T  with float operands, float
// multiply-adds on the CUDA cores and float sums.  Two kernels by the number of activation rows, each with 16-byte loads
// where all rows allow them (V = 4) and element-wise guarded ones where not (V = 1); the order of the sums is the same.
//
//   gemm_f32_rows_kernel   M <= 16: a decode step.  Bound by the stream of weights, each read once.
//   gemm_f32_tile_kernel   more rows: a prompt.  Bound by the multiply-add pipes.
#include <cooperative_groups.h>

#include "api.h"
#include "common.cuh"

namespace cg = cooperative_groups;

// Columns k .. k + 3 of a row, zeros from `end` on (V = 4: the row starts on 16 bytes and `end` is a multiple of 4).
template <int V>
__device__ __forceinline__ float4 f32_load4(const float* row, int k, int end) {
  if constexpr (V == 4) return k < end ? *reinterpret_cast<const float4*>(row + k) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  else return make_float4(k < end ? row[k] : 0.0f, k + 1 < end ? row[k + 1] : 0.0f, k + 2 < end ? row[k + 2] : 0.0f, k + 3 < end ? row[k + 3] : 0.0f);
}

// ---------------------------------------------------------------------------------------------
// Few rows.  A warp owns R weight rows and a range of K: per round every lane asks for 16 bytes of each of them (the
// next round's loads are under way while this round is multiplied) and for the same columns of every activation row,
// which come from L1.  The R * MT sums of the 32 lanes are added with halving exchanges, so that 32 of them cost 31
// shuffles and lane l ends with sum l.  KW warps of a CTA share a row group's K where there are too few row groups
// to fill the GPU; their sums meet in shared memory and are added in order.
// Measured on a B200 at 3 rows, inside a step: 4,096 and 6,144 weight rows of K 1,024 85 -> 8 us, 1,024 rows of K 2,048 and 3,072
// 216 -> 5.6 us, 151,936 rows 711 -> 101 us (6.2 TB/s); before, 64-row tiles spent their time on rows that do not exist.
#define FR_WARPS 8
template <int MT, int R, int EPI, int V>
__global__ void __launch_bounds__(FR_WARPS * 32)
gemm_f32_rows_kernel(const float* A, int lda, const float* __restrict__ W, int ldw, float* C, int ldc,
                     int M, int N, int K, int kw) {
  static_assert(R * MT == 32 || R * MT == 64, "the halving exchange ends with one or two sums a lane");
  constexpr int KEEP = R * MT / 32;
  __shared__ float red[FR_WARPS][R * MT];
  pdl_wait();
  pdl_launch();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int groups = FR_WARPS / kw;                       // row groups of this CTA
  const int part = warp % kw;
  const int n0 = (blockIdx.x * groups + warp / kw) * R;
  const float* wr[R];
#pragma unroll
  for (int r = 0; r < R; ++r) wr[r] = W + (size_t)(n0 + r < N ? n0 + r : N - 1) * ldw;
  const float* ar[MT];
#pragma unroll
  for (int m = 0; m < MT; ++m) ar[m] = A + (size_t)(m < M ? m : M - 1) * lda;

  float acc[R * MT];
#pragma unroll
  for (int i = 0; i < R * MT; ++i) acc[i] = 0.0f;
  float4 w[R], nw[R];
  const int step = kw * 128;
  auto load = [&](int k, float4* d) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if constexpr (V == 4) {
        d[r] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (k < K) asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(d[r].x), "=f"(d[r].y), "=f"(d[r].z), "=f"(d[r].w) : "l"(wr[r] + k));
      } else d[r] = f32_load4<1>(wr[r], k, K);
    }
  };
  int k = part * 128 + lane * 4;
  load(k, w);
  for (; k - lane * 4 < K; k += step) {
    load(k + step, nw);
    if (k < K) {
#pragma unroll
      for (int m0 = 0; m0 < MT; m0 += 4) {                // four rows' columns are asked for together
        float4 x[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) x[m] = f32_load4<V>(ar[m0 + m], k, K);
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
          for (int r = 0; r < R; ++r) {
            float s = acc[r * MT + m0 + m];
            s = fmaf(w[r].x, x[m].x, s);
            s = fmaf(w[r].y, x[m].y, s);
            s = fmaf(w[r].z, x[m].z, s);
            acc[r * MT + m0 + m] = fmaf(w[r].w, x[m].w, s);
          }
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) w[r] = nw[r];
  }
  // halving exchange: a lane gives away the half of its sums that the lane `o` further keeps
#pragma unroll
  for (int o = 16, n = R * MT; o > 0; o >>= 1, n >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < R * MT / 2; ++i)
      if (i < n / 2) {
        const float mine = up ? acc[i + n / 2] : acc[i], theirs = up ? acc[i] : acc[i + n / 2];
        acc[i] = mine + __shfl_xor_sync(0xffffffffu, theirs, o);
      }
  }
#pragma unroll
  for (int i = 0; i < KEEP; ++i) red[warp][lane * KEEP + i] = acc[i];
  __syncthreads();
  for (int i = threadIdx.x; i < groups * R * MT; i += FR_WARPS * 32) {
    const int g = i / (R * MT), e = i % (R * MT), m = e % MT, n = (blockIdx.x * groups + g) * R + e / MT;
    if (m >= M || n >= N) continue;
    float s = red[g * kw][e];
    for (int p = 1; p < kw; ++p) s += red[g * kw + p][e];
    float* c = C + (size_t)m * ldc + n;
    *c = EPI == HB_EPI_RESIDUAL ? *c + s : s;
  }
}

template <int MT, int R, int V>
static void f32_rows_launch(const float* A, int lda, const float* W, int ldw, float* C, int ldc, int M, int N, int K, int epi, cudaStream_t s, int sms) {
  // Warps share K only while the CTAs are fewer than two an SM (1,024 rows: 8 warps a row group, 128 CTAs).
  int kw = 1;
  while (kw < FR_WARPS && K > kw * 128 && ceil_div(N, R * (FR_WARPS / kw)) < 2 * sms) kw <<= 1;
  const dim3 grid((unsigned)ceil_div(N, R * (FR_WARPS / kw))), block(FR_WARPS * 32);
  if (epi == HB_EPI_RESIDUAL) hb_launch(gemm_f32_rows_kernel<MT, R, HB_EPI_RESIDUAL, V>, grid, block, 0, s, A, lda, W, ldw, C, ldc, M, N, K, kw);
  else hb_launch(gemm_f32_rows_kernel<MT, R, HB_EPI_STORE_F32, V>, grid, block, 0, s, A, lda, W, ldw, C, ldc, M, N, K, kw);
}

// ---------------------------------------------------------------------------------------------
// More rows.  A CTA of 128 threads owns 64 x 128 outputs, a thread 8 x 8 of them as pairs (packed multiply-adds:
// fma.rn.f32x2 rounds each half as fmaf does).  Slabs of 16 columns of K lie transposed in shared memory, two of them: the next one's
// loads are under way in registers while this one is multiplied.  A cluster of S CTAs shares a tile's K where the tiles
// alone would leave SMs idle (1,024 weight rows at 250 rows: 32 tiles x 4); each CTA then finishes 64 / S of the rows,
// adding the parts in the order of K from the other CTAs' shared memory.
// Measured on a B200 at about 250 rows, inside a step: 4,096 and 6,144 weight rows of K 1,024 247 -> 70 us (37 TFLOP/s), 1,024 rows
// of K 2,048 and 3,072 229 -> 43 us.
#define FT_M 64
#define FT_N 128
#define FT_K 16
#define FT_THREADS 128
#define FT_LDA (FT_M + 4)
#define FT_LDW (FT_N + 4)
#define FT_STAGE (FT_K * (FT_LDA + FT_LDW))      // floats of a slab of both operands

__device__ __forceinline__ unsigned long long f32x2(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

template <int EPI, int V>
__global__ void __launch_bounds__(FT_THREADS)
gemm_f32_tile_kernel(const float* A, int lda, const float* __restrict__ W, int ldw, float* C, int ldc,
                     int M, int N, int K, int S, int k_per) {
  __shared__ __align__(16) float sh[FT_M * FT_N > 2 * FT_STAGE ? FT_M * FT_N : 2 * FT_STAGE];
  pdl_wait();
  pdl_launch();
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int part = blockIdx.x % S;                        // a cluster is S neighbours along x
  const int m0 = blockIdx.y * FT_M, n0 = (blockIdx.x / S) * FT_N;
  const int kb = part * k_per, ke = kb + k_per < K ? kb + k_per : K;
  const int lr = tid >> 2, lk = (tid & 3) * 4;            // loads: 32 rows x 4 groups of 4 columns at a time
  const float* ap[2];
  const float* wp[4];
#pragma unroll
  for (int i = 0; i < 2; ++i) ap[i] = A + (size_t)min(m0 + lr + 32 * i, M - 1) * lda;
#pragma unroll
  for (int i = 0; i < 4; ++i) wp[i] = W + (size_t)min(n0 + lr + 32 * i, N - 1) * ldw;
  float4 ra[2], rw[4];
  auto load = [&](int k) {
#pragma unroll
    for (int i = 0; i < 2; ++i) ra[i] = f32_load4<V>(ap[i], k + lk, ke);      // where K is a multiple of 4 the ranges are too
#pragma unroll
    for (int i = 0; i < 4; ++i) rw[i] = f32_load4<V>(wp[i], k + lk, ke);
  };
  auto put = [&](int buf) {
    float* as = sh + buf * FT_STAGE;
    float* ws = as + FT_K * FT_LDA;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float* p = as + lk * FT_LDA + lr + 32 * i;
      p[0] = ra[i].x; p[FT_LDA] = ra[i].y; p[2 * FT_LDA] = ra[i].z; p[3 * FT_LDA] = ra[i].w;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float* p = ws + lk * FT_LDW + lr + 32 * i;
      p[0] = rw[i].x; p[FT_LDW] = rw[i].y; p[2 * FT_LDW] = rw[i].z; p[3 * FT_LDW] = rw[i].w;
    }
  };
  unsigned long long acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;

  load(kb);
  put(0);
  __syncthreads();
  int buf = 0;
  for (int k = kb; k < ke; k += FT_K, buf ^= 1) {
    const bool more = k + FT_K < ke;
    if (more) load(k + FT_K);
    const float* as = sh + buf * FT_STAGE + ty * 4;
    const float* ws = sh + buf * FT_STAGE + FT_K * FT_LDA + tx * 4;
#pragma unroll
    for (int kk = 0; kk < FT_K; ++kk) {
      const float4 a0 = *reinterpret_cast<const float4*>(as + kk * FT_LDA), a1 = *reinterpret_cast<const float4*>(as + kk * FT_LDA + 32);
      const float4 b0 = *reinterpret_cast<const float4*>(ws + kk * FT_LDW), b1 = *reinterpret_cast<const float4*>(ws + kk * FT_LDW + 64);
      const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
      const unsigned long long b[4] = {f32x2(b0.x, b0.y), f32x2(b0.z, b0.w), f32x2(b1.x, b1.y), f32x2(b1.z, b1.w)};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const unsigned long long aa = f32x2(a[i], a[i]);
#pragma unroll
        for (int j = 0; j < 4; ++j) fma2(acc[i][j], aa, b[j]);
      }
    }
    if (more) put(buf ^ 1);
    __syncthreads();
  }

  auto out = [&](int m, int n, float4 v) {                // four neighbouring columns of a row
    if (m >= M) return;
    float* c = C + (size_t)m * ldc + n;
    const float x[4] = {v.x, v.y, v.z, v.w};
    if (n + 4 <= N && ((uintptr_t)c & 15) == 0) {
      float4* c4 = reinterpret_cast<float4*>(c);
      if (EPI == HB_EPI_RESIDUAL) { const float4 o = *c4; v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w; }
      *c4 = v;
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (n + j < N) c[j] = EPI == HB_EPI_RESIDUAL ? c[j] + x[j] : x[j];
    }
  };
  auto quad = [&](int i, int j) {
    float4 v;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(acc[i][2 * j]));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.z), "=f"(v.w) : "l"(acc[i][2 * j + 1]));
    return v;
  };
  if (S == 1) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) out(m0 + (i & 4) * 8 + ty * 4 + (i & 3), n0 + 64 * j + tx * 4, quad(i, j));
    return;
  }
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) *reinterpret_cast<float4*>(sh + ((i & 4) * 8 + ty * 4 + (i & 3)) * FT_N + 64 * j + tx * 4) = quad(i, j);
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  const int rows = FT_M / S;                              // S is a power of two
  for (int i = tid; i < rows * (FT_N / 4); i += FT_THREADS) {
    const int r = part * rows + i / (FT_N / 4), c = (i % (FT_N / 4)) * 4;
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int p = 0; p < S; ++p) {
      const float4 x = *reinterpret_cast<const float4*>(cluster.map_shared_rank(sh, p) + r * FT_N + c);
      v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
    }
    out(m0 + r, n0 + c, v);
  }
  cluster.sync();                                         // nobody leaves while its part is still read
}

template <int EPI, int V>
static void f32_tile_launch(const float* A, int lda, const float* W, int ldw, float* C, int ldc, int M, int N, int K, cudaStream_t s, int sms) {
  const int tiles_m = ceil_div(M, FT_M), tiles_n = ceil_div(N, FT_N);
  // Parts of K while the CTAs are fewer than two an SM (four warps alone do not fill an SM's pipes) and a part has at least 128 columns.
  int S = 1;
  while (S < 8 && (long long)tiles_m * tiles_n * S < 2LL * sms && K >= S * 2 * 128) S <<= 1;
  const int k_per = ceil_div(ceil_div(K, S), FT_K) * FT_K;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(S * tiles_n, tiles_m);
  cfg.blockDim = dim3(FT_THREADS);
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
  cudaLaunchKernelEx(&cfg, gemm_f32_tile_kernel<EPI, V>, A, lda, W, ldw, C, ldc, M, N, K, S, k_per);
}

template <int V>
static void f32_launch(const float* A, int lda, const float* W, int ldw, float* C, int ldc, int M, int N, int K, int epi, cudaStream_t s, int sms) {
  if (M <= 4) f32_rows_launch<4, 8, V>(A, lda, W, ldw, C, ldc, M, N, K, epi, s, sms);
  else if (M <= 8) f32_rows_launch<8, 4, V>(A, lda, W, ldw, C, ldc, M, N, K, epi, s, sms);
  else if (M <= 16) f32_rows_launch<16, 4, V>(A, lda, W, ldw, C, ldc, M, N, K, epi, s, sms);
  else if (epi == HB_EPI_RESIDUAL) f32_tile_launch<HB_EPI_RESIDUAL, V>(A, lda, W, ldw, C, ldc, M, N, K, s, sms);
  else f32_tile_launch<HB_EPI_STORE_F32, V>(A, lda, W, ldw, C, ldc, M, N, K, s, sms);
}

int hb_gemm_f32(const float* A, int lda, const float* W, int ldw, float* C, int ldc, int M, int N, int K, int epi, void* stream) {
  HB_REQUIRE(ceil_div(M, FT_M) <= 65535, "gemm: too many rows (%d)", M);
  int sms = 0, dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const bool v4 = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
  if (v4) f32_launch<4>(A, lda, W, ldw, C, ldc, M, N, K, epi, (cudaStream_t)stream, sms);
  else f32_launch<1>(A, lda, W, ldw, C, ldc, M, N, K, epi, (cudaStream_t)stream, sms);
  HB_CHECK_LAUNCH("gemm_f32");
  return 0;
}
