// Rows kept in registers by the kernels that norm, gate and add whole rows.  A CTA owns a row of D floats (D a multiple
// of 128, rows 16-byte aligned); thread i holds float4s i, i + threads, ...: V of them.  Everything a row needs is asked for at once
// before the first sum (a decode step's few rows are bound by the way to memory and back, taken once here and once per
// array and pass before), and a sum over the row costs one barrier: every warp leaves its 128 columns' part, every thread
// adds the parts it needs in order.
#pragma once
#include "common.cuh"

#define RN_MAX_THREADS 512
#define RN_MAX_V 4
#define RN_MAX_D (RN_MAX_THREADS * 4 * RN_MAX_V)

template <int V> struct RowRegs { float4 v[V]; };

template <int V>
__device__ __forceinline__ void rn_load(RowRegs<V>& r, const float* p, int D) {
#pragma unroll
  for (int j = 0; j < V; ++j) {
    const int i = (j * blockDim.x + threadIdx.x) * 4;
    r.v[j] = i < D ? *reinterpret_cast<const float4*>(p + i) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  }
}
template <int V>
__device__ __forceinline__ void rn_store(float* p, const RowRegs<V>& r, int D) {
#pragma unroll
  for (int j = 0; j < V; ++j) {
    const int i = (j * blockDim.x + threadIdx.x) * 4;
    if (i < D) *reinterpret_cast<float4*>(p + i) = r.v[j];
  }
}
template <int V>
__device__ __forceinline__ void rn_store(bf16* p, const RowRegs<V>& r, int D) {
#pragma unroll
  for (int j = 0; j < V; ++j) {
    const int i = (j * blockDim.x + threadIdx.x) * 4;
    if (i >= D) continue;
    const __nv_bfloat162 lo = __floats2bfloat162_rn(r.v[j].x, r.v[j].y), hi = __floats2bfloat162_rn(r.v[j].z, r.v[j].w);
    *reinterpret_cast<uint2*>(p + i) = make_uint2(*reinterpret_cast<const unsigned*>(&lo), *reinterpret_cast<const unsigned*>(&hi));
  }
}
// f(value, j, component) for every value a thread holds
template <int V, typename F>
__device__ __forceinline__ void rn_each(RowRegs<V>& r, F f) {
#pragma unroll
  for (int j = 0; j < V; ++j) {
    r.v[j].x = f(r.v[j].x, j, 0);
    r.v[j].y = f(r.v[j].y, j, 1);
    r.v[j].z = f(r.v[j].z, j, 2);
    r.v[j].w = f(r.v[j].w, j, 3);
  }
}
__device__ __forceinline__ float rn_at(const float4& v, int c) { return c == 0 ? v.x : c == 1 ? v.y : c == 2 ? v.z : v.w; }

// Parts of a sum over the row: part[k] = the sum over columns 128 k .. 128 k + 127 of term(value), k < D / 128.  `part` is the
// caller's (V * 16 floats, one array per sum: no barrier protects one that is still read).  The barrier at the end makes the parts visible.
template <int V, typename F>
__device__ __forceinline__ void rn_parts(const RowRegs<V>& r, float* part, int D, F term) {
#pragma unroll
  for (int j = 0; j < V; ++j) {
    const float4 x = r.v[j];
    const float s = warp_sum((term(x.x) + term(x.y)) + (term(x.z) + term(x.w)));
    const int k = j * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if ((threadIdx.x & 31) == 0 && k * 128 < D) part[k] = s;
  }
  __syncthreads();
}
__device__ __forceinline__ float rn_sum(const float* part, int first, int n) {
  float s = 0.0f;
  for (int k = 0; k < n; ++k) s += part[first + k];
  return s;
}

// Whether rows of D floats take the kernels above; every array of the call has to start on 16 bytes (`bits`: their addresses
// and row strides in bytes, or-ed).
static inline bool rn_ok(int D, uintptr_t bits) { return D % 128 == 0 && D <= RN_MAX_D && (bits & 15) == 0; }
static inline int rn_threads(int D) { return D / 4 < RN_MAX_THREADS ? D / 4 : RN_MAX_THREADS; }
#define RN_GO(D, LAUNCH)                                      \
  do {                                                        \
    const int need__ = ceil_div((D) / 4, rn_threads(D));      \
    if (need__ == 1) { LAUNCH(1); }                           \
    else if (need__ == 2) { LAUNCH(2); }                      \
    else { LAUNCH(4); }                                       \
  } while (0)
