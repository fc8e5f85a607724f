// Shared device helpers for the sm_100a kernels of this library.
//
// Conventions used by every kernel file:
//  * activations and cache entries are of type T = float (32-bit path) or __nv_bfloat16;
//    sums, norms, softmax, rotation and the residual stream are always float;
//  * every launcher is `extern "C"`, takes raw device pointers plus a cudaStream_t (as void*),
//    returns 0 on success and a non-zero code after storing a message for hb_last_error();
//  * a launcher validates sizes on the host and refuses what its kernel cannot do; it never
//    launches a kernel that could give a wrong result.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

typedef __nv_bfloat16 bf16;

// ---- host-side error reporting ------------------------------------------------------------
void hb_set_error(const char* fmt, ...);
#define HB_FAIL(code, ...)            \
  do {                                \
    hb_set_error(__VA_ARGS__);        \
    return (code);                    \
  } while (0)
#define HB_REQUIRE(cond, ...)         \
  do {                                \
    if (!(cond)) HB_FAIL(2, __VA_ARGS__); \
  } while (0)
#define HB_CHECK_LAUNCH(name)                                                   \
  do {                                                                          \
    cudaError_t e__ = cudaGetLastError();                                       \
    if (e__ != cudaSuccess) HB_FAIL(3, "%s: launch failed: %s", name, cudaGetErrorString(e__)); \
  } while (0)

// ---- launching ------------------------------------------------------------------------------
// Every kernel is launched through hb_launch.  With programmatic dependent launch (hb_set_pdl; the engine switches it on, a
// launcher called alone runs without it) a kernel may be scheduled while kernels ahead of it in the stream still run.  What that rests on:
//  * Every kernel calls pdl_wait(), also one that reads nothing of its predecessor's.  The wait ends when the predecessor has ended, and
//    that one has waited for its own: so everything older has ended too.  A kernel without the wait would break the chain for the next one.
//  * Ahead of the wait a kernel touches only weights, tables and what the host copied before the step.
//  * What another kernel of a step writes is read with ordinary loads: no __ldg, no __restrict__ at its pointer.
//  * pdl_launch() tells the hardware that the next kernel may start.  It does once every CTA has called it (or ended), that is, once all of
//    them are resident: so tensor memory is taken, and whatever else an early CTA could take away, before that call.
// Most kernels trigger right after their wait, decode attention when the CTA's own loads are done.  The products of few rows
// (gemm_skinny.cu) trigger ahead of their wait, as soon as their own first loads are out: behind a chain of them several kernels sit on the SMs.
// What makes an early start pay or not is where the early CTAs come to stand: those of a kernel that leaves room for several on an SM
// crowd on the SMs that are free first and keep crowded for their whole length.  The products' CTAs leave little room on an SM; row
// kernels that trigger ahead of their wait gained the recurrent designs 1 % and cost those with experts 5 to 20 %.  Both calls are no-ops
// for a kernel launched without the attribute.
int hb_pdl_enabled(void);   // 0 off, 1 every kernel, 2 only the launches that ask for it (hb_launch_pdl)
template <typename... KArgs, typename... Args>
static inline cudaError_t hb_launch_ex(int want_pdl, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem,
                                       cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  const int mode = hb_pdl_enabled();
  cfg.numAttrs = want_pdl >= 0 && (mode == 1 || (mode == 2 && want_pdl)) ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}
template <typename... KArgs, typename... Args>
static inline cudaError_t hb_launch(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                    Args&&... args) {
  return hb_launch_ex(0, kernel, grid, block, smem, stream, static_cast<KArgs>(args)...);
}
// For kernels whose prologue is worth starting early (weight loads that do not depend on the predecessor).
template <typename... KArgs, typename... Args>
static inline cudaError_t hb_launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                        Args&&... args) {
  return hb_launch_ex(1, kernel, grid, block, smem, stream, static_cast<KArgs>(args)...);
}
// For kernels whose CTAs should spread evenly over the SMs (long ones, about one CTA an SM): never before the predecessor's end.
template <typename... KArgs, typename... Args>
static inline cudaError_t hb_launch_after(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                          Args&&... args) {
  return hb_launch_ex(-1, kernel, grid, block, smem, stream, static_cast<KArgs>(args)...);
}
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Asks for `bytes` bytes from p into L2, a line a lane (a whole warp calls it): weights that a kernel reads after its wait.
__device__ __forceinline__ void warp_prefetch_l2(const void* p, size_t bytes) {
  for (size_t b = (threadIdx.x & 31) * 128; b < bytes; b += 32 * 128) asm volatile("prefetch.global.L2 [%0];" ::"l"((const char*)p + b));
}

// ---- conversions ---------------------------------------------------------------------------
__device__ __forceinline__ float to_f32(float v) { return v; }
__device__ __forceinline__ float to_f32(bf16 v) { return __bfloat162float(v); }
template <typename T> __device__ __forceinline__ T from_f32(float v);
template <> __device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ bf16 from_f32<bf16>(float v) { return __float2bfloat16_rn(v); }

// ---- a cap on attention scores ---------------------------------------------------------------
// cap * tanh(s / cap) with tanh(x) = 1 - 2 / (1 + e^{2x}): one exponential and one division of the
// fast kind, absolute error about 1e-7 * cap (e^{2x} = inf gives 1, 0 gives -1).  The 32-bit path
// uses tanhf instead.
__device__ __forceinline__ float capped_score(float s, float cap) {
  const float e = __expf(2.0f * __fdividef(s, cap));
  return cap * (1.0f - __fdividef(2.0f, 1.0f + e));
}

// ---- reductions -----------------------------------------------------------------------------
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
// Sum over a whole block (any multiple of 32 threads up to 1024); every thread gets the result.
__device__ __forceinline__ float block_sum(float v, float* smem32) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) smem32[warp] = v;
  __syncthreads();
  float t = (lane < nwarp) ? smem32[lane] : 0.0f;
  t = warp_sum(t);
  return t;
}

static inline int ceil_div(int a, int b) { return (a + b - 1) / b; }
static inline long long ceil_div_ll(long long a, long long b) { return (a + b - 1) / b; }
