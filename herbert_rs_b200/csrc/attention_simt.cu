// Grouped-query softmax attention over the paged cache, CUDA cores only, any head size up to
// 512 and any number of heads and groups.  One CTA per (token, query head).
//
// This is the attention of the true 32-bit path (prefill and decode alike) and the any-shape
// fallback of the bfloat16 path.  It follows the reference's online-softmax form
// (generic_attention/prefill/kernel_f32.rs:61-111): for every key j in the query's range,
//   s_j = (q . k_j) * scale;  m' = max(m, s_j);  l = l*exp(m-m') + exp(s_j-m');
//   o = o*exp(m-m') + exp(s_j-m') * v_j;   result o / l,
// here taken 32 keys at a time, the runs of 32 keys dealt to the CTA's warps, whose (m, l, o) are joined in order at the end.  Range of the query at position p: keys lo..p with
// lo = max(0, p - window + 1) when window > 0, else 0 (causal; decode.rs:126-295 scans 0..=pos).
// Query head h reads key/value head h / (nh/nkv) (loader_common.rs:1003-1005).
// Two options for other designs: a cap on the scores, s <- cap * tanh(s / cap) after the scale
// (softcap > 0), and a sink, a learned number per query head whose exponential joins the softmax's
// denominator and nothing else: the running maximum starts at the sink and the running sum at 1,
// as if it were a first key without a value.  The value plane may be the key plane itself.
// A third option replaces the softmax: with `gate_bias` (a number per query head) the weight of a visible key
// is sigmoid(s_j + gate_bias[h]), used as it is (nothing is normalised over the keys): o = sum_j w_j v_j.
// And a fourth: with `out_gate` a head's result is multiplied by sigmoid(out_gate[token, head]) before it is rounded.
#include "api.h"
#include "common.cuh"

#define ATT_MAX_HD 512      // heads of up to 128 and 256 channels take instances with fewer registers for a result
#define ATT_WARPS 8

struct AttnArgs {
  const void* q;
  int ldq;
  void* out;
  int ldo;
  const void* kcache;
  const void* vcache;
  const int* tok_seq;
  const int* tok_pos;
  const int* seq_pages;
  int pages_stride;
  int n_tokens, nh, nkv, hd, page_size;
  float scale;
  int window;
  float softcap;
  const float* sink;
  const float* gate_bias;
  const float* out_gate;   // [n_tokens, ldg] or null: head h's result of token t is multiplied by sigmoid(out_gate[t * ldg + h])
  int ldg;
  int out_f32;              // the output is float whatever the activation type (something follows before it is rounded)
};

// V neighbouring elements as floats (one load where V = 4: rows then start on 4 elements)
template <int V> __device__ __forceinline__ void att_load(float* d, const float* p) {
  if constexpr (V == 4) {
    const float4 x = *reinterpret_cast<const float4*>(p);
    d[0] = x.x; d[1] = x.y; d[2] = x.z; d[3] = x.w;
  } else d[0] = p[0];
}
template <int V> __device__ __forceinline__ void att_load(float* d, const bf16* p) {
  if constexpr (V == 4) {
    const uint2 x = *reinterpret_cast<const uint2*>(p);
    const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&x.x), b = *reinterpret_cast<const __nv_bfloat162*>(&x.y);
    d[0] = __low2float(a); d[1] = __high2float(a); d[2] = __low2float(b); d[3] = __high2float(b);
  } else d[0] = to_f32(p[0]);
}

// Bound by the latency of the loads of keys and values: eight lanes share a key's row, so that a load covers whole
// 128-byte lines, a warp has the rows of several keys under way, and a CTA's eight warps take different runs of keys.
// (One warp per unit with a key a lane read a line per element and took 198 us for 3 sequences of about 150 keys, 16 heads of
// 128 float channels, on a B200; this form takes 18 us.)
template <typename T, int MAX_HD, int V>
__global__ void __launch_bounds__(ATT_WARPS * 32) attention_simt_kernel(AttnArgs a) {
  __shared__ __align__(16) float qs[MAX_HD];
  __shared__ float os[ATT_WARPS][MAX_HD];
  __shared__ float ms[ATT_WARPS], ls[ATT_WARPS];
  constexpr int NV = (MAX_HD + 32 * V - 1) / (32 * V);     // runs of V channels of a result per lane
  pdl_wait();
  pdl_launch();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = blockIdx.x / a.nh, h = blockIdx.x % a.nh;
  const int kvh = h / (a.nh / a.nkv);
  const int p = a.tok_pos[t], b = a.tok_seq[t];
  const int lo = (a.window > 0 && p - a.window + 1 > 0) ? p - a.window + 1 : 0;
  const T* qp = (const T*)a.q + (size_t)t * a.ldq + (size_t)h * a.hd;
  for (int d = threadIdx.x; d < a.hd; d += ATT_WARPS * 32) qs[d] = to_f32(qp[d]);
  __syncthreads();
  const int* pages = a.seq_pages + (size_t)b * a.pages_stride;
  const T* kc = (const T*)a.kcache;
  const T* vc = (const T*)a.vcache;

  float m = -INFINITY, l = 0.0f;
  if (a.sink != nullptr && warp == 0) { m = a.sink[h]; l = 1.0f; }
  const bool gated = a.gate_bias != nullptr;
  const float gb = gated ? a.gate_bias[h] : 0.0f;
  float o[NV * V];
#pragma unroll
  for (int i = 0; i < NV * V; ++i) o[i] = 0.0f;
  const int eight = lane & 7, quarter = lane >> 3;

  for (int j0 = lo + warp * 32; j0 <= p; j0 += ATT_WARPS * 32) {
    const int j = j0 + lane, jc = j <= p ? j : p;          // lanes past the last key read its row and drop the result
    const long long row = (((long long)pages[jc / a.page_size] * a.nkv + kvh) * a.page_size + jc % a.page_size) * a.hd;
    float s = 0.0f;
#pragma unroll
    for (int sub = 0; sub < 8; ++sub) {                    // four keys at a time, eight lanes each
      const T* kr = kc + __shfl_sync(0xffffffffu, row, sub * 4 + quarter);
      float dot = 0.0f;
#pragma unroll
      for (int i = 0; i < MAX_HD / (8 * V); ++i) {
        const int d = V * (eight + 8 * i);
        if (d < a.hd) {
          float x[V];
          att_load<V>(x, kr + d);
#pragma unroll
          for (int c = 0; c < V; ++c) dot = fmaf(qs[d + c], x[c], dot);
        }
      }
      dot += __shfl_xor_sync(0xffffffffu, dot, 1);
      dot += __shfl_xor_sync(0xffffffffu, dot, 2);
      dot += __shfl_xor_sync(0xffffffffu, dot, 4);
      const float mine = __shfl_sync(0xffffffffu, dot, (lane & 3) * 8);
      if (sub == (lane >> 2)) s = mine;
    }
    s *= a.scale;
    if (a.softcap > 0.0f) s = a.softcap * tanhf(s / a.softcap);
    if (j > p) s = -INFINITY;
    float pj;
    if (gated) {
      pj = (j <= p) ? 1.0f / (1.0f + expf(-(s + gb))) : 0.0f;
    } else {
      const float m_new = fmaxf(m, warp_max(s));
      const float corr = expf(m - m_new);  // m = -inf on the first chunk: exp(-inf) = 0
      pj = (j <= p) ? expf(s - m_new) : 0.0f;
      l = l * corr + warp_sum(pj);
      m = m_new;
#pragma unroll
      for (int i = 0; i < NV * V; ++i) o[i] *= corr;
    }
    const int nk = p - j0 + 1 < 32 ? p - j0 + 1 : 32;
#pragma unroll 4
    for (int k = 0; k < nk; ++k) {
      const float pk = __shfl_sync(0xffffffffu, pj, k);
      const T* vr = vc + __shfl_sync(0xffffffffu, row, k);
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int d = V * (lane + 32 * i);
        if (d < a.hd) {
          float x[V];
          att_load<V>(x, vr + d);
#pragma unroll
          for (int c = 0; c < V; ++c) o[i * V + c] = fmaf(pk, x[c], o[i * V + c]);
        }
      }
    }
  }
  if (lane == 0) { ms[warp] = m; ls[warp] = l; }
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int d = V * (lane + 32 * i);
    if (d < a.hd)
#pragma unroll
      for (int c = 0; c < V; ++c) os[warp][d + c] = o[i * V + c];
  }
  __syncthreads();
  float top = ms[0], inv = 1.0f, part[ATT_WARPS];
#pragma unroll
  for (int w = 1; w < ATT_WARPS; ++w) top = fmaxf(top, ms[w]);
  if (gated) {
#pragma unroll
    for (int w = 0; w < ATT_WARPS; ++w) part[w] = 1.0f;
  } else {
    float sum = 0.0f;
#pragma unroll
    for (int w = 0; w < ATT_WARPS; ++w) {
      part[w] = ms[w] == -INFINITY ? 0.0f : expf(ms[w] - top);      // a warp without keys: nothing
      sum = fmaf(ls[w], part[w], sum);
    }
    inv = sum > 0.0f ? 1.0f / sum : 0.0f;
  }
  if (a.out_gate != nullptr) inv *= 1.0f / (1.0f + expf(-a.out_gate[(size_t)t * a.ldg + h]));
  T* op = (T*)a.out + (size_t)t * a.ldo + (size_t)h * a.hd;
  float* of = (float*)a.out + (size_t)t * a.ldo + (size_t)h * a.hd;
  for (int d = threadIdx.x; d < a.hd; d += ATT_WARPS * 32) {
    float v = os[0][d] * part[0];
#pragma unroll
    for (int w = 1; w < ATT_WARPS; ++w) v = fmaf(os[w][d], part[w], v);
    if (a.out_f32) of[d] = v * inv;
    else op[d] = from_f32<T>(v * inv);
  }
}

extern "C" int hb_attention_simt(int dtype, const void* q, int ldq, void* out, int ldo, const void* kcache,
                                 const void* vcache, const int* tok_seq, const int* tok_pos,
                                 const int* seq_pages, int pages_stride, int n_tokens, int nh, int nkv,
                                 int hd, int page_size, float scale, int window, float softcap, const float* sink,
                                 const float* gate_bias, const float* out_gate, int ldg, int out_f32, void* stream) {
  HB_REQUIRE(n_tokens > 0 && nh > 0 && nkv > 0 && hd > 0 && page_size > 0, "attention: sizes must be positive");
  HB_REQUIRE(nh % nkv == 0, "attention: %d query heads are not a multiple of %d key/value heads", nh, nkv);
  HB_REQUIRE(hd <= ATT_MAX_HD, "attention: head size %d exceeds the supported maximum %d", hd, ATT_MAX_HD);
  HB_REQUIRE(window >= 0, "attention: window must be >= 0");
  HB_REQUIRE(softcap >= 0.0f, "attention: the cap on the scores must be >= 0 (0: none)");
  HB_REQUIRE(gate_bias == nullptr || sink == nullptr, "attention: sigmoid weights have no sink");
  AttnArgs a{q, ldq, out, ldo, kcache, vcache, tok_seq, tok_pos, seq_pages, pages_stride,
             n_tokens, nh, nkv, hd, page_size, scale, window, softcap, sink, gate_bias, out_gate, ldg, out_f32};
  const long long blocks = (long long)n_tokens * nh;
  HB_REQUIRE(blocks < 2147483647LL, "attention: too many (token, head) pairs");
  // four elements a load where every head's row starts on four
  const int es = dtype == HB_F32 ? 4 : 2;
  const bool v4 = hd % 4 == 0 && (((uintptr_t)kcache | (uintptr_t)vcache) & (uintptr_t)(4 * es - 1)) == 0;
#define AS_GO(T, MAX_HD, V) hb_launch(attention_simt_kernel<T, MAX_HD, V>, dim3((unsigned)blocks), dim3(ATT_WARPS * 32), 0, (cudaStream_t)stream, a)
#define AS_SIZE(T)                                                                        \
  do {                                                                                    \
    if (!v4) AS_GO(T, 512, 1);                                                            \
    else if (hd <= 128) AS_GO(T, 128, 4);                                                 \
    else if (hd <= 256) AS_GO(T, 256, 4);                                                 \
    else AS_GO(T, 512, 4);                                                                \
  } while (0)
  if (dtype == HB_F32) AS_SIZE(float); else AS_SIZE(bf16);
#undef AS_SIZE
#undef AS_GO
  HB_CHECK_LAUNCH("attention_simt");
  return 0;
}
