// Grouped-query softmax attention over the paged cache, CUDA cores only, any head size up to
// 512 and any number of heads and groups.  Eight or two warps of a CTA per (token, query head).
//
// This is the attention of the true 32-bit path (prefill and decode alike) and the any-shape
// fallback of the bfloat16 path.  It follows the reference's online-softmax form
// (generic_attention/prefill/kernel_f32.rs:61-111): for every key j in the query's range,
//   s_j = (q . k_j) * scale;  m' = max(m, s_j);  l = l*exp(m-m') + exp(s_j-m');
//   o = o*exp(m-m') + exp(s_j-m') * v_j;   result o / l,
// here taken 8 keys at a time, the runs of 8 keys dealt to the unit's warps, whose (m, l, o) are joined in order at the end.  Range of the query at position p: keys lo..p with
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
#define ATT_RUN 8           // keys that a warp takes at a time

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
// 128-byte lines, all rows of a run of eight keys are asked for at once, and a CTA's eight warps take different runs.
// (One warp per unit with a key a lane read a line per element and took 198 us for 3 sequences of about 150 keys, 16 heads of
// 128 float channels, on a B200; runs of 32 keys, four rows at a time, 18 us; this form 9.7 us.)
template <typename T, int MAX_HD, int V, int WPU>
__global__ void __launch_bounds__(ATT_WARPS * 32) attention_simt_kernel(AttnArgs a) {
  constexpr int UNITS = ATT_WARPS / WPU;                   // (token, head) pairs of this CTA
  __shared__ __align__(16) float qs_all[UNITS][MAX_HD];
  __shared__ float os[ATT_WARPS][MAX_HD];
  __shared__ float ms[ATT_WARPS], ls[ATT_WARPS];
  constexpr int NV = (MAX_HD + 32 * V - 1) / (32 * V);     // runs of V channels of a result per lane
  constexpr int KV = MAX_HD / (8 * V);                     // ... and of a key
  constexpr bool PREFETCH = MAX_HD <= 128;                 // a run's values fit the registers beside its keys
  pdl_wait();
  pdl_launch();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int mine = warp / WPU, part = warp % WPU;          // the unit of this warp, and which of its warps it is
  const long long last = (long long)a.n_tokens * a.nh - 1, want = (long long)blockIdx.x * UNITS + mine;
  const long long unit = want < last ? want : last;        // past the last unit: it once more, not stored
  const int t = (int)(unit / a.nh), h = (int)(unit % a.nh);
  const int kvh = h / (a.nh / a.nkv);
  const int p = a.tok_pos[t], b = a.tok_seq[t];
  const int lo = (a.window > 0 && p - a.window + 1 > 0) ? p - a.window + 1 : 0;
  const T* qp = (const T*)a.q + (size_t)t * a.ldq + (size_t)h * a.hd;
  float* qs = qs_all[mine];
  for (int d = part * 32 + lane; d < a.hd; d += WPU * 32) qs[d] = to_f32(qp[d]);
  __syncthreads();
  const int* pages = a.seq_pages + (size_t)b * a.pages_stride;
  const T* kc = (const T*)a.kcache;
  const T* vc = (const T*)a.vcache;

  float m = -INFINITY, l = 0.0f;
  if (a.sink != nullptr && part == 0) { m = a.sink[h]; l = 1.0f; }
  const bool gated = a.gate_bias != nullptr;
  const float gb = gated ? a.gate_bias[h] : 0.0f;
  float o[NV * V];
#pragma unroll
  for (int i = 0; i < NV * V; ++i) o[i] = 0.0f;
  const int eight = lane & 7, quarter = lane >> 3;

  for (int j0 = lo + part * ATT_RUN; j0 <= p; j0 += WPU * ATT_RUN) {
    long long row[2];                                      // this lane's keys j0 + quarter and j0 + 4 + quarter; past the last key: its row, the result dropped
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int j = j0 + 4 * u + quarter, jc = j <= p ? j : p;
      row[u] = (((long long)pages[jc / a.page_size] * a.nkv + kvh) * a.page_size + jc % a.page_size) * a.hd;
    }
    float x[2][KV][V], y[PREFETCH ? ATT_RUN : 1][NV][V];
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int i = 0; i < KV; ++i) {
        const int d = V * (eight + 8 * i);
        if (d < a.hd) att_load<V>(x[u][i], kc + row[u] + d);
      }
    if constexpr (PREFETCH) {                              // the values do not wait for the scores
#pragma unroll
      for (int k = 0; k < ATT_RUN; ++k) {
        const T* vr = vc + __shfl_sync(0xffffffffu, row[k >> 2], (k & 3) * 8);
#pragma unroll
        for (int i = 0; i < NV; ++i) {
          const int d = V * (lane + 32 * i);
          if (d < a.hd) att_load<V>(y[k][i], vr + d);
        }
      }
    }
    float s[2], pj[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      float dot = 0.0f;
#pragma unroll
      for (int i = 0; i < KV; ++i) {
        const int d = V * (eight + 8 * i);
        if (d < a.hd)
#pragma unroll
          for (int c = 0; c < V; ++c) dot = fmaf(qs[d + c], x[u][i][c], dot);
      }
      dot += __shfl_xor_sync(0xffffffffu, dot, 1);
      dot += __shfl_xor_sync(0xffffffffu, dot, 2);
      dot += __shfl_xor_sync(0xffffffffu, dot, 4);
      s[u] = dot * a.scale;
      if (a.softcap > 0.0f) s[u] = a.softcap * tanhf(s[u] / a.softcap);
      if (j0 + 4 * u + quarter > p) s[u] = -INFINITY;
    }
    if (gated) {
#pragma unroll
      for (int u = 0; u < 2; ++u) pj[u] = j0 + 4 * u + quarter <= p ? 1.0f / (1.0f + expf(-(s[u] + gb))) : 0.0f;
    } else {
      float top = fmaxf(s[0], s[1]);
      top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 8));
      top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 16));
      const float m_new = fmaxf(m, top);
      const float corr = expf(m - m_new);  // m = -inf on the first run: exp(-inf) = 0
#pragma unroll
      for (int u = 0; u < 2; ++u) pj[u] = j0 + 4 * u + quarter <= p ? expf(s[u] - m_new) : 0.0f;
      float sum = pj[0] + pj[1];
      sum += __shfl_xor_sync(0xffffffffu, sum, 8);
      sum += __shfl_xor_sync(0xffffffffu, sum, 16);
      l = l * corr + sum;
      m = m_new;
#pragma unroll
      for (int i = 0; i < NV * V; ++i) o[i] *= corr;
    }
    const int nk = p - j0 + 1 < ATT_RUN ? p - j0 + 1 : ATT_RUN;
#pragma unroll
    for (int k = 0; k < ATT_RUN; ++k) {
      const float pk = __shfl_sync(0xffffffffu, pj[k >> 2], (k & 3) * 8);
      const long long vrow = PREFETCH ? 0 : __shfl_sync(0xffffffffu, row[k >> 2], (k & 3) * 8);
      if (k < nk)
#pragma unroll
        for (int i = 0; i < NV; ++i) {
          const int d = V * (lane + 32 * i);
          if (d < a.hd) {
            if constexpr (!PREFETCH) att_load<V>(y[0][i], vc + vrow + d);
#pragma unroll
            for (int c = 0; c < V; ++c) o[i * V + c] = fmaf(pk, y[PREFETCH ? k : 0][i][c], o[i * V + c]);
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
  const int w0 = mine * WPU;                               // the unit's warps
  float top = ms[w0], inv = 1.0f, f[WPU];
#pragma unroll
  for (int w = 1; w < WPU; ++w) top = fmaxf(top, ms[w0 + w]);
  if (gated) {
#pragma unroll
    for (int w = 0; w < WPU; ++w) f[w] = 1.0f;
  } else {
    float sum = 0.0f;
#pragma unroll
    for (int w = 0; w < WPU; ++w) {
      f[w] = ms[w0 + w] == -INFINITY ? 0.0f : expf(ms[w0 + w] - top);      // a warp without keys: nothing
      sum = fmaf(ls[w0 + w], f[w], sum);
    }
    inv = sum > 0.0f ? 1.0f / sum : 0.0f;
  }
  if (want > last) return;
  if (a.out_gate != nullptr) inv *= 1.0f / (1.0f + expf(-a.out_gate[(size_t)t * a.ldg + h]));
  T* op = (T*)a.out + (size_t)t * a.ldo + (size_t)h * a.hd;
  float* of = (float*)a.out + (size_t)t * a.ldo + (size_t)h * a.hd;
  for (int d = part * 32 + lane; d < a.hd; d += WPU * 32) {
    float v = os[w0][d] * f[0];
#pragma unroll
    for (int w = 1; w < WPU; ++w) v = fmaf(os[w0 + w][d], f[w], v);
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
  const long long units = (long long)n_tokens * nh;
  // four elements a load where every head's row starts on four
  const int es = dtype == HB_F32 ? 4 : 2;
  const bool v4 = hd % 4 == 0 && (((uintptr_t)kcache | (uintptr_t)vcache) & (uintptr_t)(4 * es - 1)) == 0;
  // Eight warps share a unit's keys where units are few (a decode step); two where they fill the GPU several times over (a
  // prompt: 4,000 units of up to 150 keys 54 -> 38 us, since a unit's start and end cost as much as its keys)
  int sms = 0, dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const bool many = units >= 8LL * sms;
  HB_REQUIRE(ceil_div_ll(units, ATT_WARPS / 2) < 2147483647LL, "attention: too many (token, head) pairs");
#define AS_GO(T, MAX_HD, V)                                                                                                                  \
  do {                                                                                                                                       \
    if (many) hb_launch(attention_simt_kernel<T, MAX_HD, V, 2>, dim3((unsigned)ceil_div_ll(units, ATT_WARPS / 2)), dim3(ATT_WARPS * 32), 0, (cudaStream_t)stream, a); \
    else hb_launch(attention_simt_kernel<T, MAX_HD, V, 8>, dim3((unsigned)units), dim3(ATT_WARPS * 32), 0, (cudaStream_t)stream, a);          \
  } while (0)
#define AS_SIZE(T)                                                                        \
  do {                                                                                    \
    if (v4) { if (hd <= 128) AS_GO(T, 128, 4); else if (hd <= 256) AS_GO(T, 256, 4); else AS_GO(T, 512, 4); } \
    else { if (hd <= 128) AS_GO(T, 128, 1); else if (hd <= 256) AS_GO(T, 256, 1); else AS_GO(T, 512, 1); }    \
  } while (0)
  if (dtype == HB_F32) AS_SIZE(float); else AS_SIZE(bf16);
#undef AS_SIZE
#undef AS_GO
  HB_CHECK_LAUNCH("attention_simt");
  return 0;
}
