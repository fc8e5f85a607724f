// Attention over a cached latent (see latent_attention.cu) for prompts, on tcgen05: many (token, head) rows of a
// sequence against its cached rows [c | r], which are keys (all of them) and values (their first `rank` columns) at once.
//
// A CTA takes 128 consecutive rows (token, head), head fastest, of one sequence, and 256 of the latent's columns.  The
// queries, rounded to bfloat16 once, stay in shared memory (up to 144 KB); a tile of 64 keys (up to 72 KB) is fetched by TMA
// in blocks of 64 columns, with a barrier for each of the two kinds below.  Tensor memory holds the sums over the values (256 columns)
// and two buffers of scores.  The latent's 512 columns do not fit beside the scores, so two CTAs share a tile of
// rows and both compute its scores: half as many operations again, on a unit that is twelve times as fast as the warp-level instruction.
//   A-blocks     the columns whose values belong to the other CTA, and the rotated part: free as soon as the scores have read
//                them, so the next tile's are on their way under this tile's softmax
//   own blocks   the columns that are values here too: free when the product with P has read them
// Order of the MMA lane: A-blocks of tile j + 1, P V of tile j, own blocks of tile j + 1; so the scores of the next tile
// run while the row threads take this tile's softmax.  A thread owns a row (as in attention_prefill_tc.cu): P goes back over
// the scores, O is rescaled only when a tile's maximum exceeds the row's reference by more than 2^8.
// Bound by the reads of the queries from shared memory (4 KB per 128 x 64 x 16 product).
// Measured on a B200 inside a step, 16 heads, latent 512 + 64: four prompts of 714 to 2,000 tokens 1,057 us on mma.sync -> 421, four of 336
// to 1,500 477 -> 208; of that about 26 us a CTA go into its queries and results.  (With the weights in one part 391 and 194; so, and
// with one barrier a block of columns and a loop over the steps of K, 557 and 263: the MMA lane's own instructions were the limit;
// with 32 keys a tile and two sets of blocks 590.)
#include "api.h"
#include "common.cuh"
#include "tcgen05_utils.cuh"

#define LP_ROWS 128
#define LP_KEYS 64
#define LP_HALF 256                       // columns of the latent per CTA
#define LP_QBLOCK (LP_ROWS * 128)         // bytes of 64 columns of the queries
#define LP_KBLOCK (LP_KEYS * 128)         // ... of a tile of keys
#define LP_MAX_BLOCKS 9
#define LP_THREADS 320                    // TMA warp, MMA warp, four row warps; four more that help to bring the queries in
#define LP_RAISE 8.0f

struct LatentTcArgs {
  const float* q; int ldq;
  float* out; int ldo;
  const float* sink;
  const int* seq_start;
  const int* seq_pos0;
  const int* seq_pages;
  int pages_stride;
  int H, rank, W, page_size, window, row_tiles, halves;
  int* error_flag;
};

__device__ __forceinline__ void lp_mma_ta(unsigned tmem_d, unsigned tmem_a, unsigned long long bdesc, unsigned idesc, unsigned accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void lp_st32(unsigned taddr, const unsigned* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]),
        "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]),
        "r"(r[30]), "r"(r[31])
      : "memory");
}

__global__ void __launch_bounds__(LP_THREADS, 1)
latent_prefill_tc_kernel(const __grid_constant__ CUtensorMap map_c, LatentTcArgs a) {
  extern __shared__ unsigned char smem_raw[];
  pdl_wait();
  const int half = blockIdx.x % a.halves, b = blockIdx.x / a.halves;
  const int tile = a.row_tiles - 1 - (int)blockIdx.y;                      // the longest key ranges first
  const int tok0 = a.seq_start[b], nrows = (a.seq_start[b + 1] - tok0) * a.H, r0 = tile * LP_ROWS;
  if (r0 >= nrows) return;
  const unsigned base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  unsigned char* gen = smem_raw + (base - smem_u32(smem_raw));
  const int NB = (a.W + 63) >> 6;                                          // blocks of 64 columns; beyond W: zeros on both sides
  const unsigned q_s = base, k_s = q_s + NB * LP_QBLOCK, bars = k_s + NB * LP_KBLOCK;
  const int own0 = half * (LP_HALF / 64), nown = min(LP_HALF, a.rank - half * LP_HALF) >> 6, na = NB - nown;
  auto kfull = [&](int kind) { return bars + kind * 8; };                 // 0: a tile's A-blocks, 1: its own blocks
  const unsigned a_free = bars + 16, s_full = a_free + 8, p_ready = s_full + 16, o_full = p_ready + 8, drained = o_full + 8;
  volatile unsigned* tmem_slot = reinterpret_cast<volatile unsigned*>(gen + (drained + 8 - base));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) mbar_init(kfull(i), 1);
    mbar_init(a_free, 1);
    mbar_init(s_full, 1);
    mbar_init(s_full + 8, 1);
    mbar_init(p_ready, 4);
    mbar_init(o_full, 1);
    mbar_init(drained, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)tmem_slot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  // the queries: bfloat16, K-major with the 128-byte swizzle (16-byte piece c of row r lies at piece c ^ (r & 7))
  // 288 KB of floats a CTA: eight pieces a thread (80 KB a CTA) are asked for before the first is rounded
  const int per = NB * 8, pieces = LP_ROWS * per;
  for (int i0 = threadIdx.x; i0 < pieces; i0 += LP_THREADS * 8) {
    float4 x[8], y[8];
    int at[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int i = i0 + u * LP_THREADS, r = i / per, c = i - r * per, row = r0 + r;
      at[u] = i < pieces ? (c >> 3) * LP_QBLOCK + r * 128 + (((c & 7) ^ (r & 7)) << 4) : -1;
      x[u] = y[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (at[u] >= 0 && row < nrows && c * 8 < a.W) {                      // W is a multiple of 8
        const float* src = a.q + (size_t)(tok0 + row / a.H) * a.ldq + (size_t)(row % a.H) * a.W + c * 8;
        x[u] = *reinterpret_cast<const float4*>(src);
        y[u] = *reinterpret_cast<const float4*>(src + 4);
      }
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const __nv_bfloat162 p0 = __floats2bfloat162_rn(x[u].x, x[u].y), p1 = __floats2bfloat162_rn(x[u].z, x[u].w);
      const __nv_bfloat162 p2 = __floats2bfloat162_rn(y[u].x, y[u].y), p3 = __floats2bfloat162_rn(y[u].z, y[u].w);
      if (at[u] >= 0)
        *reinterpret_cast<uint4*>(gen + at[u]) = make_uint4(*reinterpret_cast<const unsigned*>(&p0), *reinterpret_cast<const unsigned*>(&p1),
                                                            *reinterpret_cast<const unsigned*>(&p2), *reinterpret_cast<const unsigned*>(&p3));
    }
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");             // the tensor cores read what these threads wrote
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem = *tmem_slot, tm_o = tmem, tm_s0 = tmem + LP_HALF;    // O: 256 columns, then two buffers of 64
  const int last = min(nrows - r0, LP_ROWS) - 1, pos0 = a.seq_pos0[b];
  const int p_first = pos0 + r0 / a.H, p_last = pos0 + (r0 + last) / a.H;
  const int lo_first = (a.window > 0 && p_first - a.window + 1 > 0) ? p_first - a.window + 1 : 0;
  const int lo_last = (a.window > 0 && p_last - a.window + 1 > 0) ? p_last - a.window + 1 : 0;
  const int tile0 = lo_first / LP_KEYS, n = p_last / LP_KEYS + 1 - tile0;
  auto a_block = [&](int i) { return i < own0 ? i : i + nown; };           // the i-th block that is not a value here

  if (warp == 0) {
    if (lane == 0) {
      const int* pages = a.seq_pages + (size_t)b * a.pages_stride;
      int sent_a = 0, sent_own = 0;
      for (int j = 0; j < n; ++j) {
        const int key0 = (tile0 + j) * LP_KEYS, lp = key0 / a.page_size;   // page_size is a multiple of 64: a tile lies in one page
        const int row = pages[lp < a.pages_stride ? lp : a.pages_stride - 1] * a.page_size + key0 % a.page_size;
        auto fetch = [&](int blk, unsigned full) { tma_load_2d(k_s + blk * LP_KBLOCK, &map_c, blk * 64, row, full); };
        if (na > 0 && j > 0 && !mbar_wait(a_free, (j - 1) & 1)) { atomicExch(a.error_flag, 41); break; }
        if (na > 0) mbar_expect_tx(kfull(0), na * LP_KBLOCK);
        for (int i = 0; i < na; ++i) fetch(a_block(i), kfull(0));
        ++sent_a;
        if (j > 0 && !mbar_wait(o_full, (j - 1) & 1)) { atomicExch(a.error_flag, 42); break; }
        mbar_expect_tx(kfull(1), nown * LP_KBLOCK);
        for (int i = 0; i < nown; ++i) fetch(own0 + i, kfull(1));
        ++sent_own;
      }
      // no copy is under way when the CTA ends, also after a wait that gave up (here or in another warp)
      if (na > 0 && sent_a > 0 && !mbar_wait(kfull(0), (sent_a - 1) & 1)) atomicExch(a.error_flag, 48);
      if (sent_own > 0 && !mbar_wait(kfull(1), (sent_own - 1) & 1)) atomicExch(a.error_flag, 48);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // D float, A and B bfloat16; B of the second product is MN-major (bit 16)
      const unsigned idesc_qk = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(LP_KEYS >> 3) << 17) | ((unsigned)(LP_ROWS >> 4) << 24);
      const unsigned idesc_pv = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((unsigned)(nown * 8) << 17) | ((unsigned)(LP_ROWS >> 4) << 24);
      const unsigned long long desc_q = umma_desc_sw128(q_s), desc_k = umma_desc_sw128(k_s);
      const unsigned long long desc_v = umma_desc_sw128_mn(k_s + own0 * LP_KBLOCK, LP_KBLOCK);
      auto scores = [&](int j, int blk, bool first) {
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)                                     // columns past W are zeros on both sides
          tc_mma_bf16(tm_s0 + (j & 1) * LP_KEYS, desc_q + ((blk * LP_QBLOCK + ks * 32) >> 4), desc_k + ((blk * LP_KBLOCK + ks * 32) >> 4), idesc_qk,
                      first && ks == 0 ? 0u : 1u);
      };
      bool ok = true;
      auto a_scores = [&](int j) {
        if (na > 0 && !mbar_wait(kfull(0), j & 1)) { atomicExch(a.error_flag, 43); ok = false; }
        tc_fence_after();
        for (int i = 0; i < na && ok; ++i) scores(j, a_block(i), i == 0);
        if (na > 0 && ok) tc_commit(a_free);
      };
      auto own_scores = [&](int j) {
        if (!mbar_wait(kfull(1), j & 1)) { atomicExch(a.error_flag, 43); ok = false; }
        tc_fence_after();
        for (int i = 0; i < nown && ok; ++i) scores(j, own0 + i, na == 0 && i == 0);
        if (ok) tc_commit(s_full + (j & 1) * 8);
      };
      a_scores(0);
      if (ok) own_scores(0);
      for (int j = 0; j < n && ok; ++j) {
        // these scores overwrite P of tile j - 1: the product that reads it was issued before, and the instructions of a CTA
        // execute in the order of their issue
        if (j + 1 < n) a_scores(j + 1);
        if (!ok) break;
        if (!mbar_wait(p_ready, j & 1)) { atomicExch(a.error_flag, 44); break; }
        tc_fence_after();
        for (int ks = 0; ks < LP_KEYS / 16; ++ks)                          // 16 keys of P = 8 columns of tensor memory
          for (int part = 0; part < 2; ++part)
            lp_mma_ta(tm_o, tm_s0 + (j & 1) * LP_KEYS + part * (LP_KEYS / 2) + ks * 8, desc_v + ((ks * 2048) >> 4), idesc_pv,
                      (j > 0 || ks > 0 || part > 0) ? 1u : 0u);
        tc_commit(o_full);
        if (j + 1 < n) own_scores(j + 1);
      }
      // ... and no product either: the tensor memory is given back and its operands' shared memory ends with the CTA
      tc_commit(drained);
      if (!mbar_wait(drained, 0)) atomicExch(a.error_flag, 49);
    }
  } else if (warp < 6) {
    const int quad = warp & 3, r = quad * 32 + lane, row = r0 + r;         // a warp reads the tensor memory lanes of its quadrant
    const unsigned lane_off = (unsigned)(quad * 32) << 16;
    const bool valid = row < nrows;
    const int p = valid ? pos0 + row / a.H : -1;
    const int lo = (a.window > 0 && p - a.window + 1 > 0) ? p - a.window + 1 : 0;
    const float log2e = 1.4426950408889634f;
    float m = -INFINITY, l = 0.0f;                                         // m: the maximum (log2 units) that P, l and O are scaled to
    if (valid && a.sink != nullptr) { m = a.sink[row % a.H] * log2e; l = 1.0f; }
    bool ok = true;
    for (int j = 0; j < n; ++j) {
      const int key0 = (tile0 + j) * LP_KEYS;
      const unsigned tm_s = tm_s0 + (j & 1) * LP_KEYS + lane_off;
      if (!mbar_wait(s_full + (j & 1) * 8, (j >> 1) & 1)) { if (lane == 0) atomicExch(a.error_flag, 45); ok = false; break; }
      tc_fence_after();
      float s[LP_KEYS];
      tc_ld32f(tm_s, s);
      tc_ld32f(tm_s + 32, s + 32);
      if (key0 + LP_KEYS - 1 > p_first || key0 < lo_last) {
#pragma unroll
        for (int i = 0; i < LP_KEYS; ++i) s[i] = (key0 + i <= p && key0 + i >= lo) ? s[i] : -INFINITY;
      }
      float mx = -INFINITY, my = -INFINITY;
#pragma unroll
      for (int i = 0; i < LP_KEYS; i += 2) { mx = fmaxf(mx, s[i]); my = fmaxf(my, s[i + 1]); }
      mx = fmaxf(mx, my) * log2e;
      const bool raise = mx > m + LP_RAISE || (m == -INFINITY && mx > -INFINITY);
      if (j > 0 && __any_sync(0xffffffffu, raise)) {
        // O to the new maximum (rows that keep theirs: factor 1), once the product of the tile before is complete
        if (!mbar_wait(o_full, (j - 1) & 1)) { if (lane == 0) atomicExch(a.error_flag, 46); ok = false; break; }
        tc_fence_after();
        const float f = raise ? (m == -INFINITY ? 0.0f : exp2f(m - mx)) : 1.0f;
#pragma unroll 1
        for (int c = 0; c < nown * 64; c += 16) {
          float o[16];
          tc_ld16f(tm_o + lane_off + c, o);
#pragma unroll
          for (int i = 0; i < 16; ++i) o[i] *= f;
          tc_st16f(tm_o + lane_off + c, o);
        }
      }
      if (raise) {
        l *= m == -INFINITY ? 0.0f : exp2f(m - mx);
        m = mx;
      }
      const float m_use = m == -INFINITY ? 0.0f : m;
      unsigned pk[LP_KEYS / 2], pl[LP_KEYS / 2];                           // P as two bfloat16 parts
      float sum0 = 0.0f, sum1 = 0.0f;
#pragma unroll
      for (int i = 0; i < LP_KEYS; i += 2) {
        const float e0 = fast_exp2(fmaf(s[i], log2e, -m_use)), e1 = fast_exp2(fmaf(s[i + 1], log2e, -m_use));
        const __nv_bfloat162 hi = __floats2bfloat162_rn(e0, e1);
        const __nv_bfloat162 lo = __floats2bfloat162_rn(e0 - __low2float(hi), e1 - __high2float(hi));
        sum0 += e0;
        sum1 += e1;
        pk[i >> 1] = *reinterpret_cast<const unsigned*>(&hi);
        pl[i >> 1] = *reinterpret_cast<const unsigned*>(&lo);
      }
      l += sum0 + sum1;
      lp_st32(tm_s, pk);                                                   // P where the row's scores were, its second part behind the first
      lp_st32(tm_s + LP_KEYS / 2, pl);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cta(p_ready);
    }
    if (ok) {
      if (!mbar_wait(o_full, (n - 1) & 1)) { if (lane == 0) atomicExch(a.error_flag, 47); ok = false; }
    }
    if (ok) {
      tc_fence_after();
      const float inv = l > 0.0f ? 1.0f / l : 0.0f;
      float* dst = a.out + (size_t)(tok0 + (valid ? row / a.H : 0)) * a.ldo + (size_t)(row % a.H) * a.rank + half * LP_HALF;
#pragma unroll 1
      for (int c = 0; c < nown * 64; c += 32) {
        float o[32];
        tc_ld32f(tm_o + lane_off + c, o);
        if (valid) {
#pragma unroll
          for (int i = 0; i < 32; i += 4)
            *reinterpret_cast<float4*>(dst + c + i) = make_float4(o[i] * inv, o[i + 1] * inv, o[i + 2] * inv, o[i + 3] * inv);
        }
        __syncwarp();
      }
      tc_fence_before();
    }
  }
  __syncthreads();
  pdl_launch();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

static size_t latent_tc_smem(int W) { return 1024 + (size_t)ceil_div(W, 64) * (LP_QBLOCK + LP_KBLOCK) + 256; }

// Whether these kernels serve a latent of `rank` + `rot` columns in pages of `page_size`.
extern "C" int hb_latent_prefill_tc_ok(int rank, int rot, int page_size) {
  const int W = rank + rot;
  return rank > 0 && rank % 64 == 0 && rank <= 2 * LP_HALF && rot >= 0 && rot % 16 == 0 && ceil_div(W, 64) <= LP_MAX_BLOCKS && page_size > 0 &&
         page_size % LP_KEYS == 0;
}

// cache_rows: rows of [c | r] in the whole cache plane; the other arguments as in hb_latent_attention_mma_bf16.
extern "C" int hb_latent_prefill_tc_bf16(const float* q, int ldq, float* out, int ldo, const void* cache, long long cache_rows, const float* sink,
                                         const int* seq_start, const int* seq_pos0, const int* seq_pages, int pages_stride, int n_seqs,
                                         int max_q_len, int heads, int rank, int rot, int page_size, int window, int* error_flag, void* stream) {
  HB_REQUIRE(n_seqs > 0 && max_q_len > 0 && heads > 0 && page_size > 0 && window >= 0 && pages_stride > 0, "latent_prefill_tc: bad sizes");
  HB_REQUIRE(hb_latent_prefill_tc_ok(rank, rot, page_size), "latent_prefill_tc: rank %d, rot %d and pages of %d are not served", rank, rot, page_size);
  HB_REQUIRE(cache_rows > 0 && cache_rows <= 2147483647LL && cache_rows % page_size == 0, "latent_prefill_tc: the cache's rows must be whole pages");
  HB_REQUIRE(ldq % 4 == 0 && ldo % 4 == 0 && (((uintptr_t)q | (uintptr_t)out | (uintptr_t)cache) & 15) == 0, "latent_prefill_tc: rows must start on 16 bytes");
  HB_REQUIRE(error_flag != nullptr, "latent_prefill_tc: needs an error flag");
  const int W = rank + rot, halves = ceil_div(rank, LP_HALF);
  const long long row_tiles = ceil_div_ll((long long)max_q_len * heads, LP_ROWS);
  HB_REQUIRE(row_tiles <= 65535, "latent_prefill_tc: too many rows");
  CUtensorMap map;
  const int rc = make_map_cols(&map, cache, cache_rows, W, W, LP_KEYS);
  if (rc) return rc;
  const LatentTcArgs a{q, ldq, out, ldo, sink, seq_start, seq_pos0, seq_pages, pages_stride, heads, rank, W, page_size, window, (int)row_tiles, halves, error_flag};
  const size_t smem = latent_tc_smem(W);
  cudaError_t e = cudaFuncSetAttribute(latent_prefill_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) HB_FAIL(3, "latent_prefill_tc: cannot reserve %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
  hb_launch_after(latent_prefill_tc_kernel, dim3((unsigned)(n_seqs * halves), (unsigned)row_tiles), dim3(LP_THREADS), smem, (cudaStream_t)stream, map, a);
  HB_CHECK_LAUNCH("latent_prefill_tc");
  return 0;
}
