// Causal grouped-query attention of the 32-bit path over the paged cache, keys and values of one width of 64 or 128,
// every position of the sequence visible (no window, no chunked mask): float products, float sums, on the CUDA cores.
//
// What bounds it: multiply-adds for a prompt (4 * width a visible pair and head), the cache's bytes and the length of
// a warp's chain for single tokens.  The any-shape kernel (attention_simt.cu) gives a CTA to a token and head and reads
// every key's row once for it, one warp-wide sum a score: 914 us for 500 tokens of 32 heads of 64 over 8 KV heads and
// 151 us for four single tokens behind 96 to 700 (one B200); this kernel: 80 us (13 TFLOP/s: a tile's eight warps have
// one or two chunks each, so its ends weigh) and 15.6 us.  Here the ROWS rows of a CTA are the query heads of a KV head,
// of one token or of several neighbouring ones, so that a key is read once for all of them, and scores and sums are
// register tiles: a lane holds four rows by ROWS / 4 keys of a score tile, and four rows by HD * ROWS / 128 dimensions
// of the output.
//
// Keys are taken 32 at a time in position order, chunk c of a sequence by warp c % WARPS, which brings the keys and the values
// of its chunk into a shared-memory area of its own (16-byte asynchronous copies: the next chunk's keys arrive under
// this chunk's P V, its values under the next chunk's scores; or, with more CTAs than SMs, one area for both and two CTAs an SM:
// see rl_attention_f32).  At the end the warps' (max, denominator, output)
// are merged in the order of the warps.  Chunks, their warps and the order of every sum are functions of a row's position
// alone - neither ROWS nor what shares the tile changes a bit - so a position's result does not depend on the
// batch or on how the tokens were cut into steps.  A dot product is summed in runs of 16 dimensions.
//
// Invisible keys (behind a row's position) are left out, not multiplied by zero: what a row may not see cannot reach it,
// not even as infinity or NaN.
#include <math.h>

#include "common.cuh"

namespace {

constexpr int AF_CHUNK = 32;

__device__ __forceinline__ void af_copy16(float* dst, const float* src, bool live) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int bytes = live ? 16 : 0;         // 0: sixteen bytes of zeros, nothing is read
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void af_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void af_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

struct AfArgs {
  const float* q;
  const float *k_pool, *v_pool;
  const int *page_table, *slot_of_token, *positions;
  const float *gate, *sinks;
  float* out;
  int ldq, max_pages, ldo, M, H, G, sink, ldg, gate_per_head, tokens;
  float scale, softcap;
};

// a warp's area in floats: keys (rows 16 bytes further apart than they are long: lanes that read one column of eight neighbouring
// rows meet in no bank), values, probabilities
// SHARED: the values take the place of the chunk's keys, so that two CTAs fit an SM
template <int HD, int ROWS, bool SHARED> constexpr int af_warp_floats() {
  return AF_CHUNK * (HD + 4) + (SHARED ? 0 : AF_CHUNK * HD) + ROWS * (AF_CHUNK + 4);
}
template <int HD, int ROWS, int WARPS, bool SHARED> constexpr int af_smem() {
  return (ROWS * (HD + 4) + WARPS * af_warp_floats<HD, ROWS, SHARED>()) * 4;
}

template <int HD, int ROWS, int WARPS, bool SHARED>
__global__ void __launch_bounds__(WARPS * 32, SHARED ? 2 : 1) attention_f32_kernel(const AfArgs a) {
  constexpr int RG = ROWS / 4, KG = 32 / RG;              // lanes: RG groups of rows (row = i * RG + rg) by KG groups of keys
  constexpr int NK = AF_CHUNK / KG;                       // keys a lane: kg + KG * j
  constexpr int DPL = HD / KG, VW = DPL < 4 ? DPL : 4, NV = DPL / VW;      // dimensions a lane: NV runs of VW
  static_assert(VW == 2 || VW == 4, "a lane's run of dimensions is a vector");
  constexpr int KS = HD + 4, VS = SHARED ? KS : HD, PS = AF_CHUNK + 4;
  extern __shared__ __align__(16) float af_smem_area[];
  float* Qs = af_smem_area;                               // [ROWS][KS], scaled
  __shared__ float s_max[WARPS][ROWS], s_sum[WARPS][ROWS];
  __shared__ int s_pos[ROWS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rg = lane / KG, kg = lane % KG;
  float* Ks = af_smem_area + ROWS * KS + warp * af_warp_floats<HD, ROWS, SHARED>();
  float* Vs = SHARED ? Ks : Ks + AF_CHUNK * KS;
  float* Ps = Vs + AF_CHUNK * VS;
  const int g = blockIdx.y, hpg = a.H / a.G;
  const int tile = gridDim.x - 1 - blockIdx.x;            // a prompt's last tokens have the most keys: they start first
  const int m0 = tile * a.tokens, tokens = min(a.tokens, a.M - m0), rows = tokens * hpg;

  for (int idx = threadIdx.x; idx < ROWS * (HD / 4); idx += WARPS * 32) {
    const int r = idx / (HD / 4), c = idx % (HD / 4);
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < rows) v = *reinterpret_cast<const float4*>(a.q + (size_t)(m0 + r / hpg) * a.ldq + (size_t)(g * hpg + r % hpg) * HD + 4 * c);
    *reinterpret_cast<float4*>(Qs + r * KS + 4 * c) = make_float4(v.x * a.scale, v.y * a.scale, v.z * a.scale, v.w * a.scale);
  }
  if (threadIdx.x < ROWS) s_pos[threadIdx.x] = threadIdx.x < rows ? a.positions[m0 + threadIdx.x / hpg] : -1;
  __syncthreads();

  float acc[4][NV][VW], run_max[4], run_sum[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    run_max[i] = -INFINITY;
    run_sum[i] = 0.f;
#pragma unroll
    for (int n = 0; n < NV; ++n)
#pragma unroll
      for (int e = 0; e < VW; ++e) acc[i][n][e] = 0.f;
  }
  const float inv_cap = a.softcap > 0.f ? 1.0f / a.softcap : 0.f;
  const size_t head_off = (size_t)g * RL_PAGE * HD, page_stride = (size_t)a.G * RL_PAGE * HD;

  // the tile's tokens by sequence (a slot's tokens lie side by side): as a rule one run
  for (int t0 = 0; t0 < tokens;) {
    const int slot = a.slot_of_token[m0 + t0];
    int t1 = t0 + 1;
    while (t1 < tokens && a.slot_of_token[m0 + t1] == slot) ++t1;
    // the run's largest position; a row's own (-1: not of this run; a row of the tile that is nobody's sees whatever is there)
    int last = 0, lim[4];
    for (int t = t0; t < t1; ++t) last = max(last, s_pos[t * hpg]);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = i * RG + rg;
      lim[i] = r >= rows ? 0x7fffffff : r >= t0 * hpg && r < t1 * hpg ? s_pos[r] : -1;
    }
    t0 = t1;
    const int* pages = a.page_table + (size_t)slot * a.max_pages;
    const int chunks = last / AF_CHUNK + 1;
    auto fetch = [&](float* dst, int stride, const float* pool, int c) {
      if (c < chunks) {
        const float* src = pool + (size_t)pages[c * AF_CHUNK / RL_PAGE] * page_stride + head_off + (size_t)(c * AF_CHUNK % RL_PAGE) * HD;
#pragma unroll
        for (int idx = lane; idx < AF_CHUNK * (HD / 4); idx += 32) {
          const int r = idx / (HD / 4), d = 4 * (idx % (HD / 4));
          const bool live = c * AF_CHUNK + r <= last;
          af_copy16(dst + r * stride + d, live ? src + (size_t)r * HD + d : src, live);
        }
      }
      af_commit();
    };
    fetch(Ks, KS, a.k_pool, warp);
    for (int c = warp; c < chunks; c += WARPS) {
      if constexpr (SHARED) {
        af_wait<0>();                                     // this chunk's keys
      } else {
        fetch(Vs, VS, a.v_pool, c);
        af_wait<1>();
      }
      __syncwarp();
      float s[4][NK];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < NK; ++j) s[i][j] = 0.f;
#pragma unroll
      for (int d0 = 0; d0 < HD; d0 += 16) {
        float part[4][NK];
#pragma unroll
        for (int d = 0; d < 16; d += 4) {
          float4 kk[NK];
#pragma unroll
          for (int j = 0; j < NK; ++j) kk[j] = *reinterpret_cast<const float4*>(Ks + (kg + KG * j) * KS + d0 + d);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float4 qq = *reinterpret_cast<const float4*>(Qs + (i * RG + rg) * KS + d0 + d);
#pragma unroll
            for (int j = 0; j < NK; ++j) {
              part[i][j] = d ? fmaf(qq.x, kk[j].x, part[i][j]) : qq.x * kk[j].x;
              part[i][j] = fmaf(qq.y, kk[j].y, part[i][j]);
              part[i][j] = fmaf(qq.z, kk[j].z, part[i][j]);
              part[i][j] = fmaf(qq.w, kk[j].w, part[i][j]);
            }
          }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < NK; ++j) s[i][j] += part[i][j];
      }
      __syncwarp();                                       // every lane has read the keys
      if constexpr (SHARED) fetch(Vs, VS, a.v_pool, c);
      else fetch(Ks, KS, a.k_pool, c + WARPS);
      bool whole = true;                                  // every row of this lane sees every key of the chunk
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float top = -INFINITY;
#pragma unroll
        for (int j = 0; j < NK; ++j) {
          if (a.softcap > 0.f) s[i][j] = a.softcap * tanhf(s[i][j] * inv_cap);
          if (c * AF_CHUNK + kg + KG * j > lim[i]) s[i][j] = -INFINITY;
          top = fmaxf(top, s[i][j]);
        }
        whole &= lim[i] >= c * AF_CHUNK + AF_CHUNK - 1;
#pragma unroll
        for (int o = 1; o < KG; o <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
        const float new_max = fmaxf(run_max[i], top);
        const bool any = lim[i] >= c * AF_CHUNK;          // a row that sees none of the chunk keeps what it has
        const float corr = any ? expf(run_max[i] - new_max) : 1.f;        // exp(-inf) = 0 on the warp's first chunk
#pragma unroll
        for (int j = 0; j < NK; ++j)
          Ps[(i * RG + rg) * PS + kg + KG * j] = c * AF_CHUNK + kg + KG * j <= lim[i] ? expf(s[i][j] - new_max) : 0.f;
        if (any) run_max[i] = new_max;
        run_sum[i] = __fmul_rn(run_sum[i], corr);            // (rounded by itself in every shape of the kernel)
#pragma unroll
        for (int n = 0; n < NV; ++n)
#pragma unroll
          for (int e = 0; e < VW; ++e) acc[i][n][e] *= corr;
      }
      whole = __all_sync(0xffffffffu, whole);
      if constexpr (SHARED) af_wait<0>();                 // this chunk's values
      else af_wait<1>();                                  // (the next one's keys may be on their way)
      __syncwarp();
      const int seen = min(AF_CHUNK, last + 1 - c * AF_CHUNK);
      for (int j0 = 0; j0 < seen; j0 += 4) {
        float p[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 pp = *reinterpret_cast<const float4*>(Ps + (i * RG + rg) * PS + j0);
          p[i][0] = pp.x; p[i][1] = pp.y; p[i][2] = pp.z; p[i][3] = pp.w;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float v[NV][VW];
#pragma unroll
          for (int n = 0; n < NV; ++n) {
            const float* src = Vs + (j0 + j) * VS + n * KG * VW + kg * VW;
            if constexpr (VW == 4) {
              const float4 x = *reinterpret_cast<const float4*>(src);
              v[n][0] = x.x; v[n][1] = x.y; v[n][2] = x.z; v[n][3] = x.w;
            } else {
              const float2 x = *reinterpret_cast<const float2*>(src);
              v[n][0] = x.x; v[n][1] = x.y;
            }
          }
          const int at = c * AF_CHUNK + j0 + j;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (whole || at <= lim[i]) {
              run_sum[i] = __fadd_rn(run_sum[i], p[i][j]);
#pragma unroll
              for (int n = 0; n < NV; ++n)
#pragma unroll
                for (int e = 0; e < VW; ++e) acc[i][n][e] = fmaf(p[i][j], v[n][e], acc[i][n][e]);
            }
          }
        }
      }
      __syncwarp();                                       // values and probabilities have been read by all
      if constexpr (SHARED) fetch(Ks, KS, a.k_pool, c + WARPS);
    }
    af_wait<0>();
    __syncwarp();
  }

  // ---- the warps' results, merged in the order of the warps; a warp's key area holds its output ----
  float* Os = Ks;                                         // [ROWS][HD]
  static_assert(ROWS * HD <= AF_CHUNK * KS, "a warp's output fits where its keys were");
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = i * RG + rg;
    if (kg == 0) { s_max[warp][r] = run_max[i]; s_sum[warp][r] = run_sum[i]; }
#pragma unroll
    for (int n = 0; n < NV; ++n)
#pragma unroll
      for (int e = 0; e < VW; ++e) Os[r * HD + n * KG * VW + kg * VW + e] = acc[i][n][e];
  }
  __syncthreads();
  const float* O0 = af_smem_area + ROWS * KS;
  for (int idx = threadIdx.x; idx < rows * (HD / 4); idx += WARPS * 32) {
    const int r = idx / (HD / 4), d = 4 * (idx % (HD / 4));
    const int m = m0 + r / hpg, h = g * hpg + r % hpg;
    // sink: one more term in the denominator without a value, of score 0 or the head's own
    const bool has_sink = a.sink || a.sinks != nullptr;
    const float sink_score = a.sinks ? a.sinks[h] : 0.f;
    float M = has_sink ? sink_score : -INFINITY;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) M = fmaxf(M, s_max[w][r]);
    float L = has_sink ? expf(sink_score - M) : 0.f;
    float o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      const float wgt = s_max[w][r] > -INFINITY ? expf(s_max[w][r] - M) : s_sum[w][r];       // no keys: 0 (scores that are no numbers stay so)
      L = fmaf(s_sum[w][r], wgt, L);
      const float4 x = *reinterpret_cast<const float4*>(O0 + w * af_warp_floats<HD, ROWS, SHARED>() + r * HD + d);
      o[0] = fmaf(x.x, wgt, o[0]); o[1] = fmaf(x.y, wgt, o[1]); o[2] = fmaf(x.z, wgt, o[2]); o[3] = fmaf(x.w, wgt, o[3]);
    }
    const float inv = 1.0f / L;
    float4 res = make_float4(o[0] * inv, o[1] * inv, o[2] * inv, o[3] * inv);
    if (a.gate) {
      const float* gp = a.gate + (size_t)m * a.ldg + (a.gate_per_head ? (size_t)h : (size_t)h * HD + d);
      auto sig = [&](int e) { return 1.0f / (1.0f + expf(-gp[a.gate_per_head ? 0 : e])); };
      res.x *= sig(0); res.y *= sig(1); res.z *= sig(2); res.w *= sig(3);
    }
    *reinterpret_cast<float4*>(a.out + (size_t)m * a.ldo + (size_t)h * HD + d) = res;
  }
}

template <int HD, int ROWS, int WARPS, bool SHARED>
int af_launch(const AfArgs& a, cudaStream_t stream) {
  constexpr int smem = af_smem<HD, ROWS, WARPS, SHARED>();
  static const cudaError_t e = cudaFuncSetAttribute(attention_f32_kernel<HD, ROWS, WARPS, SHARED>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  RL_REQUIRE(e == cudaSuccess, "rl_attention_f32: cannot reserve %d bytes of shared memory: %s", smem, cudaGetErrorString(e));
  attention_f32_kernel<HD, ROWS, WARPS, SHARED><<<dim3((a.M + a.tokens - 1) / a.tokens, a.G), WARPS * 32, smem, stream>>>(a);
  RL_LAUNCH_CHECK("rl_attention_f32");
  return RL_OK;
}

}  // namespace

// Whether the kernel takes these: heads of 64 or 128 (keys and values alike), up to 16 query heads a KV head, rows of q and out and
// pools that 16-byte pieces can fetch.
extern "C" int rl_attention_f32_supported(int num_heads, int num_kv_heads, int head_dim, int ldq, int ldo, const void* q, const void* k_pool,
                                          const void* v_pool, const void* out) {
  return num_kv_heads > 0 && num_heads % num_kv_heads == 0 && num_heads / num_kv_heads <= 16 && (head_dim == 64 || head_dim == 128) &&
         num_kv_heads <= 65535 && ldq % 4 == 0 && ldo % 4 == 0 && (((uintptr_t)q | (uintptr_t)k_pool | (uintptr_t)v_pool | (uintptr_t)out) & 15) == 0;
}

// q: float [M, ldq] with head h at columns [h * hd, (h + 1) * hd); out likewise, [M, ldo].  Pools: float [pages, G, RL_PAGE, hd].
// sink, sinks, gate, ldg, gate_per_head, softcap: as in rl_attention_simt_shaped.  single_tokens != 0: every sequence of the step
// brings one token (a tile is then one token's heads, whatever their number).
extern "C" int rl_attention_f32(const float* q, int ldq, const float* k_pool, const float* v_pool, const int* page_table, int max_pages,
                                const int* slot_of_token, const int* positions, float* out, int ldo, int num_tokens, int num_heads,
                                int num_kv_heads, int head_dim, float scale, int sink, const float* gate, int ldg, float softcap,
                                int gate_per_head, const float* sinks, int single_tokens, cudaStream_t stream) {
  RL_REQUIRE(num_tokens >= 0 && num_heads > 0 && num_kv_heads > 0 && max_pages > 0 && softcap >= 0.f, "rl_attention_f32: bad sizes");
  RL_REQUIRE(rl_attention_f32_supported(num_heads, num_kv_heads, head_dim, ldq, ldo, q, k_pool, v_pool, out),
             "rl_attention_f32: %d heads over %d KV heads of %d, or rows or pools 16-byte pieces cannot fetch", num_heads, num_kv_heads, head_dim);
  RL_REQUIRE(ldq >= num_heads * head_dim && ldo >= num_heads * head_dim, "rl_attention_f32: row strides too small");
  RL_REQUIRE(gate == nullptr || ldg >= (gate_per_head ? num_heads : num_heads * head_dim), "rl_attention_f32: the gate's row stride is too small");
  if (num_tokens == 0) return RL_OK;
  const int hpg = num_heads / num_kv_heads;
  // Single tokens: the rows are one token's heads, in the smallest tile that holds them (more would only be idle lanes).
  // Prompts: as many neighbouring tokens as sixteen rows hold.
  const int tokens = single_tokens ? 1 : 16 / hpg;
  const int rows = tokens * hpg;
  AfArgs a = {q, k_pool, v_pool, page_table, slot_of_token, positions, gate, sinks, out,
              ldq, max_pages, ldo, num_tokens, num_heads, num_kv_heads, sink, ldg, gate_per_head, tokens, scale, softcap};
  // More CTAs than SMs: a warp's keys and values share an area, two CTAs run on an SM, and a warp that waits for its loads leaves the SM to
  // the other CTA's (128 registers a thread at width 64, a few of 16 rows' spilled).  One B200, areas of their own against one: 32
  // heads over 8 of 64, 500 tokens 99 / 80 us, 2,000 978 / 755, 64 single tokens behind 700 59 / 43; of 128: 200 / 132, 2,333 / 1,396,
  // 115 / 71.  Just beyond the SMs: 152 CTAs of 76 tokens 14.9 / 12.4, of 19 single tokens behind 700 29.3 / 21.7 (8 heads over 8,
  // 290 tokens: 20.0 / 21.3, 310: 21.1 / 23.5 - the CTAs behind the first wave are the shortest there - 500: 38.9 / 31.8).  With an SM
  // for every CTA the second one never comes and the areas of their own win: 8 tokens behind 2,000 67.8 / 74.5.  The order of every
  // sum is the same either way.
  const bool many = (size_t)((num_tokens + tokens - 1) / tokens) * num_kv_heads > (size_t)rl_num_sms();
  if (head_dim == 64) {
    if (rows <= 4) return many ? af_launch<64, 4, 8, true>(a, stream) : af_launch<64, 4, 8, false>(a, stream);
    if (rows <= 8) return many ? af_launch<64, 8, 8, true>(a, stream) : af_launch<64, 8, 8, false>(a, stream);
    return many ? af_launch<64, 16, 8, true>(a, stream) : af_launch<64, 16, 8, false>(a, stream);
  }
  if (rows <= 4) return many ? af_launch<128, 4, 4, true>(a, stream) : af_launch<128, 4, 4, false>(a, stream);
  if (rows <= 8) return many ? af_launch<128, 8, 4, true>(a, stream) : af_launch<128, 8, 4, false>(a, stream);
  return many ? af_launch<128, 16, 4, true>(a, stream) : af_launch<128, 16, 4, false>(a, stream);
}
