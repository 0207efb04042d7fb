// out[M, N] = A[M, K] * W[N, K]^T (+ bias[N]) for up to 8 rows of floats: one pass over W.
//
// What bounds it: how many of W's bytes are on their way.  The streaming kernel of gemm_simt.cu gives 32 weight rows to a CTA and
// one row and a chain of all of K to a thread; 2,048 rows of 8,192 are then 64 CTAs that keep 1.5 MB in flight: 58 us for 67 MB at
// four tokens (1.15 TB/s).  Here a warp takes two or four weight rows, its lanes lie along K (512 neighbouring bytes a load), and 8 KB
// a warp are on their way while the 8 KB in front are multiplied: 19 us (3.5 TB/s; one token 17); 2,048 -> 16,384: 26 us against 35;
// 2,048 -> 128,256: 162 (6.5 TB/s) against 206.
//
// A lane sums its values of k in order, k = 4 lane .. 4 lane + 3, then 128 further on, and the lanes' sums are added as a tree (16, 8,
// 4, 2, 1 lanes apart): shorter chains, so smaller rounding errors than one chain over K (K = 2,048 / 8,192: 1.6e-7 / 3.0e-7 of the result's
// rms against 8.6e-7 / 1.5e-6).  Neither the number of rows a warp nor of tokens changes the order: a token's result does not depend on the batch.
#include "common.cuh"

namespace {

constexpr int FEW_WARPS = 4;

// W is read once; the load stays in front of the products it is to be hidden under
__device__ __forceinline__ float4 few_ld_w(const float* p) {
  float4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}

__device__ __forceinline__ void few_copy16(float* dst, const float* src, bool live) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int bytes = live ? 16 : 0;           // 0: sixteen bytes of zeros, nothing is read
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}

// The tokens' values come through a ring of three stages of four steps (512 values of k) in shared memory: read from L2 where they were
// used, every step waited for them (2,048 rows of 8,192, four tokens: 30 us instead of 19).
constexpr int FEW_STEPS = 4, FEW_STAGES = 3;

// R rows of W a warp, MT >= M tokens, U steps of 128 values of k on their way.  GATED: W is N / 2 gate rows and N / 2 up rows behind them; a
// warp takes R / 2 of each, and out [M, N / 2] is silu(gate) * up - the sums, and the activation on them, bit for bit those of the
// product and the activation's own kernel.
template <int R, int MT, int U, bool GATED>
__global__ void __launch_bounds__(FEW_WARPS * 32)
gemm_f32_few_kernel(const float* __restrict__ A_, const float* __restrict__ W, const float* __restrict__ bias, float* __restrict__ out_,
                    int add, int M, int N, int K, int lda, int ldo) {
  static_assert(U % FEW_STEPS == 0, "a warp's ring is whole stages");
  __shared__ __align__(16) float As[FEW_STAGES][MT][FEW_STEPS * 128];
  const int lane = threadIdx.x & 31;
  const int n0 = ((int)blockIdx.x * FEW_WARPS + (int)(threadIdx.x >> 5)) * R;
  rl_pdl_trigger();
  const float* w[R];
  const int half = N / 2;
  // the weight row of this warp's row r (a row beyond the last reads the last: not stored)
  auto row_of = [&](int r) { return GATED ? (r & 1) * half + min(n0 / 2 + r / 2, half - 1) : min(n0 + r, N - 1); };
#pragma unroll
  for (int r = 0; r < R; ++r) w[r] = W + (size_t)row_of(r) * K + lane * 4;
  const int steps = (K + 127) / 128, mine = (K - lane * 4 + 127) / 128;                    // K is a multiple of 4: a lane's piece is whole or beyond the end
  const int stages = (steps + FEW_STEPS - 1) / FEW_STEPS;
  float4 x[R][U];
  auto fetch = [&](int r, int u, int step) { x[r][u] = step < mine ? few_ld_w(w[r] + step * 128) : make_float4(0.f, 0.f, 0.f, 0.f); };
#pragma unroll
  for (int u = 0; u < U; ++u)
#pragma unroll
    for (int r = 0; r < R; ++r) fetch(r, u, u);
  rl_pdl_wait();                             // a weight is written by no kernel of a step (where W is none, see few_launch), the tokens' rows are
  const float* A = rl_behind_wait(const_cast<float*>(A_));
  float* out = rl_behind_wait(out_);
  auto fill = [&](int i) {
    if (i < stages) {
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        const int k = i * FEW_STEPS * 128 + (int)threadIdx.x * 4;
        few_copy16(&As[i % FEW_STAGES][m][threadIdx.x * 4], k < K ? A + (size_t)min(m, M - 1) * lda + k : A, k < K);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int i = 0; i < FEW_STAGES - 1; ++i) fill(i);
  float acc[R * MT];
#pragma unroll
  for (int i = 0; i < R * MT; ++i) acc[i] = 0.f;
  for (int i0 = 0; i0 < stages; i0 += U / FEW_STEPS) {
#pragma unroll
    for (int h = 0; h < U / FEW_STEPS; ++h) {
      const int i = i0 + h;
      if (i >= stages) break;
      asm volatile("cp.async.wait_group %0;" ::"n"(FEW_STAGES - 2) : "memory");
      __syncthreads();                       // stage i has arrived for every thread; stage i - 1 has been read by all
      fill(i + FEW_STAGES - 1);
#pragma unroll
      for (int v = 0; v < FEW_STEPS; ++v) {
        const int u = h * FEW_STEPS + v;
        float4 now[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          now[r] = x[r][u];
          fetch(r, u, i * FEW_STEPS + v + U);
        }
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          const float4 a = *reinterpret_cast<const float4*>(&As[i % FEW_STAGES][m][v * 128 + lane * 4]);
#pragma unroll
          for (int r = 0; r < R; ++r) {
            float t = acc[r * MT + m];
            t = fmaf(a.x, now[r].x, t);
            t = fmaf(a.y, now[r].y, t);
            t = fmaf(a.z, now[r].z, t);
            acc[r * MT + m] = fmaf(a.w, now[r].w, t);
          }
        }
      }
    }
  }
  // The lanes' sums: at every distance half of the values are handed over and half kept, until a lane holds COUNT / 32 sums (or, of
  // fewer than 32, a sum is held by several lanes).
  constexpr int COUNT = R * MT;
  int n = COUNT, first = 0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool up = lane & o;
    if (n > 1) {
      n >>= 1;
      first += up ? n : 0;
#pragma unroll
      for (int i = 0; i < COUNT / 2; ++i) {
        if (i < n) {
          const float give = up ? acc[i] : acc[i + n], keep = up ? acc[i + n] : acc[i];
          acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
      }
    } else {
      acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o);
    }
  }
  if constexpr (GATED) {
    // the gate's sum and its up's lie in lanes that the row's lowest bit parts: the second of the distances above with four rows, the first with two
    static_assert(COUNT <= 32, "a lane holds one sum");
    const int r = first / MT, m = first % MT, i = n0 / 2 + r / 2;
    const float v = acc[0] + (bias ? bias[row_of(r)] : 0.f);
    const float up = __shfl_xor_sync(0xffffffffu, v, R == 4 ? 8 : 16);
    if (lane % (32 / COUNT) == 0 && (r & 1) == 0 && i < half && m < M) out[(size_t)m * ldo + i] = v / (1.0f + expf(-v)) * up;
    return;
  }
  constexpr int HELD = COUNT > 32 ? COUNT / 32 : 1, COPIES = COUNT < 32 ? 32 / COUNT : 1;      // a sum's copies lie in neighbouring lanes
  if (lane % COPIES) return;
#pragma unroll
  for (int i = 0; i < HELD; ++i) {
    const int idx = first + i, nn = n0 + idx / MT, m = idx % MT;
    if (nn >= N || m >= M) continue;
    float v = acc[i] + (bias ? bias[nn] : 0.f);
    float* o = out + (size_t)m * ldo + nn;
    *o = add ? *o + v : v;
  }
}

template <int R, int MT, bool GATED>
int few_launch(const float* A, const float* W, const float* bias, float* out, int add, int M, int N, int K, int lda, int ldo, int early,
               cudaStream_t stream) {
  const int rows = R * FEW_WARPS;
  const dim3 grid((N + rows - 1) / rows), block(FEW_WARPS * 32);
  cudaError_t e;
  if (early) {
    e = rl_launch_pdl(gemm_f32_few_kernel<R, MT, 16 / R, GATED>, grid, block, 0, stream, A, W, bias, out, add, M, N, K, lda, ldo);
  } else {           // launched the ordinary way the kernel begins when all in front of it have ended
    gemm_f32_few_kernel<R, MT, 16 / R, GATED><<<grid, block, 0, stream>>>(A, W, bias, out, add, M, N, K, lda, ldo);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) {
    rl_set_error("rl_gemm_f32_few: %s", cudaGetErrorString(e));
    return RL_ERR_CUDA;
  }
  return RL_OK;
}

}  // namespace

// 1 where the product is taken instead of gemm_simt.cu's kernels: rows that 16-byte pieces can fetch, a K that two steps of a warp's 128
// values fill (shorter ones leave lanes idle), and up to 8 tokens: from there on the multiply-adds bound it and the product on the tensor
// cores (gemm_f32_split.cu) takes over (2,048 -> 16,384: 8 tokens 32 us against 45, 16 tokens 85 against 46).
extern "C" int rl_gemm_f32_few_supported(const void* A, const void* W, int M, int N, int K, int lda) {
  return M > 0 && M <= 8 && N > 0 && K >= 256 && K % 4 == 0 && lda % 4 == 0 && lda >= K && (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
}

template <bool GATED>
static int few_run(const float* A, const float* W, const float* bias, float* out, int add, int M, int N, int K, int lda, int ldo, int early,
                   cudaStream_t stream) {
  // Four rows a warp halve the tokens' loads a weight row; two leave more warps to stream where rows are few.  Four tokens, two / four rows:
  // 2,048 rows of 8,192 19.4 / 22.3 us, 3,072 of 2,048 7.2 / 8.3, 16,384 of 2,048 30.6 / 26.3, 128,256 of 2,048 189 / 162.
  const bool four = N >= 32 * rl_num_sms();
#define FEW_GO(MT)                                                                                                      \
  (four ? few_launch<4, MT, GATED>(A, W, bias, out, add, M, N, K, lda, ldo, early, stream)                              \
        : few_launch<2, MT, GATED>(A, W, bias, out, add, M, N, K, lda, ldo, early, stream))
  if (M == 1) return FEW_GO(1);
  if (M == 2) return FEW_GO(2);
  if (M <= 4) return FEW_GO(4);
  return FEW_GO(8);
#undef FEW_GO
}

// A: float [M, K], row stride lda; W: float [N, K] contiguous; out: float [M, N], row stride ldo; add != 0: added into out.
// early != 0: W is a weight, which no kernel that may still run writes, so it may be read before the kernels in front have ended.
extern "C" int rl_gemm_f32_few(const float* A, const float* W, const float* bias, float* out, int add, int M, int N, int K, int lda, int ldo,
                               int early, cudaStream_t stream) {
  RL_REQUIRE(rl_gemm_f32_few_supported(A, W, M, N, K, lda) && ldo >= N, "rl_gemm_f32_few: operands not supported (M=%d N=%d K=%d lda=%d ldo=%d)", M, N,
             K, lda, ldo);
  return few_run<false>(A, W, bias, out, add, M, N, K, lda, ldo, early, stream);
}

// W: float [2 I, K], gate rows first (as its bias [2 I], may be null), a weight; out: float [M, I] = silu(gate) * up.
extern "C" int rl_gemm_f32_few_swiglu(const float* A, const float* W, const float* bias, float* out, int M, int I, int K, int lda, int ldo,
                                      cudaStream_t stream) {
  RL_REQUIRE(I > 0 && I <= 1073741823 && rl_gemm_f32_few_supported(A, W, M, 2 * I, K, lda) && ldo >= I,
             "rl_gemm_f32_few_swiglu: operands not supported (M=%d I=%d K=%d lda=%d ldo=%d)", M, I, K, lda, ldo);
  return few_run<true>(A, W, bias, out, 0, M, 2 * I, K, lda, ldo, 1, stream);
}
