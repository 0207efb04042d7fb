// out[M, N] = A[M, K] * W[N, K]^T (+ bias[N]) for float operands and more than 8 rows, on the tensor cores without
// giving up float's accuracy.
//
// A float is the exact sum of three bf16 numbers: x = h + m + l, h the bf16 nearest to x, m the one nearest to what is left (below
// 2^-8 of x's power of two), l the rest (below 2^-17).  The product of two floats is taken as h h' + (h m' + m h') + (h l' + m m' + l h');
// what is left out (m l', l m', l l'; with tiles of up to 64 tokens l m' is in) is below 2^-24 of the product, of either sign: half a unit
// in the last place, a float rounding.  (Cut by truncation the residuals are twice as large and have the operand's sign: up to
// 2^-21 is left out, always towards zero.)  bf16 products are exact in the tensor core's float accumulators;
// those are only trusted with 64 values of k at a time - h h' in one, the small terms in another, so that they are not cut off against the
// large ones - and are then added to sums in registers, rounded to nearest.  The error against 64 bits
// is smaller than that of the k-ordered sum it replaces (rms over the rms of the result, K = 2,048 / 8,192: 1.3e-7 / 1.6e-7
// against 8.1e-7 / 1.6e-6; tests/test_kernels_gpu.py holds it to that, and single products to 2^-23).
//
// What bounds it: shared memory.  Per 64 values of k a tile of 128 x 128 takes 24 products of 128 x 128 x 16 (1,536 clocks of the
// tensor pipe), which read 192 KB of operands, and the cutting warps write 96 KB.  The register tile on the CUDA cores
// that this replaces (gemm_simt_big_kernel) reached 14 to 47 TFLOP/s.  500 tokens, 2,048 -> 16,384: 249 us (135 TFLOP/s)
// against 828; 8,192 -> 2,048: 121 against 1,232.
//
// Roles in a CTA: eight warps fetch floats from global memory (the next block's loads are in flight while this block is
// cut) and write the three bf16 tiles of both operands in the tensor core's swizzled layout; eight warps (four for tiles of up to 64
// tokens) add the accumulators to their registers and store; one thread issues the products: of the first summing warp, or of a warp of
// its own for tiles of up to 64 tokens.  Few tiles: the K range of a tile is cut over a cluster of
// 2 or 4 CTAs, added in order through distributed shared memory.
//
// Infinities and NaNs do not survive the cutting (inf - inf), and floats above the largest bf16 (3.39e38) are rounded to infinity, so an
// output that is no finite number is computed again, alone and in the order of k, by the plain sum.
#include <type_traits>

#include "tc_device.cuh"

namespace {

constexpr int SP_BK = 64;                                               // floats of K a stage
constexpr int SP_TILE_W = 128 * SP_BK * 2;                              // one bf16 tile of W: 128 rows of 128 bytes
// Warps: eight cut; with 128 tokens a tile eight add, the first of which also issues the products (sixteen warps, so that a
// thread may have 128 registers); with fewer four add and one more issues.
constexpr int SP_CONVERT = 8;
template <int BT> constexpr int sp_sum() { return BT > 64 ? 8 : 4; }
template <int BT> constexpr int sp_issuer() { return BT > 64 ? SP_CONVERT : SP_CONVERT + sp_sum<BT>(); }
template <int BT> constexpr int sp_threads() { return BT > 64 ? 512 : 32 * (SP_CONVERT + sp_sum<BT>() + 1); }
// Tensor memory: an accumulator is two blocks of BT columns (h h', the small terms) or, with fewer tokens, three; as many
// as 512 columns hold
template <int BT> constexpr int sp_acc_cols() { return BT > 32 ? 256 : 128; }
template <int BT> constexpr int sp_accs() { return 512 / sp_acc_cols<BT>(); }
// BT: tokens a tile.  A stage: h, m, l of W's tile, then of A's
template <int BT> constexpr int sp_stage() { return 3 * (SP_TILE_W + BT * SP_BK * 2); }
template <int BT> constexpr int sp_stages() { return BT > 64 ? 2 : 3; }
template <int BT> constexpr int sp_smem() { return sp_stages<BT>() * sp_stage<BT>() + 1024 + 256; }

// two floats -> their nearest bf16 numbers, the first in the low half
__device__ __forceinline__ uint32_t sp_round2(float x0, float x1) {
  uint32_t d;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(x1), "f"(x0));
  return d;
}

// four floats -> four bf16 of each cut
__device__ __forceinline__ void sp_cut(const float4& a, uint2& h, uint2& m, uint2& l) {
  const float x[4] = {a.x, a.y, a.z, a.w};
  uint32_t c[3][2];
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    float r0 = x[2 * p], r1 = x[2 * p + 1];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      c[i][p] = sp_round2(r0, r1);
      r0 -= __uint_as_float(c[i][p] << 16);              // exact: 16 bits are left, then 8
      r1 -= __uint_as_float(c[i][p] & 0xffff0000u);
    }
  }
  h = make_uint2(c[0][0], c[0][1]);
  m = make_uint2(c[1][0], c[1][1]);
  l = make_uint2(c[2][0], c[2][1]);
}

// A load that stays where it is written (a plain one is moved down to its use, behind the wait it was to be hidden under).
__device__ __forceinline__ float4 sp_ld(const float* p) {
  float4 v;
  asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}

__device__ __forceinline__ float sp_dsmem_ld(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}

// the sum in the order of k, for outputs that are no finite numbers
__device__ __noinline__ float sp_plain_dot(const float* x, const float* w, int K) {
  float v = 0.f;
  for (int k = 0; k < K; ++k) v = fmaf(x[k], w[k], v);
  return v;
}

template <int BT>
__global__ void __launch_bounds__(sp_threads<BT>(), 1)
gemm_f32_split_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias, float* __restrict__ out,
                      int add, int M, int N, int K, int lda, int ldo, int splits, int kb_per_split, int* __restrict__ err) {
  constexpr int STAGES = sp_stages<BT>(), ACCS = sp_accs<BT>(), SUM = sp_sum<BT>(), ISSUER = sp_issuer<BT>();
  extern __shared__ uint8_t sp_smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)sp_smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = (uint64_t*)(smem + STAGES * sp_stage<BT>());
  uint64_t* full_bar = bars;                          // [STAGES] a stage's tiles are written (one arrival a cutting warp)
  uint64_t* empty_bar = bars + STAGES;                // [STAGES] the products that read a stage are done
  uint64_t* acc_full = bars + 2 * STAGES;             // [ACCS]
  uint64_t* acc_empty = acc_full + ACCS;              // [ACCS] one arrival a summing warp
  uint32_t* tmem_slot = (uint32_t*)(acc_empty + ACCS);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int split = blockIdx.x % splits;
  const int m0 = (int)(blockIdx.x / splits) * BT, n0 = (int)blockIdx.y * 128;
  const int total_kb = (K + SP_BK - 1) / SP_BK;
  const int kb0 = split * kb_per_split, num_kb = min(kb_per_split, total_kb - kb0);

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&full_bar[s]), SP_CONVERT);
      mbar_init(smem_u32(&empty_bar[s]), 1);
    }
    for (int s = 0; s < ACCS; ++s) {
      mbar_init(smem_u32(&acc_full[s]), 1);
      mbar_init(smem_u32(&acc_empty[s]), SUM);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == SP_CONVERT) tmem_alloc(smem_u32(tmem_slot), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  auto give_up = [&](int code) {
    if (!*abort_flag) { *abort_flag = 1; atomicExch(err, code); }
  };

  // ---------------- the products of block kb (one thread) ----------------
  // Instructions that add to one accumulator run in the order they were issued in only if they have one shape, and what does not fit a
  // float is cut off: h h' has an accumulator of its own, the small terms another.  With 128 tokens two of 128 columns are all there is room for
  // (twice): six instructions for every 16 values of k (249 us where four wider ones of mixed shapes took 235).  With fewer tokens an instruction
  // takes some 100 clocks however few its columns, so the small terms' instructions multiply a cut of W with two of A's, whose tiles lie one
  // behind the other (w[2] with m as well, which costs nothing).
  auto issue = [&](int kb, int s, int phase) {
    const int b = kb % ACCS;
    if (kb >= ACCS && !mbar_wait(smem_u32(&acc_empty[b]), ((kb / ACCS) & 1) ^ 1, abort_flag)) { give_up(23); return false; }
    if (!mbar_wait(smem_u32(&full_bar[s]), phase, abort_flag)) { give_up(24); return false; }
    tc_fence_after();
    uint8_t* st = smem + s * sp_stage<BT>();
    uint64_t w[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) w[i] = make_smem_desc(smem_u32(st + i * SP_TILE_W));
    const uint64_t a = make_smem_desc(smem_u32(st + 3 * SP_TILE_W));
    const uint32_t d = tmem_base + (uint32_t)(b * sp_acc_cols<BT>());
    constexpr int TILE = BT * SP_BK * 2, SMALL = BT > 64 ? BT : 2 * BT;          // columns of the small terms
    const uint64_t am = make_smem_desc(smem_u32(st + 3 * SP_TILE_W + TILE));
    auto product = [&](uint32_t cols, uint64_t cut_w, uint64_t cut_a, int n, bool anew) {
#pragma unroll
      for (int k = 0; k < SP_BK / UMMA_K; ++k) umma_bf16(cols, cut_w + 2 * k, cut_a + 2 * k, make_idesc(128, n), anew && k == 0 ? 0u : 1u);
    };
    product(d + BT, w[2], a, SMALL, true);
    if constexpr (SMALL == BT) {
      product(d + BT, w[1], am, SMALL, false);
      product(d + BT, w[0], make_smem_desc(smem_u32(st + 3 * SP_TILE_W + 2 * TILE)), SMALL, false);
    }
    product(d + BT, w[1], a, SMALL, false);
    product(d + BT, w[0], am, SMALL, false);
    product(d, w[0], a, BT, true);
    umma_commit(smem_u32(&empty_bar[s]));
    umma_commit(smem_u32(&acc_full[b]));
    return true;
  };

  if (warp < SP_CONVERT) {
    // ---------------- fetch and cut ----------------
    // A stage is groups of four rows, 32 of W and BT / 4 of A; pass p of a warp takes group p * 8 + warp of W (p < 4), then of A.
    // Sixteen lanes read a row's 256 bytes, two rows a load, and write their four floats' cuts as 8-byte pieces.  Rows beyond
    // the last read the last: their outputs are not stored.
    constexpr int PW = 4, PASSES = PW + BT / 32;
    const int sub = lane >> 4, col = lane & 15;
    // rows 4 * warp + sub and + 2 of a group (groups of a warp are eight apart: the place among eight rows is the same in all)
    uint32_t place[2];
    const float* src[PASSES][2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int r = warp * 4 + 2 * e + sub;
      place[e] = (uint32_t)(r * 128 + (((col >> 1) ^ (r & 7)) << 4) + (col & 1) * 8);
#pragma unroll
      for (int p = 0; p < PASSES; ++p)
        src[p][e] = (p < PW ? W + (size_t)min(n0 + p * 32 + r, N - 1) * K : A + (size_t)min(m0 + (p - PW) * 32 + r, M - 1) * lda) + kb0 * SP_BK + col * 4;
    }
    float4 x[PASSES][2];
    auto load = [&](int p, int kb) {
#pragma unroll
      for (int e = 0; e < 2; ++e) x[p][e] = sp_ld(src[p][e] + kb * SP_BK);
    };
    // the last block of K may be a part of one (K is a multiple of 4: a piece is whole or beyond the end)
    const int whole_kb = (K - kb0 * SP_BK) / SP_BK;
    auto load_end = [&](int p, int kb) {
#pragma unroll
      for (int e = 0; e < 2; ++e)
        x[p][e] = (kb0 + kb) * SP_BK + col * 4 < K ? sp_ld(src[p][e] + kb * SP_BK) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
#pragma unroll
    for (int p = 0; p < PASSES; ++p) load_end(p, 0);
    int s = 0, phase = 1;
    for (int kb = 0; kb < num_kb; ++kb) {
      if (kb >= STAGES && !mbar_wait(smem_u32(&empty_bar[s]), phase, abort_flag)) { give_up(21); break; }
      uint8_t* st = smem + s * sp_stage<BT>();
      const bool next = kb + 1 < num_kb, next_whole = kb + 1 < whole_kb;
#pragma unroll
      for (int p = 0; p < PASSES; ++p) {
        uint8_t* dst = st + (p < PW ? p * 4096 : 3 * SP_TILE_W + (p - PW) * 4096);
        constexpr int cut_w = SP_TILE_W, cut_a = BT * SP_BK * 2;
        const int cut = p < PW ? cut_w : cut_a;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          uint2 h, m, l;
          sp_cut(x[p][e], h, m, l);
          uint8_t* d = dst + place[e];
          *reinterpret_cast<uint2*>(d) = h;
          *reinterpret_cast<uint2*>(d + cut) = m;
          *reinterpret_cast<uint2*>(d + 2 * cut) = l;
        }
        if (next) {
          if (next_whole) load(p, kb + 1);
          else load_end(p, kb + 1);
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");        // what the tensor core reads next
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&full_bar[s]));
      if (++s == STAGES) { s = 0; phase ^= 1; }
    }
  } else if (warp < SP_CONVERT + SUM) {
    // ---------------- sums: a warp's quarter of the rows (lanes), its share of the token columns ----------------
    constexpr int NC = BT / (SUM / 4), BLOCKS = BT > 64 ? 2 : 3;
    const int quarter = warp & 3, share = (warp - SP_CONVERT) >> 2;
    const int n = n0 + quarter * 32 + lane;
    // With up to 64 tokens a tile the bias goes in front of the last block's terms, the small ones first: it is then not one more rounding of a
    // finished sum.  (With 128 a second form of the loop below takes registers that are not there: 249 -> 282 us.)
    constexpr bool BIAS_INSIDE = BT <= 64;
    const float b = BIAS_INSIDE && bias && split == 0 && n < N ? bias[n] : 0.f;
    float acc[NC];
#pragma unroll
    for (int j = 0; j < NC; ++j) acc[j] = 0.f;
    auto add_block = [&](uint32_t t, auto last) {
#pragma unroll
      for (int q = 0; q < NC / 16; ++q) {
        uint32_t r[16], v[16];
        tmem_ld16(t + BT + q * 16, v);
        if constexpr (BLOCKS == 3) {
          tmem_ld16(t + 2 * BT + q * 16, r);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) + __uint_as_float(r[j]));
        }
        tmem_ld16(t + q * 16, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          float& sum = acc[q * 16 + j];
          if constexpr (decltype(last)::value) sum = ((sum + b) + __uint_as_float(v[j])) + __uint_as_float(r[j]);
          else sum += __uint_as_float(v[j]) + __uint_as_float(r[j]);
        }
      }
    };
    int s = 0, phase = 0;
    for (int kb = 0; kb <= num_kb; ++kb) {
      if (warp == ISSUER && kb < num_kb) {       // they run while the sums of the block in front are added
        if (lane == 0 && !*abort_flag) issue(kb, s, phase);
        __syncwarp();
        if (++s == STAGES) { s = 0; phase ^= 1; }
      }
      if (kb == 0) continue;
      const int buf = (kb - 1) % ACCS;
      if (!mbar_wait(smem_u32(&acc_full[buf]), ((kb - 1) / ACCS) & 1, abort_flag)) { give_up(22); break; }
      tc_fence_after();
      const uint32_t t = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * sp_acc_cols<BT>() + share * NC);
      if (BIAS_INSIDE && kb == num_kb) add_block(t, std::bool_constant<BIAS_INSIDE>());
      else add_block(t, std::false_type());
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&acc_empty[buf]));
    }
    if (splits > 1) {
      // the other parts' sums come through their shared memory (every product has read it: this thread has seen its part's
      // last accumulator)
      float* red = (float*)smem;                 // [NC][32 SUM]
      const int t = threadIdx.x - 32 * SP_CONVERT;
      if (split > 0 && !*abort_flag) {
#pragma unroll
        for (int j = 0; j < NC; ++j) red[j * (32 * SUM) + t] = acc[j];
      }
      __syncwarp();
      cluster_sync_all();
      if (split == 0) {
        const uint32_t local = smem_u32(red + t);
        for (int p = 1; p < splits; ++p) {       // in the order 1, 2, ...
          const uint32_t remote = dsmem_addr(local, (uint32_t)p);
#pragma unroll
          for (int j = 0; j < NC; ++j) acc[j] += sp_dsmem_ld(remote + (uint32_t)(j * (128 * SUM)));
        }
      }
      __syncwarp();
      cluster_sync_all();                        // nobody leaves while another part still reads its shared memory
    }
    if (split == 0 && n < N && !*abort_flag) {
      const float at_end = !BIAS_INSIDE && bias ? bias[n] : 0.f;
      const int j0 = m0 + share * NC;
#pragma unroll
      for (int c = 0; c < NC; c += 16) {
        float old[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) old[j] = add && j0 + c + j < M ? out[(size_t)(j0 + c + j) * ldo + n] : 0.f;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int m = j0 + c + j;
          if (m >= M) continue;
          float v = acc[c + j];
          if (!(fabsf(v) <= 3.402823466e38f)) v = sp_plain_dot(A + (size_t)m * lda, W + (size_t)n * K, K) + b;
          if constexpr (!BIAS_INSIDE) v += at_end;
          out[(size_t)m * ldo + n] = add ? old[j] + v : v;
        }
      }
    }
  } else if (lane == 0) {
    int s = 0, phase = 0;
    for (int kb = 0; kb < num_kb; ++kb) {
      if (!issue(kb, s, phase)) break;
      if (++s == STAGES) { s = 0; phase ^= 1; }
    }
  }
  if (splits > 1 && (warp < SP_CONVERT || warp >= SP_CONVERT + SUM)) {
    __syncwarp();
    cluster_sync_all();
    cluster_sync_all();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == SP_CONVERT) tmem_dealloc(tmem_base, 512);
}

// Tokens a tile: what holds them, up to 128.
int sp_token_tile(int M) { return M <= 32 ? 32 : M <= 64 ? 64 : 128; }

// The K range of a tile in as many parts (1, 2 or 4: the cluster's size) as still fit one CTA an SM, at least four blocks of 64 a
// part: 64 tiles (500 tokens, 2,048 output columns) leave more than half of the SMs idle otherwise (K = 8,192: 224 us whole,
// 122 us in two parts).  Eight parts lose: one CTA adds seven others' sums (16 tiles, K = 8,192: 90 us against 70 in four).
int sp_parts(int M, int N, int K) {
  const int bt = sp_token_tile(M), tiles = ((N + 127) / 128) * ((M + bt - 1) / bt), total_kb = (K + SP_BK - 1) / SP_BK;
  int parts = 1;
  while (parts < 4 && tiles * parts * 2 <= rl_num_sms() && total_kb / (parts * 2) >= 4) parts *= 2;
  return parts;
}

template <int BT>
int sp_launch(const float* A, const float* W, const float* bias, float* out, int add, int M, int N, int K, int lda, int ldo, int* err,
              int parts, int kb_per_part, cudaStream_t stream) {
  static const cudaError_t e0 = cudaFuncSetAttribute(gemm_f32_split_kernel<BT>, cudaFuncAttributeMaxDynamicSharedMemorySize, sp_smem<BT>());
  RL_REQUIRE(e0 == cudaSuccess, "rl_gemm_f32_split: cannot reserve %d bytes of shared memory: %s", sp_smem<BT>(), cudaGetErrorString(e0));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(parts * ((M + BT - 1) / BT), (N + 127) / 128);
  cfg.blockDim = dim3(sp_threads<BT>());
  cfg.dynamicSmemBytes = sp_smem<BT>();
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = parts;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = parts > 1 ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_f32_split_kernel<BT>, A, W, bias, out, add, M, N, K, lda, ldo, parts, kb_per_part, err);
  if (e != cudaSuccess) {
    rl_set_error("rl_gemm_f32_split: launch failed (%d parts): %s", parts, cudaGetErrorString(e));
    return RL_ERR_CUDA;
  }
  return RL_OK;
}

}  // namespace

// 1 where the split product is taken instead of the CUDA cores: rows that 16-byte pieces can fetch, a tile's width of outputs, sums from
// K = 256 on, where it is twice as exact as the ordered sum (1.1e-7 against 2.2e-7 of the result's rms; K = 64: 1.1e-7 against 1.4e-7), and more than 8 tokens (up to there gemm_f32_few.cu: see there).
extern "C" int rl_gemm_f32_split_supported(const void* A, const void* W, int M, int N, int K, int lda) {
  return M > 8 && N >= 128 && K >= 256 && K % 4 == 0 && lda % 4 == 0 && lda >= K && (((uintptr_t)A | (uintptr_t)W) & 15) == 0 &&
         (N + 127) / 128 <= 65535;
}

// A: float [M, K], row stride lda; W: float [N, K] contiguous; out: float [M, N], row stride ldo; add != 0: added into out.
// err: device int, set non-zero if a bounded wait inside the kernel ran out.  force_parts: 0 = by the rule above; 1, 2, 4, 8.
extern "C" int rl_gemm_f32_split(const float* A, const float* W, const float* bias, float* out, int add, int M, int N, int K, int lda,
                                 int ldo, int* err, int force_parts, cudaStream_t stream) {
  RL_REQUIRE(M > 0 && N > 0 && K > 0 && K % 4 == 0 && lda % 4 == 0 && lda >= K && ldo >= N && (((uintptr_t)A | (uintptr_t)W) & 15) == 0,
             "rl_gemm_f32_split: operands not supported (M=%d N=%d K=%d lda=%d ldo=%d)", M, N, K, lda, ldo);
  RL_REQUIRE((N + 127) / 128 <= 65535 && err != nullptr, "rl_gemm_f32_split: too many rows of the weight, or null error word");
  RL_REQUIRE(force_parts == 0 || force_parts == 1 || force_parts == 2 || force_parts == 4 || force_parts == 8,
             "rl_gemm_f32_split: the number of K parts must be 1, 2, 4 or 8 (0: chosen from the shapes), got %d", force_parts);
  const int total_kb = (K + SP_BK - 1) / SP_BK;
  int parts = force_parts ? force_parts : sp_parts(M, N, K);
  while (parts > 1 && (parts - 1) * ((total_kb + parts - 1) / parts) >= total_kb) parts /= 2;       // every part has a block
  const int per = (total_kb + parts - 1) / parts;
  switch (sp_token_tile(M)) {
    case 32: return sp_launch<32>(A, W, bias, out, add, M, N, K, lda, ldo, err, parts, per, stream);
    case 64: return sp_launch<64>(A, W, bias, out, add, M, N, K, lda, ldo, err, parts, per, stream);
    default: return sp_launch<128>(A, W, bias, out, add, M, N, K, lda, ldo, err, parts, per, stream);
  }
}
