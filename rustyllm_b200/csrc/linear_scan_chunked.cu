// The linear recurrences of linear_scan.cu's modes 0 and 1 over many tokens, by chunks of 64:
//
//   S_t = a_t S_{t-1} + b_t k_t v_t^T,  o_t = S_t^T q_t (+ skip_h v_t)
//
// With L_i the sum of log a over a chunk's tokens up to i and S the state in front of the chunk,
//   o_i  = exp(L_i) S^T q_i + sum_{j <= i} (q_i . k_j) exp(L_i - L_j) b_j v_j (+ skip v_i)
//   S'   = exp(L_end) S + sum_j exp(L_end - L_j) b_j k_j v_j^T
// so what a chunk adds to the state (first kernel) and its outputs (third) are products of float matrices, for every chunk and head at
// once, and only the small second kernel walks from chunk to chunk.
//
// What bounds it: multiply-adds on the CUDA cores (about 2.7 M a chunk and head of 128 x 128), where the token-by-token walk is
// bound by the latency of its chain: 2,048 tokens of 16 heads of 128 x 128: 128 us against 637; 32 heads of 128 x 64: 129 against 606.  Everything
// behind the loads is 32-bit as there; sums of logarithms are 64-bit, so that exp(L_i - L_j) is as exact for late tokens of a chunk as for early
// ones.  Outputs of a position depend on where chunks begin, that is on how a sequence was cut into steps, to rounding.  Error against 64 bits
// relative to the outputs' rms: 0.8e-7 to 1.8e-7, the walk's 0.7e-7 to 6.7e-7 (tests/test_kernels_gpu.py).
//
// Logarithms are for decays that fade: a in [0, 1], as every trained model's (mode 1 gives no others).  A head of mode 0 whose decay
// lies outside (below 0; beyond 1, where exp(L_i - L_j) would leave float's range before the recurrence does; no number) is walked
// token by token in the second kernel, with the walk's bits, and left out of the other two.
#include <math.h>

#include "common.cuh"

namespace {

constexpr int CH = 64;             // tokens a chunk
constexpr int CH_THREADS = 256;    // 16 x 16 threads over a product's tile

struct ChunkArgs {
  const void *q, *k, *v, *dt_raw;
  int ldq, ldk, ldv, lddt;
  const float *dt_bias, *rate, *skip;
  int mode, act;
  const int *cu_seqlens, *seq_slots;
  int num_seqs;
  float* state;
  long long state_stride;
  float *out, *work, *decay;       // work: [chunks, H, dv, dk], what a chunk adds to the state, then the state in front of it; decay: [chunks, H]
  int ldo, H, hpg;
};

// as linear_scan.cu: accurate in a 32-bit run, with the fast exponential and division in a bfloat16 run
__device__ __forceinline__ float ch_silu(float z, float) { return z / (1.0f + expf(-z)); }
__device__ __forceinline__ float ch_silu(float z, __nv_bfloat16) { return __fdividef(z, 1.0f + __expf(-z)); }
__device__ __forceinline__ float4 ch_ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 ch_ld4(const __nv_bfloat16* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
}
template <typename T>
__device__ __forceinline__ float4 ch_value(float4 x, int act) {
  if (act) x = make_float4(ch_silu(x.x, T()), ch_silu(x.y, T()), ch_silu(x.z, T()), ch_silu(x.w, T()));
  return x;
}
// Rows t0 .. t0 + nt of [., ld] (zeros behind) as 64 rows of W values in registers, four neighbouring ones a piece, all pieces of a thread
// on their way at once; piece p is row `row(p)`, values `col(p)` .. + 3.
template <typename T, int W>
struct ChRows {
  static constexpr int PIECES = CH * W / 4 / CH_THREADS;
  float4 x[PIECES];
  static __device__ __forceinline__ int row(int p) { return (int)(threadIdx.x + p * CH_THREADS) / (W / 4); }
  static __device__ __forceinline__ int col(int p) { return (int)(threadIdx.x + p * CH_THREADS) % (W / 4) * 4; }
  __device__ __forceinline__ void load(const T* base, int ld, int t0, int nt) {
#pragma unroll
    for (int p = 0; p < PIECES; ++p)
      x[p] = row(p) < nt ? ch_ld4(base + (size_t)(t0 + row(p)) * ld + col(p)) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
};

// chunk `index` of the step: its sequence, first token and number of tokens; false: there is none
__device__ __forceinline__ bool ch_find(const ChunkArgs& a, int index, int& t0, int& nt) {
  for (int b = 0; b < a.num_seqs; ++b) {
    const int lo = a.cu_seqlens[b], n = a.cu_seqlens[b + 1] - lo, chunks = (n + CH - 1) / CH;
    if (index < chunks) {
      t0 = lo + index * CH;
      nt = min(CH, n - index * CH);
      return true;
    }
    index -= chunks;
  }
  return false;
}

// whether the head's decays are taken by their logarithms
__device__ __forceinline__ bool ch_fades(const ChunkArgs& a, int h) { return a.mode || (a.rate[h] >= 0.f && a.rate[h] <= 1.f); }

// The chunk's sums of log a (64-bit) and step sizes b, by the first warp: two tokens a lane
template <typename T>
__device__ __forceinline__ void ch_decays(const ChunkArgs& a, int h, int t0, int nt, double* L, float* bsize) {
  if (threadIdx.x >= 32) return;
  const int lane = threadIdx.x;
  double la[2];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int i = 2 * lane + e;
    la[e] = 0.0;
    float b = 0.f;
    if (i < nt) {
      if (a.mode) {
        const float z = rl_ld((const T*)a.dt_raw + (size_t)(t0 + i) * a.lddt + h) + a.dt_bias[h];
        b = z > 20.0f ? z : log1pf(expf(z));
        const float l = -expf(a.rate[h]) * b;
        la[e] = l < -1e4f ? -1e4f : l;                 // exp(-1e4) is 0, and a difference of two such sums is no NaN
      } else {
        b = 1.f;
        const double l = log((double)a.rate[h]);
        la[e] = l < -1e4 ? -1e4 : l;
      }
    }
    bsize[i] = b;
  }
  double sum = la[0] + la[1];
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double other = __shfl_up_sync(0xffffffffu, sum, o);
    if (lane >= o) sum += other;
  }
  L[2 * lane] = sum - la[1];
  L[2 * lane + 1] = sum;
}

// ---------------- what a chunk adds to the state: U[c][n] = sum_j v_j[c] w_j k_j[n], w_j = exp(L_end - L_j) b_j ----------------
template <typename T, int DK, int DV>
__global__ void __launch_bounds__(CH_THREADS) chunk_add_kernel(const ChunkArgs a) {
  extern __shared__ __align__(16) float ch_smem[];
  float* Ks = ch_smem;                       // [CH][DK], weighted
  float* Vs = ch_smem + CH * DK;             // [CH][DV]
  __shared__ double L[CH];
  __shared__ float bsize[CH], weight[CH];
  rl_pdl_trigger();
  rl_pdl_wait();
  const int h = blockIdx.x, tid = threadIdx.x;
  int t0, nt;
  if (!ch_fades(a, h) || !ch_find(a, blockIdx.y, t0, nt)) return;
  const T *k = (const T*)a.k + (size_t)(h / a.hpg) * DK, *v = (const T*)a.v + (size_t)h * DV;
  ChRows<T, DK> kr;
  ChRows<T, DV> vr;
  kr.load(k, a.ldk, t0, nt);                 // on their way while the decays are summed
  vr.load(v, a.ldv, t0, nt);
  ch_decays<T>(a, h, t0, nt, L, bsize);
  __syncthreads();
  if (tid < CH) weight[tid] = tid < nt ? expf((float)(L[nt - 1] - L[tid])) * bsize[tid] : 0.f;
  if (tid == 0) a.decay[(size_t)blockIdx.y * a.H + h] = expf((float)L[nt - 1]);
  __syncthreads();
#pragma unroll
  for (int p = 0; p < ChRows<T, DK>::PIECES; ++p) {
    const float4 x = ch_value<T>(kr.x[p], a.act);
    const float w = weight[kr.row(p)];
    *reinterpret_cast<float4*>(Ks + kr.row(p) * DK + kr.col(p)) = make_float4(x.x * w, x.y * w, x.z * w, x.w * w);
  }
#pragma unroll
  for (int p = 0; p < ChRows<T, DV>::PIECES; ++p)
    *reinterpret_cast<float4*>(Vs + vr.row(p) * DV + vr.col(p)) = ch_value<T>(vr.x[p], a.act);
  __syncthreads();
  constexpr int NN = DK / 64, NCc = DV / 64;           // runs of four n and of four c a thread, 64 apart
  const int tx = tid & 15, ty = tid >> 4;
  float acc[NCc][4][NN][4];
#pragma unroll
  for (int i = 0; i < NCc * 4 * NN * 4; ++i) (&acc[0][0][0][0])[i] = 0.f;
#pragma unroll 4
  for (int j = 0; j < nt; ++j) {
    float kk[NN][4], vv[NCc][4];
#pragma unroll
    for (int s = 0; s < NN; ++s) {
      const float4 x = *reinterpret_cast<const float4*>(Ks + j * DK + 64 * s + 4 * tx);
      kk[s][0] = x.x; kk[s][1] = x.y; kk[s][2] = x.z; kk[s][3] = x.w;
    }
#pragma unroll
    for (int s = 0; s < NCc; ++s) {
      const float4 x = *reinterpret_cast<const float4*>(Vs + j * DV + 64 * s + 4 * ty);
      vv[s][0] = x.x; vv[s][1] = x.y; vv[s][2] = x.z; vv[s][3] = x.w;
    }
#pragma unroll
    for (int s = 0; s < NCc; ++s)
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int u = 0; u < NN; ++u)
#pragma unroll
          for (int f = 0; f < 4; ++f) acc[s][e][u][f] = fmaf(kk[u][f], vv[s][e], acc[s][e][u][f]);
  }
  float* U = a.work + ((size_t)blockIdx.y * a.H + h) * DK * DV;
#pragma unroll
  for (int s = 0; s < NCc; ++s)
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
      for (int u = 0; u < NN; ++u)
        *reinterpret_cast<float4*>(U + (size_t)(64 * s + 4 * ty + e) * DK + 64 * u + 4 * tx) =
            make_float4(acc[s][e][u][0], acc[s][e][u][1], acc[s][e][u][2], acc[s][e][u][3]);
}

// Four consecutive rows of a column of a head's state over a sequence's tokens, DK / 4 neighbouring lanes a column: the order of every
// sum is the walk's (linear_scan.cu, its shape for many tokens), so are the bits.  Eight tokens' values are on their way at once.
template <typename T, int DK, int DV>
__device__ __noinline__ void ch_walk_tokens(const ChunkArgs& a, int b, int h, int at) {
  constexpr int R = DK / 4, AHEAD = 8;
  const int col = at / DK, row = at % DK;
  const T *q = (const T*)a.q + (size_t)(h / a.hpg) * DK + row, *k = (const T*)a.k + (size_t)(h / a.hpg) * DK + row;
  const T* v = (const T*)a.v + (size_t)h * DV + col;
  float* st = a.state + (size_t)a.seq_slots[b] * a.state_stride + (size_t)h * DK * DV + at;
  const float decay = a.rate[h], skip = a.skip ? a.skip[h] : 0.f;
  float4 S = *reinterpret_cast<const float4*>(st);
  const int hi = a.cu_seqlens[b + 1];
  for (int t0 = a.cu_seqlens[b]; t0 < hi; t0 += AHEAD) {
    float4 qq[AHEAD], kk[AHEAD];
    float vv[AHEAD];
#pragma unroll
    for (int i = 0; i < AHEAD; ++i) {
      const size_t t = min(t0 + i, hi - 1);
      qq[i] = ch_ld4(q + t * a.ldq);
      kk[i] = ch_ld4(k + t * a.ldk);
      vv[i] = rl_ld(v + t * a.ldv);
    }
#pragma unroll
    for (int i = 0; i < AHEAD; ++i) {
      if (t0 + i >= hi) break;
      const float4 x = ch_value<T>(qq[i], a.act), y = ch_value<T>(kk[i], a.act);
      const float z = a.act ? ch_silu(vv[i], T()) : vv[i];
      S = make_float4(fmaf(decay, S.x, z * y.x), fmaf(decay, S.y, z * y.y), fmaf(decay, S.z, z * y.z), fmaf(decay, S.w, z * y.w));
      float p = fmaf(S.w, x.w, fmaf(S.z, x.z, fmaf(S.y, x.y, fmaf(S.x, x.x, 0.f))));
#pragma unroll
      for (int o = 1; o < R; o <<= 1) p += __shfl_xor_sync(0xffffffffu, p, o);
      if (row == 0) a.out[(size_t)(t0 + i) * a.ldo + (size_t)h * DV + col] = p + skip * z;
    }
  }
  *reinterpret_cast<float4*>(st) = S;
}

// ---------------- the walk: the state in front of every chunk in place of what the chunk adds ----------------
template <typename T, int DK, int DV>
__global__ void __launch_bounds__(256) chunk_walk_kernel(const __grid_constant__ ChunkArgs a) {
  rl_pdl_trigger();
  rl_pdl_wait();
  constexpr int size = DK * DV;
  static_assert(size % 1024 == 0, "a block's 256 threads hold four elements each");
  const int b = blockIdx.x, h = blockIdx.y, at = ((int)blockIdx.z * 256 + (int)threadIdx.x) * 4;
  if (!ch_fades(a, h)) {
    ch_walk_tokens<T, DK, DV>(a, b, h, at);
    return;
  }
  int first = 0;
  for (int i = 0; i < b; ++i) first += (a.cu_seqlens[i + 1] - a.cu_seqlens[i] + CH - 1) / CH;
  const int chunks = (a.cu_seqlens[b + 1] - a.cu_seqlens[b] + CH - 1) / CH;
  float* st = a.state + (size_t)a.seq_slots[b] * a.state_stride + (size_t)h * size + at;
  float4 S = *reinterpret_cast<const float4*>(st);
  float* u = a.work + ((size_t)first * a.H + h) * size + at;
  const float* d = a.decay + (size_t)first * a.H + h;
  const size_t step = (size_t)a.H * size;
  constexpr int AHEAD = 8;                   // chunks on their way
  float4 x[AHEAD];
  float w[AHEAD];
#pragma unroll
  for (int i = 0; i < AHEAD; ++i)
    if (i < chunks) { x[i] = *reinterpret_cast<const float4*>(u + i * step); w[i] = d[(size_t)i * a.H]; }
  for (int c0 = 0; c0 < chunks; c0 += AHEAD) {
#pragma unroll
    for (int i = 0; i < AHEAD; ++i) {
      const int c = c0 + i;
      if (c >= chunks) break;
      const float4 add = x[i];
      const float dc = w[i];
      if (c + AHEAD < chunks) { x[i] = *reinterpret_cast<const float4*>(u + (size_t)(c + AHEAD) * step); w[i] = d[(size_t)(c + AHEAD) * a.H]; }
      *reinterpret_cast<float4*>(u + (size_t)c * step) = S;
      S = make_float4(fmaf(dc, S.x, add.x), fmaf(dc, S.y, add.y), fmaf(dc, S.z, add.z), fmaf(dc, S.w, add.w));
    }
  }
  *reinterpret_cast<float4*>(st) = S;
}

// rows (row0 + ty + 16 r) of X against rows (tx + 16 s) of Y, both [., D + 4] in shared memory, summed in runs of 32
template <int D, int R, int S>
__device__ __forceinline__ void ch_dots(const float* X, const float* Y, int tx, int ty, float (&acc)[R][S]) {
  constexpr int LD = D + 4;
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int s = 0; s < S; ++s) acc[r][s] = 0.f;
  for (int n0 = 0; n0 < D; n0 += 32) {
    float part[R][S];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int s = 0; s < S; ++s) part[r][s] = 0.f;
#pragma unroll
    for (int n = 0; n < 32; n += 4) {
      float4 y[S];
#pragma unroll
      for (int s = 0; s < S; ++s) y[s] = *reinterpret_cast<const float4*>(Y + (tx + 16 * s) * LD + n0 + n);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float4 x = *reinterpret_cast<const float4*>(X + (ty + 16 * r) * LD + n0 + n);
#pragma unroll
        for (int s = 0; s < S; ++s) {
          part[r][s] = fmaf(x.x, y[s].x, part[r][s]);
          part[r][s] = fmaf(x.y, y[s].y, part[r][s]);
          part[r][s] = fmaf(x.z, y[s].z, part[r][s]);
          part[r][s] = fmaf(x.w, y[s].w, part[r][s]);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int s = 0; s < S; ++s) acc[r][s] += part[r][s];
  }
}

// ---------------- a chunk's outputs ----------------
template <int DK, int DV>
constexpr int ch_out_smem() { return (CH * (DK + 4) + CH * ((DK > DV ? DK : DV) + 4) + CH * (CH + 4)) * 4; }

template <typename T, int DK, int DV>
__global__ void __launch_bounds__(CH_THREADS, 2) chunk_out_kernel(const ChunkArgs a) {
  extern __shared__ __align__(16) float ch_smem[];
  constexpr int LQ = DK + 4, LA = CH + 4;
  float* Qs = ch_smem;                                            // [CH][LQ]
  float* X = ch_smem + CH * LQ;                                   // keys [CH][LQ], then values [CH][DV], then 64 columns of the state [64][LQ]
  float* As = X + CH * ((DK > DV ? DK : DV) + 4);                 // [CH][LA]: row i, column j
  __shared__ double L[CH];
  __shared__ float bsize[CH];
  rl_pdl_trigger();
  rl_pdl_wait();
  const int h = blockIdx.x, tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  int t0, nt;
  if (!ch_fades(a, h) || !ch_find(a, blockIdx.y, t0, nt)) return;
  const T *q = (const T*)a.q + (size_t)(h / a.hpg) * DK, *k = (const T*)a.k + (size_t)(h / a.hpg) * DK, *v = (const T*)a.v + (size_t)h * DV;
  {
    ChRows<T, DK> qr, kr;
    qr.load(q, a.ldq, t0, nt);               // on their way while the decays are summed
    kr.load(k, a.ldk, t0, nt);
    ch_decays<T>(a, h, t0, nt, L, bsize);
#pragma unroll
    for (int p = 0; p < ChRows<T, DK>::PIECES; ++p) {
      *reinterpret_cast<float4*>(Qs + qr.row(p) * LQ + qr.col(p)) = ch_value<T>(qr.x[p], a.act);
      *reinterpret_cast<float4*>(X + kr.row(p) * LQ + kr.col(p)) = ch_value<T>(kr.x[p], a.act);
    }
  }
  __syncthreads();
  {
    float s[4][4];
    ch_dots<DK, 4, 4>(Qs, X, tx, ty, s);
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int i = ty + 16 * r, j = tx + 16 * u;
        As[i * LA + j] = j <= i && i < nt ? s[r][u] * (expf((float)(L[i] - L[j])) * bsize[j]) : 0.f;
      }
  }
  __syncthreads();
  {
    ChRows<T, DV> vr;
    vr.load(v, a.ldv, t0, nt);
#pragma unroll
    for (int p = 0; p < ChRows<T, DV>::PIECES; ++p)
      *reinterpret_cast<float4*>(X + vr.row(p) * DV + vr.col(p)) = ch_value<T>(vr.x[p], a.act);
  }
  __syncthreads();
  // rows ty + 16 r, columns 64 * half + tx + 16 u: what the chunk's own tokens contribute.  Tokens behind a row's are left out, not
  // multiplied by zero: row block r of 16 sees the blocks of tokens in front of it whole and its own up to the row.
  constexpr int HALVES = DV / 64;
  float o[HALVES][4][4];
  const float skip = a.skip ? a.skip[h] : 0.f;
#pragma unroll
  for (int f = 0; f < HALVES; ++f)
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int u = 0; u < 4; ++u) o[f][r][u] = 0.f;
#pragma unroll
  for (int jb = 0; jb < 4; ++jb) {
#pragma unroll 1
    for (int jj = 0; jj < 16; jj += 4) {
      float w[4][4];
#pragma unroll
      for (int r = jb; r < 4; ++r) {
        const float4 x = *reinterpret_cast<const float4*>(As + (ty + 16 * r) * LA + 16 * jb + jj);
        w[r][0] = x.x; w[r][1] = x.y; w[r][2] = x.z; w[r][3] = x.w;
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float* vr = X + (16 * jb + jj + e) * DV + tx;
        const bool own = jj + e <= ty;
#pragma unroll
        for (int f = 0; f < HALVES; ++f)
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const float x = vr[64 * f + 16 * u];
#pragma unroll
            for (int r = jb; r < 4; ++r)
              if (r > jb || own) o[f][r][u] = fmaf(w[r][e], x, o[f][r][u]);
          }
      }
    }
  }
  float scale[4], direct[HALVES][4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int i = ty + 16 * r;
    scale[r] = i < nt ? expf((float)L[i]) : 0.f;
#pragma unroll
    for (int f = 0; f < HALVES; ++f)
#pragma unroll
      for (int u = 0; u < 4; ++u) direct[f][r][u] = skip != 0.f ? skip * X[i * DV + 64 * f + tx + 16 * u] : 0.f;
  }
  const float* S = a.work + ((size_t)blockIdx.y * a.H + h) * DK * DV;
#pragma unroll
  for (int f = 0; f < HALVES; ++f) {
    ChRows<float, DK> sr;
    sr.load(S + (size_t)(64 * f) * DK, DK, 0, 64);
    __syncthreads();                                              // the values, or the columns in front, have been read
#pragma unroll
    for (int p = 0; p < ChRows<float, DK>::PIECES; ++p) *reinterpret_cast<float4*>(X + sr.row(p) * LQ + sr.col(p)) = sr.x[p];
    __syncthreads();
    float s[4][4];
    ch_dots<DK, 4, 4>(Qs, X, tx, ty, s);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = ty + 16 * r;
      if (i >= nt) continue;
#pragma unroll
      for (int u = 0; u < 4; ++u)
        a.out[(size_t)(t0 + i) * a.ldo + (size_t)h * DV + 64 * f + tx + 16 * u] = fmaf(scale[r], s[r][u], o[f][r][u]) + direct[f][r][u];
    }
  }
}

template <typename T, int DK, int DV>
int ch_launch(const ChunkArgs& a, int chunks, cudaStream_t stream) {
  constexpr int add_smem = CH * (DK + DV) * 4, out_smem = ch_out_smem<DK, DV>();
  static const cudaError_t e0 = cudaFuncSetAttribute(chunk_add_kernel<T, DK, DV>, cudaFuncAttributeMaxDynamicSharedMemorySize, add_smem);
  static const cudaError_t e1 = cudaFuncSetAttribute(chunk_out_kernel<T, DK, DV>, cudaFuncAttributeMaxDynamicSharedMemorySize, out_smem);
  RL_REQUIRE(e0 == cudaSuccess && e1 == cudaSuccess, "rl_linear_scan_chunked: cannot reserve %d and %d bytes of shared memory", add_smem, out_smem);
  rl_launch_pdl(chunk_add_kernel<T, DK, DV>, dim3(a.H, chunks), dim3(CH_THREADS), (size_t)add_smem, stream, a);
  rl_launch_pdl(chunk_walk_kernel<T, DK, DV>, dim3(a.num_seqs, a.H, DK * DV / 1024), dim3(256), 0, stream, a);
  rl_launch_pdl(chunk_out_kernel<T, DK, DV>, dim3(a.H, chunks), dim3(CH_THREADS), (size_t)out_smem, stream, a);
  RL_LAUNCH_CHECK("rl_linear_scan_chunked");
  return RL_OK;
}

template <typename T>
int ch_dispatch(const ChunkArgs& a, int chunks, int dk, int dv, cudaStream_t stream) {
  if (dk == 64) return dv == 64 ? ch_launch<T, 64, 64>(a, chunks, stream) : ch_launch<T, 64, 128>(a, chunks, stream);
  return dv == 64 ? ch_launch<T, 128, 64>(a, chunks, stream) : ch_launch<T, 128, 128>(a, chunks, stream);
}

constexpr long long CH_WORK_LIMIT = 768LL << 20;       // bytes of work a call may take

}  // namespace

// Chunks that the chunked form of a step of num_tokens tokens is launched for (its work: chunks * heads * (dk * dv + 1) floats), or 0 where the
// form does not take the step: state widths other than 64 and 128, rows that pieces of four elements cannot fetch, fewer than 256 tokens or 32
// a sequence (16 heads of 128 x 128, one sequence, walk / chunks: 128 tokens 43 / 59 us, 256 tokens 83 / 56), or more work than 768 MiB (some
// 24,000 tokens of 32 such heads).  Whether a step that it takes is worth it is for the caller (scan_chunks_pay in kernels.py).
extern "C" int rl_linear_scan_chunks(const void* q, int ldq, const void* k, int ldk, const void* v, int ldv, int dtype, const void* state,
                                     long long state_stride, int num_tokens, int num_seqs, int num_heads, int dk, int dv) {
  if ((dk != 64 && dk != 128) || (dv != 64 && dv != 128) || num_seqs <= 0 || num_tokens < 256 || num_tokens < 32LL * num_seqs) return 0;
  const uintptr_t mask = dtype == RL_F32 ? 15 : 7;
  if ((((uintptr_t)q | (uintptr_t)k | (uintptr_t)v) & mask) || ldq % 4 || ldk % 4 || ldv % 4) return 0;
  if (((uintptr_t)state & 15) || state_stride % 4) return 0;
  const long long chunks = num_tokens / CH + num_seqs;
  return chunks <= 65535 && chunks * num_heads * ((long long)dk * dv + 1) * 4 <= CH_WORK_LIMIT ? (int)chunks : 0;
}

// As rl_linear_scan; work: see rl_linear_scan_chunks, 16-byte aligned.
extern "C" int rl_linear_scan_chunked(const void* q, int ldq, const void* k, int ldk, const void* v, int ldv, const void* dt_raw, int lddt, int dtype,
                                      const float* dt_bias, const float* rate, const float* skip, int mode, int act, const int* cu_seqlens,
                                      const int* seq_slots, int num_seqs, float* state, long long state_stride, float* out, int ldo, int num_tokens,
                                      int num_heads, int heads_per_group, int dk, int dv, float* work, cudaStream_t stream) {
  RL_REQUIRE(num_seqs > 0 && num_seqs <= 65535 && num_heads > 0 && num_heads <= 65535 && heads_per_group > 0 && num_heads % heads_per_group == 0,
             "rl_linear_scan_chunked: bad sizes");
  const int chunks = rl_linear_scan_chunks(q, ldq, k, ldk, v, ldv, dtype, state, state_stride, num_tokens, num_seqs, num_heads, dk, dv);
  RL_REQUIRE(chunks > 0, "rl_linear_scan_chunked: operands not supported (%d tokens of %d sequences, %d x %d)", num_tokens, num_seqs, dk, dv);
  RL_REQUIRE(mode == 0 || (mode == 1 && dt_raw != nullptr && dt_bias != nullptr), "rl_linear_scan_chunked: mode %d, or no step sizes", mode);
  RL_REQUIRE(rate != nullptr && state != nullptr && work != nullptr && ((uintptr_t)work & 15) == 0,
             "rl_linear_scan_chunked: no decay, no state, or no work on a 16-byte boundary");
  ChunkArgs a = {q, k, v, dt_raw, ldq, ldk, ldv, lddt, dt_bias, rate, skip, mode, act, cu_seqlens, seq_slots, num_seqs, state, state_stride,
                 out, work, work + (size_t)chunks * num_heads * dk * dv, ldo, num_heads, heads_per_group};
  if (dtype == RL_F32) return ch_dispatch<float>(a, chunks, dk, dv, stream);
  RL_REQUIRE(dtype == RL_BF16, "rl_linear_scan_chunked: unknown dtype %d", dtype);
  return ch_dispatch<__nv_bfloat16>(a, chunks, dk, dv, stream);
}
