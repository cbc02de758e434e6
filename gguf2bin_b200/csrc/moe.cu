// A routed feed-forward: every token goes through `top` of a layer's small feed-forwards.
//
//   moe_route    logits z (+ a bias per expert); scores s = softmax(z) over all experts (or sigmoid(z), each by itself) in 32-bit;
//                optionally only the experts of the best groups of neighbours stay eligible; the `top` largest of s + c
//                (c: a stored correction that steers the choice only) are chosen, ties to the
//                lower index; the weights are the chosen experts' s as they are, or divided by
//                their sum; then times `scale`.  idx [T, top], weight [T, top].
//   moe_plan     the step's (token, choice) pairs grouped by expert: how many rows every expert
//                gets, where its rows start, which pair sits in which row, and the list of row
//                tiles that the products walk.  Experts from `n_real` on have no matrices (their
//                output is their input); their pairs get no row.
//   moe_gemm     one product per expert over its rows: out = A_rows . W_e^T, the rows of A
//                gathered by the plan; with `swiglu` W_e holds gate rows then up rows and the
//                output is the gate of glu.cuh (silu(gate) * up, the
//                capped gate, ...).  32-bit accumulation; a row's sum runs over k in
//                ascending order whatever else is in the tile.
//   moe_combine  y_t = sum_j weight_tj * (row of pair (t, j), or the token's own input for an
//                expert without matrices), added in the order of j; stored, or added to what is there.
//
// Which row of an expert's range a pair lands in depends on the batch (the plan hands rows out
// with atomic counters); what is computed for the pair does not: a row of a product depends on
// that row alone, and the combination adds a token's choices in the order of the choice.
#include "common.cuh"
#include "glu.cuh"
#include "join.cuh"
#include "mma.cuh"

G2B_DEFINE_LAST_ERROR

// Row of a gate/up matrix [2N, K] that holds gate (s = 0) or up (s = 1) row n: all gates and then all ups
// (`blocked` = 0), or eight gates and the eight ups of the same outputs in turn (`blocked` = 1, the
// layout whose neighbours a tensor-core epilogue combines).  Plain matrices pass s = 0, blocked = 0.
__device__ __forceinline__ size_t gu_row(int s, int n, int N, int blocked) {
  return blocked ? (size_t)((n >> 3) << 4) + (s << 3) + (n & 7) : (size_t)s * N + n;
}

// rows gathered side by side, in the plan's order, for the kernels that fetch tiles by address
template <typename T>
__global__ void __launch_bounds__(256)
moe_gather_kernel(const T *__restrict__ A, int a_stride, const int *__restrict__ row_pair, int pairs_per_token,
                  const int *__restrict__ plan, int n_real, int K, T *__restrict__ out) {
  pdl_launch();
  pdl_wait();
  const int r = blockIdx.x;
  if (r >= plan[1 + n_real]) return;
  const T *src = A + (size_t)(row_pair[r] / pairs_per_token) * a_stride;
  T *dst = out + (size_t)r * K;
  if ((K * sizeof(T)) % 16 == 0 && (a_stride * sizeof(T)) % 16 == 0) {
    const int n16 = K * (int)sizeof(T) / 16;
    for (int i = threadIdx.x; i < n16; i += blockDim.x) ((uint4 *)dst)[i] = ((const uint4 *)src)[i];
  } else {
    for (int i = threadIdx.x; i < K; i += blockDim.x) dst[i] = src[i];
  }
}

extern "C" int g2b_moe_gather(const void *A, int dtype, int a_stride, const int *row_pair, int pairs_per_token,
                              const int *plan, int n_real, int n_rows, int K, void *out, cudaStream_t stream) {
  if (n_rows <= 0) return 0;
  if (dtype == G2B_F32)
    g2b_launch(moe_gather_kernel<float>, dim3(n_rows), dim3(256), 0, stream, (const float *)A, a_stride, row_pair,
               pairs_per_token, plan, n_real, K, (float *)out);
  else if (dtype == G2B_BF16)
    g2b_launch(moe_gather_kernel<bf16>, dim3(n_rows), dim3(256), 0, stream, (const bf16 *)A, a_stride, row_pair,
               pairs_per_token, plan, n_real, K, (bf16 *)out);
  else
    G2B_REFUSE("moe_gather: unknown dtype %d", dtype);
  return g2b_check_launch("moe_gather");
}

// ---------------------------------------------------------------------------
// router
// ---------------------------------------------------------------------------
#define ROUTE_WARPS 4
// `sigmoid`: the scores are sigmoids of the logits, each by itself, instead of a softmax over all.
// `groups` > 1: the experts form that many equal groups of neighbours; a group's score is the sum of its
// two largest scores (of score + correction); only experts of the `keep` best groups can be chosen.
struct Route {
  const float *z, *correction, *bias;
  int T, N, top, renormalise, sigmoid, groups, keep;
  int *idx;
  float *weight, scale;
};
// One warp chooses token t's experts; `s`: 2 N + groups floats of shared memory (scores, what is picked from, group scores).
__device__ __forceinline__ void route_token(const Route &a, int t, float *s) {
  const float *z = a.z, *correction = a.correction, *bias = a.bias;
  const int N = a.N, top = a.top, renormalise = a.renormalise, sigmoid = a.sigmoid, groups = a.groups, keep = a.keep;
  int *idx = a.idx;
  float *weight = a.weight;
  const float scale = a.scale;
  const int lane = threadIdx.x & 31;
  float *pick = s + N, *gs = pick + N;
  const float *zr = z + (size_t)t * N;
  if (sigmoid) {
    for (int j = lane; j < N; j += 32) {
      s[j] = 1.f / (1.f + expf(-(zr[j] + (bias ? bias[j] : 0.f))));
      pick[j] = s[j] + (correction ? correction[j] : 0.f);
    }
  } else {
    float m = -INFINITY;
    for (int j = lane; j < N; j += 32) {
      s[j] = zr[j] + (bias ? bias[j] : 0.f);
      m = fmaxf(m, s[j]);
    }
    m = warp_max(m);
    float sum = 0.f;
    for (int j = lane; j < N; j += 32) {
      const float e = expf(s[j] - m);
      s[j] = e;
      sum += e;
    }
    sum = warp_sum(sum);
    const float inv = 1.f / sum;
    for (int j = lane; j < N; j += 32) {
      s[j] *= inv;
      pick[j] = s[j] + (correction ? correction[j] : 0.f);
    }
  }
  __syncwarp();
  if (groups > 1) {
    const int per = N / groups;
    for (int g = lane; g < groups; g += 32) {     // the sum of a group's two best
      float a = -INFINITY, b = -INFINITY;
      for (int j = g * per; j < (g + 1) * per; ++j) {
        const float v = pick[j];
        if (v > a) { b = a; a = v; } else if (v > b) { b = v; }
      }
      gs[g] = per > 1 ? a + b : a;
    }
    __syncwarp();
    for (int r = 0; r < keep; ++r) {              // the best groups, one after another; ties to the lower index
      float best = -INFINITY;
      int at = 0x7fffffff;
      for (int g = lane; g < groups; g += 32)
        if (gs[g] > best) { best = gs[g]; at = g; }
      for (int off = 16; off > 0; off >>= 1) {
        const float ob = __shfl_xor_sync(0xffffffffu, best, off);
        const int oa = __shfl_xor_sync(0xffffffffu, at, off);
        if (ob > best || (ob == best && oa < at)) { best = ob; at = oa; }
      }
      if (at >= groups) break;                    // nothing left (NaN scores): every lane agrees
      if (lane == 0) gs[at] = -INFINITY;          // taken: marked by the value no score has
      __syncwarp();
    }
    for (int j = lane; j < N; j += 32)
      if (gs[j / per] != -INFINITY) pick[j] = -INFINITY;      // its group was not kept
    __syncwarp();
  }
  float chosen_sum = 0.f;
  for (int r = 0; r < top; ++r) {
    float best = -INFINITY;
    int at = 0x7fffffff;
    for (int j = lane; j < N; j += 32)
      if (pick[j] > best) { best = pick[j]; at = j; }
    for (int off = 16; off > 0; off >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, off);
      const int oa = __shfl_xor_sync(0xffffffffu, at, off);
      if (ob > best || (ob == best && oa < at)) { best = ob; at = oa; }
    }
    if (at >= N) at = 0;                        // all NaN: never read outside
    if (lane == 0) {
      idx[(size_t)t * top + r] = at;
      weight[(size_t)t * top + r] = renormalise ? s[at] : s[at] * scale;
      pick[at] = -INFINITY;
    }
    chosen_sum += s[at];
    __syncwarp();
  }
  if (renormalise && lane == 0)
    for (int r = 0; r < top; ++r)
      weight[(size_t)t * top + r] = weight[(size_t)t * top + r] / (chosen_sum + 1e-20f) * scale;
}

__global__ void __launch_bounds__(ROUTE_WARPS * 32)
moe_route_kernel(const Route a) {
  pdl_launch();
  pdl_wait();
  extern __shared__ float sm[];
  const int warp = threadIdx.x >> 5, t = blockIdx.x * ROUTE_WARPS + warp;
  if (t < a.T) route_token(a, t, sm + (size_t)warp * (2 * a.N + a.groups));
}

extern "C" int g2b_moe_route(const float *z, const float *correction, int T, int N, int top, int renormalise,
                             int *idx, float *weight, float scale, int sigmoid, int groups, int keep,
                             const float *bias, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (top < 1 || top > N) G2B_REFUSE("moe_route: %d choices among %d experts", top, N);
  if (groups < 1) groups = 1;
  if (groups > 1 && (N % groups || keep < 1 || keep > groups || top > keep * (N / groups)))
    G2B_REFUSE("moe_route: %d experts in %d groups of which %d are kept, for %d choices", N, groups, keep, top);
  const size_t smem = (size_t)ROUTE_WARPS * (2 * N + groups) * sizeof(float);
  if (smem > 48 * 1024) G2B_REFUSE("moe_route: %d experts are more than a block's shared memory holds", N);
  const Route a = {z, correction, bias, T, N, top, renormalise, sigmoid, groups, keep, idx, weight, scale};
  g2b_launch(moe_route_kernel, dim3((T + ROUTE_WARPS - 1) / ROUTE_WARPS), dim3(ROUTE_WARPS * 32), smem, stream, a);
  return g2b_check_launch("moe_route");
}

// ---------------------------------------------------------------------------
// plan: one block
// ---------------------------------------------------------------------------
#define PLAN_MAX_EXPERTS 1024
// plan layout (int32): [0] tiles in use, [1..E+1] first row of each expert (and the end),
// then the tiles as (expert, first row, rows) triples from word PLAN_TILES_AT(E) on
#define PLAN_TILES_AT(E) ((E) + 2)

__device__ __forceinline__ void make_plan(const int *idx, int n_pairs, int n_real, int tile_rows, int max_tiles, int *plan, int *row_pair,
                                          int *pair_row) {
  __shared__ int count[PLAN_MAX_EXPERTS], start[PLAN_MAX_EXPERTS + 1], cursor[PLAN_MAX_EXPERTS];
  for (int e = threadIdx.x; e < n_real; e += blockDim.x) count[e] = 0;
  __syncthreads();
  for (int p = threadIdx.x; p < n_pairs; p += blockDim.x) {
    const int e = idx[p];
    if (e >= 0 && e < n_real) atomicAdd(&count[e], 1);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int at = 0, tiles = 0;
    int *tl = plan + PLAN_TILES_AT(n_real);
    for (int e = 0; e < n_real; ++e) {
      start[e] = at;
      plan[1 + e] = at;
      for (int r = 0; r < count[e] && tiles < max_tiles; r += tile_rows, ++tiles) {
        tl[3 * tiles + 0] = e;
        tl[3 * tiles + 1] = at + r;
        tl[3 * tiles + 2] = min(tile_rows, count[e] - r);
      }
      at += count[e];
    }
    start[n_real] = at;
    plan[1 + n_real] = at;
    plan[0] = tiles;
  }
  for (int e = threadIdx.x; e < n_real; e += blockDim.x) cursor[e] = 0;
  __syncthreads();
  for (int p = threadIdx.x; p < n_pairs; p += blockDim.x) {
    const int e = idx[p];
    int row = -1;
    if (e >= 0 && e < n_real) {
      row = start[e] + atomicAdd(&cursor[e], 1);
      row_pair[row] = p;
    }
    pair_row[p] = row;
  }
}

__global__ void __launch_bounds__(1024)
moe_plan_kernel(const int *__restrict__ idx, int n_pairs, int n_real, int tile_rows, int max_tiles,
                int *__restrict__ plan, int *__restrict__ row_pair, int *__restrict__ pair_row) {
  pdl_launch();
  pdl_wait();
  make_plan(idx, n_pairs, n_real, tile_rows, max_tiles, plan, row_pair, pair_row);
}

// The few tokens of a decode step: the choice and the plan in one block, a warp a token (one launch instead of two: 5.2 us for
// one token and 18 experts, 4.0 + 2.8 apart; 5.7 for eight and 16, 4.0 + 3.2).
__global__ void __launch_bounds__(1024)
moe_route_plan_kernel(const Route a, int n_real, int tile_rows, int max_tiles, int *plan, int *row_pair, int *pair_row) {
  pdl_launch();
  pdl_wait();
  extern __shared__ float sm[];
  const int warp = threadIdx.x >> 5;
  for (int t = warp; t < a.T; t += blockDim.x >> 5) {
    route_token(a, t, sm + (size_t)warp * (2 * a.N + a.groups));
    __syncwarp();                               // the next token's scores go where this one's were
  }
  __syncthreads();                              // the choices, written to global memory, are seen by the whole block
  make_plan(a.idx, a.T * a.top, n_real, tile_rows, max_tiles, plan, row_pair, pair_row);
}

extern "C" int g2b_moe_plan(const int *idx, int n_pairs, int n_real, int tile_rows, int max_tiles, int *plan,
                            int *row_pair, int *pair_row, cudaStream_t stream) {
  if (n_pairs <= 0) return 0;
  if (n_real < 0 || n_real > PLAN_MAX_EXPERTS) G2B_REFUSE("moe_plan: %d experts outside 0..%d", n_real, PLAN_MAX_EXPERTS);
  g2b_launch(moe_plan_kernel, dim3(1), dim3(1024), 0, stream, idx, n_pairs, n_real, tile_rows, max_tiles, plan, row_pair,
             pair_row);
  return g2b_check_launch("moe_plan");
}

// Both for a step of few tokens whose scores fit one block.
extern "C" int g2b_moe_route_plan(const float *z, const float *correction, int T, int N, int top, int renormalise, int *idx,
                                  float *weight, float scale, int sigmoid, int groups, int keep, const float *bias, int n_real,
                                  int tile_rows, int max_tiles, int *plan, int *row_pair, int *pair_row, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (top < 1 || top > N) G2B_REFUSE("moe_route: %d choices among %d experts", top, N);
  if (groups < 1) groups = 1;
  if (groups > 1 && (N % groups || keep < 1 || keep > groups || top > keep * (N / groups)))
    G2B_REFUSE("moe_route: %d experts in %d groups of which %d are kept, for %d choices", N, groups, keep, top);
  if (n_real < 0 || n_real > PLAN_MAX_EXPERTS) G2B_REFUSE("moe_plan: %d experts outside 0..%d", n_real, PLAN_MAX_EXPERTS);
  const int warps = T < 8 ? 8 : T < 32 ? T : 32;
  const size_t smem = (size_t)warps * (2 * N + groups) * sizeof(float);
  if (smem > 32 * 1024) G2B_REFUSE("moe_route_plan: %d tokens of %d experts are not one block's", T, N);
  const Route a = {z, correction, bias, T, N, top, renormalise, sigmoid, groups, keep, idx, weight, scale};
  g2b_launch(moe_route_plan_kernel, dim3(1), dim3(warps * 32), smem, stream, a, n_real, tile_rows, max_tiles, plan, row_pair, pair_row);
  return g2b_check_launch("moe_route_plan");
}

// ---------------------------------------------------------------------------
// one product per expert over its rows (CUDA cores, any type)
// ---------------------------------------------------------------------------
#define MG_BM 32
#define MG_BN 64
#define MG_BK 16
// 128 threads: thread (ty, tx) = (i / 16, i % 16) owns rows ty*4..+3 and columns tx + 16*j, j < 4

template <typename T, bool SWIGLU>
__global__ void __launch_bounds__(128)
moe_gemm_kernel(const T *__restrict__ A, int a_stride, const int *__restrict__ row_pair, int pairs_per_token,
                const T *__restrict__ W, int N, int K, const int *__restrict__ plan, int n_real,
                void *__restrict__ out, int out_f32, int blocked, GluForm glu) {
  pdl_launch();
  pdl_wait();
  const int tile = blockIdx.y;
  if (tile >= plan[0]) return;
  const int *tl = plan + PLAN_TILES_AT(n_real) + 3 * tile;
  const int e = tl[0], row0 = tl[1], rows = tl[2];
  const int n0 = blockIdx.x * MG_BN;
  __shared__ float As[MG_BK][MG_BM + 1];
  __shared__ float Bs[SWIGLU ? 2 : 1][MG_BK][MG_BN + 1];
  __shared__ int src_row[MG_BM];
  const int tid = threadIdx.x;
  if (tid < MG_BM) {
    int r = -1;
    if (tid < rows) r = row_pair ? row_pair[row0 + tid] / pairs_per_token : row0 + tid;
    src_row[tid] = r;
  }
  __syncthreads();
  const int ty = tid / 16, tx = tid % 16;
  const size_t w_rows = SWIGLU ? 2 * (size_t)N : (size_t)N;
  const T *We = W + (size_t)e * w_rows * K;
  float acc[SWIGLU ? 2 : 1][4][4];
#pragma unroll
  for (int s = 0; s < (SWIGLU ? 2 : 1); ++s)
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[s][i][j] = 0.f;
  for (int k0 = 0; k0 < K; k0 += MG_BK) {
    for (int i = tid; i < MG_BM * MG_BK; i += 128) {
      const int r = i / MG_BK, kk = i % MG_BK;
      const int sr = src_row[r];
      As[kk][r] = (sr >= 0 && k0 + kk < K) ? to_f32(A[(size_t)sr * a_stride + k0 + kk]) : 0.f;
    }
    for (int i = tid; i < MG_BN * MG_BK; i += 128) {
      const int c = i / MG_BK, kk = i % MG_BK;
      const bool in = n0 + c < N && k0 + kk < K;
      Bs[0][kk][c] = in ? to_f32(We[gu_row(0, n0 + c, N, SWIGLU ? blocked : 0) * K + k0 + kk]) : 0.f;
      if (SWIGLU) Bs[1][kk][c] = in ? to_f32(We[gu_row(1, n0 + c, N, blocked) * K + k0 + kk]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < MG_BK; ++kk) {
      float av[4], bv[SWIGLU ? 2 : 1][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) av[i] = As[kk][ty * 4 + i];
#pragma unroll
      for (int s = 0; s < (SWIGLU ? 2 : 1); ++s)
#pragma unroll
        for (int j = 0; j < 4; ++j) bv[s][j] = Bs[s][kk][tx + 16 * j];
#pragma unroll
      for (int s = 0; s < (SWIGLU ? 2 : 1); ++s)
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[s][i][j] = fmaf(av[i], bv[s][j], acc[s][i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = ty * 4 + i;
    if (r >= rows) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = n0 + tx + 16 * j;
      if (c >= N) continue;
      const float v = SWIGLU ? glu_value(acc[0][i][j], acc[SWIGLU ? 1 : 0][i][j], glu) : acc[0][i][j];
      const size_t at = (size_t)(row0 + r) * N + c;
      if (out_f32) ((float *)out)[at] = v;
      else ((T *)out)[at] = from_f32<T>(v);
    }
  }
}

// ---------------------------------------------------------------------------
// the same on the tensor cores (bfloat16, mma.sync m16n8k16): a tile of 32 rows x 64 columns,
// four warps side by side, each 32 x 16
// ---------------------------------------------------------------------------
#define MT_BK 32
#define MT_PAD 8
template <bool SWIGLU>
__global__ void __launch_bounds__(128)
moe_gemm_mma_kernel(const bf16 *__restrict__ A, int a_stride, const int *__restrict__ row_pair, int pairs_per_token,
                    const bf16 *__restrict__ W, int N, int K, const int *__restrict__ plan, int n_real,
                    void *__restrict__ out, int out_f32, int blocked, GluForm glu) {
  pdl_launch();
  pdl_wait();
  const int tile = blockIdx.y;
  if (tile >= plan[0]) return;
  const int *tl = plan + PLAN_TILES_AT(n_real) + 3 * tile;
  const int e = tl[0], row0 = tl[1], rows = tl[2];
  const int n0 = blockIdx.x * MG_BN;
  constexpr int S = SWIGLU ? 2 : 1;
  __shared__ __align__(16) bf16 As[MG_BM][MT_BK + MT_PAD];
  __shared__ __align__(16) bf16 Bs[S][MG_BN][MT_BK + MT_PAD];
  __shared__ int src_row[MG_BM];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid < MG_BM) {
    int r = -1;
    if (tid < rows) r = row_pair ? row_pair[row0 + tid] / pairs_per_token : row0 + tid;
    src_row[tid] = r;
  }
  __syncthreads();
  const bf16 *We = W + (size_t)e * (size_t)S * N * K;
  float acc[S][2][2][4];                        // [gate|up][16-row block][8-column block][fragment]
#pragma unroll
  for (int s = 0; s < S; ++s)
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int f = 0; f < 4; ++f) acc[s][i][j][f] = 0.f;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  for (int k0 = 0; k0 < K; k0 += MT_BK) {       // K is a multiple of 8: 16-byte pieces
    for (int i = tid; i < MG_BM * (MT_BK / 8); i += 128) {
      const int r = i / (MT_BK / 8), p = i % (MT_BK / 8);
      const int sr = src_row[r];
      uint4 v = zero;
      if (sr >= 0 && k0 + p * 8 < K) v = *(const uint4 *)(A + (size_t)sr * a_stride + k0 + p * 8);
      *(uint4 *)&As[r][p * 8] = v;
    }
    for (int i = tid; i < S * MG_BN * (MT_BK / 8); i += 128) {
      const int s = i / (MG_BN * (MT_BK / 8)), c = (i / (MT_BK / 8)) % MG_BN, p = i % (MT_BK / 8);
      uint4 v = zero;
      if (n0 + c < N && k0 + p * 8 < K) v = *(const uint4 *)(We + gu_row(s, n0 + c, N, SWIGLU ? blocked : 0) * K + k0 + p * 8);
      *(uint4 *)&Bs[s][c][p * 8] = v;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < MT_BK; kk += 16) {
      const int g = lane >> 2, q = lane & 3;
      uint32_t a[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        a[i][0] = *(const uint32_t *)&As[16 * i + g][kk + 2 * q];
        a[i][1] = *(const uint32_t *)&As[16 * i + g + 8][kk + 2 * q];
        a[i][2] = *(const uint32_t *)&As[16 * i + g][kk + 2 * q + 8];
        a[i][3] = *(const uint32_t *)&As[16 * i + g + 8][kk + 2 * q + 8];
      }
#pragma unroll
      for (int s = 0; s < S; ++s)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int c = warp * 16 + 8 * j + g;
          uint32_t b[2];
          b[0] = *(const uint32_t *)&Bs[s][c][kk + 2 * q];
          b[1] = *(const uint32_t *)&Bs[s][c][kk + 2 * q + 8];
#pragma unroll
          for (int i = 0; i < 2; ++i) mma_bf16_16816(acc[s][i][j], a[i], b[0], b[1]);
        }
    }
    __syncthreads();
  }
  const int g = lane >> 2, q = lane & 3;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int f = 0; f < 4; ++f) {
        const int r = 16 * i + g + (f >> 1) * 8;
        const int c = n0 + warp * 16 + 8 * j + 2 * q + (f & 1);
        if (r >= rows || c >= N) continue;
        const float v = SWIGLU ? glu_value(acc[0][i][j][f], acc[S - 1][i][j][f], glu) : acc[0][i][j][f];
        const size_t at = (size_t)(row0 + r) * N + c;
        if (out_f32) ((float *)out)[at] = v;
        else ((bf16 *)out)[at] = __float2bfloat16_rn(v);
      }
}

// ---------------------------------------------------------------------------
// many rows per expert: tiles of 128 rows x 64 columns, eight warps (4 x 2, each 32 x 32), operands
// fetched one k-step ahead with cp.async, fragments read with ldmatrix
// ---------------------------------------------------------------------------
#define MW_BM 128
#define MW_BK 32
#define MW_LD (MW_BK + 8)
template <bool SWIGLU>
__global__ void __launch_bounds__(256)
moe_gemm_wide_kernel(const bf16 *__restrict__ A, int a_stride, const int *__restrict__ row_pair, int pairs_per_token,
                     const bf16 *__restrict__ W, int N, int K, const int *__restrict__ plan, int n_real,
                     void *__restrict__ out, int out_f32, int blocked, GluForm glu) {
  pdl_launch();
  pdl_wait();
  constexpr int S = SWIGLU ? 2 : 1;
  __shared__ __align__(16) bf16 As[2][MW_BM][MW_LD];
  __shared__ __align__(16) bf16 Bs[2][S][MG_BN][MW_LD];
  __shared__ int src_row[MW_BM];
  // the plan's tiles are MG_BM rows; this kernel takes MW_BM / MG_BM of them at a time when they follow
  // one another in ONE expert's range: blockIdx.y counts groups of plan tiles, and a group that starts
  // inside an expert's range but is not its first of this size is skipped
  const int per = MW_BM / MG_BM;
  const int tile = blockIdx.y;
  const int n_tiles = plan[0];
  if (tile >= n_tiles) return;
  const int *tl = plan + PLAN_TILES_AT(n_real) + 3 * tile;
  const int e = tl[0], row0 = tl[1];
  const int first = plan[1 + e], end = plan[2 + e];        // the expert's rows
  if ((row0 - first) % MW_BM) return;                      // not the first plan tile of a wide tile
  const int rows = min(MW_BM, end - row0);
  (void)per;
  const int n0 = blockIdx.x * MG_BN;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wm = warp >> 1, wn = warp & 1;
  if (tid < MW_BM) {
    int r = -1;
    if (tid < rows) r = row_pair ? row_pair[row0 + tid] / pairs_per_token : row0 + tid;
    src_row[tid] = r;
  }
  __syncthreads();
  const bf16 *We = W + (size_t)e * (size_t)S * N * K;
  float acc[S][2][4][4];
#pragma unroll
  for (int s = 0; s < S; ++s)
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int f = 0; f < 4; ++f) acc[s][i][j][f] = 0.f;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  auto load_stage = [&](int st, int k0) {
    for (int i = tid; i < MW_BM * (MW_BK / 8); i += 256) {
      const int r = i >> 2, p = i & 3;
      const int sr = src_row[r];
      bf16 *dst = &As[st][r][p * 8];
      if (sr >= 0 && k0 + p * 8 < K) cp_async_16(smem_u32(dst), A + (size_t)sr * a_stride + k0 + p * 8);
      else *(uint4 *)dst = zero;
    }
    for (int i = tid; i < S * MG_BN * (MW_BK / 8); i += 256) {
      const int s = i / (MG_BN * 4), c = (i >> 2) % MG_BN, p = i & 3;
      bf16 *dst = &Bs[st][s][c][p * 8];
      if (n0 + c < N && k0 + p * 8 < K) cp_async_16(smem_u32(dst), We + gu_row(s, n0 + c, N, SWIGLU ? blocked : 0) * K + k0 + p * 8);
      else *(uint4 *)dst = zero;
    }
    cp_async_commit();
  };
  const int KT = (K + MW_BK - 1) / MW_BK;
  load_stage(0, 0);
  for (int kt = 0; kt < KT; ++kt) {
    const int st = kt & 1;
    if (kt + 1 < KT) {
      load_stage(st ^ 1, (kt + 1) * MW_BK);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < MW_BK; kk += 16) {
      uint32_t a[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i)
        ldmatrix_x4(a[i], smem_u32(&As[st][wm * 32 + 16 * i + (lane & 15)][kk + (lane >> 4) * 8]));
#pragma unroll
      for (int s = 0; s < S; ++s)
#pragma unroll
        for (int j2 = 0; j2 < 2; ++j2) {
          uint32_t b[4];
          ldmatrix_x4(b, smem_u32(&Bs[st][s][wn * 32 + 16 * j2 + (lane & 7) + ((lane >> 4) << 3)][kk + ((lane >> 3) & 1) * 8]));
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            mma_bf16_16816(acc[s][i][2 * j2], a[i], b[0], b[1]);
            mma_bf16_16816(acc[s][i][2 * j2 + 1], a[i], b[2], b[3]);
          }
        }
    }
    __syncthreads();
  }
  const int g = lane >> 2, q = lane & 3;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int f = 0; f < 4; ++f) {
        const int r = wm * 32 + 16 * i + g + (f >> 1) * 8;
        const int c = n0 + wn * 32 + 8 * j + 2 * q + (f & 1);
        if (r >= rows || c >= N) continue;
        const float v = SWIGLU ? glu_value(acc[0][i][j][f], acc[S - 1][i][j][f], glu) : acc[0][i][j][f];
        const size_t at = (size_t)(row0 + r) * N + c;
        if (out_f32) ((float *)out)[at] = v;
        else ((bf16 *)out)[at] = __float2bfloat16_rn(v);
      }
}

// ---------------------------------------------------------------------------
// the same for a step of few rows (decoding): a warp takes four output columns of one row and
// streams their weight rows with 16-byte loads, the row's K entries dealt to the lanes
// ---------------------------------------------------------------------------
__device__ __forceinline__ float dot_chunk(const uint4 &w, const uint4 &x, float acc, bf16) {
  const uint32_t ww[4] = {w.x, w.y, w.z, w.w}, xx[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    acc = fmaf(__uint_as_float(ww[i] << 16), __uint_as_float(xx[i] << 16), acc);
    acc = fmaf(__uint_as_float(ww[i] & 0xffff0000u), __uint_as_float(xx[i] & 0xffff0000u), acc);
  }
  return acc;
}
__device__ __forceinline__ float dot_chunk(const uint4 &w, const uint4 &x, float acc, float) {
  acc = fmaf(__uint_as_float(w.x), __uint_as_float(x.x), acc);
  acc = fmaf(__uint_as_float(w.y), __uint_as_float(x.y), acc);
  acc = fmaf(__uint_as_float(w.z), __uint_as_float(x.z), acc);
  return fmaf(__uint_as_float(w.w), __uint_as_float(x.w), acc);
}

#define MV_COLS 4            // columns a warp computes at a time
template <typename T, bool SWIGLU>
__global__ void __launch_bounds__(128)
moe_gemv_kernel(const T *__restrict__ A, int a_stride, const int *__restrict__ row_pair, int pairs_per_token, int gather,
                const int *__restrict__ idx, const T *__restrict__ W, int N, int K, const int *__restrict__ plan,
                int n_real, void *__restrict__ out, int out_f32, int blocked, GluForm glu) {
  pdl_wait();
  pdl_launch();                                         // only now: see moe_stream_kernel
  const int r = blockIdx.y;
  if (r >= plan[1 + n_real]) return;                     // rows in use
  const int pair = row_pair[r];
  const int e = idx[pair];
  constexpr int EPL = 16 / sizeof(T);                    // entries per 16-byte load
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = (blockIdx.x * 4 + warp) * MV_COLS;
  if (n0 >= N) return;
  const T *a = A + (size_t)(gather ? pair / pairs_per_token : r) * a_stride;
  const T *We = W + (size_t)e * (SWIGLU ? 2 : 1) * N * K;
  const int chunks = K / EPL;
  float acc[SWIGLU ? 2 : 1][MV_COLS];
#pragma unroll
  for (int s = 0; s < (SWIGLU ? 2 : 1); ++s)
#pragma unroll
    for (int j = 0; j < MV_COLS; ++j) acc[s][j] = 0.f;
#pragma unroll 2
  for (int c = lane; c < chunks; c += 32) {
    const uint4 x = *(const uint4 *)(a + (size_t)c * EPL);
    uint4 w[SWIGLU ? 2 : 1][MV_COLS];
#pragma unroll
    for (int s = 0; s < (SWIGLU ? 2 : 1); ++s)
#pragma unroll
      for (int j = 0; j < MV_COLS; ++j) {
        const int n = min(n0 + j, N - 1);
        w[s][j] = *(const uint4 *)(We + gu_row(s, n, N, SWIGLU ? blocked : 0) * K + (size_t)c * EPL);
      }
#pragma unroll
    for (int s = 0; s < (SWIGLU ? 2 : 1); ++s)
#pragma unroll
      for (int j = 0; j < MV_COLS; ++j) acc[s][j] = dot_chunk(w[s][j], x, acc[s][j], T());
  }
#pragma unroll
  for (int j = 0; j < MV_COLS; ++j) {
    float v = warp_sum(acc[0][j]);
    if (SWIGLU) v = glu_value(v, warp_sum(acc[SWIGLU ? 1 : 0][j]), glu);
    if (lane == 0 && n0 + j < N) {
      const size_t at = (size_t)r * N + n0 + j;
      if (out_f32) ((float *)out)[at] = v;
      else ((T *)out)[at] = from_f32<T>(v);
    }
  }
}

// ---------------------------------------------------------------------------
// the same in bfloat16: an expert's matrices are read once for all of its rows
// ---------------------------------------------------------------------------
// The work is a line of items: for every eight rows of every expert in use, all quads of rows of its matrix (two gates and their
// two ups with SWIGLU) over the whole K.  A block per SM takes an equal stretch of the line, its sixteen warps an item each in turn,
// the expert's rows staged whole in shared memory.  A warp brings 512 bytes of each of its four matrix rows at a time, RING such
// blocks ahead, across items and experts, through a ring that needs no barrier: a lane reads back only what it copied, and
// multiplies it by the same eight columns of each of the expert's rows.
//
// A lane's columns, the order of its multiply-adds and the tree that adds the lanes' sums are moe_gemv_kernel's, so both kernels give
// the same bits.  On mma.m16n8k16, which cuts off what it adds instead of rounding it, sums over K = 768 to 6,000 were 1.0e-7 to
// 7.2e-7 off and always towards zero; here 0.7e-7 to 1.1e-7 and to either side.  Memory bounds one row and two, the conversions to 32 bits (half
// rate) and the multiply-adds more: hence four matrix rows a lane behind each conversion of x, and fma.rn.f32x2, which rounds each half
// by itself, for two rows of x.  A product behind a product (of a row at a time; on mma.sync), gate and up of 3072 / down, width 4096,
// eight tokens: 3 of 16 experts 118 us (6.0 TB/s) / 62 (166 / 62; 116 / 62), 8 of 16 168 / 87 (293 / 109; 134 / 71); sixteen tokens,
// 8 of 16 241 / 129 (493 / 193; 191 / 105).  One token, 4 of 16, 768 / width 2048: 6.1 / 4.7 (13.6 / 4.3; 8.7 / 7.2).
//
// The next kernel of the stream may start once every block here has seen the plan (and waited for the kernel that wrote it), not
// before.  A second product over the same plan (`plan_stands`: the down product behind gate and up) can therefore read the plan and
// fill its ring with weights while the first one still works, and waits only for the rows.
#define MS_WARPS 16
#define MS_ROWS 8
#define MS_COLS 256               // columns of a block: eight a lane
#define MS_BLOCK 2048             // bytes of a block: four rows
template <int N> struct Rows { static constexpr int value = N; };
__device__ __forceinline__ float lower_half(uint32_t two) { return __uint_as_float(two << 16); }
__device__ __forceinline__ float upper_half(uint32_t two) { return __uint_as_float(two & 0xffff0000u); }
__device__ __forceinline__ float2 fma_both(float a, const float2 &x, const float2 &acc) {      // each half rounded by itself
  float2 r;
  asm("{\n\t.reg .b64 ra, rx, rc;\n\tmov.b64 ra, {%2, %2};\n\tmov.b64 rx, {%3, %4};\n\tmov.b64 rc, {%5, %6};\n\t"
      "fma.rn.f32x2 rc, ra, rx, rc;\n\tmov.b64 {%0, %1}, rc;\n\t}\n"
      : "=f"(r.x), "=f"(r.y) : "f"(a), "f"(x.x), "f"(x.y), "f"(acc.x), "f"(acc.y));
  return r;
}
// dot_chunk of four matrix rows and 2 PAIRS rows x, two of them an instruction; acc[p][j]: rows 2p and 2p + 1 against matrix row j
template <int PAIRS>
__device__ __forceinline__ void dot_chunks(const uint4 (&w)[4], const bf16 *x, int xrow, float2 (&acc)[PAIRS][4]) {
  uint32_t xx[2 * PAIRS][4];
#pragma unroll
  for (int m = 0; m < 2 * PAIRS; ++m) {
    const uint4 v = *reinterpret_cast<const uint4 *>(x + (size_t)m * xrow);
    xx[m][0] = v.x, xx[m][1] = v.y, xx[m][2] = v.z, xx[m][3] = v.w;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      float ww[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t raw = i == 0 ? w[j].x : i == 1 ? w[j].y : i == 2 ? w[j].z : w[j].w;
        ww[j] = half ? upper_half(raw) : lower_half(raw);
      }
#pragma unroll
      for (int p = 0; p < PAIRS; ++p) {
        const float2 xp = half ? make_float2(upper_half(xx[2 * p][i]), upper_half(xx[2 * p + 1][i]))
                               : make_float2(lower_half(xx[2 * p][i]), lower_half(xx[2 * p + 1][i]));
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[p][j] = fma_both(ww[j], xp, acc[p][j]);
      }
    }
}

// The sums of N values (a power of two up to 32) over a warp, in warp_sum's tree: value i ends in the lanes whose bits from the
// highest on are i's.
template <int N>
__device__ __forceinline__ float sums_over_warp(float (&v)[N], int lane) {
  int n = N;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    if (n > 1) {
      n >>= 1;
#pragma unroll
      for (int i = 0; i < N / 2; ++i)
        if (i < n) {
          const bool upper = lane & o;
          const float keep = upper ? v[i + n] : v[i], send = upper ? v[i] : v[i + n];
          v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    }
  }
  return v[0];
}

template <bool SWIGLU, int RING>
__global__ void __launch_bounds__(MS_WARPS * 32, 1)
moe_stream_kernel(const bf16 *A, int a_stride, const int *row_pair, int pairs_per_token, int gather, const bf16 *__restrict__ W, int N,
                  int K, const int *plan, int n_real, void *out, int out_f32, GluForm glu, int plan_stands) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ int warp_units[MS_WARPS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nkb = (K + MS_COLS - 1) / MS_COLS, xrow = nkb * MS_COLS;
  const uint32_t ring = smem_u32(smem_raw) + warp * (RING * MS_BLOCK) + lane * 16, ring_end = ring + RING * MS_BLOCK;
  bf16 *xs = reinterpret_cast<bf16 *>(smem_raw + MS_WARPS * RING * MS_BLOCK);                // [8][xrow]
  int *ustart = reinterpret_cast<int *>(xs + (size_t)MS_ROWS * xrow);                       // [n_real + 1]: units in front of an expert
  const int w_rows = SWIGLU ? 2 * N : N, quads = SWIGLU ? N / 2 : (N + 3) / 4;
  if (!plan_stands) pdl_wait();
  pdl_launch();
  int before = 0;
  for (int e0 = 0; e0 < n_real; e0 += MS_WARPS * 32) {
    const int e = e0 + threadIdx.x;
    const int mine = e < n_real ? (__ldcg(plan + 2 + e) - __ldcg(plan + 1 + e) + MS_ROWS - 1) / MS_ROWS : 0;
    int upto = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    if (lane == 31) warp_units[warp] = upto;
    __syncthreads();
    int all = 0;
#pragma unroll
    for (int w = 0; w < MS_WARPS; ++w) {
      if (w < warp) upto += warp_units[w];
      all += warp_units[w];
    }
    if (e < n_real) ustart[e] = before + upto - mine;
    before += all;
    __syncthreads();
  }
  if (threadIdx.x == 0) ustart[n_real] = before;
  __syncthreads();
  const long long total = (long long)before * quads;
  const int t_begin = (int)(total * blockIdx.x / gridDim.x), t_end = (int)(total * (blockIdx.x + 1) / gridDim.x);
  if (t_begin >= t_end) {
    if (plan_stands) pdl_wait();                        // every kernel's end stands for the end of those in front
    return;
  }
  auto expert_of = [&](int unit) {                      // the last expert with no more than `unit` units in front that has any
    int lo = 0, hi = n_real;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (ustart[mid] <= unit) lo = mid;
      else hi = mid;
    }
    return lo;
  };
  // ---- the weight stream
  int p_t = t_begin + warp, p_unit = -1, p_k = lane * 8;
  uint32_t put = ring;
  const bf16 *p_matrix = nullptr, *p_w[4];
  auto aim = [&]() {
    const int unit = p_t / quads, q = p_t - unit * quads;
    if (unit != p_unit) p_matrix = W + (size_t)expert_of(unit) * w_rows * K + lane * 8;
    p_unit = unit;
#pragma unroll
    for (int j = 0; j < 4; ++j) {                       // SWIGLU: rows in blocks of eight gates and their eight ups
      const int row = SWIGLU ? (q >> 2) * 16 + (q & 3) * 2 + (j & 1) + 8 * (j >> 1) : min(4 * q + j, N - 1);
      p_w[j] = p_matrix + (size_t)row * K;
    }
  };
  auto issue = [&]() {                                  // one block (or nothing), one group
    if (p_t < t_end) {
      if (p_k < K)
#pragma unroll
        for (int j = 0; j < 4; ++j) cp_async_16(put + j * 512, p_w[j]);
#pragma unroll
      for (int j = 0; j < 4; ++j) p_w[j] += MS_COLS;
      p_k += MS_COLS;
      if (p_k - lane * 8 >= K) {
        p_k = lane * 8;
        p_t += MS_WARPS;
        if (p_t < t_end) aim();
      }
    }
    cp_async_commit();
    put += MS_BLOCK;
    if (put == ring_end) put = ring;
  };
  if (p_t < t_end) aim();
#pragma unroll 1
  for (int i = 0; i < RING; ++i) issue();
  if (plan_stands) pdl_wait();
  // ---- the products
  uint32_t get = ring;
  int t = t_begin + warp;
  for (int unit = t_begin / quads; unit * (long long)quads < t_end; ++unit) {
    const int e = expert_of(unit), r0 = plan[1 + e] + MS_ROWS * (unit - ustart[e]), rows = min(MS_ROWS, plan[2 + e] - r0);
    __syncthreads();                                    // the rows before are no longer read
    for (int m = warp & 7; m < rows; m += MS_ROWS) {    // two warps a row
      bf16 *dst = xs + (size_t)m * xrow;
      const bf16 *src = A + (size_t)(gather ? row_pair[r0 + m] / pairs_per_token : r0 + m) * a_stride;
      for (int k = ((warp >> 3) * 32 + lane) * 8; k < K; k += 512) *reinterpret_cast<uint4 *>(dst + k) = *reinterpret_cast<const uint4 *>(src + k);
    }
    __syncthreads();
    const int end = (int)min((long long)t_end, (unit + 1ll) * quads);
    auto walk = [&](auto held) {
      constexpr int HELD = decltype(held)::value, PAIRS = (HELD + 1) / 2, SUMS = 4 * HELD;      // HELD: 1, 2, 4 or 8
      for (; t < end; t += MS_WARPS) {
        float acc[SUMS];
        float2 both[PAIRS][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          acc[i] = 0.f;
#pragma unroll
          for (int p = 0; p < PAIRS; ++p) both[p][i] = make_float2(0.f, 0.f);
        }
        const bf16 *x = xs + lane * 8;
        for (int k = lane * 8; k - lane * 8 < K; k += MS_COLS, x += MS_COLS) {
          cp_async_wait<RING - 1>();                    // this lane's copies of the block have landed
          uint4 w[4];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];\n" : "=r"(w[j].x), "=r"(w[j].y), "=r"(w[j].z), "=r"(w[j].w) : "r"(get + j * 512));
          get += MS_BLOCK;
          if (get == ring_end) get = ring;
          issue();                                      // the slot just read is filled again
          if (k >= K) continue;
          if (HELD == 1) {
            const uint4 xv = *reinterpret_cast<const uint4 *>(x);
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[j] = dot_chunk(w[j], xv, acc[j], bf16());
          } else {
            dot_chunks<PAIRS>(w, x, xrow, both);
          }
        }
        if (HELD > 1)
#pragma unroll
          for (int i = 0; i < SUMS; ++i) acc[i] = i & 4 ? both[i >> 3][i & 3].y : both[i >> 3][i & 3].x;
        float v = sums_over_warp(acc, lane);
        const int value = lane / (32 / SUMS), m = value >> 2, j = value & 3, q = t - unit * quads;
        if (SWIGLU) v = glu_value(v, __shfl_xor_sync(0xffffffffu, v, 2 * (32 / SUMS)), glu);
        const int n = SWIGLU ? 2 * q + j : 4 * q + j;
        if (lane % (32 / SUMS) == 0 && m < rows && n < N && (!SWIGLU || j < 2)) {
          const size_t at = (size_t)(r0 + m) * N + n;
          if (out_f32) ((float *)out)[at] = v;
          else ((bf16 *)out)[at] = __float2bfloat16_rn(v);
        }
      }
    };
    if (rows == 1) walk(Rows<1>());
    else if (rows == 2) walk(Rows<2>());
    else if (rows <= 4) walk(Rows<4>());
    else walk(Rows<8>());
  }
  cp_async_wait<0>();
}

static size_t stream_smem(int ring, int K, int n_real) {
  return (size_t)MS_WARPS * ring * MS_BLOCK + (size_t)MS_ROWS * ((K + MS_COLS - 1) / MS_COLS * MS_COLS) * sizeof(bf16) + (size_t)(n_real + 1) * sizeof(int);
}
#define MS_SMEM_MOST (226 * 1024)
template <bool SWIGLU, int RING>
static int launch_stream(const bf16 *A, int a_stride, const int *row_pair, int pairs_per_token, int gather, const bf16 *W, int N, int K,
                         const int *plan, int n_real, int n_rows, void *out, int out_f32, GluForm glu, int plan_stands, cudaStream_t stream) {
  static G2bPerDevice done;
  const int dev = g2b_current_device();
  if (dev < 0 || !done.value[dev]) {
    if (cudaFuncSetAttribute(moe_stream_kernel<SWIGLU, RING>, cudaFuncAttributeMaxDynamicSharedMemorySize, MS_SMEM_MOST) != cudaSuccess)
      G2B_REFUSE("moe_gemv: %d bytes of shared memory are not available", MS_SMEM_MOST);
    if (dev >= 0) done.value[dev] = 1;
  }
  const long long most = (SWIGLU ? N / 2 : (N + 3ll) / 4) * n_rows;
  g2b_launch(moe_stream_kernel<SWIGLU, RING>, dim3(most < 148 ? (unsigned)most : 148u), dim3(MS_WARPS * 32), stream_smem(RING, K, n_real), stream, A,
             a_stride, row_pair, pairs_per_token, gather, W, N, K, plan, n_real, out, out_f32, glu, plan_stands);
  return g2b_check_launch("moe_gemv");
}

extern "C" int g2b_moe_tile_rows() { return MG_BM; }

template <typename T>
static void launch_gemv(const void *A, int a_stride, const int *row_pair, int pairs_per_token, int gather, const int *idx,
                        const void *W, int N, int K, const int *plan, int n_real, int n_rows, int swiglu, void *out,
                        int out_f32, int blocked, GluForm glu, cudaStream_t stream) {
  const dim3 grid((N + 4 * MV_COLS - 1) / (4 * MV_COLS), n_rows);
  if (swiglu)
    g2b_launch(moe_gemv_kernel<T, true>, grid, dim3(128), 0, stream, (const T *)A, a_stride, row_pair, pairs_per_token,
               gather, idx, (const T *)W, N, K, plan, n_real, out, out_f32, blocked, glu);
  else
    g2b_launch(moe_gemv_kernel<T, false>, grid, dim3(128), 0, stream, (const T *)A, a_stride, row_pair, pairs_per_token,
               gather, idx, (const T *)W, N, K, plan, n_real, out, out_f32, blocked, glu);
}

// Few rows: `row_pair` (row -> pair) and `idx` (pair -> expert) are both needed; `gather` says whether
// row r reads A[pair / pairs_per_token] or A[r].  `plan_stands`: this function has been called for the same plan since the plan
// was written, on the same stream.
extern "C" int g2b_moe_gemv(const void *A, int dtype, int a_stride, const int *row_pair, int pairs_per_token, int gather,
                            const int *idx, const void *W, int N, int K, const int *plan, int n_real, int n_rows,
                            int swiglu, void *out, int out_f32, int blocked, float glu_limit, float glu_offset, float glu_c1,
                            float glu_c3, int plan_stands, cudaStream_t stream) {
  const GluForm glu = {glu_limit, glu_offset, glu_c1, glu_c3};
  if (n_rows <= 0 || N <= 0) return 0;
  const int epl = dtype == G2B_BF16 ? 8 : 4;
  if (K % epl || a_stride % epl || (((uintptr_t)A | (uintptr_t)W) & 15))
    G2B_REFUSE("moe_gemv: K = %d or the rows' distance %d is no multiple of %d, or a pointer is off 16 bytes", K, a_stride, epl);
  // a ring of 128 KB where the rows leave room for it (K up to about 6,000), else of 64 (up to about 10,000)
  const long long line = (swiglu ? N / 2 : (N + 3ll) / 4) * n_rows;
  if (dtype == G2B_BF16 && (!swiglu || (blocked && N % 8 == 0)) && line < (1ll << 31) - 1024 && stream_smem(2, K, n_real) <= MS_SMEM_MOST) {
    const bool deep = stream_smem(4, K, n_real) <= MS_SMEM_MOST;
    const auto launch = swiglu ? (deep ? launch_stream<true, 4> : launch_stream<true, 2>) : (deep ? launch_stream<false, 4> : launch_stream<false, 2>);
    return launch((const bf16 *)A, a_stride, row_pair, pairs_per_token, gather, (const bf16 *)W, N, K, plan, n_real, n_rows, out, out_f32, glu,
                  plan_stands, stream);
  }
  if (dtype == G2B_F32) launch_gemv<float>(A, a_stride, row_pair, pairs_per_token, gather, idx, W, N, K, plan, n_real, n_rows, swiglu, out, out_f32, blocked, glu, stream);
  else if (dtype == G2B_BF16) launch_gemv<bf16>(A, a_stride, row_pair, pairs_per_token, gather, idx, W, N, K, plan, n_real, n_rows, swiglu, out, out_f32, blocked, glu, stream);
  else G2B_REFUSE("moe_gemv: unknown dtype %d", dtype);
  return g2b_check_launch("moe_gemv");
}

extern "C" int g2b_moe_gemm(const void *A, int dtype, int a_stride, const int *row_pair, int pairs_per_token,
                            const void *W, int N, int K, const int *plan, int n_real, int max_tiles, int swiglu,
                            void *out, int out_f32, int blocked, float glu_limit, float glu_offset, float glu_c1,
                            float glu_c3, cudaStream_t stream) {
  const GluForm glu = {glu_limit, glu_offset, glu_c1, glu_c3};
  if (max_tiles <= 0 || N <= 0) return 0;
  const dim3 grid((N + MG_BN - 1) / MG_BN, max_tiles);
  if (dtype == G2B_F32) {
    if (swiglu)
      g2b_launch(moe_gemm_kernel<float, true>, grid, dim3(128), 0, stream, (const float *)A, a_stride, row_pair,
                 pairs_per_token, (const float *)W, N, K, plan, n_real, out, out_f32, blocked, glu);
    else
      g2b_launch(moe_gemm_kernel<float, false>, grid, dim3(128), 0, stream, (const float *)A, a_stride, row_pair,
                 pairs_per_token, (const float *)W, N, K, plan, n_real, out, out_f32, blocked, glu);
  } else if (dtype == G2B_BF16) {
    const bool mma = K % 8 == 0 && a_stride % 8 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
    // many rows an expert (a prompt step): the wide tiles
    const bool wide = mma && max_tiles > 3 * n_real + 8;
    if (wide && swiglu)
      g2b_launch(moe_gemm_wide_kernel<true>, grid, dim3(256), 0, stream, (const bf16 *)A, a_stride, row_pair,
                 pairs_per_token, (const bf16 *)W, N, K, plan, n_real, out, out_f32, blocked, glu);
    else if (wide)
      g2b_launch(moe_gemm_wide_kernel<false>, grid, dim3(256), 0, stream, (const bf16 *)A, a_stride, row_pair,
                 pairs_per_token, (const bf16 *)W, N, K, plan, n_real, out, out_f32, blocked, glu);
    else if (mma && swiglu)
      g2b_launch(moe_gemm_mma_kernel<true>, grid, dim3(128), 0, stream, (const bf16 *)A, a_stride, row_pair,
                 pairs_per_token, (const bf16 *)W, N, K, plan, n_real, out, out_f32, blocked, glu);
    else if (mma)
      g2b_launch(moe_gemm_mma_kernel<false>, grid, dim3(128), 0, stream, (const bf16 *)A, a_stride, row_pair,
                 pairs_per_token, (const bf16 *)W, N, K, plan, n_real, out, out_f32, blocked, glu);
    else if (swiglu)
      g2b_launch(moe_gemm_kernel<bf16, true>, grid, dim3(128), 0, stream, (const bf16 *)A, a_stride, row_pair,
                 pairs_per_token, (const bf16 *)W, N, K, plan, n_real, out, out_f32, blocked, glu);
    else
      g2b_launch(moe_gemm_kernel<bf16, false>, grid, dim3(128), 0, stream, (const bf16 *)A, a_stride, row_pair,
                 pairs_per_token, (const bf16 *)W, N, K, plan, n_real, out, out_f32, blocked, glu);
  } else {
    G2B_REFUSE("moe_gemm: unknown dtype %d", dtype);
  }
  return g2b_check_launch("moe_gemm");
}

// ---------------------------------------------------------------------------
// combination
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
moe_combine_kernel(const float *__restrict__ rows, const int *__restrict__ pair_row, const float *__restrict__ weight,
                   const float *__restrict__ x_self, int T, int top, int Hw, float *__restrict__ out, int accumulate) {
  pdl_launch();
  pdl_wait();
  const int t = blockIdx.x;
  for (int j = threadIdx.x; j < Hw; j += blockDim.x) {
    float acc = 0.f;
    for (int r = 0; r < top; ++r) {
      const int row = pair_row[(size_t)t * top + r];
      const float v = row >= 0 ? rows[(size_t)row * Hw + j] : x_self[(size_t)t * Hw + j];
      acc = fmaf(weight[(size_t)t * top + r], v, acc);
    }
    out[(size_t)t * Hw + j] = accumulate ? out[(size_t)t * Hw + j] + acc : acc;
  }
}

// The same four neighbours a thread, the choices' rows fetched four at a time (a token of a decode step is a few threads, whose
// time is the chain from the pairs to their rows).
__global__ void __launch_bounds__(128)
moe_combine4_kernel(const float *__restrict__ rows, const int *__restrict__ pair_row, const float *__restrict__ weight,
                    const float *__restrict__ x_self, int top, int Hw, float *__restrict__ out, int accumulate) {
  pdl_launch();
  pdl_wait();
  const int t = blockIdx.x, j = (blockIdx.y * 128 + threadIdx.x) * 4;
  if (j >= Hw) return;
  float4 *to = reinterpret_cast<float4 *>(out + (size_t)t * Hw + j);
  const float4 there = accumulate ? *to : make_float4(0.f, 0.f, 0.f, 0.f);
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int r0 = 0; r0 < top; r0 += 4) {
    const float *src[4];
    float wt[4];
    float4 v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const size_t at = (size_t)t * top + min(r0 + i, top - 1);
      const int row = pair_row[at];
      wt[i] = weight[at];
      src[i] = (row >= 0 ? rows + (size_t)row * Hw : x_self + (size_t)t * Hw) + j;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = *reinterpret_cast<const float4 *>(src[i]);
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (r0 + i < top)
        a.x = fmaf(wt[i], v[i].x, a.x), a.y = fmaf(wt[i], v[i].y, a.y), a.z = fmaf(wt[i], v[i].z, a.z), a.w = fmaf(wt[i], v[i].w, a.w);
  }
  *to = accumulate ? make_float4(there.x + a.x, there.y + a.y, there.z + a.z, there.w + a.w) : a;
}

// The combination, then the sum's RMS norm (times a weight) added to the stream, and the new stream
// once more in the compute type (join.cuh): what a layer whose sublayer outputs are normed does behind its routed
// feed-forward, in one pass.
#define MCN_MOST 4096
extern "C" int g2b_moe_combine_norm_add(const float *rows, const int *pair_row, const float *weight, float *x,
                                        const float *norm_w, float eps, int T_tokens, int top, int Hw, void *cast_out,
                                        int dtype, cudaStream_t stream) {
  if (T_tokens <= 0 || Hw <= 0) return 0;
  if (Hw > MCN_MOST) G2B_REFUSE("moe_combine_norm_add: rows of %d entries (at most %d)", Hw, MCN_MOST);
  const JoinTail a = {norm_w, eps, nullptr, nullptr, 0.f, cast_out, 1};
  const JoinExperts from = {rows, pair_row, weight, nullptr, top};
  const bool aligned = !(((uintptr_t)x | (uintptr_t)rows | (uintptr_t)norm_w | (uintptr_t)cast_out) & 15);
  if (dtype == G2B_F32) launch_join<float>(x, from, a, T_tokens, Hw, aligned, stream);
  else if (dtype == G2B_BF16) launch_join<bf16>(x, from, a, T_tokens, Hw, aligned, stream);
  else G2B_REFUSE("moe_combine_norm_add: unknown dtype %d", dtype);
  return g2b_check_launch("moe_combine_norm_add");
}

extern "C" int g2b_moe_combine(const float *rows, const int *pair_row, const float *weight, const float *x_self, int T,
                               int top, int Hw, float *out, int accumulate, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (Hw % 4 == 0 && top > 0 && !(((uintptr_t)rows | (uintptr_t)x_self | (uintptr_t)out) & 15) && (Hw + 511) / 512 <= 65535) {
    g2b_launch(moe_combine4_kernel, dim3(T, (Hw + 511) / 512), dim3(128), 0, stream, rows, pair_row, weight, x_self, top, Hw, out,
               accumulate);
    return g2b_check_launch("moe_combine");
  }
  g2b_launch(moe_combine_kernel, dim3(T), dim3(256), 0, stream, rows, pair_row, weight, x_self, T, top, Hw, out, accumulate);
  return g2b_check_launch("moe_combine");
}

// The combination as the sublayer result of a layer that norms it on the way in and on the way out (join.cuh):
// y = base + sum, x += norm(y) * w (+ add), and the next sublayer's normed input.
extern "C" int g2b_moe_combine_join(const float *rows, const int *pair_row, const float *weight, const float *base, int top,
                                    float *x, const float *w, float eps, const float *add, int n_rows, int H,
                                    const float *next_w, float next_eps, void *next, int dtype, cudaStream_t stream) {
  if (n_rows <= 0 || H <= 0) return 0;
  const JoinTail a = {w, eps, add, next_w, next_eps, next, 0};
  const JoinExperts from = {rows, pair_row, weight, base, top};
  const bool aligned = !(((uintptr_t)x | (uintptr_t)rows | (uintptr_t)base | (uintptr_t)w | (uintptr_t)add | (uintptr_t)next_w |
                          (uintptr_t)next) & 15);
  if (dtype == G2B_F32) launch_join<float>(x, from, a, n_rows, H, aligned, stream);
  else if (dtype == G2B_BF16) launch_join<bf16>(x, from, a, n_rows, H, aligned, stream);
  else G2B_REFUSE("moe_combine_join: unknown dtype %d", dtype);
  return g2b_check_launch("moe_combine_join");
}
