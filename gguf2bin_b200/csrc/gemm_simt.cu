// True 32-bit matrix product on the CUDA cores (FFMA only, no tensor-core mode):
//   C[M,N] (=|+=) A[M,K] * W[N,K]^T        W row-major [out][in] as in the checkpoint,
// the layout the reference's GEMV reads (src/l3_math.c:17-20: row i at w + i*n_in).
// Elements of A and W may be float or bfloat16 and are widened exactly; every product
// and sum is 32-bit.  One output element is a sum of chunks of SUM_CHUNK consecutive k: inside a chunk
// the products are added in increasing k, from zero, and the chunks' sums in increasing order.  Every kernel
// below keeps that order, whatever M is, so a row's result does not depend on the other rows of the batch.
//
// This is the product of the float32 path of the whole model, and the fallback of the
// bfloat16 path for sizes or dtypes the tensor-core kernels refuse.
#include "common.cuh"

#include <math.h>

G2B_DEFINE_LAST_ERROR

#define BM 64
#define BN 64
#define BK 16
#define SUM_CHUNK 64

enum { EPI_STORE_F32 = 0, EPI_STORE_BF16 = 1, EPI_ACCUM_F32 = 2 };

template <int EPI>
__device__ __forceinline__ void put(void *C, size_t at, float v) {
  if (EPI == EPI_STORE_F32) ((float *)C)[at] = v;
  else if (EPI == EPI_STORE_BF16) ((bf16 *)C)[at] = __float2bfloat16_rn(v);
  else ((float *)C)[at] += v;
}

// ---- any types, strides and alignment ---------------------------------------------------------------
template <typename TA, typename TW, int EPI>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(const TA *__restrict__ A, const TW *__restrict__ W, void *__restrict__ Cv, int M,
                 int N, int K, int lda, int ldw, int ldc) {
  pdl_launch();
  pdl_wait();
  __shared__ float As[BK][BM + 4];
  __shared__ float Ws[BK][BN + 4];
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;          // 16 x 16 threads, 4 x 4 outputs each
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  float acc[4][4], sum[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = sum[i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += BK) {
    // each thread loads 4 elements of each tile: row = e/BK, col = e%BK
#pragma unroll
    for (int e = tid; e < BM * BK; e += 256) {
      const int r = e / BK, c = e % BK;
      const int gm = m0 + r, gk = k0 + c;
      As[c][r] = (gm < M && gk < K) ? to_f32(A[(size_t)gm * lda + gk]) : 0.f;
      const int gn = n0 + r;
      Ws[c][r] = (gn < N && gk < K) ? to_f32(W[(size_t)gn * ldw + gk]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float a[4], w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) w[j] = Ws[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
    }
    __syncthreads();
    if (k0 + BK >= K || (k0 + BK) % SUM_CHUNK == 0) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          sum[i][j] += acc[i][j];
          acc[i][j] = 0.f;
        }
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gm = m0 + ty * 4 + i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gn = n0 + tx * 4 + j;
      if (gn >= N) continue;
      put<EPI>(Cv, (size_t)gm * ldc + gn, sum[i][j]);
    }
  }
}

// ---- float rows that start on 16 bytes ------------------------------------------------------------
// 16 bytes from global to shared memory, of which the last 16 - `bytes` are zeros.
__device__ __forceinline__ void copy16(float *dst, const float *src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes));
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }
// bytes of the four floats at k that lie in front of K
__device__ __forceinline__ int bytes_left(int k, int K) { return max(0, min(4, K - k)) * 4; }

// Few rows: a weight matrix is read once and used for every row of A, so memory bounds it.  A block takes NB rows
// of W; a stage is CH chunks of their columns (and of A's), brought by asynchronous copies while the stage in front
// is computed; thread (chunk, row) sums its chunk for every row of A, then the chunks' sums are added in order.
// Chunks lie 4 floats apart in shared memory, so eight lanes that read eight chunks touch all banks once.  The first
// stage of weights is asked for before the wait for the kernel in front.  Two rows, inside a decode step: 5.2 us for
// 1024 x 2048 and 1024 x 3072, 10 us for 4096 x 1024 and 6144 x 1024 (220 to 330 us with 64 x 64 tiles for the two rows).
#define ROWS_MAX 32
#define CHUNK_PITCH (SUM_CHUNK + 4)
template <int NB, int CH, int MT, int EPI>
__global__ void __launch_bounds__(NB *CH)
gemm_f32_rows_kernel(const float *A, const float *__restrict__ W, void *C, int rows_all, int rows_each, int N, int K, int lda, int ldw,
                     int ldc) {
  constexpr int THREADS = NB * CH, KS = CH * SUM_CHUNK, PITCH = CH * CHUNK_PITCH;
  constexpr int OWN = (NB * ROWS_MAX + THREADS - 1) / THREADS;
  extern __shared__ __align__(16) float sm[];
  const int tid = threadIdx.x, chunk = tid % CH, row = tid / CH, n0 = blockIdx.x * NB;
  const int m_base = blockIdx.y * rows_each, M = min(rows_each, rows_all - m_base);
  A += (size_t)m_base * lda;
  float *Ws = sm, *As = Ws + 2 * NB * PITCH, *part = As + 2 * M * PITCH;          // part [M][NB][CH + 1]
  const int stages = (K + KS - 1) / KS;
  auto bring_w = [&](int s) {
    float *to = Ws + (s & 1) * NB * PITCH;
    for (int i = tid; i < NB * KS / 4; i += THREADS) {
      const int r = i / (KS / 4), q = i % (KS / 4), k = s * KS + q * 4, n = min(n0 + r, N - 1);
      const int bytes = bytes_left(k, K);
      copy16(to + r * PITCH + (q / 16) * CHUNK_PITCH + (q % 16) * 4, W + (size_t)n * ldw + (bytes ? k : 0), bytes);
    }
  };
  auto bring_a = [&](int s) {
    float *to = As + (s & 1) * M * PITCH;
    for (int i = tid; i < M * (KS / 4); i += THREADS) {
      const int r = i / (KS / 4), q = i % (KS / 4), k = s * KS + q * 4;
      const int bytes = bytes_left(k, K);
      copy16(to + r * PITCH + (q / 16) * CHUNK_PITCH + (q % 16) * 4, A + (size_t)r * lda + (bytes ? k : 0), bytes);
    }
  };
  bring_w(0);
  pdl_launch();
  pdl_wait();
  bring_a(0);
  copies_commit();
  float sum[OWN];
#pragma unroll
  for (int o = 0; o < OWN; ++o) sum[o] = 0.f;
  for (int s = 0; s < stages; ++s) {
    if (s + 1 < stages) {
      bring_w(s + 1);
      bring_a(s + 1);
    }
    copies_commit();
    copies_wait<1>();
    __syncthreads();
    const float *w = Ws + (s & 1) * NB * PITCH + row * PITCH + chunk * CHUNK_PITCH;
    const float *a = As + (s & 1) * M * PITCH + chunk * CHUNK_PITCH;
    for (int m0 = 0; m0 < M; m0 += MT) {
      float acc[MT];
#pragma unroll
      for (int m = 0; m < MT; ++m) acc[m] = 0.f;
#pragma unroll 8
      for (int k = 0; k < SUM_CHUNK; k += 4) {
        const float4 wv = *(const float4 *)(w + k);
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          const float4 av = *(const float4 *)(a + min(m0 + m, M - 1) * PITCH + k);
          acc[m] = fmaf(av.x, wv.x, acc[m]);
          acc[m] = fmaf(av.y, wv.y, acc[m]);
          acc[m] = fmaf(av.z, wv.z, acc[m]);
          acc[m] = fmaf(av.w, wv.w, acc[m]);
        }
      }
#pragma unroll
      for (int m = 0; m < MT; ++m)
        if (m0 + m < M) part[((m0 + m) * NB + row) * (CH + 1) + chunk] = acc[m];
    }
    __syncthreads();
    const int here = min(CH, (K - s * KS + SUM_CHUNK - 1) / SUM_CHUNK);
#pragma unroll
    for (int o = 0; o < OWN; ++o) {
      const int p = tid + o * THREADS;
      if (p < M * NB)
        for (int c = 0; c < here; ++c) sum[o] += part[p * (CH + 1) + c];
    }
    __syncthreads();                                       // this stage's buffers may be filled again
  }
#pragma unroll
  for (int o = 0; o < OWN; ++o) {
    const int p = tid + o * THREADS;
    if (p < M * NB && n0 + p % NB < N) put<EPI>(C, (size_t)(m_base + p / NB) * ldc + n0 + p % NB, sum[o]);
  }
}

// Up to eight rows against a K whose rows of W fit shared memory whole: a block's NB rows are asked for at once, before the wait for the kernel
// in front, so that the copies of all blocks of an SM (up to 192 KB of it) are on their way together and nothing is waited for but their
// arrival; the kernel above has one stage of 32 KB on its way in front of the wait and, with 32 chunks a stage, moved zeros for half of a K of 1,024.
// Thread (chunk, row) sums chunks c, c + CH, ... of its row for every row of A.  A chunk's 16 pieces of four floats lie in the order
// piece ^ (chunk % 8): eight lanes that read one piece of eight chunks touch all banks once, without padding.  In a chain
// of launches, two rows: 5.1 us for 4096 x 1024 (10.5 by the kernel above), 5.7 for 6144 x 1024 (9.3), 3.9 for 1024 x 2048 (4.1), 5.6 for 1024 x 3072
// (5.9), 119 for 151936 x 1024 (139); a layer's four in turn 20.3 (29.5), with one row 17.5 (24.3), with eight 41 (64).
template <int NB, int CH, int MT, int EPI>
__global__ void __launch_bounds__(NB *CH)
gemm_f32_whole_kernel(const float *A, const float *__restrict__ W, void *C, int M, int N, int K, int lda, int ldw, int ldc) {
  constexpr int THREADS = NB * CH;
  extern __shared__ __align__(16) float sm[];
  const int tid = threadIdx.x, n0 = blockIdx.x * NB, chunks = (K + SUM_CHUNK - 1) / SUM_CHUNK, pitch = chunks * SUM_CHUNK;
  float *Ws = sm, *As = Ws + NB * pitch, *part = As + M * pitch;                  // part [M][NB][chunks + 1]
  auto bring = [&](float *to, const float *from, int rows, int ld, int last) {
    for (int i = tid; i < rows * (pitch / 4); i += THREADS) {
      const int r = i / (pitch / 4), q = i % (pitch / 4), chunk = q / 16;
      const int bytes = bytes_left(q * 4, K);
      copy16(to + r * pitch + chunk * SUM_CHUNK + ((q % 16) ^ (chunk & 7)) * 4, from + (size_t)min(r, last) * ld + (bytes ? q * 4 : 0), bytes);
    }
  };
  bring(Ws, W + (size_t)n0 * ldw, NB, ldw, N - 1 - n0);
  pdl_launch();
  pdl_wait();
  bring(As, A, M, lda, M - 1);
  copies_commit();
  copies_wait<0>();
  __syncthreads();
  const int row = tid / CH;
  for (int chunk = tid % CH; chunk < chunks; chunk += CH) {
    const float *w = Ws + row * pitch + chunk * SUM_CHUNK, *a = As + chunk * SUM_CHUNK;
    const int turn = chunk & 7;
    float acc[MT];
#pragma unroll
    for (int m = 0; m < MT; ++m) acc[m] = 0.f;
#pragma unroll
    for (int q = 0; q < SUM_CHUNK / 4; ++q) {
      const int at = (q ^ turn) * 4;
      const float4 wv = *(const float4 *)(w + at);
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        const float4 av = *(const float4 *)(a + min(m, M - 1) * pitch + at);
        acc[m] = fmaf(av.x, wv.x, acc[m]);
        acc[m] = fmaf(av.y, wv.y, acc[m]);
        acc[m] = fmaf(av.z, wv.z, acc[m]);
        acc[m] = fmaf(av.w, wv.w, acc[m]);
      }
    }
#pragma unroll
    for (int m = 0; m < MT; ++m)
      if (m < M) part[(m * NB + row) * (chunks + 1) + chunk] = acc[m];
  }
  __syncthreads();
  for (int p = tid; p < M * NB; p += THREADS) {
    float sum = 0.f;
#pragma unroll 16
    for (int c = 0; c < chunks; ++c) sum += part[p * (chunks + 1) + c];
    if (n0 + p % NB < N) put<EPI>(C, (size_t)(p / NB) * ldc + n0 + p % NB, sum);
  }
}

// Many rows: 64 x 64 outputs a block, 8 x 8 a thread, so that 16 loads of 16 bytes feed 256 multiply-adds and the FFMA
// pipe bounds it.  G groups of 64 threads share a tile: group g sums chunks g, g + G, ... of it, and after every round
// all threads add the groups' sums to their share of the tile in the chunks' order.  G = 1 where the tiles alone fill
// the GPU; G = 4 keeps all four schedulers of an SM busy with one tile.  701 rows: 231 us for 4096 x 1024 and 6144 x 1024
// on average (32 TFLOP/s), 184 us for 1024 x 2048 and 1024 x 3072 (20 TFLOP/s).
#define TILE 64
#define STEP 16
#define STEP_PITCH (STEP + 4)
#define SUM_PITCH (TILE + 8)
template <int G, int EPI>
__global__ void __launch_bounds__(TILE *G, G == 1 ? 4 : 1)
gemm_f32_tile_kernel(const float *A, const float *__restrict__ W, void *C, int M, int N, int K, int lda, int ldw, int ldc) {
  constexpr int THREADS = TILE * G, STAGES = 3, STAGE = G * 2 * TILE * STEP_PITCH, PER_CHUNK = SUM_CHUNK / STEP;
  constexpr int OWN = G == 1 ? 1 : TILE * TILE / THREADS;
  extern __shared__ __align__(16) float sm[];
  float *red = sm + STAGES * STAGE;                          // [G][TILE][SUM_PITCH], G > 1 only
  const int tid = threadIdx.x, g = tid / TILE, tx = tid % 8, ty = (tid % TILE) / 8;
  const int m0 = blockIdx.y * TILE, n0 = blockIdx.x * TILE;
  const int chunks = (K + SUM_CHUNK - 1) / SUM_CHUNK, rounds = (chunks + G - 1) / G, steps = rounds * PER_CHUNK;
  auto bring = [&](int s) {
    float *to = sm + (s % STAGES) * STAGE;
    const int base = (s / PER_CHUNK) * G * SUM_CHUNK + (s % PER_CHUNK) * STEP;
#pragma unroll
    for (int i = tid; i < G * 2 * TILE * (STEP / 4); i += THREADS) {
      const int q = i % (STEP / 4), r = (i / (STEP / 4)) % (2 * TILE), gr = i / (2 * TILE * (STEP / 4));
      const int k = base + gr * SUM_CHUNK + q * 4;
      const int bytes = bytes_left(k, K);
      const float *src = r < TILE ? A + (size_t)min(m0 + r, M - 1) * lda : W + (size_t)min(n0 + r - TILE, N - 1) * ldw;
      copy16(to + (gr * 2 * TILE + r) * STEP_PITCH + q * 4, src + (bytes ? k : 0), bytes);
    }
  };
  pdl_launch();
  pdl_wait();
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < steps) bring(s);
    copies_commit();
  }
  float acc[8][8], sum[G == 1 ? 8 : 1][G == 1 ? 8 : 1], own[OWN];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      acc[i][j] = 0.f;
      if (G == 1) sum[i][j] = 0.f;
    }
#pragma unroll
  for (int o = 0; o < OWN; ++o) own[o] = 0.f;
  for (int s = 0; s < steps; ++s) {
    copies_wait<STAGES - 2>();
    __syncthreads();
    if (s + STAGES - 1 < steps) bring(s + STAGES - 1);
    copies_commit();
    const float *a = sm + (s % STAGES) * STAGE + g * 2 * TILE * STEP_PITCH + ty * STEP_PITCH;
    const float *w = sm + (s % STAGES) * STAGE + (g * 2 + 1) * TILE * STEP_PITCH + tx * STEP_PITCH;
#pragma unroll
    for (int k = 0; k < STEP; k += 4) {
      float4 av[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) av[i] = *(const float4 *)(a + i * 8 * STEP_PITCH + k);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float4 wv = *(const float4 *)(w + j * 8 * STEP_PITCH + k);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          acc[i][j] = fmaf(av[i].x, wv.x, acc[i][j]);
          acc[i][j] = fmaf(av[i].y, wv.y, acc[i][j]);
          acc[i][j] = fmaf(av[i].z, wv.z, acc[i][j]);
          acc[i][j] = fmaf(av[i].w, wv.w, acc[i][j]);
        }
      }
    }
    if (s % PER_CHUNK != PER_CHUNK - 1) continue;
    if (G == 1) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          sum[G == 1 ? i : 0][G == 1 ? j : 0] += acc[i][j];
          acc[i][j] = 0.f;
        }
    } else {
      // the barrier of the step in between lies between the last reads of `red` and these writes
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          red[(g * TILE + ty + 8 * i) * SUM_PITCH + tx + 8 * j] = acc[i][j];
          acc[i][j] = 0.f;
        }
      __syncthreads();
      const int here = min(G, chunks - (s / PER_CHUNK) * G);
#pragma unroll
      for (int o = 0; o < OWN; ++o) {
        const int e = tid + o * THREADS;
#pragma unroll
        for (int c = 0; c < G; ++c)
          if (c < here) own[o] += red[(c * TILE + e / TILE) * SUM_PITCH + e % TILE];
      }
    }
  }
  if (G == 1) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int m = m0 + ty + 8 * i, n = n0 + tx + 8 * j;
        if (m < M && n < N) put<EPI>(C, (size_t)m * ldc + n, sum[G == 1 ? i : 0][G == 1 ? j : 0]);
      }
  } else {
#pragma unroll
    for (int o = 0; o < OWN; ++o) {
      const int e = tid + o * THREADS, m = m0 + e / TILE, n = n0 + e % TILE;
      if (m < M && n < N) put<EPI>(C, (size_t)m * ldc + n, own[o]);
    }
  }
}

template <typename K>
static int allow_smem(K kernel, size_t bytes, G2bPerDevice &done, const char *what) {
  const int dev = g2b_current_device();
  if (dev >= 0 && done.value[dev]) return 0;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess)
    G2B_REFUSE("%s: %zu bytes of shared memory are not available", what, bytes);
  if (dev >= 0) done.value[dev] = 1;
  return 0;
}

template <int NB, int CH, int MT, int EPI>
static int launch_rows(const float *A, const float *W, void *C, int M, int N, int K, int lda, int ldw, int ldc, cudaStream_t stream,
                       int rows_each = 0) {
  if (!rows_each) rows_each = M;
  static G2bPerDevice done;
  const int most = MT == 8 && CH == 8 ? ROWS_MAX : MT;
  auto bytes = [](int m) { return sizeof(float) * (2 * (size_t)(NB + m) * CH * CHUNK_PITCH + (size_t)m * NB * (CH + 1)); };
  if (allow_smem(gemm_f32_rows_kernel<NB, CH, MT, EPI>, bytes(most), done, "gemm_simt")) return 1;
  g2b_launch(gemm_f32_rows_kernel<NB, CH, MT, EPI>, dim3((N + NB - 1) / NB, (M + rows_each - 1) / rows_each), dim3(NB * CH),
             bytes(rows_each), stream, A, W, C, M, rows_each, N, K, lda, ldw, ldc);
  return g2b_check_launch("gemm_simt");
}

// Rows of W a block of the kernel that keeps them whole takes: 16, or 8 or 4 where fewer would leave SMs without a block; 0 where two blocks do not
// fit an SM (then the kernel that goes through K in stages).
static size_t whole_bytes(int NB, int M, int K) {
  const size_t chunks = (K + SUM_CHUNK - 1) / SUM_CHUNK;
  return sizeof(float) * ((NB + M) * chunks * SUM_CHUNK + (size_t)M * NB * (chunks + 1));
}
static int whole_rows(int M, int N, int K) {
  if (M > 8 || K < 8 * SUM_CHUNK) return 0;        // a short K is nothing but latency: 0.2 us more here at K = 64
  for (int NB = 16; NB >= 4; NB /= 2)
    if ((NB == 4 || N >= 128 * NB) && whole_bytes(NB, M, K) <= 112 * 1024) return NB;
  return 0;
}
template <int NB, int CH, int MT, int EPI>
static int launch_whole(const float *A, const float *W, void *C, int M, int N, int K, int lda, int ldw, int ldc, cudaStream_t stream) {
  static G2bPerDevice done;
  if (allow_smem(gemm_f32_whole_kernel<NB, CH, MT, EPI>, 112 * 1024, done, "gemm_simt")) return 1;
  g2b_launch(gemm_f32_whole_kernel<NB, CH, MT, EPI>, dim3((N + NB - 1) / NB), dim3(NB * CH), whole_bytes(NB, M, K), stream, A, W, C, M, N, K, lda,
             ldw, ldc);
  return g2b_check_launch("gemm_simt");
}
template <int MT, int EPI>
static int launch_whole_rows(int NB, const float *A, const float *W, void *C, int M, int N, int K, int lda, int ldw, int ldc, cudaStream_t stream) {
  if (NB == 16) return launch_whole<16, 16, MT, EPI>(A, W, C, M, N, K, lda, ldw, ldc, stream);
  if (NB == 8) return launch_whole<8, 32, MT, EPI>(A, W, C, M, N, K, lda, ldw, ldc, stream);
  return launch_whole<4, 32, MT, EPI>(A, W, C, M, N, K, lda, ldw, ldc, stream);
}

template <int G, int EPI>
static int launch_tile(const float *A, const float *W, void *C, int M, int N, int K, int lda, int ldw, int ldc, cudaStream_t stream) {
  static G2bPerDevice done;
  const size_t bytes = sizeof(float) * (3 * (size_t)G * 2 * TILE * STEP_PITCH + (G > 1 ? (size_t)G * TILE * SUM_PITCH : 0));
  if (allow_smem(gemm_f32_tile_kernel<G, EPI>, bytes, done, "gemm_simt")) return 1;
  g2b_launch(gemm_f32_tile_kernel<G, EPI>, dim3((N + TILE - 1) / TILE, (M + TILE - 1) / TILE), dim3(TILE * G), bytes, stream, A, W, C, M,
             N, K, lda, ldw, ldc);
  return g2b_check_launch("gemm_simt");
}

// Which kernel takes float operands whose rows all start on 16 bytes.  All give the same bits, so time decides: the estimates
// below (microseconds; the sums behind them are waves of blocks times what a block takes) pick a kernel within 8 % of the quickest for 950 of
// 976 combinations of K from 16 to 4,096, N from 64 to 8,192 and 1 to 2,048 rows, timed back to back.  Where the kernel for
// any strides wins: K up to about 128 (64 x 4096, 1,024 rows: 24 us, 429 with the rows kernel, to which a rule on the matrix's size alone
// sent it; 64 x 4096, 4 rows: 4.9 and 17.7).  The rows kernel: up to about two waves of its blocks (64 x 1024, 64 rows: 37 us in
// tiles, 8 here), and up to ROWS_MAX rows.
enum { F32_GENERAL, F32_TILE1, F32_TILE4, F32_ROWS };
static double ceil_div(double a, double b) { return ceil(a / b); }
static double us_general(int M, int N, int K) {
  const double tiles = ceil_div(N, BN) * ceil_div(M, BM);
  return (1.6 + 0.055 * K) * (tiles <= 74 ? 1.0 : 1.2 + tiles / 270.0);
}
static double us_tile(int G, int M, int N, int K) {
  const double tiles = ceil_div(N, TILE) * ceil_div(M, TILE), ragged = M % TILE ? 0.0006 * N : 0.0;      // all blocks ask for the last row
  if (G == 4) return 0.6 + ragged + ceil_div(tiles, 148) * (0.2 + 9.0 * ceil_div(K, 4 * SUM_CHUNK));
  return ragged + (3.6 + 3.8 * ceil_div(K, SUM_CHUNK)) * (tiles <= 148 ? 1.0 : tiles <= 592 ? 1.65 : 1.65 * tiles / 592);
}
static double us_rows(int rows_each, int NB, int CH, int M, int N, int K) {
  const double smem = sizeof(float) * (2.0 * (NB + rows_each) * CH * CHUNK_PITCH + rows_each * NB * (CH + 1.0));
  const double per_sm = floor(227 * 1024 / (smem + 1024)), waves = ceil_div(ceil_div(N, NB) * ceil_div(M, rows_each), 148 * per_sm);
  return 0.6 + waves * (0.5 + (CH == 8 ? 1.3 + 0.17 * rows_each : 1.2 + 0.25 * rows_each) * sqrt(per_sm) * ceil_div(K, CH * SUM_CHUNK));
}
static bool four_rows_of_w(int M, int N) { return M <= 8 && N < 16 * 2 * 148; }      // where 16 would leave SMs without a block
static int choose_f32(int M, int N, int K) {
  const double general = us_general(M, N, K);
  if (M <= ROWS_MAX) {
    const bool four = four_rows_of_w(M, N);
    return general < us_rows(M, four ? 4 : 16, four ? 32 : 8, M, N, K) ? F32_GENERAL : F32_ROWS;
  }
  const double us[4] = {general, us_tile(1, M, N, K), us_tile(4, M, N, K), us_rows(8, 16, 8, M, N, K)};
  int best = 0;
  for (int i = 1; i < 4; ++i)
    if (us[i] < us[best]) best = i;
  return best == F32_ROWS && (M + 7) / 8 > 65535 ? F32_TILE4 : best;
}
extern "C" int g2b_gemm_f32_kernel(int M, int N, int K) { return choose_f32(M, N, K); }
// Nanoseconds that the kernel chosen for more than ROWS_MAX rows is estimated to take.
extern "C" int g2b_gemm_f32_estimate(int M, int N, int K) {
  const double us = fmin(fmin(us_general(M, N, K), us_rows(8, 16, 8, M, N, K)), fmin(us_tile(1, M, N, K), us_tile(4, M, N, K)));
  return us < 2e6 ? (int)(1e3 * us) : 2000000000;
}

template <int EPI>
static int launch_f32(const float *A, const float *W, void *C, int M, int N, int K, int lda, int ldw, int ldc, int which, cudaStream_t stream) {
  if (which == F32_TILE1) return launch_tile<1, EPI>(A, W, C, M, N, K, lda, ldw, ldc, stream);
  if (which == F32_TILE4) return launch_tile<4, EPI>(A, W, C, M, N, K, lda, ldw, ldc, stream);
  if (const int NB = whole_rows(M, N, K)) {
    if (M == 1) return launch_whole_rows<1, EPI>(NB, A, W, C, M, N, K, lda, ldw, ldc, stream);
    if (M == 2) return launch_whole_rows<2, EPI>(NB, A, W, C, M, N, K, lda, ldw, ldc, stream);
    if (M <= 4) return launch_whole_rows<4, EPI>(NB, A, W, C, M, N, K, lda, ldw, ldc, stream);
    return launch_whole_rows<8, EPI>(NB, A, W, C, M, N, K, lda, ldw, ldc, stream);
  }
  if (M > ROWS_MAX) return launch_rows<16, 8, 8, EPI>(A, W, C, M, N, K, lda, ldw, ldc, stream, 8);      // eight rows a block, the matrix from the L2
  if (four_rows_of_w(M, N)) {
    if (M == 1) return launch_rows<4, 32, 1, EPI>(A, W, C, M, N, K, lda, ldw, ldc, stream);
    if (M == 2) return launch_rows<4, 32, 2, EPI>(A, W, C, M, N, K, lda, ldw, ldc, stream);
    if (M <= 4) return launch_rows<4, 32, 4, EPI>(A, W, C, M, N, K, lda, ldw, ldc, stream);
    return launch_rows<4, 32, 8, EPI>(A, W, C, M, N, K, lda, ldw, ldc, stream);
  }
  if (M == 1) return launch_rows<16, 8, 1, EPI>(A, W, C, M, N, K, lda, ldw, ldc, stream);
  if (M == 2) return launch_rows<16, 8, 2, EPI>(A, W, C, M, N, K, lda, ldw, ldc, stream);
  if (M <= 4) return launch_rows<16, 8, 4, EPI>(A, W, C, M, N, K, lda, ldw, ldc, stream);
  return launch_rows<16, 8, 8, EPI>(A, W, C, M, N, K, lda, ldw, ldc, stream);
}

template <typename TA, typename TW>
static int launch(const void *A, const void *W, void *C, int M, int N, int K, int lda, int ldw,
                  int ldc, int epi, cudaStream_t stream) {
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  if (grid.y > 65535) G2B_REFUSE("gemm_simt: M=%d is too large for one launch", M);
  switch (epi) {
    case EPI_STORE_F32:
      g2b_launch(gemm_simt_kernel<TA, TW, EPI_STORE_F32>, dim3(grid), dim3(256), 0, stream, 
          (const TA *)A, (const TW *)W, C, M, N, K, lda, ldw, ldc);
      break;
    case EPI_STORE_BF16:
      g2b_launch(gemm_simt_kernel<TA, TW, EPI_STORE_BF16>, dim3(grid), dim3(256), 0, stream, 
          (const TA *)A, (const TW *)W, C, M, N, K, lda, ldw, ldc);
      break;
    case EPI_ACCUM_F32:
      g2b_launch(gemm_simt_kernel<TA, TW, EPI_ACCUM_F32>, dim3(grid), dim3(256), 0, stream, 
          (const TA *)A, (const TW *)W, C, M, N, K, lda, ldw, ldc);
      break;
    default:
      G2B_REFUSE("gemm_simt: unknown epilogue %d", epi);
  }
  return g2b_check_launch("gemm_simt");
}

// epi: 0 store float, 1 store bfloat16, 2 add into float
extern "C" int g2b_gemm_simt(const void *A, int a_dtype, const void *W, int w_dtype, void *C,
                             int M, int N, int K, int lda, int ldw, int ldc, int epi,
                             cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) G2B_REFUSE("gemm_simt: K=%d", K);
  if (a_dtype == G2B_F32 && w_dtype == G2B_F32 && lda % 4 == 0 && ldw % 4 == 0 && (uintptr_t)A % 16 == 0 && (uintptr_t)W % 16 == 0 &&
      (M + TILE - 1) / TILE <= 65535) {
    const float *a = (const float *)A, *w = (const float *)W;
    const int which = choose_f32(M, N, K);
    if (which != F32_GENERAL) {
      if (epi == EPI_STORE_F32) return launch_f32<EPI_STORE_F32>(a, w, C, M, N, K, lda, ldw, ldc, which, stream);
      if (epi == EPI_STORE_BF16) return launch_f32<EPI_STORE_BF16>(a, w, C, M, N, K, lda, ldw, ldc, which, stream);
      if (epi == EPI_ACCUM_F32) return launch_f32<EPI_ACCUM_F32>(a, w, C, M, N, K, lda, ldw, ldc, which, stream);
    }
  }
  if (a_dtype == G2B_F32 && w_dtype == G2B_F32)
    return launch<float, float>(A, W, C, M, N, K, lda, ldw, ldc, epi, stream);
  if (a_dtype == G2B_BF16 && w_dtype == G2B_BF16)
    return launch<bf16, bf16>(A, W, C, M, N, K, lda, ldw, ldc, epi, stream);
  if (a_dtype == G2B_BF16 && w_dtype == G2B_F32)
    return launch<bf16, float>(A, W, C, M, N, K, lda, ldw, ldc, epi, stream);
  if (a_dtype == G2B_F32 && w_dtype == G2B_BF16)
    return launch<float, bf16>(A, W, C, M, N, K, lda, ldw, ldc, epi, stream);
  G2B_REFUSE("gemm_simt: unknown dtypes %d, %d", a_dtype, w_dtype);
}
