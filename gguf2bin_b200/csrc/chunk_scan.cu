// The state scan of a prompt in chunks: per head a state S [V columns of D], a token at a time
//   S <- g_t S + s_t v_t k_t^T   (column c: S_c <- g_t S_c + s_t v_t[c] k_t),   o_t[c] = S_c . q_t
// with g, s numbers per token and head (or one g per head and s = 1).  seq_mix.cu has the recurrence as it stands; a prompt
// of thousands of tokens is a chain of dependent steps there, whatever the GPU could do beside it.
//
// Here a sequence is cut into chunks of 64 tokens, and inside a chunk the recurrence is products:
//   with D_ij = g_(j+1) ... g_i, c_i = g_0 ... g_i (from the chunk's start) and the state S at the chunk's start
//   o_i = c_i (S q_i) + sum_(j<=i) (q_i . k_j) D_ij s_j v_j,      S' = c_last S + sum_j D_(last,j) s_j v_j k_j^T.
// The decays are products of the g's themselves, in the order of the tokens (no logarithms, no quotients), so a g of zero is
// exact.  They are taken in 64 bits and rounded once, and what carries a state over a chunk is a pair of floats: the
// rounding of one factor would fall on a whole state, again with every chunk.  All else is 32-bit multiply-adds, in sums of 16
// that are added up, which rounds less than the chain of single tokens does (decay per head, 2,048 tokens, against 64 bits:
// outputs 1.5e-7, states 1.2e-7, token by token 4.9e-7 and 5.7e-7; gates 0.9e-7 and 0.8e-7, 1.3e-7 and 0.9e-7).
//   1. chunk_kernel<false>: every chunk by itself from a zero state: its own contribution, and the product of its g's
//   2. chunk_carry: along a sequence, S at every chunk's start from the contributions; the sequence's state in the end
//   3. chunk_kernel<true>: every chunk from its start state: the outputs
// A block of 256 threads takes a chunk of one head and 64 columns.  Its phases (the loads, the decays, the products, the way out) bound it, so two
// blocks share an SM: the outputs keep their products where the queries were and values in 16 bits as they came (one block an SM: 276 us a layer for
// four prompts of 203 to 1,501 tokens, 64 heads of 128 x 64, now 233), and begin while half of the rows are on their way; the contributions'
// multiply-adds go two an instruction (161 us, now 136).  The whole scan there 0.46 ms (0.53; 0.89 token by token); 2,048 tokens, 8 heads of 128 x 256:
// 156 us (178; 486).  Chunks grouped into segments of up to 256 tokens, whose states alone went through memory: 189 and 709 us.
//
// Which sequences of a step come here is the caller's rule: those of more than `over` tokens, and sequence `pad`.  Of the
// others nothing is read or written.
#include "common.cuh"
#include <math.h>
#include <algorithm>
#include <exception>
#include <functional>
#include <type_traits>
#include <queue>
#include <vector>

G2B_DEFINE_LAST_ERROR

#define CHUNK 64
#define COLS 64
#define THREADS 256
#define MAX_D 128
#define P_PITCH (CHUNK + 4)

struct Members {
  const int *meta;            // [n_seqs, 4]: first row, tokens, past, slot
  int n_seqs, over, pad;
  // chunks of `size` tokens of sequence b
  __device__ __forceinline__ int chunks(int b, int size) const {
    const int n = meta[4 * b + 1];
    return n > over || b == pad ? (n + size - 1) / size : 0;
  }
};

struct ChunkArgs {
  const float *qf, *kf;       // [T, G, D] prepared
  const void *v;              // compute type, rows of a wider buffer
  int v_stride, H, G, D, V, Vin;        // V: columns of a head's state; Vin: value size in `v` (columns beyond: 1)
  const float *decay;         // [H], or null:
  const float *gates;         // [T, 2H]: g, then s
  float *state;               // [slots, H, V, D]
  Members seqs;
  int base, chunks;           // the launch's chunks: so many from this one of the step on
  float *parts;               // [chunks, H, V, D]: contributions, then start states
  float2 *part_decay;         // [chunks, H]: the product of the g's, and what its rounding left
  float *out;                 // [T, H*V]
};

// The sequence and the place in it of chunk `idx` of the step (sequences one after another); false behind the last one.
__device__ __forceinline__ bool find_chunk(const Members &seqs, int size, int idx, int &b, int &place) {
  const int lane = threadIdx.x & 31;
  int before = 0;
  for (int b0 = 0; b0 < seqs.n_seqs; b0 += 32) {
    const int mine = b0 + lane < seqs.n_seqs ? seqs.chunks(b0 + lane, size) : 0;
    int upto = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    const unsigned behind = __ballot_sync(0xffffffffu, before + upto > idx);
    if (behind) {
      const int at = __ffs(behind) - 1;
      b = b0 + at;
      place = idx - before - __shfl_sync(0xffffffffu, upto - mine, at);
      return true;
    }
    before += __shfl_sync(0xffffffffu, upto, 31);
  }
  return false;
}
// Chunks of the sequences in front of b; every lane has the sum.
__device__ __forceinline__ int chunks_before(const Members &seqs, int size, int b, int lane) {
  int before = 0;
  for (int b0 = 0; b0 < b; b0 += 32) {
    int c = b0 + lane < b ? seqs.chunks(b0 + lane, size) : 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    before += c;
  }
  return before;
}

__device__ __forceinline__ void copy16(float *dst, const float *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ float dot4(const float4 &a, const float4 &b, float acc) {
  return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, acc))));
}
__device__ __forceinline__ void add4(float4 &a, float f, const float4 &b) { fma4(a, make_float4(f, f, f, f), b); }

__device__ __forceinline__ float2 two_floats(double x) {
  const float hi = (float)x;
  return make_float2(hi, (float)(x - (double)hi));
}
__device__ __forceinline__ float carry1(float a, float2 f, float b) {         // f a + b; what f's rounding left changes no infinite a
  return fmaf(f.x, a, fmaf(f.y, isinf(a) ? 0.f : a, b));
}
__device__ __forceinline__ float4 carry4(const float4 &a, float2 f, const float4 &b) {
  return make_float4(carry1(a.x, f, b.x), carry1(a.y, f, b.y), carry1(a.z, f, b.z), carry1(a.w, f, b.w));
}
__device__ __forceinline__ float4 sum4(const float4 &a, const float4 &b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

template <typename T, bool OUT>
__global__ void __launch_bounds__(THREADS, 2)
chunk_kernel(const ChunkArgs a) {
  pdl_launch();
  pdl_wait();
  extern __shared__ __align__(16) float sm[];
  const int D = a.D, pitch = D + 4, V = a.V, H = a.H, h = blockIdx.y, col0 = blockIdx.x * COLS;
  int b, place;
  if (!find_chunk(a.seqs, CHUNK, a.base + blockIdx.z, b, place)) return;
  const int first = a.seqs.meta[4 * b] + place * CHUNK, n = min(CHUNK, a.seqs.meta[4 * b + 1] - place * CHUNK);
  const int qk_head = h / (H / a.G), tid = threadIdx.x;
  typedef typename std::conditional<OUT, T, float>::type Value;
  float *K = sm;
  Value *Vs = reinterpret_cast<Value *>(K + CHUNK * pitch);
  // decays and strengths of the chunk's tokens; from the token on: to the end of its sixteen, of the chunk times its strength;
  // up to the token: from its sixteen's start; the sixteens' products; in_block[B][i][j] = D_ij inside sixteen B
  double *tail16 = reinterpret_cast<double *>(Vs + CHUNK * COLS), *head = tail16 + CHUNK, *block = head + CHUNK;
  float *g = reinterpret_cast<float *>(block + 4), *s = g + CHUNK, *in_block = s + CHUNK, *tail = in_block + CHUNK * 17;
  float *Q = tail, *S = Q + CHUNK * pitch, *P = Q;       // OUT only (where there is no `tail`); the products where the queries were
  float *part = a.parts + ((size_t)blockIdx.z * H + h) * ((size_t)V * D);
  // the outputs start on the first 64 entries of keys, queries and states while the others are on their way
  const int D1 = OUT ? min(D, 64) : D;
  auto bring = [&](int d0, int d1) {
    const int quads = (d1 - d0) / 4;
    for (int i = tid; i < CHUNK * quads; i += THREADS) {
      const int r = i / quads, c = d0 + i % quads * 4;
      float *kd = K + r * pitch + c, *qd = Q + r * pitch + c, *sd = S + r * pitch + c;
      const size_t at = ((size_t)(first + r) * a.G + qk_head) * D + c;
      const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r < n) {
        copy16(kd, a.kf + at);
        if (OUT) copy16(qd, a.qf + at);
      } else {
        *reinterpret_cast<float4 *>(kd) = zero;
        if (OUT) *reinterpret_cast<float4 *>(qd) = zero;
      }
      if (OUT) {                                           // column col0 + r of the state at the chunk's start
        if (col0 + r < V) copy16(sd, part + (size_t)(col0 + r) * D + c);
        else *reinterpret_cast<float4 *>(sd) = zero;
      }
    }
    asm volatile("cp.async.commit_group;\n" ::);
  };
  bring(0, D1);
  if (OUT) bring(D1, D);
  {
    const int c = col0 + (tid & 63);
    const T *vg = (const T *)a.v;
    T rv[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {                       // nothing here waits for a load
      const int r = (tid >> 6) + 4 * i;
      rv[i] = from_f32<T>(c < V && c >= a.Vin ? 1.f : 0.f);
      if (r < n && c < a.Vin) rv[i] = vg[(size_t)(first + r) * a.v_stride + (size_t)h * a.Vin + c];
    }
    if (tid < CHUNK) {
      float rg = 1.f, rs = tid < n ? 1.f : 0.f;
      if (tid < n) {
        const size_t at = (size_t)(first + tid) * 2 * H + h;
        if (a.decay) rg = a.decay[h];
        else rg = a.gates[at], rs = a.gates[at + H];
      }
      g[tid] = rg;
      s[tid] = rs;
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) Vs[((tid >> 6) + 4 * i) * COLS + (tid & 63)] = from_f32<Value>(to_f32(rv[i]));
  }
  if (OUT) asm volatile("cp.async.wait_group 1;\n" ::: "memory");
  else asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
  if (tid < CHUNK) {                                     // the decays from token `tid` on, to the end of its sixteen
    const int b16 = tid & ~15, j = tid & 15;
    double d = 1.0;
    in_block[tid * 17 + j] = 1.f;                        // row i of its sixteen: in_block[(b16 + i) * 17 + j]
    if (j == 0) head[tid] = g[tid];
    for (int i = j + 1; i < 16; ++i) {
      d *= g[b16 + i];
      in_block[(b16 + i) * 17 + j] = (float)d;
      if (j == 0) head[b16 + i] = g[b16] * d;
    }
    tail16[tid] = d;
    if (j == 0) block[tid >> 4] = g[b16] * d;
  }
  if (OUT) {
    const int tx = tid & 15, ty = tid >> 4;              // tokens ty + 16 i, columns (or keys) tx + 16 j
    float p[4][4], o[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) p[i][j] = o[i][j] = 0.f;
#pragma unroll 1
    for (int d0 = 0; d0 < D; d0 += 16) {
      if (d0 == 64) {
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();
      }
      float p16[4][4], o16[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) p16[i][j] = o16[i][j] = 0.f;
      const int d1 = min(d0 + 16, D);
#pragma unroll 2
      for (int d = d0; d < d1; d += 4) {
        float4 q[4], k[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) q[i] = *reinterpret_cast<const float4 *>(Q + (ty + 16 * i) * pitch + d);
#pragma unroll
        for (int j = 0; j < 4; ++j) k[j] = *reinterpret_cast<const float4 *>(K + (tx + 16 * j) * pitch + d);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (j <= i) p16[i][j] = dot4(q[i], k[j], p16[i][j]);   // later keys are not seen
#pragma unroll
        for (int j = 0; j < 4; ++j) k[j] = *reinterpret_cast<const float4 *>(S + (tx + 16 * j) * pitch + d);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) o16[i][j] = dot4(q[i], k[j], o16[i][j]);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) p[i][j] += p16[i][j], o[i][j] += o16[i][j];
    }
    __syncthreads();                                     // all decays stand, and the queries are read
    double before = 1.0;                                 // the sixteens in front
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = ty + 16 * i;
      const double up = head[r];
      const float from_start = (float)(before * up);
#pragma unroll
      for (int j = 0; j < 4; ++j) o[i][j] *= from_start;
      before *= block[i];
      double between = up;                               // the sixteens between the key's and the row's, and the row's up to it
#pragma unroll
      for (int j = 3; j >= 0; --j) {
        if (j > i) continue;
        const int t = tx + 16 * j;
        if (j == i) {
          p[i][j] = tx <= ty ? p[i][j] * (in_block[r * 17 + tx] * s[t]) : 0.f;
        } else {
          p[i][j] *= (float)(tail16[t] * between * (double)s[t]);
          between *= block[j];
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j <= i; ++j) P[(ty + 16 * i) * P_PITCH + tx + 16 * j] = p[i][j];
    __syncwarp();                                        // a row's 16 threads are one half of a warp
    // sixteen tokens at a time, for the rows that see them; later values are not touched, whatever they hold
#pragma unroll
    for (int tb = 0; tb < 4; ++tb) {
      float o16[4][4];
#pragma unroll
      for (int i = tb; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) o16[i][j] = 0.f;
#pragma unroll 1
      for (int t = 16 * tb; t < 16 * tb + 16; t += 4) {
        float x[4][4];
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
          for (int j = 0; j < 4; ++j) x[e][j] = to_f32(Vs[(t + e) * COLS + tx + 16 * j]);
#pragma unroll
        for (int i = tb; i < 4; ++i) {
          const int r = ty + 16 * i;
          const float4 w = *reinterpret_cast<const float4 *>(P + r * P_PITCH + t);
          const bool all = i > tb;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (all || t <= r) o16[i][j] = fmaf(w.x, x[0][j], o16[i][j]);
            if (all || t + 1 <= r) o16[i][j] = fmaf(w.y, x[1][j], o16[i][j]);
            if (all || t + 2 <= r) o16[i][j] = fmaf(w.z, x[2][j], o16[i][j]);
            if (all || t + 3 <= r) o16[i][j] = fmaf(w.w, x[3][j], o16[i][j]);
          }
        }
      }
#pragma unroll
      for (int i = tb; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) o[i][j] += o16[i][j];
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int r = ty + 16 * i, c = col0 + tx + 16 * j;
        if (r < n && c < V) a.out[(size_t)(first + r) * H * V + (size_t)h * V + c] = o[i][j];
      }
    return;
  }
  __syncthreads();                                       // all decays stand
  if (tid < CHUNK) {
    double f = (double)s[tid] * tail16[tid];
    for (int B = (tid >> 4) + 1; B < 4; ++B) f *= block[B];
    tail[tid] = (float)f;
  }
  __syncthreads();                                       // `tail` stands
  // this thread's share of the state: columns 4 vy .. + 3, entries 4 dx .. + 3 and 64 further
  const int dx = tid & 15, vy = tid >> 4;
  float4 st[4][2];
#pragma unroll 1
  for (int tb = 0; tb < n; tb += 16) {
    float4 sum[4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int m = 0; m < 2; ++m) sum[i][m] = make_float4(0.f, 0.f, 0.f, 0.f);
    const int t1 = min(tb + 16, n);
#pragma unroll 4
    for (int t = tb; t < t1; ++t) {
      const float f = tail[t];
      const float4 x = *reinterpret_cast<const float4 *>(Vs + t * COLS + 4 * vy);
#pragma unroll
      for (int m = 0; m < 2; ++m)
        if (4 * dx + 64 * m < D) {
          const float4 k = *reinterpret_cast<const float4 *>(K + t * pitch + 4 * dx + 64 * m);
          add4(sum[0][m], f * x.x, k);
          add4(sum[1][m], f * x.y, k);
          add4(sum[2][m], f * x.z, k);
          add4(sum[3][m], f * x.w, k);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int m = 0; m < 2; ++m) st[i][m] = tb ? sum4(st[i][m], sum[i][m]) : sum[i][m];
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const int c = col0 + 4 * vy + i, d = 4 * dx + 64 * m;
      if (c < V && d < D) *reinterpret_cast<float4 *>(part + (size_t)c * D + d) = st[i][m];
    }
  if (tid == 0 && blockIdx.x == 0) a.part_decay[(size_t)blockIdx.z * H + h] = two_floats((block[0] * block[1]) * (block[2] * block[3]));
}

// Four neighbours of a sequence's state a thread, along the sequence's chunks.
__global__ void __launch_bounds__(THREADS)
chunk_carry_kernel(const ChunkArgs a) {
  pdl_launch();
  pdl_wait();
  // `chunks` of the sequence's are the launch's, in places from `before` on
  const int b = blockIdx.y, place = chunks_before(a.seqs, CHUNK, b, threadIdx.x & 31) - a.base, before = max(place, 0);
  const int chunks = min(a.seqs.chunks(b, CHUNK) - max(0, -place), a.chunks - before);
  const size_t size = (size_t)a.H * a.V * a.D, e = ((size_t)blockIdx.x * THREADS + threadIdx.x) * 4;
  if (chunks <= 0 || e >= size) return;
  const int h = (int)(e / ((size_t)a.V * a.D));
  float4 *kept = reinterpret_cast<float4 *>(a.state + (size_t)a.seqs.meta[4 * b + 3] * size + e);
  float4 s = *kept;
  for (int i0 = 0; i0 < chunks; i0 += 4) {
    float4 x[4];
    float2 g[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const size_t at = (size_t)before + min(i0 + i, chunks - 1);
      x[i] = *reinterpret_cast<const float4 *>(a.parts + at * size + e);
      g[i] = a.part_decay[at * a.H + h];
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (i0 + i < chunks) {
        *reinterpret_cast<float4 *>(a.parts + ((size_t)before + i0 + i) * size + e) = s;
        s = carry4(s, g[i], x[i]);
      }
  }
  *kept = s;
}

template <typename T, bool OUT>
static int launch_chunks(const ChunkArgs &a, dim3 grid, cudaStream_t stream) {
  static G2bPerDevice done;
  auto bytes = [](int D) {
    const size_t rows = sizeof(float) * CHUNK * (size_t)(D + 4), products = sizeof(float) * CHUNK * P_PITCH;       // (where the queries were)
    return rows + CHUNK * COLS * (OUT ? sizeof(T) : sizeof(float)) + sizeof(float) * (6 * CHUNK + 8 + CHUNK * 17) +
           (OUT ? std::max(rows, products) + std::max(rows, sizeof(float) * COLS * (size_t)(D + 4)) : sizeof(float) * CHUNK);
  };
  const int dev = g2b_current_device();
  if (dev < 0 || !done.value[dev]) {
    if (cudaFuncSetAttribute(chunk_kernel<T, OUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes(MAX_D)) != cudaSuccess)
      G2B_REFUSE("chunk_scan: %zu bytes of shared memory are not available", bytes(MAX_D));
    if (dev >= 0) done.value[dev] = 1;
  }
  g2b_launch(chunk_kernel<T, OUT>, grid, dim3(THREADS), bytes(a.D), stream, a);
  return g2b_check_launch("chunk_scan");
}

// Chunks base .. base + chunks - 1 of those (of 64 tokens) of all sequences that go here, whose states stand behind the chunks in
// front; parts [chunks, H, V, D], part_decay [chunks, H, 2].
extern "C" int g2b_chunk_scan(int dtype, const float *qf, const float *kf, const void *v, int v_stride, int H, int G, int D, int Vin, int extra_one,
                              const float *decay, const float *gates, float *state, const int *seq_meta, int n_seqs, int over, int pad,
                              int base, int chunks, float *parts, float2 *part_decay, float *out, cudaStream_t stream) {
  const int V = Vin + (extra_one ? 1 : 0);
  if (n_seqs <= 0 || chunks <= 0) return 0;
  if (dtype != G2B_F32 && dtype != G2B_BF16) G2B_REFUSE("chunk_scan: unknown dtype %d", dtype);
  if (D <= 0 || D > MAX_D || D % 4) G2B_REFUSE("chunk_scan: key size %d (a multiple of 4 up to %d)", D, MAX_D);
  if (G <= 0 || H % G) G2B_REFUSE("chunk_scan: %d heads are not a multiple of %d query/key heads", H, G);
  if (!decay == !gates) G2B_REFUSE("chunk_scan: a decay per head or gates, not both");
  if (H > 65535 || chunks > 65535 || n_seqs > 65535) G2B_REFUSE("chunk_scan: %d heads, %d chunks are too many", H, chunks);
  if (((uintptr_t)qf | (uintptr_t)kf | (uintptr_t)state | (uintptr_t)parts) & 15) G2B_REFUSE("chunk_scan: a buffer is off 16 bytes");
  const ChunkArgs a = {qf, kf, v, v_stride, H, G, D, V, Vin, decay, gates, state, {seq_meta, n_seqs, over, pad}, base, chunks, parts, part_decay, out};
  const dim3 grid((V + COLS - 1) / COLS, H, chunks);
  if (int rc = dtype == G2B_F32 ? launch_chunks<float, false>(a, grid, stream) : launch_chunks<bf16, false>(a, grid, stream)) return rc;
  const size_t quads = (size_t)H * V * D / 4;
  g2b_launch(chunk_carry_kernel, dim3((unsigned)((quads + THREADS - 1) / THREADS), n_seqs), dim3(THREADS), 0, stream, a);
  if (int rc = g2b_check_launch("chunk_scan")) return rc;
  return dtype == G2B_F32 ? launch_chunks<float, true>(a, grid, stream) : launch_chunks<bf16, true>(a, grid, stream);
}

// ---------------------------------------------------------------------------------------------------------
// the gated delta rule in chunks
// ---------------------------------------------------------------------------------------------------------
//   S <- g_t S;  u_t = b_t (v_t - S k_t);  S <- S + u_t k_t^T;  o_t = S q_t
// Inside a chunk of 32 tokens, with D_ij and c_i as above and the state S at the chunk's start, the u solve a triangular system
//   u_i + sum_(j<i) A_ij u_j = b_i v_i - b_i c_i S k_i,   A_ij = b_i D_ij (k_i . k_j),
// whose right side is linear in S: U = U0 - W S^T with (I + A) U0 = (b_i v_i) and (I + A) W = (b_i c_i k_i).
//   1. delta_chunk: every chunk by itself (none needs the state): U0, W by substitution, a column a thread, and the
//      products P_ij = D_ij (q_i . k_j) of the outputs
//   2. delta_walk: along the sequence, a chunk a step: U = U0 - W S^T, o_i = c_i S q_i + sum_(j<=i) P_ij u_j,
//      S' = c_last S + sum_j D_(last,j) u_j k_j^T.  A block has 8 columns of a head; the next chunk's operands are on their way.
// The substitution takes the tokens in their order, as the recurrence does; decays and sums as above (errors against 64 bits as
// token by token: outputs 1.5e-7, states 1.1e-7).  The walk's chain of products, read
// from shared memory, bounds it.  2,048 tokens, 8 heads of 128 x 128: 261 us, of which the walk 237 (713 us a token after a token).
#define DELTA_CHUNK 32
#define DELTA_COLS 8
#define DELTA_WALK 128
#define DELTA_DECAYS (2 * DELTA_CHUNK + 4)

struct DeltaArgs {
  const float *qf, *kf;       // [T, G, D] prepared
  const void *v;              // compute type, rows of a wider buffer
  int v_stride, H, G, D, V;
  const float *ab;            // [T, 2H]: decay input, then write-strength input
  const float *A_log, *dt_bias;
  float *state;               // [slots, H, V, D]
  Members seqs;
  int base, chunks;           // the launch's chunks: so many from this one of the step on
  float *U0, *W, *P, *decays; // [chunks, H, 32, V], [.., 32, D], [.., 32, 32], [.., 68]: c, the decays to the chunk's end, what c_last's rounding left
  float *out;                 // [T, H*V]
};

template <typename T>
__global__ void __launch_bounds__(THREADS)
delta_chunk_kernel(const DeltaArgs a) {
  pdl_launch();
  pdl_wait();
  extern __shared__ __align__(16) float sm[];
  __shared__ __align__(16) float M[DELTA_CHUNK][DELTA_CHUNK + 4];         // D_ij, then A_ij
  __shared__ float g[DELTA_CHUNK], beta[DELTA_CHUNK], beta_c[DELTA_CHUNK];
  const int D = a.D, pitch = D + 4, V = a.V, H = a.H, h = blockIdx.y, tid = threadIdx.x, qk_head = h / (H / a.G);
  int b, place;
  if (!find_chunk(a.seqs, DELTA_CHUNK, a.base + blockIdx.x, b, place)) return;
  const int first = a.seqs.meta[4 * b] + place * DELTA_CHUNK, nt = min(DELTA_CHUNK, a.seqs.meta[4 * b + 1] - place * DELTA_CHUNK);
  float *K = sm, *Q = K + DELTA_CHUNK * pitch;
  for (int i = tid; i < DELTA_CHUNK * (D / 4); i += THREADS) {
    const int r = i / (D / 4), d = i % (D / 4) * 4;
    const size_t at = ((size_t)(first + r) * a.G + qk_head) * D + d;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    *reinterpret_cast<float4 *>(K + r * pitch + d) = r < nt ? *reinterpret_cast<const float4 *>(a.kf + at) : zero;
    *reinterpret_cast<float4 *>(Q + r * pitch + d) = r < nt ? *reinterpret_cast<const float4 *>(a.qf + at) : zero;
  }
  if (tid < DELTA_CHUNK) {
    float x = 1.f, y = 0.f;
    if (tid < nt) {
      const float *ab = a.ab + (size_t)(first + tid) * 2 * H;
      const float z = ab[h] + a.dt_bias[h];
      x = expf(-expf(a.A_log[h]) * (fmaxf(z, 0.f) + log1pf(expf(-fabsf(z)))));
      y = 1.f / (1.f + expf(-ab[H + h]));
    }
    g[tid] = x;
    beta[tid] = y;
  }
  __syncthreads();
  const size_t item = (size_t)blockIdx.x * H + h;
  if (tid < DELTA_CHUNK) {
    float *decays = a.decays + item * DELTA_DECAYS;
    double d = 1.0;
    M[tid][tid] = 1.f;
    for (int i = tid + 1; i < DELTA_CHUNK; ++i) {
      d *= g[i];
      M[i][tid] = (float)d;
    }
    decays[DELTA_CHUNK + tid] = (float)d;
    d = g[0];
    for (int i = 1; i <= tid; ++i) d *= g[i];
    decays[tid] = (float)d;
    beta_c[tid] = (float)(d * beta[tid]);
    if (tid == DELTA_CHUNK - 1) decays[2 * DELTA_CHUNK] = two_floats(d).y;
  }
  const int i = tid >> 3, j0 = tid & 7;
  float kk[4] = {0.f, 0.f, 0.f, 0.f}, qk[4] = {0.f, 0.f, 0.f, 0.f};
  for (int d0 = 0; d0 < D; d0 += 16) {
    float kk16[4] = {0.f, 0.f, 0.f, 0.f}, qk16[4] = {0.f, 0.f, 0.f, 0.f};
    const int d1 = min(d0 + 16, D);
#pragma unroll 4
    for (int d = d0; d < d1; d += 4) {
      const float4 ki = *reinterpret_cast<const float4 *>(K + i * pitch + d), qi = *reinterpret_cast<const float4 *>(Q + i * pitch + d);
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const float4 kj = *reinterpret_cast<const float4 *>(K + (j0 + 8 * m) * pitch + d);
        kk16[m] = dot4(ki, kj, kk16[m]);
        qk16[m] = dot4(qi, kj, qk16[m]);
      }
    }
#pragma unroll
    for (int m = 0; m < 4; ++m) kk[m] += kk16[m], qk[m] += qk16[m];
  }
  __syncthreads();                                       // the decays stand
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    const int j = j0 + 8 * m;
    const float d = j <= i ? M[i][j] : 0.f;
    a.P[(item * DELTA_CHUNK + i) * DELTA_CHUNK + j] = j <= i ? d * qk[m] : 0.f;
    M[i][j] = j < i ? beta[i] * d * kk[m] : 0.f;
  }
  __syncthreads();
  const T *vg = (const T *)a.v;
  for (int col = tid; col < V + D; col += THREADS) {
    float x[DELTA_CHUNK];
#pragma unroll
    for (int r = 0; r < DELTA_CHUNK; ++r) {
      float y;
      if (col < V) y = r < nt ? beta[r] * to_f32(vg[(size_t)(first + r) * a.v_stride + (size_t)h * V + col]) : 0.f;
      else y = beta_c[r] * K[r * pitch + col - V];
      x[r] = y;
    }
#pragma unroll
    for (int r = 1; r < DELTA_CHUNK; ++r) {
      float y[2] = {0.f, 0.f};                           // of the first sixteen tokens, of the others
#pragma unroll
      for (int j = 0; j < r; j += 4) {
        const float4 m = *reinterpret_cast<const float4 *>(&M[r][j]);
        float &to = y[j >> 4];
        to = fmaf(m.x, x[j], to);
        if (j + 1 < r) to = fmaf(m.y, x[j + 1], to);
        if (j + 2 < r) to = fmaf(m.z, x[j + 2], to);
        if (j + 3 < r) to = fmaf(m.w, x[j + 3], to);
      }
      x[r] -= y[0] + y[1];
    }
    float *to = col < V ? a.U0 + item * DELTA_CHUNK * V + col : a.W + item * DELTA_CHUNK * D + col - V;
    const int step = col < V ? V : D;
#pragma unroll
    for (int r = 0; r < DELTA_CHUNK; ++r) to[(size_t)r * step] = x[r];
  }
}

// (two blocks of an SM asked for: without, ptxas settles on half the registers and loads later, 270 us for 237)
__global__ void __launch_bounds__(DELTA_WALK, 2)
delta_walk_kernel(const DeltaArgs a) {
  pdl_launch();
  pdl_wait();
  extern __shared__ __align__(16) float sm[];
  const int D = a.D, pitch = D + 4, V = a.V, H = a.H, h = blockIdx.y, b = blockIdx.z, tid = threadIdx.x;
  const int qk_head = h / (H / a.G), col0 = blockIdx.x * DELTA_COLS;
  // the sequence's n tokens from row `first` on are the launch's, its chunks in places from `before` on
  const int place = chunks_before(a.seqs, DELTA_CHUNK, b, tid & 31) - a.base, skip = max(0, -place) * DELTA_CHUNK, before = max(place, 0);
  const int first = a.seqs.meta[4 * b] + skip, slot = a.seqs.meta[4 * b + 3];
  const int n = min(a.seqs.meta[4 * b + 1] - skip, (a.chunks - before) * DELTA_CHUNK);
  if (n <= 0 || !a.seqs.chunks(b, DELTA_CHUNK)) return;
  // two buffers, each: W, Q, K [32, pitch], P [32, 36], U0 [32, 8], decays [68]
  const int rows = DELTA_CHUNK * pitch, P_AT = 3 * rows, U_AT = P_AT + DELTA_CHUNK * 36, G_AT = U_AT + DELTA_CHUNK * DELTA_COLS,
            SIZE = G_AT + DELTA_DECAYS;
  float *S = sm + 2 * SIZE, *U = S + DELTA_COLS * pitch;                 // S [8, pitch], U [32, 8]
  auto fetch = [&](int t0, int buf) {
    float *to = sm + buf * SIZE;
    const size_t item = (size_t)(before + t0 / DELTA_CHUNK) * H + h;
    const int nt = min(DELTA_CHUNK, n - t0);
    for (int i = tid; i < DELTA_CHUNK * (D / 4); i += DELTA_WALK) {
      const int r = i / (D / 4), d = i % (D / 4) * 4;
      const size_t at = ((size_t)(first + t0 + min(r, nt - 1)) * a.G + qk_head) * D + d;      // rows behind the last are not used
      copy16(to + r * pitch + d, a.W + (item * DELTA_CHUNK + r) * D + d);
      copy16(to + rows + r * pitch + d, a.qf + at);
      copy16(to + 2 * rows + r * pitch + d, a.kf + at);
    }
    for (int i = tid; i < DELTA_CHUNK * (DELTA_CHUNK / 4); i += DELTA_WALK)
      copy16(to + P_AT + (i / 8) * 36 + (i % 8) * 4, a.P + item * DELTA_CHUNK * DELTA_CHUNK + i * 4);
    if (tid < DELTA_CHUNK * 2) {
      const int r = tid >> 1, q = (tid & 1) * 4;
      if (col0 + q < V) copy16(to + U_AT + r * DELTA_COLS + q, a.U0 + (item * DELTA_CHUNK + r) * V + col0 + q);
    }
    if (tid >= 64 && tid < 64 + DELTA_DECAYS / 4) copy16(to + G_AT + (tid - 64) * 4, a.decays + item * DELTA_DECAYS + (tid - 64) * 4);
    asm volatile("cp.async.commit_group;\n" ::);
  };
  // this thread's share of the state: column cs, entries 4 dx .. + 3 and 64 further
  const int cs = tid >> 4, dx = tid & 15;
  float *kept = a.state + (((size_t)slot * H + h) * V + col0 + cs) * D;
  float4 st[2];
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    const int d = 4 * dx + 64 * m;
    st[m] = col0 + cs < V && d < D ? *reinterpret_cast<const float4 *>(kept + d) : make_float4(0.f, 0.f, 0.f, 0.f);
    if (d < D) *reinterpret_cast<float4 *>(S + cs * pitch + d) = st[m];
  }
  for (int i = tid; i < 2 * DELTA_CHUNK * DELTA_COLS; i += DELTA_WALK)   // columns behind the last hold zeros
    sm[(i / (DELTA_CHUNK * DELTA_COLS)) * SIZE + U_AT + i % (DELTA_CHUNK * DELTA_COLS)] = 0.f;
  __syncthreads();
  fetch(0, 0);
  const int r0 = tid >> 3, cc = tid & 7;                 // tokens r0 and r0 + 16, column cc
  int buf = 0;
  for (int t0 = 0; t0 < n; t0 += DELTA_CHUNK, buf ^= 1) {
    const int nt = min(DELTA_CHUNK, n - t0);
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();                                     // the chunk's operands and S are in place
    if (t0 + DELTA_CHUNK < n) fetch(t0 + DELTA_CHUNK, buf ^ 1);
    const float *W = sm + buf * SIZE, *Q = W + rows, *K = Q + rows, *P = W + P_AT, *U0 = W + U_AT, *G = W + G_AT;
    float ws[2] = {0.f, 0.f}, qs[2] = {0.f, 0.f};
    for (int d0 = 0; d0 < D; d0 += 16) {
      float ws16[2] = {0.f, 0.f}, qs16[2] = {0.f, 0.f};
      const int d1 = min(d0 + 16, D);
#pragma unroll 4
      for (int d = d0; d < d1; d += 4) {
        const float4 s = *reinterpret_cast<const float4 *>(S + cc * pitch + d);
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          ws16[m] = dot4(*reinterpret_cast<const float4 *>(W + (r0 + 16 * m) * pitch + d), s, ws16[m]);
          qs16[m] = dot4(*reinterpret_cast<const float4 *>(Q + (r0 + 16 * m) * pitch + d), s, qs16[m]);
        }
      }
#pragma unroll
      for (int m = 0; m < 2; ++m) ws[m] += ws16[m], qs[m] += qs16[m];
    }
#pragma unroll
    for (int m = 0; m < 2; ++m) U[(r0 + 16 * m) * DELTA_COLS + cc] = U0[(r0 + 16 * m) * DELTA_COLS + cc] - ws[m];
    __syncthreads();                                     // U stands, and S is read
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const int r = r0 + 16 * m;
      float o[2] = {0.f, 0.f};                           // of the first sixteen tokens, of the others
#pragma unroll
      for (int j = 0; j < 16 + 16 * m; j += 4) {
        const float4 p = *reinterpret_cast<const float4 *>(P + r * 36 + j);
        float &to = o[j >> 4];
        if (j <= r) to = fmaf(p.x, U[j * DELTA_COLS + cc], to);          // later tokens are not touched, whatever they hold
        if (j + 1 <= r) to = fmaf(p.y, U[(j + 1) * DELTA_COLS + cc], to);
        if (j + 2 <= r) to = fmaf(p.z, U[(j + 2) * DELTA_COLS + cc], to);
        if (j + 3 <= r) to = fmaf(p.w, U[(j + 3) * DELTA_COLS + cc], to);
      }
      if (r < nt && col0 + cc < V) a.out[(size_t)(first + t0 + r) * H * V + (size_t)h * V + col0 + cc] = fmaf(G[r], qs[m], o[0] + o[1]);
    }
    const float2 all = make_float2(G[DELTA_CHUNK - 1], G[2 * DELTA_CHUNK]);
#pragma unroll
    for (int jb = 0; jb < DELTA_CHUNK; jb += 16) {
      float4 sum[2];
      sum[0] = sum[1] = make_float4(0.f, 0.f, 0.f, 0.f);
      const int j1 = min(jb + 16, nt);
#pragma unroll 4
      for (int j = jb; j < j1; ++j) {
        const float f = G[DELTA_CHUNK + j] * U[j * DELTA_COLS + cs];
#pragma unroll
        for (int m = 0; m < 2; ++m)
          if (4 * dx + 64 * m < D) add4(sum[m], f, *reinterpret_cast<const float4 *>(K + j * pitch + 4 * dx + 64 * m));
      }
#pragma unroll
      for (int m = 0; m < 2; ++m) st[m] = jb ? sum4(st[m], sum[m]) : carry4(st[m], all, sum[m]);
    }
#pragma unroll
    for (int m = 0; m < 2; ++m)
      if (4 * dx + 64 * m < D) *reinterpret_cast<float4 *>(S + cs * pitch + 4 * dx + 64 * m) = st[m];
  }
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    const int d = 4 * dx + 64 * m;
    if (col0 + cs < V && d < D) *reinterpret_cast<float4 *>(kept + d) = st[m];
  }
}

// Chunks base .. base + chunks - 1 of those (of 32 tokens) of all sequences that go here, whose states stand behind the chunks in front.
extern "C" int g2b_delta_scan(int dtype, const float *qf, const float *kf, const void *v, int v_stride, int H, int G, int D, int V,
                              const float *ab, const float *A_log, const float *dt_bias, float *state, const int *seq_meta, int n_seqs,
                              int over, int pad, int base, int chunks, float *U0, float *W, float *P, float *decays, float *out, cudaStream_t stream) {
  if (n_seqs <= 0 || chunks <= 0) return 0;
  if (dtype != G2B_F32 && dtype != G2B_BF16) G2B_REFUSE("delta_scan: unknown dtype %d", dtype);
  if (D <= 0 || D > MAX_D || D % 4 || V <= 0 || V % 4) G2B_REFUSE("delta_scan: key size %d (a multiple of 4 up to %d), value size %d (of 4)", D, MAX_D, V);
  if (G <= 0 || H % G) G2B_REFUSE("delta_scan: %d heads are not a multiple of %d query/key heads", H, G);
  if (H > 65535 || n_seqs > 65535) G2B_REFUSE("delta_scan: %d heads, %d sequences are too many", H, n_seqs);
  if (((uintptr_t)qf | (uintptr_t)kf | (uintptr_t)state | (uintptr_t)U0 | (uintptr_t)W | (uintptr_t)P | (uintptr_t)decays) & 15)
    G2B_REFUSE("delta_scan: a buffer is off 16 bytes");
  const DeltaArgs a = {qf, kf, v, v_stride, H, G, D, V, ab, A_log, dt_bias, state, {seq_meta, n_seqs, over, pad}, base, chunks, U0, W, P, decays, out};
  auto prep_bytes = [](int d) { return sizeof(float) * (size_t)2 * DELTA_CHUNK * (d + 4); };
  auto walk_bytes = [](int d) {
    return sizeof(float) * ((size_t)2 * (3 * DELTA_CHUNK * (d + 4) + DELTA_CHUNK * 36 + DELTA_CHUNK * DELTA_COLS + DELTA_DECAYS) + DELTA_COLS * (d + 4) +
                            DELTA_CHUNK * DELTA_COLS);
  };
  static G2bPerDevice done;
  const int dev = g2b_current_device();
  if (dev < 0 || !done.value[dev]) {
    if (cudaFuncSetAttribute(delta_walk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)walk_bytes(MAX_D)) != cudaSuccess)
      G2B_REFUSE("delta_scan: %zu bytes of shared memory are not available", walk_bytes(MAX_D));
    if (dev >= 0) done.value[dev] = 1;
  }
  if (dtype == G2B_F32) g2b_launch(delta_chunk_kernel<float>, dim3(chunks, H), dim3(THREADS), prep_bytes(D), stream, a);
  else g2b_launch(delta_chunk_kernel<bf16>, dim3(chunks, H), dim3(THREADS), prep_bytes(D), stream, a);
  if (int rc = g2b_check_launch("delta_scan")) return rc;
  g2b_launch(delta_walk_kernel, dim3((V + DELTA_COLS - 1) / DELTA_COLS, H, n_seqs), dim3(DELTA_WALK), walk_bytes(D), stream, a);
  return g2b_check_launch("delta_scan");
}

// ---------------------------------------------------------------------------------------------------------
// which sequences go in chunks (host; gates on 64 heads: 64 prompts of up to 600 tokens 0.11 ms, 256 of up to 200 1.7 ms)
// ---------------------------------------------------------------------------------------------------------
#define LENGTH_STEP 32            // prompt lengths are told apart in steps of this many tokens
#define SMS 148                   // of the B200 that the times below were taken on; the rule is also asked where no GPU is

struct ScanKind { int mode, heads, cols, dim; };      // mode: 0 a decay a head, 1 the delta rule, 2 gates

// About what the scan of a token after a token takes for sequences of these lengths, in microseconds: blocks of 128 threads start
// in the sequences' order as slots of the GPU come free, and a token costs a block more the fewer lanes a column has and the more
// blocks share its SM.  (The lanes and the shared memory are seq_mix.cu's, `n_seqs` the sequences they are chosen for.)  Beyond `most`
// the estimate ends early.
static double chain_us(const std::vector<double> &lens, int n_seqs, const ScanKind &k, double most) {
  int lanes = 8;
  while (lanes * 16 < k.dim) lanes *= 2;
  while (lanes < 32 && (double)n_seqs * k.heads * k.cols * lanes * 2 <= 76800) lanes *= 2;
  const long long padded = (k.dim + 4 * lanes - 1) / (4 * lanes) * 4 * lanes, tile = padded <= 128 ? 16 : padded <= 256 ? 8 : 4;
  const long long groups = 128 / lanes, blocks = k.heads * ((k.cols + groups - 1) / groups);
  const long long per_sm = std::min(16ll, 227 * 1024 / (4 * tile * (4 * padded + 2 * (groups + 2) + 128) + 1024));
  const int wide = lanes == 8 ? 0 : lanes == 16 ? 1 : 2;
  static const double one[2][3] = {{0.25, 0.20, 0.15}, {0.42, 0.33, 0.31}}, more[2][3] = {{0.045, 0.03, 0.03}, {0.04, 0.03, 0.03}};
  const double token = one[k.mode == 1][wide] +
                       more[k.mode == 1][wide] * std::min((double)(blocks * (long long)lens.size()) / SMS, (double)per_sm);
  typedef std::pair<double, long long> Slots;           // when they come free, and how many
  std::priority_queue<Slots, std::vector<Slots>, std::greater<Slots>> free;
  free.push({0.0, SMS * per_sm});
  double end = 0.0;
  for (const double n : lens) {
    if (6.0 + end >= most) break;
    for (long long left = blocks; left > 0;) {
      const Slots s = free.top();
      free.pop();
      const long long take = std::min(s.second, left);
      left -= take;
      if (s.second > take) free.push({s.first, s.second - take});
      free.push({s.first + n * token, take});
      end = std::max(end, s.first + n * token);
    }
  }
  return 6.0 + end;
}

// Sequences of more tokens than the number returned go in chunks; 0: none does.  A token after a token costs the longest chain's latency, several
// times over once the sequences' blocks fill the GPU; chunks cost all tokens alike, but up to twice as much as a chain that
// fills the GPU.  So a few long prompts gain and large batches lose (microseconds a layer, a token after a token and in chunks:
// 8 heads of 128 x 256 with a decay, 2,048 tokens 486 and 184, 100 tokens 33 and 33, 11 x 200 186 and 230; the delta rule with 8
// heads of 128 x 128, 2,048 tokens 713 and 261, 8 x 512 303 and 506).  The times of chunks below are fitted to such measurements;
// lengths count in steps, which a step's graph is captured for.
static int chunks_over(const int *tokens, int n, const ScanKind &k) {
  std::vector<int> classes(n), cuts;                    // those of a few tokens as of four
  std::vector<double> lens(n), few;
  for (int i = 0; i < n; ++i) {
    classes[i] = tokens[i] > 8 ? (tokens[i] + LENGTH_STEP - 1) / LENGTH_STEP : 0;
    lens[i] = classes[i] ? (classes[i] - 0.5) * LENGTH_STEP : 4.0;
    if (classes[i] * LENGTH_STEP > CHUNK) cuts.push_back(classes[i]);
  }
  std::sort(cuts.begin(), cuts.end());
  cuts.erase(std::unique(cuts.begin(), cuts.end()), cuts.end());
  if (cuts.empty()) return 0;
  const double wide = (double)k.heads * ((k.cols + COLS - 1) / COLS) * COLS * k.dim;
  const double link = k.mode == 1 ? 0.04 + 0.0006 * k.dim : 0.0, token = k.mode == 1 ? (double)k.heads * k.cols * k.dim * 0.95e-6 : wide * 3.3e-7;
  double best = 0.95 * chain_us(lens, n, k, HUGE_VAL);            // chunks where they are quicker by more than the fit's error
  int over = 0;
  const int places = std::min<int>(8, (int)cuts.size());      // eight places to cut at are enough to choose from
  for (int c = 0; c < places; ++c) {
    const int cut = cuts[(size_t)c * cuts.size() / places];
    double longest = 0.0, sum = 0.0;
    int below = 0;
    few.clear();
    for (int i = 0; i < n; ++i) {
      if (classes[i] < cut) {
        few.push_back(lens[i]);
        below = std::max(below, classes[i] * LENGTH_STEP);
      } else {
        const double whole = (double)((classes[i] * LENGTH_STEP + CHUNK - 1) / CHUNK * CHUNK);
        longest = std::max(longest, whole);
        sum += whole;
      }
    }
    double us = 22.0 + std::max(longest * link, sum * token);
    if (!few.empty() && us < best) us += chain_us(few, n, k, best - us);
    if (us < best) best = us, over = std::max(below, CHUNK);
  }
  return over;
}

// `tokens` [n]: the lengths of a step's sequences, without padding.
extern "C" int g2b_scan_chunks_over(const int *tokens, int n, int mode, int heads, int cols, int dim, int *over) {
  if (n <= 0 || heads <= 0 || cols <= 0 || dim <= 0 || dim > MAX_D)
    G2B_REFUSE("chunk_scan: no rule for %d sequences on %d heads of %d x %d", n, heads, dim, cols);
  try {
    *over = chunks_over(tokens, n, {mode, heads, cols, dim});
  } catch (const std::exception &e) {
    G2B_REFUSE("chunk_scan: %s", e.what());
  }
  return 0;
}
