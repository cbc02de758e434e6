// What the decode attention kernels (attn_decode.cu, attn_decode_short.cu) share: pages in shared memory, the query tile, scores, and
// the merge of a token's chunks of CHUNK_KEYS keys that lie in scratch.  HD and CHUNK_KEYS are the including file's.
#pragma once
#include "common.cuh"
#include "mma.cuh"

constexpr int PAGE = 64;                       // keys per page
constexpr int ROW_BYTES = HD * 2;
constexpr int ROW_CHUNKS = HD / 8;             // 16-byte pieces per row
constexpr int KSTEPS = HD / 16;                // k-steps of q.k over the head size
constexpr int DTILES = HD / 8;                 // n-tiles of the output over the head size
constexpr float LOG2E = 1.4426950408889634f;

// byte offset of (row, 16-byte piece) in a swizzled panel
__device__ __forceinline__ uint32_t swz(int row, int piece) {
  return (uint32_t)(row * ROW_BYTES + ((piece ^ (row & 7)) << 4));
}

// a load that is neither cached in registers across the dependency line nor merged with another
__device__ __forceinline__ int ld_volatile(const int *p) {
  int v;
  asm volatile("ld.volatile.global.s32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// The query rows of a tile as A fragments: head = kvh * group + ht * 16 + row.
__device__ __forceinline__ void load_q_tile(uint32_t (&qa)[KSTEPS][4], const bf16 *__restrict__ q, int t,
                                            int q_stride, int kvh, int group, int ht, int g, int c) {
  const int row0 = ht * 16 + g, row1 = row0 + 8;
  const bf16 *q0 = q + (size_t)t * q_stride + ((size_t)kvh * group + row0) * HD;
  const bf16 *q1 = q0 + 8 * HD;
#pragma unroll
  for (int ks = 0; ks < KSTEPS; ++ks) {
    const int d = ks * 16 + 2 * c;
    qa[ks][0] = row0 < group ? *reinterpret_cast<const uint32_t *>(q0 + d) : 0u;
    qa[ks][1] = row1 < group ? *reinterpret_cast<const uint32_t *>(q1 + d) : 0u;
    qa[ks][2] = row0 < group ? *reinterpret_cast<const uint32_t *>(q0 + d + 8) : 0u;
    qa[ks][3] = row1 < group ? *reinterpret_cast<const uint32_t *>(q1 + d + 8) : 0u;
  }
}

// How a raw score becomes an exponent (log2 domain): times the scale, or capped first.
struct ScoreMap {
  float scale_log2;      // scale * log2(e)
  float cap_in;          // scale / softcap (0: no cap)
  float cap_log2;        // softcap * log2(e)
  __device__ __forceinline__ float operator()(float s) const {
    return cap_in > 0.f ? cap_log2 * tanhf(s * cap_in) : s * scale_log2;
  }
};

// ---- a token's chunks ---------------------------------------------------------------------------------
// The chunks that hold a key that the token at `pos` sees, counted through as 0 .. total - 1: with kept first
// tokens those in front of the window's that hold one come first (0 .. nk - 1), then c0 .. c1.
struct Chunks {
  int c0, nk, total;
  __device__ __forceinline__ Chunks(int pos, int lo, int kept_end) {
    c0 = lo / CHUNK_KEYS;
    nk = min((kept_end + CHUNK_KEYS - 1) / CHUNK_KEYS, c0);
    total = nk + (pos / CHUNK_KEYS - c0 + 1);
  }
  __device__ __forceinline__ int operator()(int idx) const { return idx < nk ? idx : c0 + idx - nk; }
};
__device__ __forceinline__ int kept_keys(int lo, int keep_first) {         // keys below it are seen behind the window
  return (keep_first > 0 && lo > 0) ? min(keep_first, lo) : 0;
}

// What the end of a merge does with a head's denominator: the sink, a learned logit, taken as it is, that adds nothing to the
// sum; with a gate the head's output times sigmoid(gate), i.e. the denominator times (1 + exp(-gate)).
struct Finish {
  const float *sink;             // [nh] or null
  const bf16 *gate;              // [T, nh], rows gate_stride apart, or null
  int gate_stride;
  __device__ __forceinline__ float operator()(float den, float M, int t, int h) const {
    if (sink) den += exp2f(sink[h] * LOG2E - M);
    if (gate) den *= 1.f + __expf(-__bfloat162float(gate[(size_t)t * gate_stride + h]));
    return den;
  }
};

// out[t, h, :] = sum_i 2^(m_i - M) o_i / sum_i 2^(m_i - M) l_i over the token's chunks.  One block of
// four warps per (token, head): warp w adds the chunks c0 + w, c0 + w + 4, ... in that order, a lane
// four neighbouring elements of the head; the four sums are then added in the order of the warps.
// The order depends on the token's position only.
constexpr int COMBINE_WARPS = 4;
__global__ void __launch_bounds__(COMBINE_WARPS * 32)
attn_combine_kernel(const float *__restrict__ part_o, const float2 *__restrict__ part_ml,
                    const int *__restrict__ tok_pos, int nh, int window, int n_chunks,
                    bf16 *__restrict__ out, Finish finish, int keep_first) {
  pdl_launch();
  pdl_wait();
  __shared__ float s_max[COMBINE_WARPS];
  __shared__ float s_acc[COMBINE_WARPS][HD + 1];
  const size_t th = blockIdx.x;                                // t * nh + h
  const int t = (int)(th / nh);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Without a window a token's chunks are 0, 1, ...: those of a short table are asked for before the position is there (what lies
  // behind the token's last is not used), so that one round of loads is waited for instead of three: 2.9 us for eight tokens at 2,048 keys (3.2).
  const float2 *ml = part_ml + th * n_chunks;
  const bool active = 4 * lane < HD;
  constexpr int AHEAD = 8;
  const bool ahead = window == 0 && n_chunks <= AHEAD * COMBINE_WARPS;
  float2 own = make_float2(-INFINITY, 0.f), mlv[AHEAD];
  float4 ov[AHEAD];
  if (ahead) {
    if ((int)threadIdx.x < n_chunks) own = ml[threadIdx.x];
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      const int i = warp + u * COMBINE_WARPS;
      if (i < n_chunks) {
        mlv[u] = ml[i];
        if (active) ov[u] = *reinterpret_cast<const float4 *>(part_o + (th * n_chunks + i) * HD + 4 * lane);
      }
    }
  }
  const int pos = tok_pos[t];
  const int lo = first_visible_key(pos, window);
  const Chunks chunk_of(pos, lo, kept_keys(lo, keep_first));
  const int total = chunk_of.total;
  float M = -INFINITY;
  if (ahead) M = (int)threadIdx.x < total ? own.x : -INFINITY;
  else
    for (int i = (int)threadIdx.x; i < total; i += COMBINE_WARPS * 32) M = fmaxf(M, ml[chunk_of(i)].x);
  M = warp_max(M);
  if (lane == 0) s_max[warp] = M;
  __syncthreads();
  M = fmaxf(fmaxf(s_max[0], s_max[1]), fmaxf(s_max[2], s_max[3]));
  float4 num = make_float4(0.f, 0.f, 0.f, 0.f);
  float den = 0.f;
  // eight chunks' loads in flight at a time (a token far into its sequence has hundreds of chunks,
  // and one load after the other cost 20 us at 65,536 keys); they are added in the same order
  for (int i0 = warp; i0 < total; i0 += AHEAD * COMBINE_WARPS) {
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      if (!ahead && i0 + u * COMBINE_WARPS < total) {
        const int i = chunk_of(i0 + u * COMBINE_WARPS);
        mlv[u] = ml[i];
        if (active) ov[u] = *reinterpret_cast<const float4 *>(part_o + (th * n_chunks + i) * HD + 4 * lane);
      }
    }
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      if (i0 + u * COMBINE_WARPS < total) {
        const float w = fast_exp2(mlv[u].x - M);
        if (active) {
          num.x = fmaf(w, ov[u].x, num.x); num.y = fmaf(w, ov[u].y, num.y);
          num.z = fmaf(w, ov[u].z, num.z); num.w = fmaf(w, ov[u].w, num.w);
        }
        den = fmaf(w, mlv[u].y, den);
      }
    }
  }
  if (active) {
    s_acc[warp][4 * lane] = num.x; s_acc[warp][4 * lane + 1] = num.y;
    s_acc[warp][4 * lane + 2] = num.z; s_acc[warp][4 * lane + 3] = num.w;
  }
  if (lane == 0) s_acc[warp][HD] = den;
  __syncthreads();
  for (int d = threadIdx.x; d < HD; d += COMBINE_WARPS * 32) {
    const float n = ((s_acc[0][d] + s_acc[1][d]) + s_acc[2][d]) + s_acc[3][d];
    const float dn = finish(((s_acc[0][HD] + s_acc[1][HD]) + s_acc[2][HD]) + s_acc[3][HD], M, t, (int)(th % nh));
    out[th * HD + d] = __float2bfloat16_rn(n / dn);
  }
}

