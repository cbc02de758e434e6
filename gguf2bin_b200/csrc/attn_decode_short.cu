// Decode attention of steps with little to read: few sequences, few heads or few keys.  Latency is what such a step waits for (a round of
// loads, the chain of products of a segment, the merge, a launch), so the keys are spread as widely as the sums allow, and what stands in
// front of the attention and behind it runs in the same launch.
//
// Every token t of the step attends to the keys 0..pos_t of its sequence in the paged bfloat16 cache (or those that its window leaves),
// as in attn_decode.cu, whose formula, options and layout these are.  Grid (chunk of 128 keys, kv head x head tile, token): chunks start at
// absolute positions, a CTA takes one for ALL query heads that share the kv head (the rows of a 16-row tensor-core tile), and each of its
// eight warps takes 16 keys: 16 rows of K and V, copied with 16-byte cp.async, read back with ldmatrix.  Scores, softmax statistics and the
// output are 32-bit; probabilities are rounded to bfloat16 for the P.V product.  The warps' partial outputs are added in warp order.
//
// How the chunks of a token meet.  Where the caller passes no scratch, they are one thread-block cluster (up to CLUSTER_MOST chunks, 2,048 keys): every CTA sends each
// CTA of the cluster its share of the partial output (and all maxima and sums) through distributed
// shared memory, and after one cluster barrier the CTAs write a share of the heads each.  Else the chunks
// leave unnormalised partial outputs with their maxima and sums (log2 domain) in scratch, which
// `attn_combine_kernel` merges.  Both add in the same order, which depends on the token's position only.
//
// What stands in front of it.  `g2b_attn_decode_short_qkv` takes the token's projection [q heads | k heads | v heads]: norm and
// rotation of the heads are done here, row by row as qknorm_rope_fast_kernel (elementwise.cu) does them, in every CTA that needs the row; the
// token's own key and value are put among the rows of the cache from shared memory, and the warp whose keys they follow writes them to the cache.
//
// Measured in a chain of launches, norm, rotation and merge included, 16 query heads of 128 on 8: one sequence at 550 keys 3.9 us (8.4 by
// qknorm_rope_fast_kernel, attn_decode_kernel with two warps of 64 keys and attn_combine_kernel), at 2,000 keys 5.9 (8.4), at 4,000 keys
// 7.5 (9.3); two at 1,000 keys 4.8 (8.8), four at 500 4.9 (8.9), eight at 500 6.7 (9.9), sixteen at 200 6.2 (10.1).  Not for clusters or CTAs that
// have to wait for others to end (`decode_plan` in kernels_bf16.py draws the line), nor for steps whose keys fill the memory's rate (8 sequences at
// 2,048 keys): there the three launches leave the memory time to run ahead, and one launch in their place was slower (90 ms against 82 for eight
// requests of 64 tokens).
//
// Formula: src/l5_model.c:518, 559-577 of AnonymoDGH/gguf2bin.  Compiled per head size (-DHD=64 or 128); the page size is 64 keys.
#include "common.cuh"

G2B_DEFINE_LAST_ERROR

#ifndef HD
#define HD 128
#endif
static_assert(HD == 64 || HD == 128, "attn_decode_short: head sizes 64 and 128");
constexpr int CHUNK_KEYS = 128;
#include "attn_decode_common.cuh"

constexpr int SEG = 16;                        // keys of a warp
constexpr int WARPS = CHUNK_KEYS / SEG;
constexpr int THREADS = WARPS * 32;
constexpr int SEG_BYTES = SEG * ROW_BYTES;
constexpr int CLUSTER_MOST = 16;               // chunks of a token that are merged inside a cluster

// Rows [from, to) of a segment, asynchronously; `rows` is the segment's first row.
__device__ __forceinline__ void load_rows(uint32_t panel, const bf16 *rows, int from, int to, int lane) {
#pragma unroll
  for (int i = 0; i < SEG * ROW_CHUNKS / 32; ++i) {
    const int idx = i * 32 + lane;
    const int row = idx / ROW_CHUNKS, piece = idx % ROW_CHUNKS;
    if (row >= from && row < to) cp_async_16(panel + swz(row, piece), rows + (size_t)row * HD + piece * 8);
  }
}

__device__ __forceinline__ void st_shared16(uint32_t addr, uint4 v) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};\n" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// Rows from `from` on hold no key that the token may see: zeros, so that a weight of zero meets a finite value.
__device__ __forceinline__ void zero_rows(uint32_t panel, int from, int lane) {
  for (int idx = from * ROW_CHUNKS + lane; idx < SEG * ROW_CHUNKS; idx += 32)
    st_shared16(panel + swz(idx / ROW_CHUNKS, idx % ROW_CHUNKS), make_uint4(0, 0, 0, 0));
}
// The token's own key or value in its row.
__device__ __forceinline__ void own_row(uint32_t panel, int row, const bf16 *own, int lane) {
  if (lane < ROW_CHUNKS) st_shared16(panel + swz(row, lane), *reinterpret_cast<const uint4 *>(own + lane * 8));
}
// What a warp makes of its segment: the unnormalised output of the tile's 16 query rows
// (lane (g, c) holds rows g and g + 8, columns 8n + 2c, 8n + 2c + 1), their maxima (log2 domain) and sums.
struct Partial {
  float o[DTILES][4];
  float m[2], l[2];
};

// A key is visible if it is at most `pos` and either at least `lo` or below `kept_end`; the segment holds one that is.  The
// copies of K and V are under way, V's in a group of their own behind K's.
__device__ __forceinline__ void attend(Partial &acc, const uint32_t (&qa)[KSTEPS][4], uint32_t k_smem, uint32_t v_smem, int key0, int pos, int lo,
                                       int kept_end, ScoreMap score, int lane) {
  const int c = lane & 3;
  cp_async_wait<1>();                      // K has landed
  __syncwarp();
  float s[SEG / 8][4] = {};
#pragma unroll
  for (int kp = 0; kp < KSTEPS / 2; ++kp) {          // the chains of the two tiles of 8 keys side by side
    uint32_t kb[SEG / 8][4];
#pragma unroll
    for (int j = 0; j < SEG / 8; ++j) ldmatrix_x4(kb[j], k_smem + swz(8 * j + (lane & 7), 4 * kp + (lane >> 3)));
#pragma unroll
    for (int j = 0; j < SEG / 8; ++j) mma_bf16_16816(s[j], qa[2 * kp], kb[j][0], kb[j][1]);
#pragma unroll
    for (int j = 0; j < SEG / 8; ++j) mma_bf16_16816(s[j], qa[2 * kp + 1], kb[j][2], kb[j][3]);
  }
  // scale (log2 domain), mask, maximum and sum
  float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
  for (int j = 0; j < SEG / 8; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int key = key0 + 8 * j + 2 * c + (e & 1);
      s[j][e] = (key <= pos && (key >= lo || key < kept_end)) ? score(s[j][e]) : -INFINITY;
      mx[e >> 1] = fmaxf(mx[e >> 1], s[j][e]);
    }
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
    acc.m[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
    acc.l[r] = 0.f;
  }
  uint32_t pa[4];
#pragma unroll
  for (int j = 0; j < SEG / 8; ++j) {
    const float p0 = fast_exp2(s[j][0] - acc.m[0]), p1 = fast_exp2(s[j][1] - acc.m[0]);
    const float p2 = fast_exp2(s[j][2] - acc.m[1]), p3 = fast_exp2(s[j][3] - acc.m[1]);
    acc.l[0] += p0 + p1;
    acc.l[1] += p2 + p3;
    pa[j * 2 + 0] = pack_bf16(p0, p1);
    pa[j * 2 + 1] = pack_bf16(p2, p3);
  }
  cp_async_wait<0>();                      // V has landed
  __syncwarp();
#pragma unroll
  for (int dp = 0; dp < DTILES / 2; ++dp) {
    uint32_t vb[4];
    // matrices: (keys +0..7, d tile 2dp), (keys +8..15, d tile 2dp), (keys +0..7, 2dp+1), (+8..15, 2dp+1)
    const int mi = lane >> 3;
    ldmatrix_x4_trans(vb, v_smem + swz((mi & 1) * 8 + (lane & 7), 2 * dp + (mi >> 1)));
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      acc.o[2 * dp + u][0] = acc.o[2 * dp + u][1] = acc.o[2 * dp + u][2] = acc.o[2 * dp + u][3] = 0.f;
      mma_bf16_16816(acc.o[2 * dp + u], pa, vb[2 * u], vb[2 * u + 1]);
    }
  }
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    acc.l[r] += __shfl_xor_sync(0xffffffffu, acc.l[r], 1);
    acc.l[r] += __shfl_xor_sync(0xffffffffu, acc.l[r], 2);
  }
}

// ---- clusters -----------------------------------------------------------------------------------------
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory"); }
__device__ __forceinline__ uint32_t in_cta(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_cluster(uint32_t addr, float4 v) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};\n" ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
__device__ __forceinline__ void st_cluster(uint32_t addr, float2 v) {
  asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};\n" ::"r"(addr), "f"(v.x), "f"(v.y) : "memory");
}

// ---- norm and rotation of the token's own rows -------------------------------------------------------------
struct Prologue {
  const bf16 *qkv;               // [T, (nh + 2 nkv) * HD]
  const float *q_w, *k_w;        // [HD] or null: no norm
  const float2 *rope;            // [T, HD / 2] (cos, sin) or null: no rotation
  float eps;
};
constexpr int ROW_LANES = HD / 8;                          // lanes a row: four elements of either half each
constexpr int ROWS_AT_ONCE = THREADS / ROW_LANES;

// Shared memory: the warps' K and V segments (later their partial outputs), the warps' maxima and sums, the query tile with the token's
// own key and value behind it (OWN), what the cluster's CTAs send (CLUSTER).
constexpr int STATS_AT = WARPS * 2 * SEG_BYTES;
constexpr int TILE_AT = STATS_AT + WARPS * 16 * 8;
constexpr int TILE_BYTES = 16 * ROW_BYTES, OWN_BYTES = 2 * ROW_BYTES;
static_assert(WARPS * 16 * HD * 4 <= STATS_AT, "the partial outputs lie where the segments were");
template <bool OWN> __host__ __device__ constexpr int received_at() { return TILE_AT + (OWN ? TILE_BYTES + OWN_BYTES : 0); }
struct Received {                                          // [source][share] float4, then [source][rows] (maximum, sum)
  int share;
  __host__ __device__ Received(int rows, int n) : share((rows * HD / 4 + n - 1) / n) {}
  __host__ __device__ int out(int source, int unit) const { return (source * share + unit) * 16; }
  __host__ __device__ int stats(int n, int source, int row, int rows) const { return n * share * 16 + (source * rows + row) * 8; }
  __host__ __device__ int bytes(int n, int rows) const { return stats(n, n, 0, rows); }
};

// One element of a head from the partial outputs of its chunks: numbers 0, 4, ..., then 1, 5, ..., and so on, and the four sums in
// that order, as attn_combine_kernel adds them; eight chunks are read at once.
template <typename Stats, typename Out>
__device__ __forceinline__ float merge_chunks(const Chunks &chunks, Stats stats, Out part, const Finish &finish, int t, int h) {
  float M = -INFINITY, num[4] = {0.f, 0.f, 0.f, 0.f}, den[4] = {0.f, 0.f, 0.f, 0.f};
  float2 ml[8];
  float v[8];
  auto read = [&](int i0) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      ml[i] = make_float2(-INFINITY, 0.f);
      v[i] = 0.f;
      if (i0 + i < chunks.total) {
        ml[i] = stats(chunks(i0 + i));
        v[i] = part(chunks(i0 + i));
      }
    }
  };
  read(0);
#pragma unroll
  for (int i = 0; i < 8; ++i) M = fmaxf(M, ml[i].x);
  for (int i = 8; i < chunks.total; ++i) M = fmaxf(M, stats(chunks(i)).x);
  for (int i0 = 0;;) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float f = fast_exp2(ml[i].x - M);
      num[i % 4] = fmaf(f, v[i], num[i % 4]);
      den[i % 4] = fmaf(f, ml[i].y, den[i % 4]);
    }
    i0 += 8;
    if (i0 >= chunks.total) break;
    read(i0);
  }
  return (((num[0] + num[1]) + num[2]) + num[3]) / finish(((den[0] + den[1]) + den[2]) + den[3], M, t, h);
}

template <bool OWN, bool CLUSTER>
__global__ void __launch_bounds__(THREADS, 2)
attn_decode_short_kernel(const bf16 *__restrict__ q, Prologue pro, bf16 *cache,
                   const int *__restrict__ tok_pos, const int *__restrict__ tok_seq,
                   const int *__restrict__ page_table, int P, int nh, int nkv, int window,
                   ScoreMap score, float *part_o, float2 *part_ml, bf16 *__restrict__ out, Finish finish,
                   int n_chunks, int planes, int q_stride, int keep_first, int v_heads) {
  pdl_launch();
  extern __shared__ __align__(128) unsigned char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, c = lane & 3;
  const int group = nh / nkv;
  const int head_tiles = (group + 15) / 16;
  const int chunk = blockIdx.x;
  const int kvh = blockIdx.y / head_tiles, ht = blockIdx.y % head_tiles;
  const int rows = min(16, group - ht * 16);     // query heads of this tile
  const int t = blockIdx.z;
  const int key_begin = chunk * CHUNK_KEYS;
  const int key0 = key_begin + warp * SEG;       // the warp's first key
  const uint32_t k_smem = smem_u32(smem) + warp * 2 * SEG_BYTES, v_smem = k_smem + SEG_BYTES;
  unsigned char *const tile = smem + TILE_AT;
  const bf16 *const own = reinterpret_cast<const bf16 *>(tile + TILE_BYTES);
  const Received rx(rows, CLUSTER ? n_chunks : 1);

  // Before the kernels in front of this one are done (they compute this token's query and
  // may write its key and value), the warp's first segment can already be on its way as far as its keys are
  // OLD: below the token's position and therefore completed by an
  // earlier step.  The position itself is moved on the device by earlier kernels (one forward
  // at the end of every step; one back when a step that was launched ahead is taken back), so
  // what is read here is a hint: it may lag behind by any number of steps, which is harmless
  // (whichever value is seen was written after every key below it), and it may be one too
  // large while a take-back is still on its way, which the "- 1" allows for.  Not with a
  // window, whose lower edge moves with the position.
  const int hint = ld_volatile(tok_pos + t);
  // the batch's layout (which sequence, which pages) was copied to the device before the step's
  // first kernel was launched, so it may be read above the dependency line
  const int b = tok_seq[t];
  const size_t panel_elems = (size_t)PAGE * HD;
  const int vh = kvh % v_heads;                  // several key heads may share one value head
  const int phys = page_table[(size_t)b * P + min(key0 / PAGE, P - 1)];
  // planes == 1: the page's one panel per kv head is read as keys and again as values
  const size_t row0 = (size_t)(key0 % PAGE) * HD;
  bf16 *const k_rows = cache + ((size_t)phys * planes * nkv + kvh) * panel_elems + row0;
  bf16 *const v_rows = planes == 1 ? k_rows : cache + (((size_t)phys * 2 + 1) * nkv + vh) * panel_elems + row0;
  const int early = window == 0 ? max(0, min(SEG, hint - 1 - key0)) : 0;
  if (early > 0) {
    load_rows(k_smem, k_rows, 0, early, lane);
    cp_async_commit();
    load_rows(v_smem, v_rows, 0, early, lane);
    cp_async_commit();
  }
  // row r of the prologue: the tile's query heads, then the token's key and value
  const int sub = threadIdx.x / ROW_LANES, j4 = 4 * (threadIdx.x % ROW_LANES);
  float wq[8], wk[8];
  if (OWN) {
    if (pro.q_w) {
      *reinterpret_cast<float4 *>(wq) = *reinterpret_cast<const float4 *>(pro.q_w + j4);
      *reinterpret_cast<float4 *>(wq + 4) = *reinterpret_cast<const float4 *>(pro.q_w + HD / 2 + j4);
    }
    if (pro.k_w) {
      *reinterpret_cast<float4 *>(wk) = *reinterpret_cast<const float4 *>(pro.k_w + j4);
      *reinterpret_cast<float4 *>(wk + 4) = *reinterpret_cast<const float4 *>(pro.k_w + HD / 2 + j4);
    }
    for (int i = rows * ROW_CHUNKS + threadIdx.x; i < 16 * ROW_CHUNKS; i += THREADS)      // rows that no head fills
      *reinterpret_cast<uint4 *>(tile + i * 16) = make_uint4(0, 0, 0, 0);
  }
  if (CLUSTER) cluster_arrive();           // this CTA runs: the others may write to its shared memory
  pdl_wait();
  const int pos = ld_volatile(tok_pos + t);
  // What depends on the token alone is asked for while its position is on the way: its query, or its rows of the projection.
  uint32_t qa[KSTEPS][4];
  uint2 first, second;
  float4 turn[2];
  const bf16 *const src = OWN ? pro.qkv + (size_t)t * (nh + 2 * nkv) * HD + j4 : nullptr;
  auto fetch = [&](int r) {
    r = min(r, rows + 1);
    const int head = r < rows ? kvh * group + ht * 16 + r : (r == rows ? nh + kvh : nh + nkv + kvh);
    first = *reinterpret_cast<const uint2 *>(src + (size_t)head * HD);
    second = *reinterpret_cast<const uint2 *>(src + (size_t)head * HD + HD / 2);
  };
  if (OWN) {
    if (pro.rope) {
      const float4 *r = reinterpret_cast<const float4 *>(pro.rope + (size_t)t * (HD / 2) + j4);
      turn[0] = r[0];
      turn[1] = r[1];
    }
    fetch(sub);
  } else {
    load_q_tile(qa, q, t, q_stride, kvh, group, ht, g, c);
  }
  const int lo = first_visible_key(pos, window);
  const int kept_end = kept_keys(lo, keep_first);
  // no key of this chunk is seen (then nothing was fetched early)
  const bool seen = !(key_begin > pos || (key_begin + CHUNK_KEYS <= lo && key_begin >= kept_end));
  if (!CLUSTER && !seen) return;
  const Chunks chunks(pos, lo, kept_end);
  Partial acc;
#pragma unroll
  for (int n = 0; n < DTILES; ++n) acc.o[n][0] = acc.o[n][1] = acc.o[n][2] = acc.o[n][3] = 0.f;
  acc.m[0] = acc.m[1] = -INFINITY;
  acc.l[0] = acc.l[1] = 0.f;
  if (seen) {
    const bool active = key0 <= pos && (key0 + SEG > lo || key0 < kept_end);          // the warp's keys hold a visible one
    const int end = (OWN ? pos : pos + 1) - key0;        // rows below it are in the cache
    const bool ends = active && end < SEG;
    if (active && early < min(end, SEG)) load_rows(k_smem, k_rows, early, end, lane);
    cp_async_commit();
    if (active && early < min(end, SEG)) load_rows(v_smem, v_rows, early, end, lane);
    cp_async_commit();
    if (ends) {
      zero_rows(k_smem, end + OWN, lane);
      zero_rows(v_smem, end + OWN, lane);
    }
    if (OWN) {
      for (int r0 = 0; r0 < rows + 2; r0 += ROWS_AT_ONCE) {
        const int r = r0 + sub;
        const float2 x0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&first.x));
        const float2 x1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&first.y));
        const float2 y0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&second.x));
        const float2 y1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&second.y));
        if (r0 + ROWS_AT_ONCE < rows + 2) fetch(r + ROWS_AT_ONCE);
        float a[4] = {x0.x, x0.y, x1.x, x1.y}, h[4] = {y0.x, y0.y, y1.x, y1.y};
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          ss = fmaf(a[i], a[i], ss);
          ss = fmaf(h[i], h[i], ss);
        }
#pragma unroll
        for (int d = ROW_LANES / 2; d > 0; d >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, d);
        if (r < rows ? pro.q_w != nullptr : (r == rows && pro.k_w)) {
          const float inv = 1.f / sqrtf(ss / (float)HD + pro.eps);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            a[i] = ((r < rows ? wq[i] : wk[i]) * a[i]) * inv;
            h[i] = ((r < rows ? wq[4 + i] : wk[4 + i]) * h[i]) * inv;
          }
        }
        if (pro.rope && r <= rows) {
#pragma unroll
          for (int i = 0; i < 4; i += 2) {
            const float4 cs = turn[i / 2];
            const float a0 = a[i], b0 = h[i], a1 = a[i + 1], b1 = h[i + 1];
            a[i] = a0 * cs.x - b0 * cs.y;
            h[i] = a0 * cs.y + b0 * cs.x;
            a[i + 1] = a1 * cs.z - b1 * cs.w;
            h[i + 1] = a1 * cs.w + b1 * cs.z;
          }
        }
        if (r < rows + 2) {
          unsigned char *to_a, *to_h;
          if (r < rows) {
            to_a = tile + swz(r, j4 / 8) + (j4 % 8) * 2;
            to_h = tile + swz(r, (HD / 2 + j4) / 8) + (j4 % 8) * 2;
          } else {
            to_a = tile + TILE_BYTES + (r - rows) * ROW_BYTES + j4 * 2;
            to_h = to_a + HD;
          }
          *reinterpret_cast<uint2 *>(to_a) = make_uint2(pack_bf16(a[0], a[1]), pack_bf16(a[2], a[3]));
          *reinterpret_cast<uint2 *>(to_h) = make_uint2(pack_bf16(h[0], h[1]), pack_bf16(h[2], h[3]));
        }
      }
      __syncthreads();
#pragma unroll
      for (int ks = 0; ks < KSTEPS; ++ks) ldmatrix_x4(qa[ks], smem_u32(tile) + swz((lane & 7) + ((lane >> 3) & 1) * 8, 2 * ks + (lane >> 4)));
      if (ends) {                                // the token's own row, here and, by its first head tile, in the cache
        own_row(k_smem, end, own, lane);
        own_row(v_smem, end, own + HD, lane);
        if (ht == 0 && lane < ROW_CHUNKS) {
          *reinterpret_cast<uint4 *>(k_rows + (size_t)end * HD + lane * 8) = *reinterpret_cast<const uint4 *>(own + lane * 8);
          *reinterpret_cast<uint4 *>(v_rows + (size_t)end * HD + lane * 8) = *reinterpret_cast<const uint4 *>(own + HD + lane * 8);
        }
      }
    }
    if (active) attend(acc, qa, k_smem, v_smem, key0, pos, lo, kept_end, score, lane);
  }

  // The warps' partial outputs through shared memory (the segments are no longer needed), added in warp order.
  float *const xo = reinterpret_cast<float *>(smem);                       // [WARPS][rows][HD]
  float2 *const xml = reinterpret_cast<float2 *>(smem + STATS_AT);         // [WARPS][rows]
  if (seen) {
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int row = g + 8 * r;
      if (row >= rows) continue;
      float *po = xo + ((size_t)warp * rows + row) * HD;
#pragma unroll
      for (int n = 0; n < DTILES; ++n)
        *reinterpret_cast<float2 *>(po + 8 * n + 2 * c) = make_float2(acc.o[n][2 * r], acc.o[n][2 * r + 1]);
      if (c == 0) xml[warp * rows + row] = make_float2(acc.m[r], acc.l[r]);
    }
  }
  __syncthreads();
  if (CLUSTER) cluster_wait();                   // all CTAs of the cluster run (they arrived above the dependency line)
  unsigned char *const received = smem + received_at<OWN>();
  const uint32_t rx_at = smem_u32(received);
  const int units = rows * (HD / 4);             // pieces of four elements
  auto slot_of = [&](int row, int of) { return ((size_t)t * nh + (size_t)kvh * group + ht * 16 + row) * n_chunks + of; };
  if (seen) {
    for (int u = threadIdx.x; u < units; u += THREADS) {
      const int row = u / (HD / 4), col = 4 * (u % (HD / 4));
      float2 ml[WARPS];
      float4 v[WARPS];
#pragma unroll
      for (int w = 0; w < WARPS; ++w) {
        ml[w] = xml[w * rows + row];
        v[w] = *reinterpret_cast<const float4 *>(xo + ((size_t)w * rows + row) * HD + col);
      }
      float M = -INFINITY;
#pragma unroll
      for (int w = 0; w < WARPS; ++w) M = fmaxf(M, ml[w].x);
      float4 num = make_float4(0.f, 0.f, 0.f, 0.f);
      float den = 0.f;
#pragma unroll
      for (int w = 0; w < WARPS; ++w) {
        const float f = ml[w].x == -INFINITY ? 0.f : fast_exp2(ml[w].x - M);
        num.x = fmaf(f, v[w].x, num.x); num.y = fmaf(f, v[w].y, num.y);
        num.z = fmaf(f, v[w].z, num.z); num.w = fmaf(f, v[w].w, num.w);
        den = fmaf(f, ml[w].y, den);
      }
      if (CLUSTER) {
        const int whose = u / rx.share;
        st_cluster(in_cta(rx_at + rx.out(chunk, u - whose * rx.share), whose), num);
        if (col < 4 * n_chunks) st_cluster(in_cta(rx_at + rx.stats(n_chunks, chunk, row, rows), col / 4), make_float2(M, den));
      } else {
        const size_t slot = slot_of(row, chunk);
        __stcg(reinterpret_cast<float4 *>(part_o + slot * HD + col), num);
        if (col == 0) __stcg(part_ml + slot, make_float2(M, den));
      }
    }
  }
  if (!CLUSTER) return;
  const int head0 = kvh * group + ht * 16;
  bf16 *const to = out + ((size_t)t * nh + head0) * HD;
  cluster_arrive();
  cluster_wait();
  const int e0 = 4 * chunk * rx.share, e1 = min(4 * units, e0 + 4 * rx.share);                // this CTA's share
  for (int e = e0 + threadIdx.x; e < e1; e += THREADS)
    to[e] = __float2bfloat16_rn(merge_chunks(
        chunks, [&](int of) { return *reinterpret_cast<const float2 *>(received + rx.stats(n_chunks, of, e / HD, rows)); },
        [&](int of) { return *reinterpret_cast<const float *>(received + rx.out(of, 0) + (e - e0) * 4); }, finish, t, head0 + e / HD));
}

// Scratch; without it (null) the chunks of a token, CLUSTER_MOST at most, are merged in a cluster: part_o float [T*nh*n_chunks*HD], part_ml float2 [T*nh*n_chunks], with
// n_chunks = ceil(max_kv_len / 128).  q, out [T, nh*HD] bfloat16.
// With programmatic dependent launch on (g2b_set_pdl(1)) the kernel reads tok_pos once above
// the dependency line, as a hint for which old keys it may fetch early.  A caller whose own
// kernels move tok_pos while this one may already have started must keep to what the library
// does: positions grow, and shrink by at most one (a step taken back) between two launches.
// With ordinary launches (the default of a freshly loaded object) there is no such rule.
struct DecodeCall {
  const bf16 *q;
  Prologue pro;
  bf16 *out, *cache;
  const int *tok_pos, *tok_seq, *page_table;
  int P, T, nh, nkv, window;
  ScoreMap score;
  int n_chunks;
  float *part_o;
  float2 *part_ml;
  Finish finish;
  int planes, q_stride, keep_first, v_heads;
};

// Shared memory of a launch, and the most that any launch of the kernel asks for: what is allowed once per device, so that threads that meet in
// their first calls cannot lower it for one another.
template <bool OWN, bool CLUSTER> static int launch_smem(int rows, int last, int n) {
  const int a = Received(rows, n).bytes(n, rows), b = Received(last, n).bytes(n, last);
  return received_at<OWN>() + (CLUSTER ? (a > b ? a : b) : 0);
}
template <bool OWN, bool CLUSTER> static int most_smem() {
  int most = 0;
  for (int n = 1; n <= (CLUSTER ? CLUSTER_MOST : 1); ++n)
    for (int rows = 1; rows <= 16; ++rows) {
      const int need = launch_smem<OWN, CLUSTER>(rows, rows, n);
      most = need > most ? need : most;
    }
  return most;
}
template <bool OWN, bool CLUSTER> static int allow() {
  static G2bPerDevice configured;
  const int dev = g2b_current_device();
  if (dev < 0 || !configured.value[dev]) {
    cudaError_t e = cudaFuncSetAttribute(attn_decode_short_kernel<OWN, CLUSTER>, cudaFuncAttributeMaxDynamicSharedMemorySize, most_smem<OWN, CLUSTER>());
    if (e == cudaSuccess && CLUSTER)                                          // more than 8 CTAs
      e = cudaFuncSetAttribute(attn_decode_short_kernel<OWN, CLUSTER>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess)
      G2B_REFUSE("attn_decode_short: shared memory of %d bytes refused: %s", most_smem<OWN, CLUSTER>(), cudaGetErrorString(e));
    if (dev >= 0) configured.value[dev] = 1;
  }
  return 0;
}

template <bool OWN, bool CLUSTER>
static int launch_decode(const DecodeCall &c, cudaStream_t stream) {
  const int group = c.nh / c.nkv, head_tiles = (group + 15) / 16, rows = group < 16 ? group : 16;
  const int n = CLUSTER ? c.n_chunks : 1;
  const int last = (group - 1) % 16 + 1;         // heads of a kv head's last tile
  const int smem = launch_smem<OWN, CLUSTER>(rows, last, n);
  if (allow<OWN, CLUSTER>()) return 1;
  g2b_launch_cluster(attn_decode_short_kernel<OWN, CLUSTER>, dim3(c.n_chunks, c.nkv * head_tiles, c.T), dim3(THREADS), smem, stream,
                     (unsigned)n, c.q, c.pro, c.cache, c.tok_pos, c.tok_seq, c.page_table, c.P, c.nh, c.nkv, c.window, c.score, c.part_o,
                     c.part_ml, c.out, c.finish, c.n_chunks, c.planes, c.q_stride, c.keep_first, c.v_heads);
  const int rc = g2b_check_launch("attn_decode_short");
  if (rc || CLUSTER) return rc;
  g2b_launch(attn_combine_kernel, dim3((unsigned)((size_t)c.T * c.nh)), dim3(COMBINE_WARPS * 32), 0, stream,
             c.part_o, (const float2 *)c.part_ml, c.tok_pos, c.nh, c.window, c.n_chunks, c.out, c.finish, c.keep_first);
  return g2b_check_launch("attn_combine");
}

// What the device allows the form (own: with the prologue; cluster: merged in clusters) behind a launch of it, and the most that it may ask for.
extern "C" int g2b_attn_decode_short_smem(int own, int cluster, int *allowed, int *most) {
  const void *kernel = own ? (cluster ? (const void *)attn_decode_short_kernel<true, true> : (const void *)attn_decode_short_kernel<true, false>)
                           : (cluster ? (const void *)attn_decode_short_kernel<false, true> : (const void *)attn_decode_short_kernel<false, false>);
  cudaFuncAttributes attr;
  const cudaError_t e = cudaFuncGetAttributes(&attr, kernel);
  if (e != cudaSuccess) G2B_REFUSE("attn_decode_short: %s", cudaGetErrorString(e));
  *allowed = attr.maxDynamicSharedSizeBytes;
  *most = own ? (cluster ? most_smem<true, true>() : most_smem<true, false>()) : (cluster ? most_smem<false, true>() : most_smem<false, false>());
  return 0;
}

static int check_sizes(int T, int nh, int nkv, int hd, int page_size, int max_kv_len, float softcap, int window, int keep_first) {
  if (softcap < 0.f || keep_first < 0 || (keep_first > 0 && window <= 0))
    G2B_REFUSE("attn_decode_short: a cap of %g, %d first tokens kept with a window of %d", softcap, keep_first, window);
  if (hd != HD) G2B_REFUSE("attn_decode_short: built for head_dim %d, got %d", HD, hd);
  if (page_size != PAGE) G2B_REFUSE("attn_decode_short: page size must be %d, got %d", PAGE, page_size);
  if (nkv <= 0 || nh % nkv) G2B_REFUSE("attn_decode_short: %d heads are not a multiple of %d kv heads", nh, nkv);
  if (T > 65535) G2B_REFUSE("attn_decode_short: %d tokens in one step (at most 65535)", T);
  const int group = nh / nkv, head_tiles = (group + 15) / 16;
  if ((long long)nkv * head_tiles > 65535) G2B_REFUSE("attn_decode_short: too many kv heads (%d)", nkv);
  if (max_kv_len <= 0) G2B_REFUSE("attn_decode_short: max_kv_len %d", max_kv_len);
  return 0;
}
static int chunks_of(int max_kv_len) { return (max_kv_len + CHUNK_KEYS - 1) / CHUNK_KEYS; }
static int check_form(const DecodeCall &c) {
  if (!c.part_o && c.n_chunks > CLUSTER_MOST) G2B_REFUSE("attn_decode_short: %d chunks are more than a cluster (%d) and there is no scratch", c.n_chunks, CLUSTER_MOST);
  if (c.part_o && !c.part_ml) G2B_REFUSE("attn_decode_short: no scratch for the statistics");
  return 0;
}

// How many clusters of n_chunks CTAs the device holds at once; 0 where it holds none (own: with the prologue).
template <bool OWN> static int count_clusters(int n) {
  if (n > CLUSTER_MOST || allow<OWN, true>()) return 0;
  int smem = 0, clusters = 0;
  for (int rows = 1; rows <= 16; ++rows) smem = max(smem, launch_smem<OWN, true>(rows, rows, n));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(n), cfg.blockDim = dim3(THREADS), cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = n, attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr, cfg.numAttrs = 1;
  if (cudaOccupancyMaxActiveClusters(&clusters, attn_decode_short_kernel<OWN, true>, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return clusters;
}
extern "C" int g2b_attn_decode_short_clusters(int own, int max_kv_len) {
  const int n = max_kv_len > 0 ? chunks_of(max_kv_len) : 0;
  return n <= 0 ? 0 : own ? count_clusters<true>(n) : count_clusters<false>(n);
}

// Arguments as g2b_attn_decode_ex (attn_decode.cu); scratch null: clusters merge.
extern "C" int g2b_attn_decode_short(const void *q, void *out, const void *cache, const int *tok_pos,
                                  const int *tok_seq, const int *page_table, int P, int T, int nh,
                                  int nkv, int hd, int page_size, int window, float scale,
                                  int max_kv_len, float *part_o, float *part_ml,
                                  const float *sink, int planes, int q_stride, const void *gate,
                                  int gate_stride, float softcap, int keep_first, int v_heads, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (v_heads <= 0) v_heads = nkv;
  if (nkv > 0 && (v_heads > nkv || nkv % v_heads)) G2B_REFUSE("attn_decode_short: %d key heads on %d value heads", nkv, v_heads);
  if (planes != 1 && planes != 2) G2B_REFUSE("attn_decode_short: %d panels per page and kv head (1 or 2)", planes);
  if (q_stride < nh * hd || q_stride % 2) G2B_REFUSE("attn_decode_short: query rows %d elements apart", q_stride);
  if (check_sizes(T, nh, nkv, hd, page_size, max_kv_len, softcap, window, keep_first)) return 1;
  const DecodeCall call = {(const bf16 *)q, Prologue{}, (bf16 *)out, (bf16 *)const_cast<void *>(cache), tok_pos, tok_seq, page_table, P, T,
                           nh, nkv, window, ScoreMap{scale * LOG2E, softcap > 0.f ? scale / softcap : 0.f, softcap * LOG2E},
                           chunks_of(max_kv_len), part_o, (float2 *)part_ml,
                           Finish{sink, (const bf16 *)gate, gate_stride}, planes, q_stride, keep_first, v_heads};
  if (check_form(call)) return 1;
  return call.part_o ? launch_decode<false, false>(call, stream) : launch_decode<false, true>(call, stream);
}

// The same from the projection of the step's tokens, qkv [T, (nh + 2 nkv) * HD] = [q heads | k heads | v heads] as g2b_qknorm_rope_cache
// (elementwise.cu) takes it: norm of the q and k heads by q_w and k_w [HD] (null: none), rotation of whole heads by the
// step's table rope [T, HD / 2, 2] (null: none), the token's key and value written to the layer's cache.  All pointers on 16 bytes.
extern "C" int g2b_attn_decode_short_qkv(const void *qkv, const float *q_w, const float *k_w, float eps, const float *rope, void *out,
                                   void *cache, const int *tok_pos, const int *tok_seq, const int *page_table, int P, int T, int nh,
                                   int nkv, int hd, int page_size, int window, float scale, int max_kv_len, float *part_o,
                                   float *part_ml, const float *sink, float softcap, int keep_first,
                                   cudaStream_t stream) {
  if (T <= 0) return 0;
  if (check_sizes(T, nh, nkv, hd, page_size, max_kv_len, softcap, window, keep_first)) return 1;
  if (((uintptr_t)qkv | (uintptr_t)q_w | (uintptr_t)k_w | (uintptr_t)rope | (uintptr_t)cache | (uintptr_t)out) & 15)
    G2B_REFUSE("attn_decode_short: operands must be 16-byte aligned");
  const DecodeCall call = {nullptr, Prologue{(const bf16 *)qkv, q_w, k_w, (const float2 *)rope, eps}, (bf16 *)out, (bf16 *)cache, tok_pos,
                           tok_seq, page_table, P, T, nh, nkv, window,
                           ScoreMap{scale * LOG2E, softcap > 0.f ? scale / softcap : 0.f, softcap * LOG2E},
                           chunks_of(max_kv_len), part_o, (float2 *)part_ml, Finish{sink, nullptr, 0}, 2, 0, keep_first,
                           nkv};
  if (check_form(call)) return 1;
  return call.part_o ? launch_decode<true, false>(call, stream) : launch_decode<true, true>(call, stream);
}
