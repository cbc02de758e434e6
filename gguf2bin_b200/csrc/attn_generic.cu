// Causal grouped-query attention over the paged cache, 32-bit arithmetic, any head size
// up to 512: one warp per (token, query head).  It serves prompts and single tokens
// alike (every token carries its own position), is the attention of the float32 path,
// and the fallback of the bfloat16 path for head sizes the tensor-core kernels refuse.
//
// Formula (src/l5_model.c:518, 559-577 of AnonymoDGH/gguf2bin): kv head = head / group;
// s_t = (q . K_t) * scale for t <= pos (the loop bound is the causal mask); softmax with
// the maximum subtracted (src/l3_math.c:52-56); o = sum_t p_t V_t.  `window` > 0 keeps
// only the keys with pos - window < t <= pos; `chunk` > 0 keeps only the keys of the token's own
// chunk, floor(pos / chunk) * chunk <= t <= pos (chunks count from position 0 of the sequence).
//
// Keys are visited in chunks of 32 that start at absolute positions that are multiples
// of 32, with a running maximum and sum, so the arithmetic for a (token, head) depends
// only on its own position: not on how the tokens were cut into steps, nor on the batch.
//
// Two options for other kinds of attention.  `sink` (one float per query head, or null): the
// softmax's denominator is sum_j exp(s_j) + exp(sink_h): the sink takes probability, adds
// nothing to the output, and is used as it is (the score scale does not apply).  `planes` = 1: a page holds one panel per kv head that serves as keys AND as
// values (attention over cached latents); 2: a panel of keys and a panel of values.
// `q_stride`: elements between the query rows of two tokens (the queries may be columns of a wider
// product's output).  `gate` (one number per token and head, or null): the head's output is
// multiplied by its sigmoid.
//
// `softcap` > 0: a score s becomes softcap tanh(s / softcap) after the scale.  `keep_first` > 0 (with a
// window): the keys at positions below it stay visible to every later token, at their true
// positions; they are visited first, in chunks of 32 from position 0.  `v_heads` < nkv: key head g
// reads the values of head g mod v_heads (several score maps over one set of values).
//
// `pool` > 0 (with a window): in front of the window's keys a token also sees one key and value for
// every block of `pool` positions that lies wholly before the window, block b if
// b pool + pool - 1 <= pos - window; they come from a second store (`pooled`, [pages, 2, nkv,
// pool_rows, hd]; block b in the page of its first position at row b - ceil(that page's first
// position / pool)) and share the softmax with the window's keys.  Blocks are visited first, in
// chunks of 32 from block 0, so the order still depends on the token's position only.
#include "common.cuh"

G2B_DEFINE_LAST_ERROR

#define AG_MAX_HD 512
#define AG_WARPS 4

template <typename T>
__global__ void __launch_bounds__(AG_WARPS * 32)
attn_generic_kernel(const T *__restrict__ q, T *__restrict__ out, const T *__restrict__ cache,
                    const int *__restrict__ tok_pos, const int *__restrict__ tok_seq,
                    const int *__restrict__ page_table, int P, int n_tokens, int nh, int nkv,
                    int hd, int page_size, int window, float scale,
                    const float *__restrict__ sink, int planes, int q_stride,
                    const T *__restrict__ gate, int gate_stride, int chunk, const T *__restrict__ pooled,
                    int pool, int pool_rows, float softcap, int keep_first, int v_heads) {
  pdl_launch();
  pdl_wait();
  __shared__ float qs[AG_WARPS][AG_MAX_HD];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long item = (long long)blockIdx.x * AG_WARPS + warp;
  if (item >= (long long)n_tokens * nh) return;
  const int t = (int)(item / nh), h = (int)(item % nh);
  const int pos = tok_pos[t], b = tok_seq[t];
  const int kvh = h / (nh / nkv);
  const int vh = kvh % v_heads;                                   // several key heads may share one value head
  const int lo = chunk > 0 ? (pos / chunk) * chunk : (window > 0 ? max(0, pos - window + 1) : 0);

  const T *qp = q + (size_t)t * q_stride + (size_t)h * hd;
  for (int j = lane; j < hd; j += 32) qs[warp][j] = to_f32(qp[j]);
  __syncwarp();

  float m = -INFINITY, l = 0.f;
  float acc[AG_MAX_HD / 32];
#pragma unroll
  for (int i = 0; i < AG_MAX_HD / 32; ++i) acc[i] = 0.f;

  const size_t head_stride = (size_t)page_size * hd;              // one (page, K|V, kv head) panel
  if (pool > 0) {
    const int n_blocks = max(0, (pos - window + 1) / pool);       // window > 0 (the launcher checks)
    const size_t pstride = (size_t)pool_rows * hd;
    auto row_of = [&](int blk, const T *&kr, const T *&vr) {
      const int home = (blk * pool) / page_size;
      const int row = blk - (home * page_size + pool - 1) / pool;
      const size_t page = (size_t)page_table[(size_t)b * P + home];
      kr = pooled + ((page * 2 + 0) * nkv + kvh) * pstride + (size_t)row * hd;
      vr = pooled + ((page * 2 + 1) * nkv + kvh) * pstride + (size_t)row * hd;
    };
    for (int base = 0; base < n_blocks; base += 32) {
      const bool valid = base + lane < n_blocks;
      float s = -INFINITY;
      if (valid) {
        const T *kr, *vr;
        row_of(base + lane, kr, vr);
        float dot = 0.f;
        for (int j = 0; j < hd; ++j) dot = fmaf(qs[warp][j], to_f32(kr[j]), dot);
        s = dot * scale;
      }
      const float m_new = fmaxf(m, warp_max(s));                  // finite: block `base` is valid
      const float p = valid ? expf(s - m_new) : 0.f;
      const float corr = expf(m - m_new);
      l = l * corr + warp_sum(p);
#pragma unroll
      for (int i = 0; i < AG_MAX_HD / 32; ++i) acc[i] *= corr;
      const int n_here = min(32, n_blocks - base);
      for (int j = 0; j < n_here; ++j) {
        const float pj = __shfl_sync(0xffffffffu, p, j);
        const T *kr, *vr;
        row_of(base + j, kr, vr);
#pragma unroll
        for (int i = 0; i < AG_MAX_HD / 32; ++i) {
          const int d = lane + 32 * i;
          if (d < hd) acc[i] = fmaf(pj, to_f32(vr[d]), acc[i]);
        }
      }
      m = m_new;
    }
  }
  // keys base .. base + 31 that lie in first .. last
  auto visit = [&](int base, int first, int last) {
    const int page = page_table[(size_t)b * P + base / page_size];
    const T *kpanel = cache + (((size_t)page * planes + 0) * nkv + kvh) * head_stride;
    const T *vpanel = cache + (((size_t)page * planes + (planes - 1)) * nkv + (planes == 2 ? vh : kvh)) * head_stride;
    const int in_page = base % page_size;                         // chunk lies inside one page
    const int key = base + lane;
    const bool valid = key >= first && key <= last;
    float s = -INFINITY;
    if (valid) {
      const T *kr = kpanel + (size_t)(in_page + lane) * hd;
      float dot = 0.f;
      for (int j = 0; j < hd; ++j) dot = fmaf(qs[warp][j], to_f32(kr[j]), dot);
      s = dot * scale;
      if (softcap > 0.f) s = softcap * tanhf(s / softcap);
    }
    const float m_new = fmaxf(m, warp_max(s));                    // finite: key `last` or `base` valid
    const float p = valid ? expf(s - m_new) : 0.f;
    const float corr = expf(m - m_new);                           // 0 on the first chunk
    l = l * corr + warp_sum(p);
#pragma unroll
    for (int i = 0; i < AG_MAX_HD / 32; ++i) acc[i] *= corr;
    const int n_keys = min(32, last - base + 1);
    for (int j = 0; j < n_keys; ++j) {
      const float pj = __shfl_sync(0xffffffffu, p, j);
      if (base + j < first) continue;
      const T *vr = vpanel + (size_t)(in_page + j) * hd;
#pragma unroll
      for (int i = 0; i < AG_MAX_HD / 32; ++i) {
        const int d = lane + 32 * i;
        if (d < hd) acc[i] = fmaf(pj, to_f32(vr[d]), acc[i]);
      }
    }
    m = m_new;
  };
  if (keep_first > 0 && lo > 0) {                                 // the first tokens stay visible behind the window
    const int last = min(keep_first, lo) - 1;
    for (int base = 0; base <= last; base += 32) visit(base, 0, last);
  }
  for (int base = (lo / 32) * 32; base <= pos; base += 32) visit(base, lo, pos);
  T *op = out + (size_t)t * nh * hd + (size_t)h * hd;
  if (sink) l += expf(sink[h] - m);                                // m is finite: the token's own key
  float inv_l = 1.f / l;
  if (gate) inv_l *= 1.f / (1.f + expf(-to_f32(gate[(size_t)t * gate_stride + h])));   // the head's output gate
#pragma unroll
  for (int i = 0; i < AG_MAX_HD / 32; ++i) {
    const int d = lane + 32 * i;
    if (d < hd) op[d] = from_f32<T>(acc[i] * inv_l);
  }
}

// ---------------------------------------------------------------------------------------------------
// The same attention in float for pages of 64 keys, head sizes up to 256 that are multiples of 4, and no pooled blocks:
// a page's keys (a segment) are brought to shared memory once and serve many rows.  A score is the sum of four partial
// dot products (d mod 4, each in increasing d); a segment's scores have one maximum; its probabilities are added pairwise
// by a warp (keys i and i + 32 first); its weighted values are added in the order of the keys; segments are merged one after
// the other from the lowest.  Both kernels keep that order, so a row's result does not depend on which of the two computes it.
//
//   tile    a block per (32 rows of one prompt, query head) that walks the segments: prompts
//   split   a block per (token, kv head, segment), for all query heads of the kv head, and a merge: single tokens, whose
//           few rows leave the GPU to the segments
//
// 16 heads of 128 on 8 kv heads: two tokens behind 200 and 500 keys 7.4 + 4.2 us in a decode step (850 us with a warp a token
// and head, whose lanes read rows of 512 bytes each for themselves); prompts of 201 and 500 tokens 123 us.
#define SEG 64
#define F32_MAX_HD 256
#define F32_MAX_GROUP 32
#define F32_PART_EXTRA 2                                            // maximum and sum in front of a part's values

struct F32Attn {
  const float *q, *cache, *sink, *gate;
  float *out, *parts;
  const int *tok_pos, *tok_seq, *page_table, *tiles;
  int P, nh, nkv, hd, window, planes, q_stride, gate_stride, chunk, keep_first, v_heads, segments;
  float scale, softcap;
};

__device__ __forceinline__ int lowest_key(const F32Attn &p, int pos) {
  return p.chunk > 0 ? (pos / p.chunk) * p.chunk : (p.window > 0 ? max(0, pos - p.window + 1) : 0);
}
// may a token whose window starts at `lo` see `key` (at most the token's own position)?
__device__ __forceinline__ bool sees(const F32Attn &p, int lo, int key) { return key >= lo || key < p.keep_first; }
__device__ __forceinline__ bool sees_segment(const F32Attn &p, int lo, int pos, int seg) {
  return seg * SEG <= pos && (seg * SEG + SEG > lo || seg * SEG < p.keep_first);
}

__device__ __forceinline__ void bring_panel(float *to, const float *from, int hd, int tid, int threads) {
  for (int i = tid; i < SEG * (hd / 4); i += threads) {
    const int r = i / (hd / 4), c = i % (hd / 4) * 4;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(to + r * (hd + 4) + c)),
                 "l"(from + (size_t)r * hd + c));
  }
  asm volatile("cp.async.commit_group;\n" ::);
}
__device__ __forceinline__ const float *panel_of(const F32Attn &p, int seq, int seg, int kvh, bool values) {
  const size_t page = (size_t)p.page_table[(size_t)seq * p.P + seg];
  const int plane = values ? p.planes - 1 : 0, head = values && p.planes == 2 ? kvh % p.v_heads : kvh;
  return p.cache + ((page * p.planes + plane) * p.nkv + head) * ((size_t)SEG * p.hd);
}
__device__ __forceinline__ float scored(const F32Attn &p, float4 d) {
  const float s = ((d.x + d.y) + (d.z + d.w)) * p.scale;
  return p.softcap > 0.f ? p.softcap * tanhf(s / p.softcap) : s;
}
__device__ __forceinline__ void dot4(float4 &d, const float4 a, const float4 b) { fma4(d, a, b); }
// One warp: a row's 64 scores in shared memory become probabilities against the maximum of those that the token at `pos` sees, and
// HIDDEN where it does not.  What is hidden is decided by the positions alone: a score or a value that is NaN or infinite and
// seen, whatever its weight, reaches the result.
#define HIDDEN -1.f
__device__ __forceinline__ void soften(const F32Attn &p, float *row, int lane, int seg, int pos, float &m, float &l) {
  const int lo = lowest_key(p, pos), key = seg * SEG + lane;
  const bool see_a = key <= pos && sees(p, lo, key), see_b = key + 32 <= pos && sees(p, lo, key + 32);
  const float a = see_a ? row[lane] : -INFINITY, b = see_b ? row[lane + 32] : -INFINITY;
  m = warp_max(fmaxf(a, b));
  const float pa = a == -INFINITY ? 0.f : expf(a - m), pb = b == -INFINITY ? 0.f : expf(b - m);
  row[lane] = see_a ? pa : HIDDEN;
  row[lane + 32] = see_b ? pb : HIDDEN;
  l = warp_sum(pa + pb);
}
__device__ __forceinline__ bool hidden(float probability) { return probability < 0.f; }
// Adds a part (maximum m_part) to a running one: the factors for what is there and for what comes.  Where the maxima are equal both
// factors are 1, also in front of the first part and behind parts whose every score is -inf.
__device__ __forceinline__ void merge_factors(float &m, float m_part, float &old_factor, float &new_factor) {
  const float m_new = fmaxf(m, m_part);
  old_factor = m == m_new ? 1.f : expf(m - m_new);
  new_factor = m_part == m_new ? 1.f : expf(m_part - m_new);
  m = m_new;
}
__device__ __forceinline__ float merged(float there, float old_factor, float part, float new_factor) {
  return fmaf(part, new_factor, __fmul_rn(there, old_factor));
}
__device__ __forceinline__ float last_factor(const F32Attn &p, int t, int h, float m, float l) {
  if (p.sink) l += expf(p.sink[h] - m);
  float f = 1.f / l;
  if (p.gate) f *= 1.f / (1.f + expf(-p.gate[(size_t)t * p.gate_stride + h]));
  return f;
}

// Prompts: half a tile (32 rows) and a query head a block, two blocks an SM at head sizes up to 128, so that one's softmax and waits lie
// beside the other's products and a long prompt's last tiles are dealt out in halves.  A segment's keys are asked for as soon as the scores
// of the one in front are taken, its values behind that one's last sum.  All heads of the longest tiles come first: with head after head the last head's
// longest tiles began when the rest was done, and the SMs idled for 0.31 of the time (1,024 tokens).  Multiply-adds go two an instruction, since a warp's
// chain of instructions is what is waited for (131 and 804 us with one).  Prompts of 201 and 500 tokens 123 us (183 with 64 rows a block of 256 threads,
// panels brought when they were needed, head after head), one of 2,048 737 us (1,097).
#define F32_ROWS 32
#define F32_THREADS 128
template <bool B> struct Flag { static constexpr bool value = B; };
template <int HD4>                                                  // float4 columns of a row per thread: ceil(hd / 64)
__global__ void __launch_bounds__(F32_THREADS, HD4 <= 2 ? 2 : 1)
attn_f32_tile_kernel(F32Attn p) {
  pdl_launch();
  pdl_wait();
  extern __shared__ __align__(16) float sm[];
  constexpr int RS = F32_THREADS / 16, PITCH = SEG + 4;             // a thread's rows are ty, ty + RS, ...
  const int hd = p.hd, pitch = hd + 4;
  float *Qs = sm, *Ks = Qs + F32_ROWS * pitch, *Vs = Ks + SEG * pitch, *Ps = Vs + SEG * pitch;
  float *row_m = Ps + F32_ROWS * PITCH, *row_l = row_m + F32_ROWS, *old_f = row_l + F32_ROWS, *new_f = old_f + F32_ROWS;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, tx = tid & 15, ty = tid >> 4;
  const int half = blockIdx.x / p.nh, h = blockIdx.x % p.nh;        // all heads of the longest tiles first
  const int *tile = p.tiles + 4 * (half / 2);
  const int skip = F32_ROWS * (half % 2), rows = min(F32_ROWS, tile[2] - skip);
  if (rows <= 0) return;
  const int seq = tile[0], t0 = tile[1] + skip, pos0 = tile[3] + skip, kvh = h / (p.nh / p.nkv);
  const int last_pos = pos0 + rows - 1, lo0 = lowest_key(p, pos0);  // the first row's window starts lowest
  auto next_of = [&](int seg) {
    do ++seg;
    while (seg * SEG <= last_pos && !sees_segment(p, lo0, last_pos, seg));
    return seg;
  };
  int seg = next_of(-1);                                            // there is one: the rows' own
  bring_panel(Ks, panel_of(p, seq, seg, kvh, false), hd, tid, F32_THREADS);
  bring_panel(Vs, panel_of(p, seq, seg, kvh, true), hd, tid, F32_THREADS);
  for (int i = tid; i < F32_ROWS * (hd / 4); i += F32_THREADS) {
    const int r = i / (hd / 4), c = i % (hd / 4) * 4;
    *(float4 *)(Qs + r * pitch + c) =
        r < rows ? *(const float4 *)(p.q + (size_t)(t0 + r) * p.q_stride + (size_t)h * hd + c) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  if (tid < F32_ROWS) {
    row_m[tid] = -INFINITY;
    row_l[tid] = 0.f;
  }
  float4 O[4][HD4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < HD4; ++j) O[i][j] = make_float4(0.f, 0.f, 0.f, 0.f);
  while (seg * SEG <= last_pos) {
    const int next = next_of(seg);
    const bool more = next * SEG <= last_pos;
    asm volatile("cp.async.wait_group 1;\n" ::);                    // the keys; the values may be on their way
    __syncthreads();
    float4 S[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) S[i][j] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
    for (int d = 0; d < hd; d += 4) {
      float4 k[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) k[j] = *(const float4 *)(Ks + (tx + 16 * j) * pitch + d);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 q = *(const float4 *)(Qs + (ty + RS * i) * pitch + d);
#pragma unroll
        for (int j = 0; j < 4; ++j) dot4(S[i][j], q, k[j]);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) Ps[(ty + RS * i) * PITCH + tx + 16 * j] = scored(p, S[i][j]);
    __syncthreads();                                                // the keys are read
    if (more) bring_panel(Ks, panel_of(p, seq, next, kvh, false), hd, tid, F32_THREADS);
    else asm volatile("cp.async.commit_group;\n" ::);
#pragma unroll 4
    for (int r = warp; r < F32_ROWS; r += F32_THREADS / 32) {
      float m, l;                                                   // rows behind the last see nothing, like rows before a window
      soften(p, Ps + r * PITCH, lane, seg, r < rows ? pos0 + r : -1, m, l);
      if (lane == 0) {
        float there = row_m[r], of, nf;
        merge_factors(there, m, of, nf);
        row_m[r] = there;
        row_l[r] = merged(row_l[r], of, l, nf);
        old_f[r] = of;
        new_f[r] = nf;
      }
    }
    asm volatile("cp.async.wait_group 1;\n" ::);                    // the values; the next keys may be on their way
    __syncthreads();
    float4 acc[4][HD4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < HD4; ++j) acc[i][j] = make_float4(0.f, 0.f, 0.f, 0.f);
    // four keys at a time; a probability of 0 for a key behind n_keys is HIDDEN already
    auto weigh = [&](auto all_seen, int n_keys) {
      for (int key = 0; key < n_keys; key += 4) {
        float4 pr[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) pr[i] = *(const float4 *)(Ps + (ty + RS * i) * PITCH + key);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          float4 v[HD4];
#pragma unroll
          for (int j = 0; j < HD4; ++j)
            if (64 * j + 4 * tx < hd) v[j] = *(const float4 *)(Vs + (key + u) * pitch + 64 * j + 4 * tx);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float w = u == 0 ? pr[i].x : (u == 1 ? pr[i].y : (u == 2 ? pr[i].z : pr[i].w));
            if (decltype(all_seen)::value || !hidden(w))            // a value that is not seen is not touched, whatever it holds
#pragma unroll
              for (int j = 0; j < HD4; ++j)
                if (64 * j + 4 * tx < hd) fma4(acc[i][j], make_float4(w, w, w, w), v[j]);
          }
        }
      }
    };
    if (rows == F32_ROWS && seg * SEG + SEG - 1 <= pos0 && seg * SEG >= lowest_key(p, last_pos)) weigh(Flag<true>(), SEG);
    else weigh(Flag<false>(), min(SEG, last_pos - seg * SEG + 1));
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float of = old_f[ty + RS * i], nf = new_f[ty + RS * i];
#pragma unroll
      for (int j = 0; j < HD4; ++j) {
        O[i][j].x = merged(O[i][j].x, of, acc[i][j].x, nf);
        O[i][j].y = merged(O[i][j].y, of, acc[i][j].y, nf);
        O[i][j].z = merged(O[i][j].z, of, acc[i][j].z, nf);
        O[i][j].w = merged(O[i][j].w, of, acc[i][j].w, nf);
      }
    }
    __syncthreads();                                                // the values, the probabilities and the factors are read
    if (more) bring_panel(Vs, panel_of(p, seq, next, kvh, true), hd, tid, F32_THREADS);
    else asm volatile("cp.async.commit_group;\n" ::);
    seg = next;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = ty + RS * i;
    if (r >= rows) continue;
    const float f = last_factor(p, t0 + r, h, row_m[r], row_l[r]);
    float *op = p.out + (size_t)(t0 + r) * p.nh * hd + (size_t)h * hd;
#pragma unroll
    for (int j = 0; j < HD4; ++j)
      if (64 * j + 4 * tx < hd)
        *(float4 *)(op + 64 * j + 4 * tx) = make_float4(O[i][j].x * f, O[i][j].y * f, O[i][j].z * f, O[i][j].w * f);
  }
}

__global__ void __launch_bounds__(128)
attn_f32_split_kernel(F32Attn p) {
  pdl_launch();
  pdl_wait();
  extern __shared__ __align__(16) float sm[];
  const int hd = p.hd, pitch = hd + 4, group = p.nh / p.nkv, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int seg = blockIdx.x, kvh = blockIdx.y, t = blockIdx.z;
  const int pos = p.tok_pos[t], seq = p.tok_seq[t], lo = lowest_key(p, pos);
  if (!sees_segment(p, lo, pos, seg)) return;
  float *Ks = sm, *Vs = Ks + SEG * pitch, *Qs = Vs + SEG * pitch, *Ps = Qs + group * pitch;
  bring_panel(Ks, panel_of(p, seq, seg, kvh, false), hd, tid, 128);
  bring_panel(Vs, panel_of(p, seq, seg, kvh, true), hd, tid, 128);
  for (int i = tid; i < group * (hd / 4); i += 128) {
    const int r = i / (hd / 4), c = i % (hd / 4) * 4;
    *(float4 *)(Qs + r * pitch + c) = *(const float4 *)(p.q + (size_t)t * p.q_stride + (size_t)(kvh * group + r) * hd + c);
  }
  asm volatile("cp.async.wait_group 1;\n" ::);
  __syncthreads();
  const int j = tid & (SEG - 1);
  for (int r = tid / SEG; r < group; r += 128 / SEG) {
    float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (int c = 0; c < hd; c += 4) dot4(d, *(const float4 *)(Qs + r * pitch + c), *(const float4 *)(Ks + j * pitch + c));
    Ps[r * (SEG + 4) + j] = scored(p, d);
  }
  __syncthreads();
  const size_t part_size = hd + F32_PART_EXTRA;
  float *part = p.parts + (((size_t)t * p.nh + kvh * group) * p.segments + seg) * part_size;
  for (int r = warp; r < group; r += 4) {
    float m, l;
    soften(p, Ps + r * (SEG + 4), lane, seg, pos, m, l);
    if (lane == 0) {
      part[r * p.segments * part_size] = m;
      part[r * p.segments * part_size + 1] = l;
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::);
  __syncthreads();
  const int n_keys = min(SEG, pos - seg * SEG + 1);
  for (int i = tid; i < group * hd; i += 128) {
    const int r = i / hd, d = i % hd;
    float acc = 0.f;
#pragma unroll 8
    for (int k = 0; k < n_keys; ++k) {
      const float pr = Ps[r * (SEG + 4) + k];
      if (!hidden(pr)) acc = fmaf(pr, Vs[k * pitch + d], acc);
    }
    part[r * p.segments * part_size + F32_PART_EXTRA + d] = acc;
  }
}

// a block per (token, head); a thread per value
__global__ void __launch_bounds__(F32_MAX_HD)
attn_f32_merge_kernel(F32Attn p) {
  pdl_launch();
  pdl_wait();
  const int t = blockIdx.x / p.nh, h = blockIdx.x % p.nh, d = threadIdx.x;
  const int pos = p.tok_pos[t], lo = lowest_key(p, pos);
  const size_t part_size = p.hd + F32_PART_EXTRA;
  const float *part = p.parts + (size_t)blockIdx.x * p.segments * part_size;
  float m = -INFINITY, l = 0.f, o = 0.f;
#pragma unroll 4
  for (int seg = 0; seg * SEG <= pos; ++seg) {
    if (!sees_segment(p, lo, pos, seg)) continue;
    const float *s = part + seg * part_size;
    const float part_m = s[0], part_l = s[1], v = d < p.hd ? s[F32_PART_EXTRA + d] : 0.f;
    float of, nf;
    merge_factors(m, part_m, of, nf);
    l = merged(l, of, part_l, nf);
    o = merged(o, of, v, nf);
  }
  if (d < p.hd) p.out[(size_t)t * p.nh * p.hd + (size_t)h * p.hd + d] = o * last_factor(p, t, h, m, l);
}

template <int HD4>
static int launch_f32_tiles(const F32Attn &p, int n_tiles, cudaStream_t stream) {
  static G2bPerDevice done;
  auto bytes = [](int hd) { return sizeof(float) * ((size_t)(F32_ROWS + 2 * SEG) * (hd + 4) + F32_ROWS * (SEG + 4) + 4 * F32_ROWS); };
  const int dev = g2b_current_device();
  if (dev < 0 || !done.value[dev]) {
    if (cudaFuncSetAttribute(attn_f32_tile_kernel<HD4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes(64 * HD4)) != cudaSuccess)
      G2B_REFUSE("attn_f32: %zu bytes of shared memory are not available", bytes(64 * HD4));
    if (dev >= 0) done.value[dev] = 1;
  }
  g2b_launch(attn_f32_tile_kernel<HD4>, dim3(2u * n_tiles * p.nh), dim3(F32_THREADS), bytes(p.hd), stream, p);
  return g2b_check_launch("attn_f32");
}

// Float attention over pages of 64 keys (see above).  `tiles` [n_tiles, 4] (sequence, first token, rows up to 64, position of
// the first row): the step's rows in tiles; null: a token by itself, with `parts` of n_tokens * nh * segments * (hd + 2)
// floats for the segments, of which there are as many as the longest sequence has pages.
extern "C" int g2b_attn_f32(const float *q, float *out, const float *cache, const int *tok_pos, const int *tok_seq,
                            const int *page_table, int P, int n_tokens, int nh, int nkv, int hd, int window, float scale,
                            const float *sink, int planes, int q_stride, const float *gate, int gate_stride, int chunk, float softcap,
                            int keep_first, int v_heads, const int *tiles, int n_tiles, float *parts, int segments,
                            cudaStream_t stream) {
  if (n_tokens <= 0) return 0;
  if (v_heads <= 0) v_heads = nkv;
  if (hd <= 0 || hd > F32_MAX_HD || hd % 4 || q_stride % 4 || (uintptr_t)q % 16 || (uintptr_t)out % 16 || (uintptr_t)cache % 16)
    G2B_REFUSE("attn_f32: head size %d (a multiple of 4 up to %d) with rows on 16 bytes", hd, F32_MAX_HD);
  if (nkv <= 0 || nh % nkv || nh / nkv > F32_MAX_GROUP) G2B_REFUSE("attn_f32: %d heads on %d kv heads", nh, nkv);
  if (v_heads > nkv || nkv % v_heads) G2B_REFUSE("attn_f32: %d key heads on %d value heads", nkv, v_heads);
  if (chunk < 0 || (chunk > 0 && window > 0)) G2B_REFUSE("attn_f32: a chunk of %d keys with a window of %d", chunk, window);
  if (keep_first < 0 || (keep_first > 0 && window <= 0)) G2B_REFUSE("attn_f32: %d first tokens kept need a window", keep_first);
  if (planes != 1 && planes != 2) G2B_REFUSE("attn_f32: %d panels per page and kv head (1 or 2)", planes);
  const F32Attn p{q, cache, sink, gate, out, parts, tok_pos, tok_seq, page_table, tiles, P, nh, nkv, hd, window, planes, q_stride, gate_stride,
                  chunk, keep_first, v_heads, segments, scale, softcap};
  if (tiles) {
    if (hd <= 64) return launch_f32_tiles<1>(p, n_tiles, stream);
    if (hd <= 128) return launch_f32_tiles<2>(p, n_tiles, stream);
    return launch_f32_tiles<4>(p, n_tiles, stream);
  }
  if (!parts || segments <= 0 || segments > P) G2B_REFUSE("attn_f32: %d segments of a table of %d pages need their parts", segments, P);
  if (n_tokens > 65535 || nkv > 65535) G2B_REFUSE("attn_f32: %d tokens of %d kv heads are too many for one launch", n_tokens, nkv);
  static G2bPerDevice done;
  auto bytes = [](int d, int group) { return sizeof(float) * ((size_t)(2 * SEG + group) * (d + 4) + group * (SEG + 4)); };
  const int dev = g2b_current_device();
  if (dev < 0 || !done.value[dev]) {
    const size_t most = bytes(F32_MAX_HD, F32_MAX_GROUP);
    if (cudaFuncSetAttribute(attn_f32_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most) != cudaSuccess)
      G2B_REFUSE("attn_f32: %zu bytes of shared memory are not available", most);
    if (dev >= 0) done.value[dev] = 1;
  }
  g2b_launch(attn_f32_split_kernel, dim3(segments, nkv, n_tokens), dim3(128), bytes(hd, nh / nkv), stream, p);
  if (int rc = g2b_check_launch("attn_f32")) return rc;
  g2b_launch(attn_f32_merge_kernel, dim3(n_tokens * nh), dim3((hd + 31) / 32 * 32), 0, stream, p);
  return g2b_check_launch("attn_f32");
}

extern "C" int g2b_attn_generic(const void *q, void *out, int dtype, const void *cache,
                                const int *tok_pos, const int *tok_seq, const int *page_table,
                                int P, int n_tokens, int nh, int nkv, int hd, int page_size,
                                int window, float scale, const float *sink, int planes, int q_stride,
                                const void *gate, int gate_stride, int chunk, const void *pooled, int pool,
                                int pool_rows, float softcap, int keep_first, int v_heads, cudaStream_t stream) {
  if (n_tokens <= 0) return 0;
  if (pool < 0 || (pool > 0 && (window <= 0 || !pooled || planes != 2 || pool_rows < (page_size + pool - 1) / pool)))
    G2B_REFUSE("attn_generic: pooled blocks of %d need a window, their store and %d rows a page", pool,
               pool > 0 ? (page_size + pool - 1) / pool : 0);
  if (chunk < 0 || (chunk > 0 && window > 0)) G2B_REFUSE("attn_generic: a chunk of %d keys with a window of %d", chunk, window);
  if (v_heads <= 0) v_heads = nkv;
  if (v_heads > nkv || nkv % v_heads) G2B_REFUSE("attn_generic: %d key heads on %d value heads", nkv, v_heads);
  if (keep_first < 0 || (keep_first > 0 && (window <= 0 || pool > 0)))
    G2B_REFUSE("attn_generic: %d first tokens kept need a window, and go with no pooled blocks", keep_first);
  if (planes != 1 && planes != 2) G2B_REFUSE("attn_generic: %d panels per page and kv head (1 or 2)", planes);
  if (hd <= 0 || hd > AG_MAX_HD) G2B_REFUSE("attn_generic: head_dim %d outside 1..%d", hd, AG_MAX_HD);
  if (nkv <= 0 || nh % nkv) G2B_REFUSE("attn_generic: %d heads are not a multiple of %d kv heads", nh, nkv);
  if (page_size <= 0 || page_size % 32)
    G2B_REFUSE("attn_generic: page size %d must be a multiple of 32", page_size);
  const long long items = (long long)n_tokens * nh;
  const unsigned blocks = (unsigned)((items + AG_WARPS - 1) / AG_WARPS);
  if (dtype == G2B_F32)
    g2b_launch(attn_generic_kernel<float>, dim3(blocks), dim3(AG_WARPS * 32), 0, stream, 
        (const float *)q, (float *)out, (const float *)cache, tok_pos, tok_seq, page_table, P,
        n_tokens, nh, nkv, hd, page_size, window, scale, sink, planes, q_stride, (const float *)gate, gate_stride, chunk, (const float *)pooled, pool, pool_rows, softcap, keep_first, v_heads);
  else if (dtype == G2B_BF16)
    g2b_launch(attn_generic_kernel<bf16>, dim3(blocks), dim3(AG_WARPS * 32), 0, stream, 
        (const bf16 *)q, (bf16 *)out, (const bf16 *)cache, tok_pos, tok_seq, page_table, P,
        n_tokens, nh, nkv, hd, page_size, window, scale, sink, planes, q_stride, (const bf16 *)gate, gate_stride, chunk, (const bf16 *)pooled, pool, pool_rows, softcap, keep_first, v_heads);
  else
    G2B_REFUSE("attn_generic: unknown dtype %d", dtype);
  return g2b_check_launch("attn_generic");
}
