// float32 products of many rows on the 5th-generation tensor cores:  C[M,N] (=|+=) A[M,K] * W[N,K]^T, everything float.
//
// A float is the sum of three bfloat16, x = x1 + x2 + x3, each the rest of the one before rounded to nearest (7 + 8 + 8 bits and two
// signs hold all 24).  Of the nine products of two such sums the six largest,
//   a1 w3 + a3 w1 + a2 w2 + a1 w2 + a2 w1 + a1 w1,
// are exact in 32 bits; the three left out are below 2^-23 of a1 w1, 2^-26 in the mean square.  The tensor cores' own sums cut low bits off: always
// toward zero, which sums of one sign do not average out.  So they are kept short: for every 32 of K the small products and then the a1 w1 are
// added in a fresh accumulator (the cuts then fall on a small sum and on the two last products, of which first parts of seven bits leave less to
// cut), and its sum is added, rounded to nearest, to a sum in registers that carries along what rounding takes from it, as two bfloat16 a register.
// Relative error against 64 bits (2-norm), K = 64 to 3,072 and 17,408, gemm_simt.cu's in brackets:
//   normal entries 0.6 to 0.8e-7 (1.4 to 3.3); their magnitudes 0.5 to 0.6e-7 (0.7 to 2.5); 1 + 0.1 normal 0.5 to 0.6e-7 (0.6 to 2.4); behind SiLU
//   0.6 to 0.7e-7 (0.7 to 2.5).  Log-normal entries over ten powers of e, where a few products decide: 0.4 to 0.8e-7 (0.4 to 1.6).
// Results of one sign are too small by 4 to 5e-8 in the mean, whatever K is (gemm_simt.cu: by nothing); with 64 of K an accumulator, eight-bit first
// parts and sums without rests by 8e-8, and the 2-norm error came to 1.6 of gemm_simt.cu's there.
//
// Two launches.  `split_kernel` writes the three parts of A and W, [3 * rows][K] each, a warp a row, and says for every row whether the sum of
// three is good for it.  `gemm_f32_tc_kernel`: a pair of CTAs takes a 256 x 256 tile (cta_group::2: each brings its own 128 rows of A and half
// of W's 256) and, where the tiles are fewer than the SMs, a part of K (up to four pairs in a cluster, each of which adds all pairs' sums, in
// their order, for a range of columns).  Roles by warp:
//   warp 8   copies: per block of K the three parts of A and of W (128-byte swizzle), two blocks in flight; a part's place is filled again
//            as soon as the last product that reads it is done
//   warp 9   products, in the pair's first CTA: 12 tcgen05.mma (kind::f16, M = N = 256, K = 16) for either half of a block, into one of two accumulators
//   warps 0-7  add: warp w reads lanes 32 (w % 4) .. + 31 and columns 128 (w / 4) .. + 127 of a finished accumulator and adds them to its
//              128 floats a thread, while the other accumulator is filled; at the end they write C, through shared memory, in rows
//
// Rows with an entry that is not finite, of 2^50 and more (sums of the products of smaller ones stay below 2^127 for any K) or below
// 2^-103 but not zero (its last bit is under 2^-126, the smallest normal number, so a part would lose bits) are flagged; an output of a flagged
// row of A or W is summed from the floats themselves in the order of gemm_simt.cu, by the warp that would have written it.  701 rows by 6144 x 1024
// (90 us; 235 by multiply-adds): 206 with a flagged row, 116 with a column, 277 with every 32nd row, 817 with all (950, 940, 910 and 6,800 by a lane
// an output).
//
// What bounds it: the tensor cores do six products for one and need a block's 24 in 3,072 cycles (128 x 256 x 64 a CTA at 8,192 operations a
// cycle); the adders, whose loads from tensor memory and sums with rests come one after another in two warps a scheduler, take about 1.4 times that
// for its two accumulators.  Sums without rests 54 us where this takes 62, one accumulator a block as well 45: the errors above forbid both.  Two accumulators
// for either half of the columns, emptied together, 72 (as 48 products of 128 columns, A is read from shared memory twice).  An adder's arrival
// that released its stores to the cluster cost 20 us.
// Measured: 701 rows, parts included: 62 us for 4096 x 1024, 67 for 6144 x 1024, 47 for 1024 x 2048, 64 for 1024 x 3072 (229, 230, 140 and 209 by
// gemm_f32_tile_kernel); 2,100 rows: 172 us for 6144 x 1024 (674).
//
// Every wait gives up after a bounded number of polls and leaves a code in `*status`, as in gemm_tc.cu.
#include "common.cuh"
#include "mma.cuh"
#include "tc_common.cuh"

#include <math.h>

#include <type_traits>

G2B_DEFINE_LAST_ERROR

using namespace tc;

constexpr int BM = 128, BN = 256, BK = 64;               // BM: rows of a CTA
constexpr int PART_BYTES = BM * BK * 2;                  // one part of a CTA's rows of A, or of its half of W
static_assert(BN / 2 == BM, "the parts of A and W have one size");
constexpr int STAGES = 2, SLOT_BYTES = 2 * PART_BYTES;   // a slot: the part p of A and of W; slots [stage][p]
constexpr int ADDERS = 8, THREADS = (ADDERS + 4) * 32;    // the last two warps only complete a group of four
// Registers: 384 threads start with 168 each (64,512); the adders hold 128 sums and their 64 pairs of rests and take 232, the others keep 40:
// 256 * 232 + 128 * 40 = 64,512.
constexpr int ADDER_REGS = 232, OTHER_REGS = 40;
constexpr int COLS = BN / 2;                             // columns of an adder
constexpr int AT_ONCE = 16;                              // columns read from an accumulator at a time
constexpr int SPLIT_MOST = 4;
constexpr int SUM_CHUNK = 64;
constexpr int RING_BYTES = STAGES * 3 * SLOT_BYTES;
constexpr int PITCH = 36;                                // floats a row of an adder's 32 x 32 outputs on their way to C
constexpr int OUT_BYTES = ADDERS * 32 * PITCH * 4;
constexpr int RECEIVED_BYTES = (SPLIT_MOST - 1) * (BN / SPLIT_MOST) * BM * 4;          // 96 KB; 64 with two parts
constexpr int SMEM = RING_BYTES + 1024 + 256;            // + the swizzle's alignment, + barriers
static_assert(RECEIVED_BYTES + OUT_BYTES <= RING_BYTES, "both lie where the ring was");
enum { ST_PRODUCER_TIMEOUT = 21, ST_MMA_TIMEOUT = 22, ST_ADDER_TIMEOUT = 23 };

// ---- parts ---------------------------------------------------------------------------------------------
// Two floats as their parts, packed pairs of bfloat16; the first is rounded to seven bits.
__device__ __forceinline__ float seven_bits(float x) {
  const uint32_t u = __float_as_uint(x);
  return __uint_as_float((u + 0xffffu + (u >> 17 & 1)) & 0xfffe0000u);
}
__device__ __forceinline__ void split2(float x, float y, uint32_t (&p)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    p[i] = i == 0 ? pack_bf16(seven_bits(x), seven_bits(y)) : pack_bf16(x, y);
    x -= __uint_as_float(p[i] << 16);
    y -= __uint_as_float(p[i] & 0xffff0000u);
  }
}

// Three parts do not hold it, or its products (NaN too).
__device__ __forceinline__ bool out_of_range(float x) {
  const float size = fabsf(x);
  return !(size < 0x1p50f) || (size < 0x1p-103f && size != 0.f);
}

// A warp a row of A (rows 0 .. M - 1) or of W (M .. M + N - 1); `ld` is the parts' row length, a multiple of 8, zeros behind K.
__global__ void __launch_bounds__(256)
split_kernel(const float *A, const float *__restrict__ W, int M, int N, int K, int lda, int ldw, bf16 *parts_a, bf16 *parts_w, int ld, int *flags) {
  pdl_launch();
  const long long r = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  pdl_wait();
  if (r >= M + N) return;
  const bool of_a = r < M;
  const float *x = of_a ? A + (size_t)r * lda : W + (size_t)(r - M) * ldw;
  const size_t plane = (size_t)(of_a ? M : N) * ld;
  bf16 *to = (of_a ? parts_a + (size_t)r * ld : parts_w + (size_t)(r - M) * ld);
  bool odd = false;
  constexpr int AHEAD = 2;
  for (int k0 = lane * 8; k0 < ld; k0 += 256 * AHEAD) {
    float4 v[AHEAD][2];
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      const int k = k0 + 256 * u;                        // K is a multiple of 4
      v[u][0] = k < K ? *reinterpret_cast<const float4 *>(x + k) : make_float4(0.f, 0.f, 0.f, 0.f);
      v[u][1] = k + 4 < K ? *reinterpret_cast<const float4 *>(x + k + 4) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      const int k = k0 + 256 * u;
      if (k >= ld) continue;
      uint32_t p[4][3];
      split2(v[u][0].x, v[u][0].y, p[0]);
      split2(v[u][0].z, v[u][0].w, p[1]);
      split2(v[u][1].x, v[u][1].y, p[2]);
      split2(v[u][1].z, v[u][1].w, p[3]);
#pragma unroll
      for (int i = 0; i < 3; ++i) *reinterpret_cast<uint4 *>(to + i * plane + k) = make_uint4(p[0][i], p[1][i], p[2][i], p[3][i]);
#pragma unroll
      for (int i = 0; i < 2; ++i) odd |= out_of_range(v[u][i].x) | out_of_range(v[u][i].y) | out_of_range(v[u][i].z) | out_of_range(v[u][i].w);
    }
  }
  odd = __any_sync(0xffffffffu, odd);
  if (lane == 0) flags[r] = odd;
}

// ---- the product -----------------------------------------------------------------------------------------
__device__ __forceinline__ void st_cluster16(uint32_t addr, float4 v) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};\n" ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}

// sum += v, two of each, with what was lost to rounding so far added to v first and what is lost now kept.
__device__ __forceinline__ void add_with_rest(float &s0, float &s1, uint32_t &rest, float2 v) {
  const float2 s = make_float2(s0, s1);
  v = add2(v, make_float2(__uint_as_float(rest << 16), __uint_as_float(rest & 0xffff0000u)));
  const float2 t = add2(s, v);
  const float2 minus = make_float2(-1.f, -1.f);
  const float2 lost = fma2(fma2(s, minus, t), minus, v);           // v - (t - s)
  rest = pack_bf16(lost.x, lost.y);
  s0 = t.x, s1 = t.y;
}

// D (+)= A * B of a pair; the descriptors' low words (their high words are one constant), so that the issuing thread keeps few registers
template <bool ACC>
__device__ __forceinline__ void umma_pair_lo(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc) {
  constexpr uint32_t HIGH = (1024 >> 4) | (1u << 14) | (2u << 29);
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "mov.b64 da, {%1, %4};\n\t"
      "mov.b64 db, {%2, %4};\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %3, p;\n\t}\n"
      ::"r"(d), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(HIGH), "n"(ACC ? 1 : 0)
      : "memory");
}

// One arrival on a barrier of the pair: says that this warp's reads of tensor memory are done (they are waited for) and hands over no data, so it is no
// release to the cluster, which waits for every store under way.
__device__ __forceinline__ void arrive_read(uint32_t cluster_bar) {
  asm volatile("mbarrier.arrive.release.cta.shared::cluster.b64 _, [%0];\n" ::"r"(cluster_bar) : "memory");
}

// Maps of the parts: [3 M][K] and [3 N][K], boxes of 128 rows.  Rows behind the last of a part belong to the next one (or are zeros):
// they fill rows and columns of the tile that are not written.
template <bool ACCUM, int SPLIT>
__global__ void __launch_bounds__(THREADS, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const float *A,
                   const float *__restrict__ W, float *C, int M, int N, int K, int lda, int ldw, int ldc, const int *flags,
                   int *__restrict__ status) {
  pdl_launch();
  extern __shared__ unsigned char smem_raw[];
  unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + RING_BYTES);
  const uint32_t full0 = smem_addr(bars), empty0 = full0 + 8 * 3 * STAGES, sum_full0 = empty0 + 8 * 3 * STAGES, sum_empty0 = sum_full0 + 16;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 6 * STAGES + 4);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank(), half = rank & 1, first = rank & ~1u;          // the pair's first CTA issues its products
  const int part = (int)(rank >> 1);
  const int n0 = (int)(blockIdx.x / (2 * SPLIT)) * BN, m0 = (int)blockIdx.y * 2 * BM + (int)half * BM;
  const int all = (K + BK - 1) / BK, per = (all + SPLIT - 1) / SPLIT;
  const int kb0 = part * per, nkb = max(0, min(all, kb0 + per) - kb0);
  if (threadIdx.x == 0) {
    for (int s = 0; s < 3 * STAGES; ++s) {
      mbar_init(full0 + 8 * s, 1);               // in the first CTA, with both CTAs' bytes
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(sum_full0 + 8 * b, 1);
      mbar_init(sum_empty0 + 8 * b, 2 * ADDERS); // in the first CTA: both CTAs' adders
    }
    mbar_init_fence();
  }
  if (warp == ADDERS + 1) tmem_alloc_pair(smem_addr(tmem_slot), 2 * BN);
  tc_fence_before();
  cluster_sync_all();                            // both CTAs' barriers and tensor memory exist
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_wait();

  const int row0 = 32 * (warp % 4), col0 = COLS * (warp / 4);                // an adder's first row and column of the CTA's tile
  uint32_t row_flags = 0, col_flags[COLS / 32] = {};       // a bit a row, a bit a column
  // Parts of K: pair p owns range p of SPLIT ranges of columns; every pair sends the others theirs, and a pair adds them in the order of
  // the parts.
  if (warp >= ADDERS) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(OTHER_REGS));
    if (warp == ADDERS && lane == 0 && PRODUCER_RUNS) {
      const uint32_t first_full0 = map_to_cta(full0, first);
      bool ok = true;
      for (int i = 0; i < nkb && ok; ++i) {
        const int k = (kb0 + i) * BK;
#pragma unroll
        for (int p = 2; p >= 0; --p) {           // in the order in which the places become free
          const int s = (i % STAGES) * 3 + p;
          if (i >= STAGES && !mbar_wait(empty0 + 8 * s, (i / STAGES - 1) & 1)) {
            atomicExch(status, ST_PRODUCER_TIMEOUT);
            ok = false;
            break;
          }
          const uint32_t to = smem_addr(smem + s * SLOT_BYTES);
          if (half == 0) mbar_expect_tx(full0 + 8 * s, 2 * SLOT_BYTES);
          tma_load_2d_pair(to, &map_a, k, p * M + m0, first_full0 + 8 * s);
          tma_load_2d_pair(to + PART_BYTES, &map_w, k, p * N + n0 + (int)half * BM, first_full0 + 8 * s);
        }
      }
    }
    if (warp == ADDERS + 1 && lane == 0 && half == 0) {
      constexpr uint32_t idesc = instr_desc(2 * BM, BN, false);
      const std::true_type yes;                  // the first of a sum
      const std::false_type no;
      const uint16_t both = (uint16_t)(3u << rank);
      bool ok = true;
      for (int i = 0; i < nkb && ok; ++i) {
        const int s0 = (i % STAGES) * 3;
        const uint32_t at = smem_addr(smem + s0 * SLOT_BYTES), parity = (i / STAGES) & 1;
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {            // the halves of the block; a part is there for the second when it was for the first
          auto arrived = [&](int p) { return h || mbar_wait(full0 + 8 * (s0 + p), parity); };
          const uint32_t to = tmem + h * BN;
          uint32_t lo = ((at & 0x3FFFF) >> 4 | 1u << 16) + 4 * h;
          asm volatile("" : "+r"(lo));           // or all descriptors are kept over the blocks, in memory
          auto products = [&](int pa, int pw, auto fresh) {
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              const uint32_t da = lo + pa * (SLOT_BYTES / 16) + 2 * k, db = lo + (pw * SLOT_BYTES + PART_BYTES) / 16 + 2 * k;
              if (decltype(fresh)::value && k == 0) umma_pair_lo<false>(to, da, db, idesc);
              else umma_pair_lo<true>(to, da, db, idesc);
            }
          };
          ok = (i < 1 || mbar_wait_cluster(sum_empty0 + 8 * h, (i - 1) & 1)) && arrived(2) && arrived(0);
          if (ok) {
            tc_fence_after();
            products(0, 2, yes);
            products(2, 0, no);
            if (h) umma_commit_pair(empty0 + 8 * (s0 + 2), both);
            ok = arrived(1);
          }
          if (!ok) {
            atomicExch(status, ST_MMA_TIMEOUT);
            break;
          }
          tc_fence_after();
          products(1, 1, no);
          products(0, 1, no);
          products(1, 0, no);
          if (h) umma_commit_pair(empty0 + 8 * (s0 + 1), both);
          products(0, 0, no);
          if (h) umma_commit_pair(empty0 + 8 * s0, both);
          umma_commit_pair(sum_full0 + 8 * h, both);
        }
      }
    }
    __syncwarp();
    if (SPLIT > 1) {
      cluster_sync_all();
      cluster_sync_all();
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(ADDER_REGS));
    float sum[COLS];
#pragma unroll
    for (int j = 0; j < COLS; ++j) sum[j] = 0.f;
    row_flags = __ballot_sync(0xffffffffu, m0 + row0 + lane < M && flags[m0 + row0 + lane] != 0);
#pragma unroll
    for (int h = 0; h < COLS / 32; ++h) {
      const int n = n0 + col0 + 32 * h + lane;
      col_flags[h] = __ballot_sync(0xffffffffu, n < N && flags[M + n] != 0);
    }
    const uint32_t first_empty0 = map_to_cta(sum_empty0, first);
    const uint32_t from0 = tmem + ((uint32_t)row0 << 16) + col0;
    uint32_t rest[COLS / 2];                               // what rounding has taken from the sums, two bfloat16 a register
#pragma unroll
    for (int j = 0; j < COLS / 2; ++j) rest[j] = 0u;
    bool ok = true;
    for (int i = 0; i < nkb && ok; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (ok && !mbar_wait(sum_full0 + 8 * h, i & 1)) {
          if (lane == 0) atomicExch(status, ST_ADDER_TIMEOUT);
          ok = false;
        }
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < COLS; c += AT_ONCE) {
          uint32_t x[AT_ONCE];
          tmem_ld16(from0 + h * BN + c, x);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < AT_ONCE; j += 2)
            add_with_rest(sum[c + j], sum[c + j + 1], rest[(c + j) / 2], make_float2(__uint_as_float(x[j]), __uint_as_float(x[j + 1])));
          if (K < 0) break;                                // never: the pieces one after another, or the compiler mixes them and keeps 240 registers in memory
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) arrive_read(first_empty0 + 8 * h);
      }
    constexpr int RANGE = BN / SPLIT, OWN = COLS < RANGE ? COLS : RANGE;         // columns of a pair, of them in an adder's reach
    if (SPLIT > 1) {
      cluster_sync_all();                                  // all rings are free
      // [source among the others][piece of four columns of the range][row] float4
      auto place = [&](int source, int col) { return ((source * (RANGE / 4) + col % RANGE / 4) * BM + row0 + lane) * 16; };
#pragma unroll
      for (int j0 = 0; j0 < COLS; j0 += OWN) {
        const int to = (col0 + j0) / RANGE;
        if (to == part) continue;
        const uint32_t at = map_to_cta(smem_addr(smem) + place(part - (part > to), col0 + j0), 2 * to + half);
#pragma unroll
        for (int j = 0; j < OWN; j += 4) st_cluster16(at + j / 4 * BM * 16, make_float4(sum[j0 + j], sum[j0 + j + 1], sum[j0 + j + 2], sum[j0 + j + 3]));
      }
      cluster_sync_all();
#pragma unroll
      for (int j0 = 0; j0 < COLS; j0 += OWN) {
        if ((col0 + j0) / RANGE != part) continue;
        const unsigned char *at = smem + place(0, col0 + j0);
#pragma unroll
        for (int j = 0; j < OWN; j += 4) {
          float4 v[SPLIT];
#pragma unroll
          for (int o = 0; o < SPLIT - 1; ++o) v[o] = *reinterpret_cast<const float4 *>(at + ((o * (RANGE / 4) + j / 4) * BM) * 16);
          const float4 mine4 = make_float4(sum[j0 + j], sum[j0 + j + 1], sum[j0 + j + 2], sum[j0 + j + 3]);
          float4 t = part == 0 ? mine4 : v[0];
#pragma unroll
          for (int o = 1; o < SPLIT; ++o) {
            const float4 x = o == part ? mine4 : (o < part ? v[o] : v[o - 1]);
            t.x += x.x; t.y += x.y; t.z += x.z; t.w += x.w;
          }
          sum[j0 + j] = t.x; sum[j0 + j + 1] = t.y; sum[j0 + j + 2] = t.z; sum[j0 + j + 3] = t.w;
        }
      }
    }
    if (m0 + row0 < M) {
      float *const mid = reinterpret_cast<float *>(smem + RECEIVED_BYTES) + warp * 32 * PITCH;
      const bool vector = ldc % 4 == 0 && ((uintptr_t)C & 15) == 0;
#pragma unroll
      for (int h = 0; h < COLS / 32; ++h) {
        if ((col0 + 32 * h) / RANGE != part) continue;
#pragma unroll
        for (int j = 0; j < 8; ++j)
          *reinterpret_cast<float4 *>(mid + lane * PITCH + 4 * j) =
              make_float4(sum[32 * h + 4 * j], sum[32 * h + 4 * j + 1], sum[32 * h + 4 * j + 2], sum[32 * h + 4 * j + 3]);
        __syncwarp();
        const int c = 4 * (lane % 8), n = n0 + col0 + 32 * h + c;               // a lane's columns: eight lanes a row
        const uint32_t flagged = col_flags[h] >> c & 15;
        if (n < N) {
#pragma unroll 4
          for (int i = 0; i < 8; ++i) {
            const int r = 4 * i + lane / 8, m = m0 + row0 + r;
            if (m >= M) break;
            float4 v = *reinterpret_cast<const float4 *>(mid + r * PITCH + c);
            float *to = C + (size_t)m * ldc + n;
            const uint32_t odd = flagged | (row_flags >> r & 1 ? 15u : 0u);
            if (vector && !odd && n + 4 <= N) {
              if (ACCUM) {
                const float4 old = *reinterpret_cast<const float4 *>(to);
                v.x += old.x; v.y += old.y; v.z += old.z; v.w += old.w;
              }
              *reinterpret_cast<float4 *>(to) = v;
            } else {
              const float each[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                if (n + e < N && !(odd >> e & 1)) to[e] = ACCUM ? to[e] + each[e] : each[e];
              }
            }
          }
        }
        __syncwarp();
      }
      // Outputs of flagged rows and columns, in the order of gemm_simt.cu: a few columns one after another, a lane a row; rows, and many
      // columns, eight rows at a time, a lane every 32nd column.
      constexpr int FEW = 8;
      constexpr int PER_LANE = OWN / 32;
#pragma unroll 1
      for (int c0 = 0; c0 < COLS; c0 += OWN) {
        if ((col0 + c0) / RANGE != part) continue;
        const float *w[PER_LANE];
        uint32_t own = 0, found[PER_LANE];                 // the lane's flagged columns, a bit each, and everybody's
        int count = 0;
#pragma unroll
        for (int j = 0; j < PER_LANE; ++j) {
          const int n = n0 + col0 + c0 + 32 * j + lane;
          w[j] = W + (size_t)min(n, N - 1) * ldw;
          found[j] = __ballot_sync(0xffffffffu, n < N && flags[M + n] != 0);
          own |= (found[j] >> lane & 1) << j;
          count += __popc(found[j]);
        }
        if (count <= FEW) {
          const float *a = A + (size_t)min(m0 + row0 + lane, M - 1) * lda;
#pragma unroll
          for (int j = 0; j < PER_LANE; ++j)
            for (uint32_t left = found[j]; left; left &= left - 1) {
              const int n = n0 + col0 + c0 + 32 * j + __ffs(left) - 1;
              const float *wn = W + (size_t)n * ldw;
              float total = 0.f;
              for (int k0 = 0; k0 < K; k0 += SUM_CHUNK) {
                float chunk = 0.f;
#pragma unroll 8
                for (int k = k0; k < min(K, k0 + SUM_CHUNK); k += 4) {
                  const float4 wk = *reinterpret_cast<const float4 *>(wn + k), ak = *reinterpret_cast<const float4 *>(a + k);
                  chunk = fmaf(ak.w, wk.w, fmaf(ak.z, wk.z, fmaf(ak.y, wk.y, fmaf(ak.x, wk.x, chunk))));
                }
                total += chunk;
              }
              if (m0 + row0 + lane < M && !(row_flags >> lane & 1)) {
                float *to = C + (size_t)(m0 + row0 + lane) * ldc + n;
                *to = ACCUM ? *to + total : total;
              }
            }
          own = 0;
        }
#pragma unroll 1
        for (int r0 = 0; r0 < 32; r0 += 8) {
          const int m = m0 + row0 + r0;
          if (m >= M || !(count > FEW || (row_flags >> r0 & 255))) continue;
          float total[8][PER_LANE] = {};
          for (int k0 = 0; k0 < K; k0 += SUM_CHUNK) {
            float chunk[8][PER_LANE] = {};
#pragma unroll 4
            for (int k = k0; k < min(K, k0 + SUM_CHUNK); k += 4) {
              float4 wk[PER_LANE];
#pragma unroll
              for (int j = 0; j < PER_LANE; ++j) wk[j] = *reinterpret_cast<const float4 *>(w[j] + k);
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const float4 ak = *reinterpret_cast<const float4 *>(A + (size_t)min(m + i, M - 1) * lda + k);
#pragma unroll
                for (int j = 0; j < PER_LANE; ++j)
                  chunk[i][j] = fmaf(ak.w, wk[j].w, fmaf(ak.z, wk[j].z, fmaf(ak.y, wk[j].y, fmaf(ak.x, wk[j].x, chunk[i][j]))));
              }
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
              for (int j = 0; j < PER_LANE; ++j) total[i][j] += chunk[i][j];
          }
#pragma unroll
          for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < PER_LANE; ++j) {
              const int n = n0 + col0 + c0 + 32 * j + lane;
              if (m + i < M && n < N && ((own >> j | row_flags >> (r0 + i)) & 1)) {
                float *to = C + (size_t)(m + i) * ldc + n;
                *to = ACCUM ? *to + total[i][j] : total[i][j];
              }
            }
        }
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  cluster_sync_all();                            // neither CTA's products, copies and arrivals meet a peer that is gone
  if (warp == ADDERS + 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem, 2 * BN);
  }
}

template <bool ACCUM, int SPLIT>
static cudaError_t allow(int &clusters) {
  cudaError_t e = cudaFuncSetAttribute(gemm_f32_tc_kernel<ACCUM, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * SPLIT), cfg.blockDim = dim3(THREADS), cfg.dynamicSmemBytes = SMEM;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = 2 * SPLIT, attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr, cfg.numAttrs = 1;
  return cudaOccupancyMaxActiveClusters(&clusters, gemm_f32_tc_kernel<ACCUM, SPLIT>, &cfg);
}
// How many clusters of one, two and four pairs the device holds at once.
struct Clusters { int of[SPLIT_MOST + 1]; };
static int count_clusters(Clusters &out) {
  static G2bPerDevice configured;
  static Clusters kept[G2B_MAX_DEVICES];
  const int dev = g2b_current_device();
  if (dev >= 0 && __atomic_load_n(&configured.value[dev], __ATOMIC_ACQUIRE)) {
    out = kept[dev];
    return 0;
  }
  cudaError_t e = allow<false, 1>(out.of[1]);
  if (e == cudaSuccess) e = allow<true, 1>(out.of[1]);
  if (e == cudaSuccess) e = allow<false, 2>(out.of[2]);
  if (e == cudaSuccess) e = allow<true, 2>(out.of[2]);
  if (e == cudaSuccess) e = allow<false, 4>(out.of[4]);
  if (e == cudaSuccess) e = allow<true, 4>(out.of[4]);
  if (e != cudaSuccess || out.of[1] < 1) G2B_REFUSE("gemm_f32_tc: %d bytes of shared memory: %s", SMEM, cudaGetErrorString(e));
  if (dev >= 0) {
    kept[dev] = out;                             // (two threads in their first calls write the same)
    __atomic_store_n(&configured.value[dev], 1, __ATOMIC_RELEASE);
  }
  return 0;
}

// Pairs per tile.  A round takes its blocks of K and about as long as two and a half more for what stands around them, four with parts.
static double rounds_of_blocks(int s, int tiles, int blocks, const Clusters &clusters) {
  return (double)((tiles + clusters.of[s] - 1) / clusters.of[s]) * ((blocks + s - 1) / s + (s > 1 ? 4.0 : 2.5));
}
static int pick_split(int tiles, int blocks, const Clusters &clusters) {
  int best = 1;
  for (int s = 2; s <= SPLIT_MOST; s *= 2)
    if (blocks >= 2 * s && clusters.of[s] > 0 && rounds_of_blocks(s, tiles, blocks, clusters) < rounds_of_blocks(best, tiles, blocks, clusters)) best = s;
  return best;
}
static int tiles_of(int M, int N) { return ((M + 2 * BM - 1) / (2 * BM)) * ((N + BN - 1) / BN); }

// Nanoseconds that both launches are estimated to take: the parts at 6.7 TB/s, a block 2.8 us, and what a launch
// takes whatever it does (within 0.13 of the time at 35 sizes of 64 to 2,100 rows, K = 1,024 to 4,096).
extern "C" int g2b_gemm_f32_tc_estimate(int M, int N, int K) {
  Clusters clusters;
  if (count_clusters(clusters)) return 2000000000;
  const int tiles = tiles_of(M, N), blocks = (K + BK - 1) / BK;
  const double us = 7.0 + 1.5e-6 * ((double)M + N) * K + 2.8 * rounds_of_blocks(pick_split(tiles, blocks, clusters), tiles, blocks, clusters);
  return us < 2e6 ? (int)(1e3 * us) : 2000000000;
}

template <int SPLIT>
static void launch_product(bool accumulate, dim3 tiles, cudaStream_t stream, const CUtensorMap &map_a, const CUtensorMap &map_w, const float *A,
                           const float *W, float *C, int M, int N, int K, int lda, int ldw, int ldc, const int *flags, int *status) {
  const dim3 grid(tiles.x * 2 * SPLIT, tiles.y);
  if (accumulate)
    g2b_launch_cluster(gemm_f32_tc_kernel<true, SPLIT>, grid, dim3(THREADS), SMEM, stream, 2u * SPLIT, map_a, map_w, A, W, C, M, N, K, lda, ldw,
                       ldc, flags, status);
  else
    g2b_launch_cluster(gemm_f32_tc_kernel<false, SPLIT>, grid, dim3(THREADS), SMEM, stream, 2u * SPLIT, map_a, map_w, A, W, C, M, N, K, lda, ldw,
                       ldc, flags, status);
}

// Rows of A and W on 16 bytes, K a multiple of 4.  parts: bfloat16 [3 (M + N) * ld], ld = K rounded up to 8; flags: int [M + N].
// accumulate: add into C.
extern "C" int g2b_gemm_f32_tc(const float *A, const float *W, float *C, int M, int N, int K, int lda, int ldw, int ldc, int accumulate,
                               void *parts, int *flags, int *status, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || K % 4 || lda % 4 || ldw % 4 || (((uintptr_t)A | (uintptr_t)W | (uintptr_t)parts) & 15))
    G2B_REFUSE("gemm_f32_tc: K=%d and row strides (%d, %d) must be multiples of 4, rows on 16 bytes", K, lda, ldw);
  const int ld = (K + 7) / 8 * 8, tiles_m = (M + 2 * BM - 1) / (2 * BM), tiles_n = (N + BN - 1) / BN;
  if (3ll * M > INT32_MAX || 3ll * N > INT32_MAX || (long long)M + N > INT32_MAX || tiles_m > 65535)
    G2B_REFUSE("gemm_f32_tc: M=%d, N=%d are too large for one launch", M, N);
  bf16 *parts_a = (bf16 *)parts, *parts_w = parts_a + (size_t)3 * M * ld;
  CUtensorMap map_a, map_w;
  int rc = get_map(&map_a, parts_a, 3ll * M, ld, ld, BM);
  if (!rc) rc = get_map(&map_w, parts_w, 3ll * N, ld, ld, BM);
  if (rc) G2B_REFUSE("gemm_f32_tc: cuTensorMapEncodeTiled failed (%d)", rc);
  Clusters clusters;
  if (count_clusters(clusters)) return 1;
  g2b_launch(split_kernel, dim3((unsigned)((M + (long long)N + 7) / 8)), dim3(256), 0, stream, A, W, M, N, K, lda, ldw, parts_a, parts_w, ld,
             flags);
  rc = g2b_check_launch("gemm_f32_tc split");
  if (rc) return rc;
  const int split = pick_split(tiles_of(M, N), (K + BK - 1) / BK, clusters);
  const dim3 tiles((unsigned)tiles_n, (unsigned)tiles_m);
  auto *launch = split == 4 ? launch_product<4> : (split == 2 ? launch_product<2> : launch_product<1>);
  launch(accumulate != 0, tiles, stream, map_a, map_w, A, W, C, M, N, K, lda, ldw, ldc, flags, status);
  return g2b_check_launch("gemm_f32_tc");
}
