// Causal grouped-query attention over the paged cache, one warp per (token, query head).
//
// The kernel of the true 32-bit path for prompts and for decoding alike, and the bfloat16
// path's fallback for head sizes its tensor-core kernels refuse.  For query head h of a token at
// position p in sequence s:  score_t = (q_h . K_t[kv(h)]) * scale over the keys t in [lo, p],
// lo = 0 or p - window + 1;  probabilities by softmax;  o_h = sum_t prob_t V_t[kv(h)]
// (stratum/native/stratum_arch_llama.inc.c:435-514; kv(h) = h / (Nq/Nk), :444).
//
// Three kernels.  float32 with heads of 64 or 128 (a Llama's): pages of 64 keys counted from position 0, two kernels of one
// arithmetic (below: "float32 by pages").  Everything else: the kernel that follows here.
//
// Keys are visited in chunks of 32 whose boundaries are multiples of 32 from position 0, and the
// running maximum, denominator and output are updated once per chunk in key order, all in
// float32.  So the result at a position does not depend on how the tokens were cut into steps,
// on the other sequences of the step, or on which pages hold the keys.
//
// q comes from the fused projection buffer [tokens][ldq] (already rotated); the cache is
// [pages][Nk][page_tokens][Hd]; page of position t = block_table[seq][t / page_tokens].
#include <cooperative_groups.h>
#include <math.h>

#include "common.cuh"

namespace cg = cooperative_groups;

#define AS_WARPS 4
#define AS_MAX_HD 256

template <typename T>
__global__ void __launch_bounds__(AS_WARPS * 32)
attention_simple_kernel(const T* __restrict__ q, int ldq, const T* __restrict__ k_cache,
                        const T* __restrict__ v_cache, const int* __restrict__ token_pos,
                        const int* __restrict__ token_seq, const int* __restrict__ block_table, int bt_stride,
                        T* __restrict__ out, int ldo, int n_tokens, int n_q, int n_kv, int head_dim,
                        int page_tokens, int window, float scale) {
  __shared__ float qs[AS_WARPS][AS_MAX_HD];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long item = (long long)blockIdx.x * AS_WARPS + warp;
  if (item >= (long long)n_tokens * n_q) return;
  const int t = (int)(item / n_q), h = (int)(item - (long long)t * n_q);
  const int seq = token_seq[t];
  if (seq < 0) return;                       // padding token
  const int pos = token_pos[t];
  const int kvh = h / (n_q / n_kv);
  const T* qp = q + (size_t)t * ldq + (size_t)h * head_dim;
  for (int d = lane; d < head_dim; d += 32) qs[warp][d] = to_float(qp[d]);
  __syncwarp();

  const int lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
  const int* bt = block_table + (size_t)seq * bt_stride;
  const size_t head_off = (size_t)kvh * page_tokens * head_dim;
  const size_t page_stride = (size_t)n_kv * page_tokens * head_dim;

  float m = -INFINITY, l = 0.f;
  float acc[AS_MAX_HD / 32];
#pragma unroll
  for (int i = 0; i < AS_MAX_HD / 32; i++) acc[i] = 0.f;

  for (int base = (lo / 32) * 32; base <= pos; base += 32) {
    const int key = base + lane;
    const bool valid = key >= lo && key <= pos;
    const int page = bt[base / page_tokens];          // page_tokens is a multiple of 32: one page per chunk
    const size_t chunk_off = (size_t)page * page_stride + head_off + (size_t)(base % page_tokens) * head_dim;
    float s = -INFINITY;
    if (valid) {
      const T* kr = k_cache + chunk_off + (size_t)lane * head_dim;
      float dot = 0.f;
      for (int d = 0; d < head_dim; d++) dot = fmaf(qs[warp][d], to_float(kr[d]), dot);
      s = dot * scale;
    }
    const float m_new = fmaxf(m, warp_max(s));        // finite: every chunk visited holds a valid key
    const float corr = expf(m - m_new);               // exp(-inf) = 0 on the first chunk
    const float p = valid ? expf(s - m_new) : 0.f;
    // denominator: add this chunk's 32 probabilities in key order
    float chunk_sum = 0.f;
#pragma unroll
    for (int j = 0; j < 32; j++) chunk_sum += __shfl_sync(0xffffffffu, p, j);
    l = l * corr + chunk_sum;
#pragma unroll
    for (int i = 0; i < AS_MAX_HD / 32; i++) acc[i] *= corr;
    const T* vr = v_cache + chunk_off;
    const int n_here = min(32, pos - base + 1);
    for (int j = 0; j < n_here; j++) {
      const float pj = __shfl_sync(0xffffffffu, p, j);
#pragma unroll
      for (int i = 0; i < AS_MAX_HD / 32; i++) {
        const int d = lane + 32 * i;
        if (d < head_dim) acc[i] = fmaf(pj, to_float(vr[(size_t)j * head_dim + d]), acc[i]);
      }
    }
    m = m_new;
  }
  const float inv = 1.0f / l;
  T* op = out + (size_t)t * ldo + (size_t)h * head_dim;
#pragma unroll
  for (int i = 0; i < AS_MAX_HD / 32; i++) {
    const int d = lane + 32 * i;
    if (d < head_dim) op[d] = from_float<T>(acc[i] * inv);
  }
}

// ---------------------------------------------------------------- float32 by pages
// For one (token, head) and one page of 64 keys:  s_j = (sum over even d of q_d k_jd + the same over odd d) * scale, each
// sum one chain of FMA;  M = max s_j;  p_j = exp(s_j - M);  L = (p_j + p_j+32) over a fixed tree of 32;  O_d = one chain
// of FMA over j.  Pages are then merged in order: m' = max(m, M), a = exp(m - m'), b = exp(M - m'), l = l a + L b,
// o = o a + O b.  Keys outside [lo, pos] take no part, and neither do pages without a key inside.  Both kernels below
// do exactly this, so a token's result is the same bits in a prompt and in a decode step, wherever its pages lie.
//
//   attention_f32_tile_kernel     64 rows (tokens x heads of a kv head's group) a block, keys and values of a page in shared
//                                 memory once for all of them, both products on register tiles: bound by the FMA units
//   attention_f32_cluster_kernel  one (token, kv head) a cluster of up to eight blocks, which take a page each at a time
//                                 and merge them through distributed shared memory: a few tokens fill the GPU, whatever
//                                 their length, in one launch and without scratch.  It takes the tokens whose pages no
//                                 tile could share: steps of one token a sequence, and of steps that mix such sequences
//                                 with prompts those that bring AF_SHORT_RUN tokens or fewer (AF_SCATTERED)
//
// Measured against one warp per (token, head) with a key a lane, which was the only kernel once (us, in brackets):
//                                              32 heads of 64, 8 of keys    32 heads of 128, each its own keys
//   a prompt of 611 tokens                        182 (1,835)                  387 (3,234)
//   1 token behind 2,000                           35 (859)                     57 (1,423)
//   64 x 1 behind 1,500                           194 (1,743)                1,212 (2,734)   as tiles 5,826 and 36,482
//   20 x 1 behind 1,500 and a prompt of 600       374 (2,258)                  930 (3,643)   as tiles 5,856 and 11,716
//   100 x 2 behind 700                            280 (1,775)                2,160 (2,794)
//   5 x 1 behind 1,500 and a prompt of 600      1,224 (1,829)                2,116 (3,329)
//   40 prompts of 9 tokens                         44 (35)                     283 (55)
#define AF_PAGE 64
#define AF_MAX_GROUP 8          // heads per kv head the cluster kernel takes
#define AF_FEW_TOKENS 32        // steps of at most this many tokens take it
#define AF_SHORT_RUN 4          // (100 x 4 behind 300: 1,936 us by token, 2,128 by tiles; 30 x 16 behind 200 1,524 and 559)
#define AF_SCATTERED 64         // steps of fewer tokens than this a sequence on the average look for short runs (with more of
                                // them the blocks that find none cost more: 5 prompts of 548 tokens, 9 us of 71)

typedef unsigned long long f32x2;
__device__ __forceinline__ void fma2(f32x2& acc, f32x2 a, f32x2 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float lo_of(f32x2 v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float hi_of(f32x2 v) { return __uint_as_float((unsigned)(v >> 32)); }
__device__ __forceinline__ f32x2 twice(float v) {
  const f32x2 b = __float_as_uint(v);
  return b << 32 | b;
}

struct PagedF32 {
  const float *q, *k, *v;
  const int *token_pos, *token_seq, *block_table;
  float* out;
  int ldq, ldo, bt_stride, n_tokens, n_q, n_kv, page_tokens, window;
  float scale;
  int short_run;                // > 0: tokens of runs (neighbours of one sequence) of at most this many are the cluster kernel's,
};                              // the others the tile kernel's; 0: the kernel that is launched takes all

__device__ __forceinline__ bool in_short_run(const PagedF32& p, int t) {
  const int seq = p.token_seq[t];
  int n = 1;
  for (int i = t - 1; i >= 0 && n <= p.short_run && p.token_seq[i] == seq; i--) n++;
  for (int i = t + 1; i < p.n_tokens && n <= p.short_run && p.token_seq[i] == seq; i++) n++;
  return n <= p.short_run;
}

// A page's keys (or values) of one kv head into shared memory, rows of HD + 4 floats.  Halves of 32 keys without a key of
// [first, last] are zeros: their pages may be nobody's.
template <int HD>
__device__ __forceinline__ void fetch_page(float* dst, const float* cache, const PagedF32& p, const int* bt, int kvh,
                                           int base, int first, int last) {
  constexpr int CHUNKS = HD / 4;
  for (int c = threadIdx.x; c < AF_PAGE * CHUNKS; c += 128) {
    const int row = c / CHUNKS, col = (c % CHUNKS) * 4, half = base + (row & 32);
    const bool there = half <= last && half + 31 >= first;
    const float* src = cache;
    if (there)
      src += (((size_t)bt[half / p.page_tokens] * p.n_kv + kvh) * p.page_tokens + (base + row) % p.page_tokens) * HD + col;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst + row * (HD + 4) + col)),
                 "l"(src), "r"(there ? 16 : 0)
                 : "memory");
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// A row's scores of a page -> its probabilities, by one warp: keys [j0, j1] count.  M and L come back.
__device__ __forceinline__ void page_softmax(float* s, int j0, int j1, float& M, float& L) {
  const int lane = threadIdx.x & 31;
  const bool in0 = lane >= j0 && lane <= j1, in1 = lane + 32 >= j0 && lane + 32 <= j1;
  const float s0 = in0 ? s[lane] : -INFINITY, s1 = in1 ? s[lane + 32] : -INFINITY;
  M = warp_max(fmaxf(s0, s1));
  const float p0 = in0 ? expf(__fsub_rn(s0, M)) : 0.f, p1 = in1 ? expf(__fsub_rn(s1, M)) : 0.f;
  s[lane] = p0;
  s[lane + 32] = p1;
  L = warp_sum(__fadd_rn(p0, p1));
}

// The running maximum and denominator take a page in; a and b are the factors of what was there and of the page.
__device__ __forceinline__ void merge_page(float& m, float& l, float M, float L, float& a, float& b) {
  const float m_new = fmaxf(m, M);
  a = expf(__fsub_rn(m, m_new));                 // 0 on the first page
  b = expf(__fsub_rn(M, m_new));
  l = __fmaf_rn(l, a, __fmul_rn(L, b));
  m = m_new;
}

template <int HD>
__global__ void __launch_bounds__(128)
attention_f32_tile_kernel(const PagedF32 p, const int tokens_per_block) {
  constexpr int PITCH = HD + 4, SP = AF_PAGE + 4, NV = HD / 32;           // NV: float4 of the output a thread holds per row
  extern __shared__ __align__(16) float smem[];
  float *qs = smem, *ks = qs + 64 * PITCH, *vs = ks + 64 * PITCH, *ss = vs + 64 * PITCH;
  __shared__ float rm[64], rl[64], ra[64], rb[64];
  __shared__ int rpos[64], rseq[64], rj0[64], rj1[64];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int group = p.n_q / p.n_kv, kvh = blockIdx.y;
  const int t0 = (gridDim.x - 1 - blockIdx.x) * tokens_per_block;         // a prompt's last tokens, which see most, first
  const int n_tok = min(tokens_per_block, p.n_tokens - t0), rows = n_tok * group;

  if (tid < 64) {                                // row = token * group + head of the group
    const int t = tid / group;
    rseq[tid] = tid < rows ? p.token_seq[t0 + t] : -1;
    rpos[tid] = tid < rows ? p.token_pos[t0 + t] : 0;
    rm[tid] = -INFINITY;
    rl[tid] = 0.f;
  }
  for (int c = tid; c < 64 * (HD / 4); c += 128) {
    const int row = c / (HD / 4), col = (c % (HD / 4)) * 4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row < rows)
      v = *reinterpret_cast<const float4*>(p.q + (size_t)(t0 + row / group) * p.ldq +
                                           (size_t)(kvh * group + row % group) * HD + col);
    *reinterpret_cast<float4*>(qs + row * PITCH + col) = v;
  }
  __syncthreads();

  const int tr = tid >> 3, tc = tid & 7;         // rows tr + 16 i; keys tc + 8 j; output columns 4 tc + 32 n
  f32x2 o[4][NV][2];
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int n = 0; n < NV; n++) o[i][n][0] = o[i][n][1] = 0;

  // one sequence of the block's tokens after the other (a step's tokens are packed: runs of equal sequences); where there
  // are many, gridDim.z blocks share them, every gridDim.z-th to each
  for (int a0 = 0, run = 0; a0 < n_tok; run++) {
    const int seq = rseq[a0 * group];
    int a1 = a0, last = 0, first = 0x7fffffff;
    for (; a1 < n_tok && rseq[a1 * group] == seq; a1++) {
      const int pos = rpos[a1 * group];
      last = max(last, pos);
      first = min(first, p.window > 0 && pos - p.window + 1 > 0 ? pos - p.window + 1 : 0);
    }
    const int r0 = a0 * group, r1 = a1 * group;
    a0 = a1;
    if (p.short_run > 0 && seq >= 0 && in_short_run(p, t0 + r0 / group)) continue;
    if (seq < 0 || run % (int)gridDim.z != (int)blockIdx.z) continue;     // padding tokens, or another block's
    const int* bt = p.block_table + (size_t)seq * p.bt_stride;
    for (int base = first / AF_PAGE * AF_PAGE; base <= last; base += AF_PAGE) {
      fetch_page<HD>(ks, p.k, p, bt, kvh, base, first, last);
      fetch_page<HD>(vs, p.v, p, bt, kvh, base, first, last);
      bool whole = true;                         // every row of this sequence sees every key of the page
      if (tid < 64) {
        const int pos = rpos[tid], lo = p.window > 0 && pos - p.window + 1 > 0 ? pos - p.window + 1 : 0;
        const bool mine = tid >= r0 && tid < r1;
        rj0[tid] = mine ? max(lo - base, 0) : 64;
        rj1[tid] = mine ? min(pos - base, 63) : -1;
        whole = !mine || (lo <= base && pos >= base + 63);
      }
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      const bool all_whole = __syncthreads_and(whole);

      f32x2 s[4][8];
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) s[i][j] = 0;
#pragma unroll 4
      for (int d = 0; d < HD; d += 4) {
        ulonglong2 a[4];
#pragma unroll
        for (int i = 0; i < 4; i++) a[i] = *reinterpret_cast<const ulonglong2*>(qs + (tr + 16 * i) * PITCH + d);
#pragma unroll
        for (int j = 0; j < 8; j++) {
          const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(ks + (tc + 8 * j) * PITCH + d);
#pragma unroll
          for (int i = 0; i < 4; i++) fma2(s[i][j], a[i].x, b.x);
#pragma unroll
          for (int i = 0; i < 4; i++) fma2(s[i][j], a[i].y, b.y);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 8; j++)
          ss[(tr + 16 * i) * SP + tc + 8 * j] = __fmul_rn(__fadd_rn(lo_of(s[i][j]), hi_of(s[i][j])), p.scale);
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();

      for (int r = warp; r < 64; r += 4) {
        const int j0 = rj0[r], j1 = rj1[r];
        float a = 1.f, b = 0.f;                  // no key of this page: the row stays as it is
        if (j0 <= j1) {
          float M, L, m = rm[r], l = rl[r];
          page_softmax(ss + r * SP, j0, j1, M, L);
          merge_page(m, l, M, L, a, b);
          __syncwarp();
          if (lane == 0) { rm[r] = m; rl[r] = l; }
        }
        if (lane == 0) { ra[r] = a; rb[r] = b; }
      }
      __syncthreads();

      f32x2 u[4][NV][2];
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int n = 0; n < NV; n++) u[i][n][0] = u[i][n][1] = 0;
      auto values = [&](int j_begin, int j_end, auto seen) {
#pragma unroll 2
        for (int j = j_begin; j < j_end; j += 4) {
          float4 w[4];
#pragma unroll
          for (int i = 0; i < 4; i++) w[i] = *reinterpret_cast<const float4*>(ss + (tr + 16 * i) * SP + j);
#pragma unroll
          for (int jj = 0; jj < 4; jj++) {
            ulonglong2 b[NV];
#pragma unroll
            for (int n = 0; n < NV; n++) b[n] = *reinterpret_cast<const ulonglong2*>(vs + (j + jj) * PITCH + 4 * tc + 32 * n);
#pragma unroll
            for (int i = 0; i < 4; i++) {
              if (!seen(i, j + jj)) continue;
              const f32x2 pp = twice(jj == 0 ? w[i].x : jj == 1 ? w[i].y : jj == 2 ? w[i].z : w[i].w);
#pragma unroll
              for (int n = 0; n < NV; n++) { fma2(u[i][n][0], pp, b[n].x); fma2(u[i][n][1], pp, b[n].y); }
            }
          }
        }
      };
      if (all_whole) {
        values(0, AF_PAGE, [](int, int) { return true; });
      } else {                                   // a key that a row does not see is not multiplied by 0 but left out: its
        int j0[4], j1[4];                        // value may be another token's NaN, or nothing that was ever written
#pragma unroll
        for (int i = 0; i < 4; i++) { j0[i] = rj0[tr + 16 * i]; j1[i] = rj1[tr + 16 * i]; }
        values(max(first - base, 0) & ~3, min(last - base, AF_PAGE - 1) + 1,
               [&](int i, int j) { return j >= j0[i] && j <= j1[i]; });
      }
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int r = tr + 16 * i;
        if (rj0[r] > rj1[r]) continue;
        const float a = ra[r], b = rb[r];
#pragma unroll
        for (int n = 0; n < NV; n++)
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const float x = __fmaf_rn(lo_of(o[i][n][h]), a, __fmul_rn(lo_of(u[i][n][h]), b));
            const float y = __fmaf_rn(hi_of(o[i][n][h]), a, __fmul_rn(hi_of(u[i][n][h]), b));
            o[i][n][h] = (f32x2)__float_as_uint(y) << 32 | __float_as_uint(x);
          }
      }
      __syncthreads();                           // before the next page's copies
    }
  }
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int r = tr + 16 * i;
    if (rl[r] == 0.f) continue;                  // not a row of this block (a token sees itself at least: its sum is not zero)
    const float inv = 1.0f / rl[r];
    float* to = p.out + (size_t)(t0 + r / group) * p.ldo + (size_t)(kvh * group + r % group) * HD;
#pragma unroll
    for (int n = 0; n < NV; n++)
      *reinterpret_cast<float4*>(to + 4 * tc + 32 * n) =
          make_float4(lo_of(o[i][n][0]) * inv, hi_of(o[i][n][0]) * inv, lo_of(o[i][n][1]) * inv, hi_of(o[i][n][1]) * inv);
  }
}

template <int HD, int C>
__global__ void __cluster_dims__(C, 1, 1) __launch_bounds__(128)
attention_f32_cluster_kernel(const PagedF32 p) {
  constexpr int PITCH = HD + 4, SP = AF_PAGE + 4, LANES = HD;             // threads side by side over the output's columns
  constexpr int MINE = (AF_MAX_GROUP * HD + 128 * C - 1) / (128 * C);     // output elements a thread merges at most
  extern __shared__ __align__(16) float smem[];
  __shared__ float part_m[2][AF_MAX_GROUP], part_l[2][AF_MAX_GROUP];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int t = blockIdx.y, kvh = blockIdx.z, group = p.n_q / p.n_kv;
  float *qs = smem, *ks = qs + group * HD, *vs = ks + 64 * PITCH, *ss = vs + 64 * PITCH, *part_o = ss + group * SP;   // [2][group][HD]
  pdl_trigger();
  const int seq = p.token_seq[t], pos = p.token_pos[t];
  pdl_wait();                                    // queries and the newest keys and values come from kernels before this one
  if (seq < 0 || (p.short_run > 0 && !in_short_run(p, t))) return;        // (of the whole cluster)
  const int lo = p.window > 0 && pos - p.window + 1 > 0 ? pos - p.window + 1 : 0;
  const int* bt = p.block_table + (size_t)seq * p.bt_stride;
  for (int c = tid; c < group * HD; c += 128) qs[c] = ld_fresh(p.q + (size_t)t * p.ldq + (size_t)kvh * group * HD + c);

  const int first_page = lo / AF_PAGE, last_page = pos / AF_PAGE;
  const int share = group * HD / C;              // of the output elements, for this block to merge
  float m[MINE], l[MINE], acc[MINE];
#pragma unroll
  for (int i = 0; i < MINE; i++) { m[i] = -INFINITY; l[i] = acc[i] = 0.f; }
  int buf = 0;
  for (int page0 = first_page; page0 <= last_page; page0 += C, buf ^= 1) {
    const int page = page0 + rank, base = page * AF_PAGE;
    if (page <= last_page) {
      fetch_page<HD>(ks, p.k, p, bt, kvh, base, lo, pos);
      fetch_page<HD>(vs, p.v, p, bt, kvh, base, lo, pos);
      const int j0 = max(lo - base, 0), j1 = min(pos - base, 63);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      __syncthreads();
      {
        const int j = tid & 63, half = tid >> 6;
        f32x2 s[AF_MAX_GROUP / 2];
#pragma unroll
        for (int i = 0; i < AF_MAX_GROUP / 2; i++) s[i] = 0;
#pragma unroll 4
        for (int d = 0; d < HD; d += 4) {
          const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(ks + j * PITCH + d);
#pragma unroll
          for (int i = 0; i < AF_MAX_GROUP / 2; i++)
            if (2 * i + half < group) {
              const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(qs + (2 * i + half) * HD + d);
              fma2(s[i], a.x, b.x);
              fma2(s[i], a.y, b.y);
            }
        }
#pragma unroll
        for (int i = 0; i < AF_MAX_GROUP / 2; i++)
          if (2 * i + half < group)
            ss[(2 * i + half) * SP + j] = __fmul_rn(__fadd_rn(lo_of(s[i]), hi_of(s[i])), p.scale);
      }
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();
      for (int r = warp; r < group; r += 4) {
        float M, L;
        page_softmax(ss + r * SP, j0, j1, M, L);
        if (lane == 0) { part_m[buf][r] = M; part_l[buf][r] = L; }
      }
      __syncthreads();
      for (int r = tid / LANES; r < group; r += 128 / LANES) {
        const int d = tid % LANES;
        float u = 0.f;
#pragma unroll 8
        for (int j = j0; j <= j1; j++) u = __fmaf_rn(ss[r * SP + j], vs[j * PITCH + d], u);
        part_o[(buf * group + r) * HD + d] = u;
      }
    }
    if constexpr (C > 1) cluster.sync();         // the round's parts are there (and those of the round before read)
    else __syncthreads();
#pragma unroll
    for (int i = 0; i < MINE; i++) {
      const int e = rank * share + tid + 128 * i, row = e / HD;
      if (tid + 128 * i >= share) break;
#pragma unroll
      for (int q = 0; q < C; q++) {
        if (page0 + q > last_page) break;
        float a, b;
        merge_page(m[i], l[i], *cluster.map_shared_rank(&part_m[buf][row], q), *cluster.map_shared_rank(&part_l[buf][row], q), a, b);
        acc[i] = __fmaf_rn(acc[i], a, __fmul_rn(*cluster.map_shared_rank(&part_o[buf * group * HD + e], q), b));
      }
    }
  }
#pragma unroll
  for (int i = 0; i < MINE; i++)
    if (tid + 128 * i < share)
      p.out[(size_t)t * p.ldo + (size_t)kvh * group * HD + rank * share + tid + 128 * i] = acc[i] * (1.0f / l[i]);
  if constexpr (C > 1) cluster.sync();           // nobody leaves while another reads its parts
}

template <int HD, int C>
static int launch_attention_f32_cluster(const PagedF32& p, cudaStream_t stream) {
  const int group = p.n_q / p.n_kv, smem = (3 * group * HD + 2 * 64 * (HD + 4) + group * (AF_PAGE + 4)) * 4;
  const cudaError_t e = cudaFuncSetAttribute(attention_f32_cluster_kernel<HD, C>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  return launch_pdl(attention_f32_cluster_kernel<HD, C>, dim3(C, p.n_tokens, p.n_kv), 128, smem, stream, p);
}

template <int HD>
static int launch_attention_f32(PagedF32 p, int n_seqs, bool all_single, cudaStream_t stream) {
  const int group = p.n_q / p.n_kv, per = 64 / group;
  const bool scattered = n_seqs > 1 && p.n_tokens < AF_SCATTERED * (long long)n_seqs;
  const bool by_token = group <= AF_MAX_GROUP && p.n_tokens <= 65535;
  const bool all_by_token = by_token && (all_single || p.n_tokens <= AF_FEW_TOKENS);
  // blocks to a token: eight, four or one, as many as fill the GPU a few times over (blocks with heads of 64 come five to an
  // SM, with heads of 128 two or three, and idle ones cost as much): 8 x 1 behind 1,500 with eight / four / one, heads of
  // 64 41 / 56 / 147 us, 32 of 128 with their own keys 299 / 283 / 228; 200 x 1 behind 700 421 / 313 / 267 and 4,745 /
  // 3,231 / 2,283
  if (all_by_token || (by_token && scattered)) {
    p.short_run = all_by_token ? 0 : AF_SHORT_RUN;
    const long long walks = (long long)p.n_tokens * p.n_kv;
    const long long most = HD == 64 ? 2048 : 296;
    const int st = walks * 8 <= most   ? launch_attention_f32_cluster<HD, 8>(p, stream)
                   : walks * 4 <= most ? launch_attention_f32_cluster<HD, 4>(p, stream)
                                       : launch_attention_f32_cluster<HD, 1>(p, stream);
    if (st || all_by_token) return st;
  }
  const int smem = (3 * 64 * (HD + 4) + 64 * (AF_PAGE + 4)) * 4;
  const cudaError_t e = cudaFuncSetAttribute(attention_f32_tile_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  // as many blocks to a tile as it has sequences on the average, and with groups that the cluster kernel does not take as it
  // may have: every run is a walk through all of its sequence's pages
  const long long runs = !by_token ? n_seqs : ((long long)n_seqs * per + p.n_tokens - 1) / p.n_tokens;
  const int most = n_seqs < per ? n_seqs : per, z = runs < most ? (int)runs : most;
  attention_f32_tile_kernel<HD><<<dim3((p.n_tokens + per - 1) / per, p.n_kv, z < 1 ? 1 : z), 128, smem, stream>>>(p, per);
  return launch_status();
}

// n_seqs (the rows of the block table) and all_single (every token is the only one of its sequence) say how the step's tokens
// share pages, for the choice of kernel alone.
STRATUM_EXPORT int stratum_attention_simple(const void* q, int ldq, const void* k_cache, const void* v_cache,
                                            int dtype, const int* token_pos, const int* token_seq,
                                            const int* block_table, int bt_stride, void* out, int ldo,
                                            int n_tokens, int n_q, int n_kv, int head_dim, int page_tokens,
                                            int window, float scale, int n_seqs, int all_single,
                                            cudaStream_t stream) {
  if (n_tokens <= 0) return 0;
  if (head_dim < 1 || head_dim > AS_MAX_HD) return STRATUM_ERR_LIMIT;
  if (n_kv < 1 || n_q % n_kv != 0 || page_tokens % 32 != 0) return STRATUM_ERR_SHAPE;
  const long long items = (long long)n_tokens * n_q;
  const long long blocks = (items + AS_WARPS - 1) / AS_WARPS;
  if (blocks > 0x7fffffffLL) return STRATUM_ERR_LIMIT;
  // (all that decides is the model's: a step's shape never moves a token from one arithmetic to the other)
  if (dtype == STRATUM_DT_F32 && (head_dim == 64 || head_dim == 128) && n_q / n_kv <= 64 && n_kv <= 65535 && ldq % 4 == 0 &&
      ldo % 4 == 0 && ((uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)out) % 16 == 0) {
    const PagedF32 p = {(const float*)q, (const float*)k_cache, (const float*)v_cache, token_pos, token_seq, block_table,
                        (float*)out, ldq, ldo, bt_stride, n_tokens, n_q, n_kv, page_tokens, window, scale, 0};
    return head_dim == 64 ? launch_attention_f32<64>(p, n_seqs, all_single != 0, stream)
                          : launch_attention_f32<128>(p, n_seqs, all_single != 0, stream);
  }
  if (dtype == STRATUM_DT_F32)
    attention_simple_kernel<float><<<(unsigned)blocks, AS_WARPS * 32, 0, stream>>>(
        (const float*)q, ldq, (const float*)k_cache, (const float*)v_cache, token_pos, token_seq, block_table,
        bt_stride, (float*)out, ldo, n_tokens, n_q, n_kv, head_dim, page_tokens, window, scale);
  else if (dtype == STRATUM_DT_BF16)
    attention_simple_kernel<bf16><<<(unsigned)blocks, AS_WARPS * 32, 0, stream>>>(
        (const bf16*)q, ldq, (const bf16*)k_cache, (const bf16*)v_cache, token_pos, token_seq, block_table,
        bt_stride, (bf16*)out, ldo, n_tokens, n_q, n_kv, head_dim, page_tokens, window, scale);
  else
    return STRATUM_ERR_DTYPE;
  return launch_status();
}
