// Picking the next token from float32 logits: greedy argmax and temperature sampling with
// optional top-k / top-p filtering.  Rows of 8,192 logits or more are cut over 32 thread blocks each
// (argmax_split_kernel, sample_split_kernel); shorter rows, and rows the split sampling kernel marks,
// get one block (argmax_kernel, sample_kernel).
//
// Greedy: the largest logit, the lowest index among equals (stratum/native/stratum_engine.h:429-463).
// Sampling (stratum/native/stratum_arch_qwen35.inc.c:14023-14109): probabilities
// exp((l - max) / T) normalised; a draw u in [0,1) picks the first candidate whose cumulative
// probability exceeds u, the last candidate if rounding leaves none.  Without filters the
// candidates are all ids in id order.  With top-k and/or top-p they are the k largest logits
// (at most SAMPLE_CAND_MAX, the reference's own cap of 512 candidates, :14019) by descending
// logit, lower id first among equals, cut after the first prefix whose probability reaches top_p,
// and renormalised.  The uniform u comes from the host (one PCG32 stream per sequence), so a
// sequence's draws do not depend on what else is in the batch.
#include <float.h>
#include <math.h>

#include "common.cuh"

#define SAMPLE_THREADS 1024
#define SAMPLE_CAND_MAX 512
static_assert(SAMPLE_THREADS == 1024 && SAMPLE_CAND_MAX % 32 == 0, "the sampling kernel counts on 32 warps");

struct MaxIdx { float v; int i; };

__device__ __forceinline__ MaxIdx better(MaxIdx a, MaxIdx b) {
  if (b.v > a.v || (b.v == a.v && b.i < a.i)) return b;
  return a;
}

__device__ __forceinline__ MaxIdx block_argmax(MaxIdx mine, MaxIdx* scratch /* 33 */) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    MaxIdx other;
    other.v = __shfl_xor_sync(0xffffffffu, mine.v, o);
    other.i = __shfl_xor_sync(0xffffffffu, mine.i, o);
    mine = better(mine, other);
  }
  __syncthreads();
  if (lane == 0) scratch[warp] = mine;
  __syncthreads();
  if (warp == 0) {
    MaxIdx t = lane < n_warps ? scratch[lane] : MaxIdx{-INFINITY, 0x7fffffff};
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      MaxIdx other;
      other.v = __shfl_xor_sync(0xffffffffu, t.v, o);
      other.i = __shfl_xor_sync(0xffffffffu, t.i, o);
      t = better(t, other);
    }
    if (lane == 0) scratch[32] = t;
  }
  __syncthreads();
  return scratch[32];
}

// f(i, logit) for every logit of the row, 16 bytes per load where the row allows it.  A thread meets its ids in
// ascending order; which thread meets which id depends on the row's alignment, so only order-free work goes here.
template <typename F>
__device__ __forceinline__ void for_each_logit(const float* __restrict__ row, int vocab, F f) {
  if ((reinterpret_cast<uintptr_t>(row) & 15) == 0) {
    const int n4 = vocab >> 2;
    // four loads in flight per thread before the first is used (one block reads a whole row: latency bounds it)
    for (int q0 = threadIdx.x; q0 < n4; q0 += 4 * blockDim.x) {
      float4 v[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int q = q0 + j * blockDim.x;
        if (q < n4) v[j] = ld_fresh(reinterpret_cast<const float4*>(row) + q);
      }
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int q = q0 + j * blockDim.x;
        if (q < n4) { f(4 * q, v[j].x); f(4 * q + 1, v[j].y); f(4 * q + 2, v[j].z); f(4 * q + 3, v[j].w); }
      }
    }
    for (int i = 4 * n4 + threadIdx.x; i < vocab; i += blockDim.x) f(i, ld_fresh(row + i));
  } else {
    for (int i = threadIdx.x; i < vocab; i += blockDim.x) f(i, ld_fresh(row + i));
  }
}

__device__ __forceinline__ MaxIdx row_argmax(const float* __restrict__ row, int vocab, MaxIdx* scratch) {
  MaxIdx mine{-INFINITY, 0x7fffffff};
  for_each_logit(row, vocab, [&](int i, float v) {
    if (v > mine.v) { mine.v = v; mine.i = i; }      // ascending i per thread: first of equals is kept
  });
  MaxIdx r = block_argmax(mine, scratch);
  if (r.i == 0x7fffffff) { r.i = 0; r.v = ld_fresh(row + (0)); }  // every logit is -inf or NaN: index 0, as a scalar scan would give
  return r;
}

__global__ void __launch_bounds__(SAMPLE_THREADS)
argmax_kernel(const float* __restrict__ logits, int ld, int vocab, int* __restrict__ ids,
              float* __restrict__ values) {
  __shared__ MaxIdx scratch[33];
  pdl_trigger();
  pdl_wait();
  const int r = blockIdx.x;
  const MaxIdx best = row_argmax(logits + (size_t)r * ld, vocab, scratch);
  if (threadIdx.x == 0) {
    ids[r] = best.i;
    if (values) values[r] = best.v;
  }
}

// The same over ARGMAX_SPLITS blocks per row: each block finds the best of its stretch of the row; the block
// that finishes last (a counter per row tells) picks among the stretches, lowest index first among equals,
// and resets the counter, so the scratch needs zeroing only once, when it is made.
#define ARGMAX_SPLITS 32
__global__ void __launch_bounds__(256)
argmax_split_kernel(const float* __restrict__ logits, int ld, int vocab, int* __restrict__ ids,
                    float* __restrict__ values, float* __restrict__ part_v, int* __restrict__ part_i,
                    unsigned* __restrict__ counters) {
  __shared__ MaxIdx scratch[33];
  __shared__ bool last;
  pdl_trigger();
  pdl_wait();
  const int r = blockIdx.x, sp = blockIdx.y;
  const float* row = logits + (size_t)r * ld;
  const int chunk = (vocab + ARGMAX_SPLITS - 1) / ARGMAX_SPLITS;
  const int b = sp * chunk, e = min(vocab, b + chunk);
  MaxIdx mine{-INFINITY, 0x7fffffff};
  for (int i = b + threadIdx.x; i < e; i += blockDim.x) {
    const float v = ld_fresh(row + (i));
    if (v > mine.v) { mine.v = v; mine.i = i; }
  }
  const MaxIdx best = block_argmax(mine, scratch);
  if (threadIdx.x == 0) {
    part_v[r * ARGMAX_SPLITS + sp] = best.v;
    part_i[r * ARGMAX_SPLITS + sp] = best.i;
    __threadfence();
    last = atomicAdd(&counters[r], 1u) == ARGMAX_SPLITS - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (threadIdx.x < 32) {
    MaxIdx t{-INFINITY, 0x7fffffff};
    if (threadIdx.x < ARGMAX_SPLITS) {
      t.v = __ldcg(&part_v[r * ARGMAX_SPLITS + threadIdx.x]);
      t.i = __ldcg(&part_i[r * ARGMAX_SPLITS + threadIdx.x]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      MaxIdx other;
      other.v = __shfl_xor_sync(0xffffffffu, t.v, o);
      other.i = __shfl_xor_sync(0xffffffffu, t.i, o);
      t = better(t, other);
    }
    if (threadIdx.x == 0) {
      if (t.i == 0x7fffffff) { t.i = 0; t.v = ld_fresh(row + (0)); }
      ids[r] = t.i;
      if (values) values[r] = t.v;
      counters[r] = 0;
    }
  }
}

// scratch (optional): part_v float[n_rows*32], part_i int[n_rows*32], counters unsigned[n_rows] zeroed once by
// the caller; with it, large rows are searched by 32 blocks each.
STRATUM_EXPORT int stratum_argmax(const float* logits, int ld, int n_rows, int vocab, int* ids, float* values,
                                  float* part_v, int* part_i, unsigned* counters, cudaStream_t stream) {
  if (n_rows <= 0) return 0;
  if (vocab < 1) return STRATUM_ERR_SHAPE;
  if (part_v && part_i && counters && vocab >= 8192)
    return launch_pdl(argmax_split_kernel, dim3(n_rows, ARGMAX_SPLITS), 256, 0, stream, logits, ld, vocab, ids, values,
                      part_v, part_i, counters);
  return launch_pdl(argmax_kernel, n_rows, SAMPLE_THREADS, 0, stream, logits, ld, vocab, ids, values);
}

// ---------------------------------------------------------------- temperature sampling
// Per-row parameters (so one launch serves sequences with different settings):
//   temperature[r] <= 0 -> greedy;  top_k[r] <= 0 -> off;  top_p[r] >= 1 -> off;  uniform[r] in [0,1).
// Every sum is taken in an order that depends on the sizes only, so a row's pick is the same in every batch and run.

// order-preserving map float -> uint32 (larger float, larger key; the two zeros are equals), and back
__device__ __forceinline__ uint32_t float_key(float f) {
  const uint32_t u = f == 0.f ? 0u : __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_float(uint32_t key) {
  return __uint_as_float((key & 0x80000000u) ? (key ^ 0x80000000u) : ~key);
}

// Inclusive prefix sum over the lanes of a warp (lane 0 first).
template <typename T>
__device__ __forceinline__ T warp_incl_scan(T v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  return v;
}

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ int warp_min(int v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Exclusive prefix sum of one value per thread over the block (thread 0 first); *total gets the sum of all.
// scratch: 33 values.  Every thread of the block calls it.
template <typename T>
__device__ __forceinline__ T block_excl_scan(T v, T* scratch, T* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
  const T incl = warp_incl_scan(v);
  __syncthreads();
  if (lane == 31) scratch[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const T w = lane < n_warps ? scratch[lane] : T(0);
    const T wi = warp_incl_scan(w);
    scratch[lane] = wi - w;
    if (lane == 31) scratch[32] = wi;
  }
  __syncthreads();
  *total = scratch[32];
  return scratch[warp] + incl - v;
}

// One warp: lane l holds the PER consecutive candidates from its first on (n_cand <= 32 PER, sorted: descending
// logit, ascending id among equals; cand_e their weights, zero beyond n_cand); sums in float64: their total, the
// top-p cut over the normalised weights, and the draw among what is kept.
template <int PER>
__device__ __forceinline__ void draw_from(const float* cand_v, const int* cand_i, const float* cand_e,
                                                     int n_cand, float tp, float u, int r, int* ids, float* values) {
  const int lane = threadIdx.x & 31;
  const int c0 = lane * PER;
  double own = 0.0;
#pragma unroll
  for (int j = 0; j < PER; j++) own += (double)cand_e[c0 + j];
  const double sum = warp_sum(own);
  int keep = n_cand;
  if (tp < 1.0f) {
    double q[PER], own_q = 0.0;
#pragma unroll
    for (int j = 0; j < PER; j++) { q[j] = (double)(float)((double)cand_e[c0 + j] / sum); own_q += q[j]; }
    double cum = warp_incl_scan(own_q) - own_q;
    int first = 0x7fffffff;
#pragma unroll
    for (int j = 0; j < PER; j++) {
      cum += q[j];
      if (first == 0x7fffffff && c0 + j < n_cand && cum >= (double)tp) first = c0 + j;
    }
    first = warp_min(first);
    if (first != 0x7fffffff) keep = first + 1;
  }
  double own_kept = 0.0;
#pragma unroll
  for (int j = 0; j < PER; j++) own_kept += (c0 + j < keep) ? (double)cand_e[c0 + j] : 0.0;
  const double kept = warp_sum(own_kept);
  const double target = (double)u * kept;
  double cum = warp_incl_scan(own_kept) - own_kept;
  int first = 0x7fffffff;
#pragma unroll
  for (int j = 0; j < PER; j++) {
    if (c0 + j < keep) {
      cum += (double)cand_e[c0 + j];
      if (first == 0x7fffffff && target < cum) first = c0 + j;
    }
  }
  first = warp_min(first);
  const int pick = first == 0x7fffffff ? keep - 1 : first;
  if (lane == 0) {
    ids[r] = cand_i[pick];
    if (values) values[r] = cand_v[pick];
  }
}

// (a lane's share follows from the number of candidates: 50 of them in shares of 16 kept four lanes busy; shares of 2
// take a row's draw with a top-p cut from 32 to 21 us in all)
__device__ __forceinline__ void draw_from_candidates(const float* cand_v, const int* cand_i, const float* cand_e,
                                                     int n_cand, float tp, float u, int r, int* ids, float* values) {
  static_assert(SAMPLE_CAND_MAX == 16 * 32, "the largest share");
  if (n_cand <= 64) draw_from<2>(cand_v, cand_i, cand_e, n_cand, tp, u, r, ids, values);
  else if (n_cand <= 128) draw_from<4>(cand_v, cand_i, cand_e, n_cand, tp, u, r, ids, values);
  else if (n_cand <= 256) draw_from<8>(cand_v, cand_i, cand_e, n_cand, tp, u, r, ids, values);
  else draw_from<16>(cand_v, cand_i, cand_e, n_cand, tp, u, r, ids, values);
}

// The rows' numbers as part of the launch itself, one temperature, top_k and top_p for all of them (rows > 0): a caller that
// draws on the host then copies nothing to the device and does not wait for it (24 rows of 128,256 logits, a pick among
// others: 31 us; with a copy of four numbers a row, which waited for the picks before, 58).
#define SAMPLE_GIVEN_MAX 256
struct SampleGiven {
  int rows, top_k;
  float temperature, top_p;
  float uniform[SAMPLE_GIVEN_MAX];
};

__global__ void __launch_bounds__(SAMPLE_THREADS)
sample_kernel(const float* __restrict__ logits, int ld, int vocab, const float* __restrict__ temperature,
              const int* __restrict__ top_k, const float* __restrict__ top_p, const float* __restrict__ uniform,
              int* __restrict__ ids, float* __restrict__ values, const int* redo, const __grid_constant__ SampleGiven given) {
  __shared__ MaxIdx mi_scratch[33];
  __shared__ float f_scratch[33];
  __shared__ unsigned u_scratch[33];
  __shared__ float cand_e[SAMPLE_CAND_MAX];
  __shared__ unsigned hist[256];
  __shared__ float cand_v[SAMPLE_CAND_MAX];
  __shared__ int cand_i[SAMPLE_CAND_MAX];
  __shared__ unsigned sh_prefix, sh_remaining, sh_count, sh_equal_total;
  __shared__ int sh_owner;

  pdl_trigger();
  pdl_wait();
  const int r = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (redo && !__ldcg(redo + r)) return;       // behind the 32-block kernel: only the rows it marked
  const float* row = logits + (size_t)r * ld;
  const float temp = given.rows ? given.temperature : temperature[r];
  const MaxIdx best = row_argmax(row, vocab, mi_scratch);
  if (!(temp > 0.f)) {
    if (tid == 0) { ids[r] = best.i; if (values) values[r] = best.v; }
    return;
  }
  const float inv_t = 1.0f / temp;
  const float u = given.rows ? given.uniform[r] : uniform[r];
  int k = given.rows ? given.top_k : top_k[r];
  const float tp = given.rows ? given.top_p : top_p[r];
  const bool filtered = (k > 0) || (tp < 1.0f);

  if (!filtered) {
    // Every id in id order.  Warp w owns the contiguous ids [w*seg, (w+1)*seg) and reads them 32 at a time; the
    // warps' sums are added in warp order, which gives the warp that holds the draw; that warp then walks its
    // stretch again, 32 ids at a time, until the running sum passes the draw.
    const int n_warps = SAMPLE_THREADS / 32;
    const int seg = (((vocab + n_warps - 1) / n_warps) + 31) & ~31;
    const int b = min(vocab, warp * seg), e = min(vocab, b + seg);
    float s = 0.f;
    for (int i = b + lane; i < e; i += 32) s += expf((ld_fresh(row + i) - best.v) * inv_t);
    s = warp_sum(s);
    __syncthreads();
    if (lane == 0) f_scratch[warp] = s;
    if (tid == 0) sh_owner = -1;
    __syncthreads();
    if (warp == 0) {
      const float w = f_scratch[lane];                 // n_warps == 32
      const float incl = warp_incl_scan(w);
      const float total = __shfl_sync(0xffffffffu, incl, 31);
      const float target = u * total;
      const unsigned hit = __ballot_sync(0xffffffffu, target < incl);
      if (lane == 0) {
        sh_owner = hit ? (__ffs(hit) - 1) : -1;
        f_scratch[32] = target;
      }
      f_scratch[lane] = incl - w;                      // the sum of the warps before
    }
    __syncthreads();
    const int owner = sh_owner;
    if (owner < 0) {                                   // rounding left no warp: the last id
      if (tid == 0) { ids[r] = vocab - 1; if (values) values[r] = ld_fresh(row + (vocab - 1)); }
      return;
    }
    if (warp != owner) return;
    const float target = f_scratch[32];
    float carry = f_scratch[owner];
    int pick = e - 1;                                  // rounding left no id in the stretch: its last
    for (int base = b; base < e; base += 4 * 32) {
      float x[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int i = base + 32 * j + lane;
        x[j] = i < e ? expf((ld_fresh(row + i) - best.v) * inv_t) : 0.f;
      }
      bool found = false;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        if (!found) {
          const float incl = carry + warp_incl_scan(x[j]);
          const unsigned hit = __ballot_sync(0xffffffffu, target < incl && base + 32 * j + lane < e);
          if (hit) { pick = base + 32 * j + __ffs(hit) - 1; found = true; }
          carry = __shfl_sync(0xffffffffu, incl, 31);
        }
      }
      if (found) break;
    }
    if (lane == 0) { ids[r] = pick; if (values) values[r] = ld_fresh(row + pick); }
    return;
  }

  // ---- filtered: the k largest logits, k <= SAMPLE_CAND_MAX
  if (k <= 0 || k > SAMPLE_CAND_MAX) k = SAMPLE_CAND_MAX;
  if (k > vocab) k = vocab;
  // radix select, 8 bits a pass from the top: find the key of the k-th largest.  Lanes that meet the same bucket
  // add to it once (the first pass sees nearly every logit in two or three buckets).
  if (tid == 0) { sh_prefix = 0; sh_remaining = (unsigned)k; }
  __syncthreads();
  for (int pass = 0; pass < 4; pass++) {
    const int shift = 24 - 8 * pass;
    if (tid < 256) hist[tid] = 0;
    __syncthreads();
    const unsigned prefix = sh_prefix;
    const unsigned mask = pass == 0 ? 0u : (0xFFFFFFFFu << (shift + 8));
    for_each_logit(row, vocab, [&](int, float v) {
      const uint32_t key = float_key(v);
      if ((key & mask) == prefix) {
        const unsigned bucket = (key >> shift) & 255u;
        const unsigned peers = __match_any_sync(__activemask(), bucket);
        if (__ffs(peers) - 1 == lane) atomicAdd(&hist[bucket], (unsigned)__popc(peers));
      }
    });
    __syncthreads();
    {
      // thread t < 256 looks at bucket 255 - t: the bucket that holds the k-th largest is the one whose count, added
      // to the counts of the buckets above it, first reaches what is still wanted (one thread walking the 256
      // buckets cost 4 us a pass)
      const int b = 255 - tid;
      const unsigned cnt = tid < 256 ? hist[b] : 0u;
      const unsigned remaining = sh_remaining;
      unsigned all;
      const unsigned above = block_excl_scan(cnt, u_scratch, &all);
      if (tid < 256 && above < remaining && remaining <= above + cnt) {
        sh_prefix = prefix | ((unsigned)b << shift);
        sh_remaining = remaining - above;   // how many of the k lie in the chosen bucket
        sh_equal_total = cnt;               // after the last pass: how many logits equal the k-th largest
      }
    }
    __syncthreads();
  }
  const uint32_t kth_key = sh_prefix;       // key of the k-th largest logit
  const unsigned n_equal_wanted = sh_remaining;
  // gather: everything above the k-th key, then the lowest ids among those equal to it.  When all
  // the equal ones are wanted (no tie straddles the cut) they are gathered in the same pass.
  const bool take_all_equal = sh_equal_total == n_equal_wanted;
  if (tid == 0) sh_count = 0;
  __syncthreads();
  for_each_logit(row, vocab, [&](int i, float v) {
    const uint32_t key = float_key(v);
    if (key > kth_key || (take_all_equal && key == kth_key)) {
      const unsigned slot = atomicAdd(&sh_count, 1u);
      cand_v[slot] = v;
      cand_i[slot] = i;
    }
  });
  __syncthreads();
  if (!take_all_equal) {
    // a tie straddles the cut: thread t counts the equal ones among its contiguous ids, the counts are summed in
    // thread order, and the first n_equal_wanted of them in id order are taken
    const unsigned above = sh_count;
    const int chunk = (vocab + SAMPLE_THREADS - 1) / SAMPLE_THREADS;
    const int b = min(vocab, tid * chunk), e = min(vocab, b + chunk);
    unsigned mine = 0;
    for (int i = b; i < e; i++) mine += float_key(ld_fresh(row + i)) == kth_key;
    unsigned all;
    unsigned rank = block_excl_scan(mine, u_scratch, &all);
    for (int i = b; i < e && rank < n_equal_wanted; i++) {
      const float v = ld_fresh(row + i);
      if (float_key(v) == kth_key) { cand_v[above + rank] = v; cand_i[above + rank] = i; rank++; }
    }
    __syncthreads();
    if (tid == 0) sh_count = above + n_equal_wanted;
    __syncthreads();
  }
  const int n_cand = (int)sh_count;        // == k
  // pad to a power of two and sort: descending logit, ascending id among equals (bitonic, in shared memory)
  int n_sort = 1;
  while (n_sort < n_cand) n_sort <<= 1;
  for (int i = n_cand + tid; i < n_sort; i += blockDim.x) { cand_v[i] = -INFINITY; cand_i[i] = 0x7fffffff; }
  __syncthreads();
  for (int size = 2; size <= n_sort; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int i = tid; i < n_sort; i += blockDim.x) {
        const int j = i ^ stride;
        if (j > i) {
          const bool up = (i & size) == 0;      // this run is sorted "first comes first"
          const bool i_first = cand_v[i] > cand_v[j] || (cand_v[i] == cand_v[j] && cand_i[i] < cand_i[j]);
          if (i_first != up) {
            const float tv = cand_v[i]; cand_v[i] = cand_v[j]; cand_v[j] = tv;
            const int ti = cand_i[i]; cand_i[i] = cand_i[j]; cand_i[j] = ti;
          }
        }
      }
      __syncthreads();
    }
  }
  // weights of the candidates, then (one warp, lane l holding the 16 consecutive candidates from 16 l on, sums
  // in float64): their total, the top-p cut over the normalised weights, and the draw among what is kept
  const float top = cand_v[0];
  for (int i = tid; i < SAMPLE_CAND_MAX; i += blockDim.x) cand_e[i] = i < n_cand ? expf((cand_v[i] - top) * inv_t) : 0.f;
  __syncthreads();
  if (warp != 0) return;
  draw_from_candidates(cand_v, cand_i, cand_e, n_cand, tp, u, r, ids, values);
}

// ---------------------------------------------------------------- the same, a row cut over 32 blocks
// One block per row reads the row five or six times and is bound by what one SM draws from L2: 36 us with a
// temperature alone, 100 to 130 us with filters, whatever the batch.  Here a row is cut into SS_SPLITS stretches
// of consecutive ids.  A block takes one stretch into shared memory and leaves: its largest logit (greedy rows,
// and the row's maximum); without filters, the sums of its weights exp((l - its maximum) / T) over eight
// sub-stretches; with filters, at least its own min(k, SS_KEEP) largest logits (gather_largest), the key that all it left
// out lie below and how many it kept.  The block that finishes last (a counter per row tells; no block waits) does the
// rest from those leavings: the row's maximum, then either the sub-stretch that holds the draw and a walk through it, or
// the k largest of the 32 lists (in shared memory), sorted, cut by top-p and drawn from, as above.
//
// For k above SS_KEEP any number of the row's k largest could lie in one stretch.  So the last block checks: a stretch has
// nothing hidden among the row's k largest if the key its leavings out lie below is at most the key of the k-th largest of
// all lists.  With 128,256 logits and k = 512 the k-th largest is the 99.6th percentile of the row, a stretch's 64th
// largest the 98.4th of its own, so the check holds unless the large logits crowd in one stretch; when it does not hold
// the row is marked and the one-block kernel, launched behind this one for marked rows only, does the row by itself.
//
// 128,256 logits, top-k 50, top-p 0.95 (us, 1 / 24 / 64 rows): 21 / 31 / 48; with two radix selections and lists in id
// order it took 36 / 61 / 113, and one block a row takes 87.  k = 512: 43 / 54 / 72 against 47 / 72 / 125.
// Sums are taken in an order that depends on the sizes only.
#define SS_SPLITS 32
#define SS_THREADS 256
#define SS_WARPS (SS_THREADS / 32)
static_assert(SS_THREADS == 256, "one thread per bucket of the radix passes");
#define SS_CHUNK_MAX 8192
#define SS_KEEP 64
#define SS_LIST 128              // room of a stretch's list
#define SS_LIST_MAX (SS_SPLITS * SS_LIST)
#define SS_FEW 128               // up to this k the last block places the candidates by counting

struct SsScratch {               // in global memory, per row (counters zeroed once; every launch leaves them at zero)
  float* part_v; int* part_i;    // [rows][SS_SPLITS] largest logit of the stretch and its id
  float* part_e;                 // [rows][SS_SPLITS][SS_WARPS] sums of the sub-stretches' weights (stretch's own maximum)
  unsigned* part_key;            // [rows][SS_SPLITS] what the stretch did not keep lies below this key (0: it kept all)
  float* cand_v; int* cand_i;    // [rows][SS_SPLITS][SS_LIST]: the stretches' lists, keys (as bits) and ids; the number
                                 // of entries lies in part_e, as bits, at the stretch's first place
  unsigned* counters;            // [rows]
  int* redo;                     // [rows] 1: the one-block kernel does this row
};

// The key of the k-th largest of n keys, 1 <= k <= n, by a radix select; *equals: how many have that key.  Returns how many
// of those belong to the k largest.  Every thread of the block calls it.  hist: 256 words, sh: 2.
template <typename Key>
__device__ unsigned radix_kth(Key key_of, int n, int k, unsigned* hist, unsigned* sh, unsigned* w_scratch33, uint32_t* kth,
                              uint32_t* equals) {
  const int tid = threadIdx.x;
  if (tid == 0) { sh[0] = 0; sh[1] = (unsigned)k; }
  __syncthreads();
  for (int pass = 0; pass < 4; pass++) {          // radix select, 8 bits a pass from the top
    const int shift = 24 - 8 * pass;
    hist[tid] = 0;                                 // (SS_THREADS == 256 buckets)
    __syncthreads();
    const unsigned prefix = sh[0];
    const unsigned mask = pass == 0 ? 0u : (0xFFFFFFFFu << (shift + 8));
    for (int j = tid; j < n; j += SS_THREADS) {
      const uint32_t key = key_of(j);
      if ((key & mask) == prefix) atomicAdd(&hist[(key >> shift) & 255u], 1u);
    }
    __syncthreads();
    {
      // thread t looks at bucket 255 - t: the bucket that holds the k-th largest is the one whose count, added to
      // the counts of the buckets above it, first reaches what is still wanted
      const int b = 255 - tid;
      const unsigned cnt = hist[b];
      const unsigned remaining = sh[1];
      unsigned all;
      const unsigned above = block_excl_scan(cnt, w_scratch33, &all);
      if (above < remaining && remaining <= above + cnt) {
        sh[0] = prefix | ((unsigned)b << shift);
        sh[1] = remaining - above;                 // how many of the k lie in the chosen bucket
      }
    }
    __syncthreads();
  }
  *kth = sh[0];
  *equals = hist[sh[0] & 255u];                    // the last pass's bucket
  return sh[1];
}

// Among n values in ascending id order (val(j), id(j)), the k largest, k < n, the lowest ids first among equals at the
// cut, written in ascending id order to out_v / out_i; *kth_key gets the key of the smallest of them.  Every thread of the
// block calls it.  hist: 256 words, sh: 2, w_scratch: 2 * SS_WARPS.
template <typename Val, typename Id>
__device__ void select_in_order(Val val, Id id, int n, int k, float* out_v, int* out_i, unsigned* hist, unsigned* sh,
                               unsigned* w_scratch, unsigned* w_scratch33, uint32_t* kth_key) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t kth, equals;
  const unsigned want_eq = radix_kth([&](int j) { return float_key(val(j)); }, n, k, hist, sh, w_scratch33, &kth, &equals);
  // in id order, 256 ids a round: an element's rank among the equal ones and its place in the output are counts of
  // the elements before it (votes inside a warp, the warps' counts through shared memory)
  unsigned eq_before = 0, out_before = 0;
  const unsigned lt = (1u << lane) - 1u;
  for (int j0 = 0; j0 < n; j0 += SS_THREADS) {
    const int j = j0 + tid;
    const float v = j < n ? val(j) : 0.f;
    const uint32_t key = j < n ? float_key(v) : 0u;
    const bool eq = j < n && key == kth;
    const unsigned eq_votes = __ballot_sync(0xffffffffu, eq);
    if (lane == 0) w_scratch[warp] = (unsigned)__popc(eq_votes);
    __syncthreads();
    unsigned eq_rank = eq_before + (unsigned)__popc(eq_votes & lt), eq_round = 0;
    for (int w = 0; w < SS_WARPS; w++) { const unsigned c = w_scratch[w]; if (w < warp) eq_rank += c; eq_round += c; }
    const bool take = j < n && (key > kth || (eq && eq_rank < want_eq));
    const unsigned take_votes = __ballot_sync(0xffffffffu, take);
    if (lane == 0) w_scratch[SS_WARPS + warp] = (unsigned)__popc(take_votes);
    __syncthreads();
    unsigned place = out_before + (unsigned)__popc(take_votes & lt), take_round = 0;
    for (int w = 0; w < SS_WARPS; w++) { const unsigned c = w_scratch[SS_WARPS + w]; if (w < warp) place += c; take_round += c; }
    if (take) { out_v[place] = v; out_i[place] = id(j); }
    eq_before += eq_round;
    out_before += take_round;
  }
  __syncthreads();
  *kth_key = kth;
}

// At least the k largest of n, k <= SS_THREADS, by their keys: thread t's largest element is one of SS_THREADS maxima, and
// the k-th largest of those is at most the k-th largest of all.  put(slot, key, j) is called for every element that
// reaches it (a little more than k of them as a rule, in any order; all of those with that key) whose slot is below
// `room`.  Returns how many there are; *least_of gets the key.  Three barriers in place of the radix passes' 24 and two
// per 256 elements.  maxima: SS_THREADS words; sh: 2.
template <typename Key, typename Put>
__device__ __forceinline__ unsigned gather_largest(Key key, Put put, int n, int k, unsigned room, uint32_t* maxima,
                                                   unsigned* sh, uint32_t* least_of) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t mine = 0u;
  for (int j = tid; j < n; j += SS_THREADS) mine = max(mine, key(j));
  if (tid == 0) sh[1] = 0u;
  // every maximum's rank: its place in its warp's, sorted by shuffles, and searches through the other warps'
  uint32_t v = mine;
#pragma unroll
  for (int size = 2; size <= 32; size <<= 1)
#pragma unroll
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      const uint32_t other = __shfl_xor_sync(0xffffffffu, v, stride);
      const bool larger = ((lane & stride) == 0) == ((lane & size) == 0);      // descending in the end
      v = larger ? max(v, other) : min(v, other);
    }
  maxima[tid] = v;
  __syncthreads();
  int before = lane;
#pragma unroll
  for (int w = 0; w < SS_WARPS; w++) {
    if (w == warp) continue;
    const uint32_t* list = maxima + 32 * w;
    int lo = 0;                                    // how many of warp w's come before v (equal ones of lower warps do)
#pragma unroll
    for (int step = 16; step > 0; step >>= 1) {
      const uint32_t o = list[lo + step - 1];
      if (o > v || (o == v && w < warp)) lo += step;
    }
    const uint32_t o = list[lo];                   // lo <= 31 after five steps
    before += lo + (o > v || (o == v && w < warp));
  }
  if (before == k - 1) sh[0] = v;
  __syncthreads();
  const uint32_t least = sh[0];
  if (mine >= least)
    for (int j = tid; j < n; j += SS_THREADS) {
      const uint32_t kj = key(j);
      if (kj < least) continue;
      const unsigned slot = atomicAdd(&sh[1], 1u);
      if (slot < room) put(slot, kj, j);
    }
  __syncthreads();
  *least_of = least;
  return sh[1];
}
// How many of the n gathered elements come before element i: larger keys, then lower ids.
__device__ __forceinline__ int place_of(const uint32_t* f_key, const int* f_id, int n, int i) {
  const uint32_t mine = f_key[i];
  const int id = f_id[i];
  int before = 0;
#pragma unroll 4
  for (int j = 0; j < n; j++) before += f_key[j] > mine || (f_key[j] == mine && f_id[j] < id);
  return before;
}

__global__ void __launch_bounds__(SS_THREADS)
sample_split_kernel(const float* __restrict__ logits, int ld, int vocab, const float* __restrict__ temperature,
                    const int* __restrict__ top_k, const float* __restrict__ top_p,
                    const float* __restrict__ uniform, int* __restrict__ ids, float* __restrict__ values,
                    const SsScratch Q, const __grid_constant__ SampleGiven given) {
  extern __shared__ __align__(16) float lv[];      // the stretch's logits; in the last block, the lists: values, ids
  __shared__ MaxIdx mi_scratch[33];
  __shared__ float f_scratch[SS_THREADS + 2];
  __shared__ unsigned w_scratch[2 * SS_WARPS];
  __shared__ unsigned u_scratch[33];
  __shared__ unsigned hist[256];
  __shared__ unsigned sh[2];
  __shared__ float cand_e[SAMPLE_CAND_MAX];
  __shared__ float cand_v[SAMPLE_CAND_MAX];
  __shared__ int cand_i[SAMPLE_CAND_MAX];
  __shared__ uint32_t f_key[SS_THREADS];
  __shared__ int f_id[SS_THREADS];
  __shared__ int list_at[SS_SPLITS + 1];
  __shared__ int sh_owner;
  __shared__ bool last;

  pdl_trigger();
  pdl_wait();
  const int r = blockIdx.x, sp = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float* row = logits + (size_t)r * ld;
  const float temp = given.rows ? given.temperature : temperature[r];
  const bool sampled = temp > 0.f;
  const float inv_t = sampled ? 1.0f / temp : 0.f;
  int k = given.rows ? given.top_k : top_k[r];
  const float tp = given.rows ? given.top_p : top_p[r];
  const bool filtered = sampled && ((k > 0) || (tp < 1.0f));
  if (k <= 0 || k > SAMPLE_CAND_MAX) k = SAMPLE_CAND_MAX;
  if (k > vocab) k = vocab;
  const int k1 = min(k, SS_KEEP);                  // what a stretch keeps
  const int chunk = (vocab + SS_SPLITS - 1) / SS_SPLITS;
  auto stretch_len = [&](int s2) { return min(vocab, (s2 + 1) * chunk) - min(vocab, s2 * chunk); };
  const int b0 = min(vocab, sp * chunk), n = stretch_len(sp);
  const int part = r * SS_SPLITS + sp;
  // the sub-stretch of warp w: ids [w sub, (w+1) sub) of the stretch
  const int sub = (chunk + SS_WARPS - 1) / SS_WARPS;

  // ---- this block's stretch
  MaxIdx mine{-INFINITY, 0x7fffffff};
#pragma unroll 4
  for (int j = tid; j < n; j += SS_THREADS) {
    const float v = ld_fresh(row + b0 + j);
    lv[j] = v;
    if (v > mine.v) { mine.v = v; mine.i = b0 + j; }              // ascending ids per thread: the first of equals stays
  }
  const MaxIdx local = block_argmax(mine, mi_scratch);
  if (tid == 0) { Q.part_v[part] = local.v; Q.part_i[part] = local.i; }
  if (sampled && !filtered) {
    float e = 0.f;
    if (local.i != 0x7fffffff)
      for (int j = warp * sub + lane; j < min(n, (warp + 1) * sub); j += 32) e += expf((lv[j] - local.v) * inv_t);
    e = warp_sum(e);
    if (lane == 0) Q.part_e[(size_t)part * SS_WARPS + warp] = e;
  } else if (filtered) {
    float* to_v = Q.cand_v + (size_t)part * SS_LIST;
    int* to_i = Q.cand_i + (size_t)part * SS_LIST;
    auto put = [&](unsigned slot, uint32_t key, int j) {
      to_v[slot] = __uint_as_float(key);
      to_i[slot] = b0 + j;
    };
    uint32_t below;                                 // (a stretch has more ids than are kept of it: the launcher's least vocabulary)
    unsigned kept = gather_largest([&](int j) { return float_key(lv[j]); }, put, n, k1, SS_LIST, hist, sh, &below);
    if (kept > SS_LIST) {                           // a crowd of equals: exactly k1, the lowest ids first among equals
      __syncthreads();                              // (everyone knows how many were gathered)
      uint32_t kth;
      select_in_order([&](int j) { return lv[j]; }, [&](int j) { return b0 + j; }, n, k1, cand_v, cand_i, hist, sh, w_scratch,
                      u_scratch, &kth);
      kept = k1;
      for (int j = tid; j < k1; j += SS_THREADS) { to_v[j] = __uint_as_float(float_key(cand_v[j])); to_i[j] = cand_i[j]; }
      below = kth == 0xffffffffu ? kth : kth + 1;
    }
    if (tid == 0) {
      Q.part_key[part] = below;
      Q.part_e[(size_t)part * SS_WARPS] = __uint_as_float(kept);
    }
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) last = atomicAdd(&Q.counters[r], 1u) == SS_SPLITS - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();

  // ---- the block that finished last: the row's maximum (the lowest id among equals: stretches are in id order)
  if (warp == 0) {
    MaxIdx t{-INFINITY, 0x7fffffff};
    if (lane < SS_SPLITS) { t.v = __ldcg(Q.part_v + r * SS_SPLITS + lane); t.i = __ldcg(Q.part_i + r * SS_SPLITS + lane); }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      MaxIdx other;
      other.v = __shfl_xor_sync(0xffffffffu, t.v, o);
      other.i = __shfl_xor_sync(0xffffffffu, t.i, o);
      t = better(t, other);
    }
    if (lane == 0) {
      if (t.i == 0x7fffffff) { t.i = 0; t.v = ld_fresh(row + 0); }   // every logit is -inf or NaN: index 0
      mi_scratch[32] = t;
      Q.counters[r] = 0;
      Q.redo[r] = 0;
    }
  }
  __syncthreads();
  const MaxIdx best = mi_scratch[32];
  if (!sampled) {
    if (tid == 0) { ids[r] = best.i; if (values) values[r] = best.v; }
    return;
  }
  const float u = given.rows ? given.uniform[r] : uniform[r];

  if (!filtered) {
    // thread t: sub-stretch t % 8 of stretch t / 8; their sums brought to the row's maximum, added in id order
    const int s_of = tid / SS_WARPS;
    const bool any = __ldcg(Q.part_i + r * SS_SPLITS + s_of) != 0x7fffffff;
    const float m_s = __ldcg(Q.part_v + r * SS_SPLITS + s_of);
    const float scale = any ? expf((m_s - best.v) * inv_t) : 0.f;
    const float w = any ? __ldcg(Q.part_e + (size_t)r * SS_SPLITS * SS_WARPS + tid) * scale : 0.f;
    float total;
    const float before = block_excl_scan(w, f_scratch, &total);
    const float target = u * total;
    if (tid == 0) sh_owner = 0x7fffffff;
    __syncthreads();
    // the first sub-stretch whose running sum passes the draw
    if (target < before + w) atomicMin(&sh_owner, tid);
    __syncthreads();
    const int owner = sh_owner;
    if (owner == 0x7fffffff) {                         // rounding left none: the last id
      if (tid == 0) { ids[r] = vocab - 1; if (values) values[r] = ld_fresh(row + (vocab - 1)); }
      return;
    }
    if (tid == owner) { f_scratch[SS_THREADS] = before; f_scratch[SS_THREADS + 1] = scale; mi_scratch[0].v = m_s; }
    __syncthreads();
    if (warp != 0) return;
    const float carry0 = f_scratch[SS_THREADS], scale_o = f_scratch[SS_THREADS + 1], m_o = mi_scratch[0].v;
    const int so = owner / SS_WARPS, wo = owner % SS_WARPS;
    const int sb = min(vocab, so * chunk), sn = stretch_len(so);
    const int b = sb + min(sn, wo * sub), e = sb + min(sn, (wo + 1) * sub);
    float carry = carry0;
    int pick = e - 1;                                  // rounding left no id in the sub-stretch: its last
    for (int base = b; base < e; base += 4 * 32) {
      float x[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int i = base + 32 * j + lane;
        x[j] = i < e ? expf((ld_fresh(row + i) - m_o) * inv_t) * scale_o : 0.f;
      }
      bool found = false;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        if (!found) {
          const float incl = carry + warp_incl_scan(x[j]);
          const unsigned hit = __ballot_sync(0xffffffffu, target < incl && base + 32 * j + lane < e);
          if (hit) { pick = base + 32 * j + __ffs(hit) - 1; found = true; }
          carry = __shfl_sync(0xffffffffu, incl, 31);
        }
      }
      if (found) break;
    }
    if (lane == 0) { ids[r] = pick; if (values) values[r] = ld_fresh(row + pick); }
    return;
  }

  // ---- filtered: the lists' keys, one list after another, into shared memory; the k largest of them
  if (warp == 0) {
    const int mine_n = (int)__float_as_uint(__ldcg(Q.part_e + (size_t)(r * SS_SPLITS + lane) * SS_WARPS));
    const int upto = warp_incl_scan(mine_n);
    list_at[lane] = upto - mine_n;
    if (lane == 31) list_at[SS_SPLITS] = upto;
  }
  __syncthreads();
  uint32_t* lk = reinterpret_cast<uint32_t*>(lv);
#pragma unroll
  for (int s2 = warp; s2 < SS_SPLITS; s2 += SS_WARPS) {
    const int at = list_at[s2], len = list_at[s2 + 1] - at;
#pragma unroll
    for (int i = 0; i < SS_LIST; i += 32)
      if (i + lane < len) lk[at + i + lane] = __float_as_uint(__ldcg(Q.cand_v + (size_t)(r * SS_SPLITS + s2) * SS_LIST + i + lane));
  }
  const int n_all = list_at[SS_SPLITS];
  auto id_of = [&](int j) {                          // the id that belongs to lk[j]: in the last list that begins at or before j
    int s2 = 0;                                      // (empty lists begin where the next one does)
#pragma unroll
    for (int step = SS_SPLITS / 2; step > 0; step >>= 1)
      if (list_at[s2 + step] <= j) s2 += step;
    return __ldcg(Q.cand_i + (size_t)(r * SS_SPLITS + s2) * SS_LIST + j - list_at[s2]);
  };
  __syncthreads();
  const int n_cand = k;
  uint32_t kth = 0u;
  bool sorted = false;                               // (the lists hold k in all: 32 min(k, SS_KEEP) at least)
  if (k <= SS_FEW) {
    uint32_t least;
    const unsigned found = gather_largest([&](int j) { return lk[j]; },
                                          [&](unsigned slot, uint32_t key, int j) { f_key[slot] = key; f_id[slot] = id_of(j); },
                                          n_all, k, SS_THREADS, hist, sh, &least);
    if (found <= SS_THREADS) {
      const int place = tid < (int)found ? place_of(f_key, f_id, found, tid) : k;
      if (place < k) { cand_v[place] = key_float(f_key[tid]); cand_i[place] = f_id[tid]; }
      if (place == k - 1) sh[0] = f_key[tid];
      __syncthreads();
      kth = sh[0];
      sorted = true;
    }
    __syncthreads();                                 // (everyone knows how many were gathered, and the k-th key)
  }
  uint32_t equals = 0u;
  const unsigned wanted = sorted ? 0u : radix_kth([&](int j) { return lk[j]; }, n_all, k, hist, sh, u_scratch, &kth, &equals);
  // is anything that a stretch did not keep among the row's k largest?
  if (__syncthreads_or(tid < SS_SPLITS && k1 < k && __ldcg(Q.part_key + r * SS_SPLITS + tid) > kth)) {
    if (tid == 0) Q.redo[r] = 1;
    return;
  }
  if (!sorted) {
    uint32_t last_id = 0u;                           // (ids turned round: of equals the lower id is the larger)
    if (wanted != equals) {                          // equals straddle the cut: the lowest ids of them, by one more selection
      uint32_t one;
      radix_kth([&](int j) { return lk[j] == kth ? ~(uint32_t)id_of(j) : 0u; }, n_all, wanted, hist, sh, u_scratch, &last_id, &one);
      __syncthreads();
    }
    if (tid == 0) sh[0] = 0u;
    __syncthreads();
    for (int j = tid; j < n_all; j += SS_THREADS)
      if (lk[j] >= kth) {
        const int id = id_of(j);
        if (lk[j] == kth && ~(uint32_t)id < last_id) continue;
        const unsigned slot = atomicAdd(&sh[0], 1u);
        cand_v[slot] = key_float(lk[j]);
        cand_i[slot] = id;
      }
    __syncthreads();
  }
  // pad to a power of two and sort: descending logit, ascending id among equals (bitonic, in shared memory)
  int n_sort = 1;
  while (!sorted && n_sort < n_cand) n_sort <<= 1;
  for (int i = n_cand + tid; i < n_sort; i += blockDim.x) { cand_v[i] = -INFINITY; cand_i[i] = 0x7fffffff; }
  __syncthreads();
  for (int size = 2; size <= n_sort; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int i = tid; i < n_sort; i += blockDim.x) {
        const int j = i ^ stride;
        if (j > i) {
          const bool up = (i & size) == 0;
          const bool i_first = cand_v[i] > cand_v[j] || (cand_v[i] == cand_v[j] && cand_i[i] < cand_i[j]);
          if (i_first != up) {
            const float tv = cand_v[i]; cand_v[i] = cand_v[j]; cand_v[j] = tv;
            const int ti = cand_i[i]; cand_i[i] = cand_i[j]; cand_i[j] = ti;
          }
        }
      }
      __syncthreads();
    }
  }
  const float top = cand_v[0];
  for (int i = tid; i < SAMPLE_CAND_MAX; i += blockDim.x) cand_e[i] = i < n_cand ? expf((cand_v[i] - top) * inv_t) : 0.f;
  __syncthreads();
  if (warp != 0) return;
  draw_from_candidates(cand_v, cand_i, cand_e, n_cand, tp, u, r, ids, values);
}

static int sample_rows(const float* logits, int ld, int n_rows, int vocab, const float* temperature, const int* top_k,
                       const float* top_p, const float* uniform, int* ids, float* values, const SsScratch& Q,
                       const SampleGiven& given, cudaStream_t stream) {
  if (n_rows <= 0) return 0;
  if (vocab < 1) return STRATUM_ERR_SHAPE;
  if (Q.part_v && Q.part_i && Q.part_e && Q.part_key && Q.cand_v && Q.cand_i && Q.counters && Q.redo && vocab >= 8192 &&
      vocab <= SS_SPLITS * SS_CHUNK_MAX) {
    const size_t chunk_bytes = (size_t)((vocab + SS_SPLITS - 1) / SS_SPLITS) * sizeof(float);
    const size_t list_bytes = (size_t)SS_LIST_MAX * sizeof(uint32_t);
    const size_t smem = chunk_bytes > list_bytes ? chunk_bytes : list_bytes;
    int st = launch_pdl(sample_split_kernel, dim3(n_rows, SS_SPLITS), SS_THREADS, smem, stream, logits, ld, vocab,
                        temperature, top_k, top_p, uniform, ids, values, Q, given);
    if (st != 0) return st;
    return launch_pdl(sample_kernel, n_rows, SAMPLE_THREADS, 0, stream, logits, ld, vocab, temperature, top_k, top_p,
                      uniform, ids, values, (const int*)Q.redo, given);
  }
  return launch_pdl(sample_kernel, n_rows, SAMPLE_THREADS, 0, stream, logits, ld, vocab, temperature, top_k, top_p,
                    uniform, ids, values, (const int*)nullptr, given);
}

// scratch (optional, all eight or none): see SsScratch; with it, rows of 8,192 to 262,144 logits are cut over 32
// blocks each, and the one-block kernel runs behind for the rows that were marked.
STRATUM_EXPORT int stratum_sample(const float* logits, int ld, int n_rows, int vocab, const float* temperature,
                                  const int* top_k, const float* top_p, const float* uniform, int* ids,
                                  float* values, float* part_v, int* part_i, float* part_e, unsigned* part_key,
                                  float* cand_v, int* cand_i, unsigned* counters, int* redo, cudaStream_t stream) {
  static const SampleGiven none = {};
  return sample_rows(logits, ld, n_rows, vocab, temperature, top_k, top_p, uniform, ids, values,
                     SsScratch{part_v, part_i, part_e, part_key, cand_v, cand_i, counters, redo}, none, stream);
}

// The same for up to 256 rows of one temperature, top_k and top_p, with the uniforms in host memory.
STRATUM_EXPORT int stratum_sample_given(const float* logits, int ld, int n_rows, int vocab, float temperature, int top_k,
                                        float top_p, const float* host_uniforms, int* ids, float* values, float* part_v,
                                        int* part_i, float* part_e, unsigned* part_key, float* cand_v, int* cand_i,
                                        unsigned* counters, int* redo, cudaStream_t stream) {
  if (n_rows > SAMPLE_GIVEN_MAX) return STRATUM_ERR_LIMIT;
  if (n_rows > 0 && !host_uniforms) return STRATUM_ERR_SHAPE;
  SampleGiven given = {};
  given.rows = n_rows;
  given.temperature = temperature; given.top_k = top_k; given.top_p = top_p;
  for (int i = 0; i < n_rows; i++) given.uniform[i] = host_uniforms[i];
  return sample_rows(logits, ld, n_rows, vocab, nullptr, nullptr, nullptr, nullptr, ids, values,
                     SsScratch{part_v, part_i, part_e, part_key, cand_v, cand_i, counters, redo}, given, stream);
}

// ---------------------------------------------------------------- feeding picked ids back on the device
// ids[i] = prev[feed[i]] where feed[i] >= 0; elsewhere ids[i] stays what the host wrote.  It lets the next decode
// step be launched before the host has read what this one picked (the reference queues its decode steps on the
// GPU the same way, with the token ring on the device: stratum/native/stratum_arch_llama.inc.c:1992-2030).
__global__ void feed_ids_kernel(int* __restrict__ ids, const int* __restrict__ feed, const int* prev, int n) {
  pdl_trigger();
  pdl_wait();                                      // `prev` is the work of the step before
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int f = feed[i];
  if (f >= 0) ids[i] = __ldcg(prev + f);
}

STRATUM_EXPORT int stratum_feed_ids(int* ids, const int* feed, const int* prev, int n, cudaStream_t stream) {
  if (n <= 0) return 0;
  return launch_pdl(feed_ids_kernel, (n + 127) / 128, 128, 0, stream, ids, feed, prev, n);
}

