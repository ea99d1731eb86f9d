// y = x W^T (+ bias) for any sizes, on CUDA cores, float32 accumulation in a fixed order.
//
// This is the whole linear layer of the true 32-bit path (no tensor-core mode of reduced
// precision anywhere), and the fallback of the bfloat16 path for shapes the tensor-core
// kernels refuse.  W is row-major [N][K] as stored in the file: y[m][n] = sum_k x[m][k] W[n][k]
// (stratum/native/stratum_linear.h:491-507).
//
// The order of a sum follows from K alone, so a value does not depend on M, on the tile it falls in,
// or on what else is in the step, and prompts and decode steps give the same bits:
//   bfloat16: one chain of fused multiply-adds over k = 0..K-1;
//   float32:  K is cut into at most eight segments (f32_segment); inside a segment the even and the odd k are a
//             chain each, then even + odd; the segments are added in order.  Even and odd are the two halves of
//             fma.rn.f32x2, whose operands then are two neighbouring values of a row as they lie in memory, and the
//             segments are what few rows of x, or few tiles, are spread over the GPU by.
//
// Epilogues: 0 store as x's type; 1 add into a float32 tensor in place (the residual stream);
//            2 store as float32 (logits).
#include "common.cuh"

// ---------------------------------------------------------------- bfloat16: one chain per output
#define LS_BM 64
#define LS_BN 64
#define LS_BK 16
#define LS_TM 4
#define LS_TN 4

template <int EPI>
__global__ void __launch_bounds__(256)
linear_simple_kernel(const bf16* __restrict__ x, const bf16* __restrict__ w, const float* __restrict__ bias,
                     void* __restrict__ out, int M, int N, int K, int ldx, int ldo, int x_step, long long w_step,
                     int o_step, int act) {
  __shared__ float xs[LS_BK][LS_BM + 1];
  __shared__ float ws[LS_BK][LS_BN + 1];
  const int tid = threadIdx.x;
  // one product per blockIdx.z (the heads of linear_heads): operands and result move on by their steps
  x += (size_t)blockIdx.z * x_step;
  w += (size_t)blockIdx.z * w_step;
  const size_t o_shift = (size_t)blockIdx.z * o_step;
  const int m0 = blockIdx.y * LS_BM, n0 = blockIdx.x * LS_BN;
  const int tm = (tid / 16) * LS_TM, tn = (tid % 16) * LS_TN;
  float acc[LS_TM][LS_TN];
#pragma unroll
  for (int i = 0; i < LS_TM; i++)
#pragma unroll
    for (int j = 0; j < LS_TN; j++) acc[i][j] = 0.f;

  // each thread loads 4 elements of each tile per step: row = tid / 4, k = (tid % 4) * 4 .. +3
  const int lr = tid / 4, lk = (tid % 4) * 4;
  for (int k0 = 0; k0 < K; k0 += LS_BK) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int k = k0 + lk + j;
      const int m = m0 + lr, n = n0 + lr;
      xs[lk + j][lr] = (m < M && k < K) ? to_float(x[(size_t)m * ldx + k]) : 0.f;
      ws[lk + j][lr] = (n < N && k < K) ? to_float(w[(size_t)n * K + k]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < LS_BK; kk++) {
      float a[LS_TM], b[LS_TN];
#pragma unroll
      for (int i = 0; i < LS_TM; i++) a[i] = xs[kk][tm + i];
#pragma unroll
      for (int j = 0; j < LS_TN; j++) b[j] = ws[kk][tn + j];
#pragma unroll
      for (int i = 0; i < LS_TM; i++)
#pragma unroll
        for (int j = 0; j < LS_TN; j++) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < LS_TM; i++) {
    const int m = m0 + tm + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < LS_TN; j++) {
      const int n = n0 + tn + j;
      if (n >= N) continue;
      float v = acc[i][j];
      if (bias) v += bias[n];
      const size_t o = (size_t)m * ldo + n + o_shift;
      if (EPI == 0) ((bf16*)out)[o] = __float2bfloat16_rn(activate(v, act));
      else if (EPI == 1) ((float*)out)[o] += v;
      else ((float*)out)[o] = v;
    }
  }
}

static int launch_linear_simple(const void* x, const void* w, const float* bias, void* out, int epilogue,
                                int M, int N, int K, int ldx, int ldo, cudaStream_t stream, int heads = 1,
                                int x_step = 0, long long w_step = 0, int o_step = 0, int act = 0) {
  dim3 grid((N + LS_BN - 1) / LS_BN, (M + LS_BM - 1) / LS_BM, heads);
  if (epilogue == 0)
    linear_simple_kernel<0><<<grid, 256, 0, stream>>>((const bf16*)x, (const bf16*)w, bias, out, M, N, K, ldx, ldo,
                                                      x_step, w_step, o_step, act);
  else if (epilogue == 1)
    linear_simple_kernel<1><<<grid, 256, 0, stream>>>((const bf16*)x, (const bf16*)w, bias, out, M, N, K, ldx, ldo,
                                                      x_step, w_step, o_step, act);
  else if (epilogue == 2)
    linear_simple_kernel<2><<<grid, 256, 0, stream>>>((const bf16*)x, (const bf16*)w, bias, out, M, N, K, ldx, ldo,
                                                      x_step, w_step, o_step, act);
  else
    return STRATUM_ERR_SHAPE;
  return launch_status();
}

// ---------------------------------------------------------------- float32
// Two kernels, chosen by the rows of x (launch_f32): up to F32_FEW_ROWS one that streams W, above it one that holds
// tiles of 64 or 32 rows by 128 columns in registers.  Measured by themselves with a cold L2 (us; the one kernel of scalar
// FMA on 64 x 64 tiles that served every shape before in brackets):
//   rows of x               1            8            64           611
//   N 3072   K 2048      14 (176)     18 (176)     38 (181)    192 (488)
//   N 16384  K 2048      45 (254)     51 (257)    128 (278)    949 (2079)
//   N 2048   K 8192      25 (706)     31 (707)     67 (721)    462 (1427)
//   N 128256 K 2048     219 (1431)   285 (1455)
// and the error against 64 bits is 2.1e-7 (8.1e-7) at K 2048, 4.1e-7 (1.6e-6) at 8192: shorter chains.  The line between
// the two lies at eight rows: 13 rows as two groups of eight took 90, 50 and 605 us on the last three shapes, 17 rows on
// a tile of 32 rows 77, 48 and 432.

#define F32_BK 32             // k per stage of either kernel: 128 bytes of a row
#define F32_PITCH 36          // floats between rows in shared memory: 16-byte loads of eight neighbouring rows are conflict-free
#define F32_FEW_ROWS 8
#define F32_TILE_STAGES 2
#define F32_MAX_SEGMENTS 8

// k per segment: 256, or an eighth of K (rounded up to a stage) where that is more
static __host__ __device__ __forceinline__ int f32_segment(int K) {
  const int eighth = ((K + F32_MAX_SEGMENTS - 1) / F32_MAX_SEGMENTS + F32_BK - 1) / F32_BK * F32_BK;
  return eighth > 256 ? eighth : 256;
}

typedef unsigned long long f32x2;
__device__ __forceinline__ void fma2(f32x2& acc, f32x2 a, f32x2 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float even_plus_odd(f32x2 v) {
  return __fadd_rn(__uint_as_float((unsigned)v), __uint_as_float((unsigned)(v >> 32)));
}

// four floats of a row from column k on into shared memory, zeros where the row ends (`row` false: none of it is there).
// VEC = false goes through L1: for a kernel launched ahead of the end of the one before, weights only.
template <bool VEC>
__device__ __forceinline__ void copy4(float* dst, const float* src, int k, int K, bool row) {
  const unsigned to = (unsigned)__cvta_generic_to_shared(dst);
  if (VEC) {                                     // K is a multiple of 4: all four or none
    const int bytes = row && k < K ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(bytes ? src + k : src), "r"(bytes)
                 : "memory");
  } else {
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int bytes = row && k + i < K ? 4 : 0;
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(to + 4 * i), "l"(bytes ? src + k + i : src),
                   "r"(bytes)
                   : "memory");
    }
  }
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

struct F32Product {
  const float *x, *w, *bias;
  float *out, *parts;           // parts: [heads][segments][M][N], where the segments of a tile are cut over several blocks
  int M, N, K, ldx, ldo, x_step, o_step, act, epilogue, segment, segments;
  long long w_step;
};

__device__ __forceinline__ void f32_finish(const F32Product& p, int head, int m, int n, float v) {
  if (p.bias) v += p.bias[n];
  float* o = p.out + (size_t)m * p.ldo + n + (size_t)head * p.o_step;
  if (p.epilogue == 1) *o = ld_fresh(o) + v;
  else *o = p.epilogue == 0 ? activate(v, p.act) : v;
}

// Few rows of x: bound by the bytes of W.  A thread owns one (row of W, segment) and all MR rows of x; a warp streams
// its 32 stretches of W through a ring of its own (cp.async, 4 KB a stage), so nothing but the sum over the segments needs
// the block.  The rows of x come with W's stages.  A block goes from tile to tile (of 128 / segments rows of W) with
// its ring full, and fills it before it waits for the kernel in front of it.  STAGES: 4, two blocks to an SM; where the
// tiles are fewer than the SMs 8, so that the one block of an SM still has 130 KB in flight.
// In a chain of launches, 1 / 3 / 8 rows of x: 16,384 x 2,048 28 / 32 / 41 us (4.8 / 4.2 / 3.3 TB/s of W), 128,256 x 2,048
// 198 / 213 / 276, 2,048 x 8,192 16 / 20 / 23.  (Two rows of W a thread, for half as many loads of x, and half as many warps:
// 26 / 33 / 38, 188 / 209 / 261 and 18 / 23 / 31.)
template <int MR, bool VEC, int STAGES>
__global__ void __launch_bounds__(128)
linear_f32_few_kernel(const F32Product p, const int rows_per_block /* 128 / segments rounded up to a power of two */) {
  constexpr int W_FLOATS = 32 * F32_PITCH, X_FLOATS = 2 * MR * F32_PITCH;
  extern __shared__ __align__(16) float smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, head = blockIdx.z;
  float* sums = smem;                            // [MR][128]
  float* ring = smem + MR * 128 + warp * STAGES * (W_FLOATS + X_FLOATS);
  const float* w = p.w + (size_t)head * p.w_step;
  const float* x = p.x + (size_t)head * p.x_step;
  const int tiles = (p.N + rows_per_block - 1) / rows_per_block, iters = p.segment / F32_BK;
  const int my_tiles = (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x, total = my_tiles * iters;
  const int warp_segments = rows_per_block < 32 ? 32 / rows_per_block : 1;      // 1 or 2
  const int first_segment = warp * 32 / rows_per_block;
  // what this lane copies of W in each of eight rounds: 16 bytes of row (round * 4 + lane / 8) of the warp's 32.  The rows'
  // places are worked out once: in every stage they were half of the kernel's instructions, and its bound (51 against 42 us
  // for 16,384 + 3,072 rows of 2,048).
  const int ck = (lane & 7) * 4, row0 = lane >> 3;
  long long place[8];
#pragma unroll
  for (int r = 0; r < 8; r++) {
    const int id = warp * 32 + r * 4 + row0;
    place[r] = (long long)(id % rows_per_block) * p.K + (id / rows_per_block) * p.segment;
  }
  const bool whole = VEC && p.K == p.segments * p.segment && rows_per_block * p.segments == 128 && p.N % rows_per_block == 0;

  auto fetch_w = [&](int tile, int it, int stage) {
    float* st = ring + stage * (W_FLOATS + X_FLOATS) + row0 * F32_PITCH + ck;
    if (whole) {                                 // every copy is there
      const float* from = w + (size_t)tile * rows_per_block * p.K + it * F32_BK + ck;
      const unsigned to = (unsigned)__cvta_generic_to_shared(st);
#pragma unroll
      for (int r = 0; r < 8; r++)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + r * 16 * F32_PITCH), "l"(from + place[r]) : "memory");
      return;
    }
#pragma unroll
    for (int r = 0; r < 8; r++) {
      const int id = warp * 32 + r * 4 + row0;
      const int n = tile * rows_per_block + id % rows_per_block, s = id / rows_per_block;
      copy4<VEC>(st + r * 4 * F32_PITCH, w + (size_t)(n < p.N ? n : 0) * p.K, s * p.segment + it * F32_BK + ck, p.K,
                 n < p.N && s < p.segments);
    }
  };
  auto fetch_x = [&](int it, int stage) {
    float* st = ring + stage * (W_FLOATS + X_FLOATS) + W_FLOATS;
    for (int c = lane; c < warp_segments * MR * 8; c += 32) {
      const int row = c >> 3, m = row % MR, s = first_segment + row / MR;
      const int k = s * p.segment + it * F32_BK + (c & 7) * 4;
      const float* from = x + (size_t)(m < p.M ? m : 0) * p.ldx;
      float* to = st + row * F32_PITCH + (c & 7) * 4;
      if (VEC) {
        copy4<true>(to, from, k, p.K, m < p.M && s < p.segments);
      } else {                                   // not by 4-byte copies: they go through L1, where a line of x may be an
#pragma unroll                                   // earlier kernel's
        for (int i = 0; i < 4; i++) to[i] = m < p.M && s < p.segments && k + i < p.K ? ld_fresh(from + k + i) : 0.f;
      }
    }
  };
  pdl_trigger();
  // the next stage to ask for: tile, stage of it, place in the ring
  int f_tile = blockIdx.x, f_it = 0, f_stage = 0;
  auto next = [&]() {
    if (++f_it == iters) { f_it = 0; f_tile += gridDim.x; }
    f_stage = f_stage + 1 == STAGES ? 0 : f_stage + 1;
  };
  for (int j = 0; j < STAGES - 1 && j < total; j++, next()) fetch_w(f_tile, f_it, f_stage);
  pdl_wait();                                    // x, and what is added into, are the work of kernels before this one
  for (int j = 0, it = 0; j < STAGES - 1; j++, it = it + 1 == iters ? 0 : it + 1) {
    if (j < total) fetch_x(it, j);
    copies_commit();
  }
  f32x2 acc[MR];
#pragma unroll
  for (int m = 0; m < MR; m++) acc[m] = 0;
  const int x_off = W_FLOATS + (tid / rows_per_block - first_segment) * MR * F32_PITCH;
  int tile = blockIdx.x, it = 0, stage = 0;
  for (int j = 0; j < total; j++) {
    copies_wait<STAGES - 2>();
    __syncwarp();
    if (j + STAGES - 1 < total) {
      fetch_w(f_tile, f_it, f_stage);
      fetch_x(f_it, f_stage);
      next();
    }
    copies_commit();
    const float* st = ring + stage * (W_FLOATS + X_FLOATS);
#pragma unroll
    for (int c = 0; c < F32_BK / 4; c++) {
      const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(st + lane * F32_PITCH + c * 4);
#pragma unroll
      for (int m = 0; m < MR; m++) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(st + x_off + m * F32_PITCH + c * 4);
        fma2(acc[m], a.x, b.x);
        fma2(acc[m], a.y, b.y);
      }
    }
    stage = stage + 1 == STAGES ? 0 : stage + 1;
    if (++it < iters) continue;
    __syncthreads();                             // the tile before this one has been added up
#pragma unroll
    for (int m = 0; m < MR; m++) { sums[m * 128 + tid] = even_plus_odd(acc[m]); acc[m] = 0; }
    __syncthreads();
    for (int i = tid; i < MR * rows_per_block; i += 128) {
      const int m = i / rows_per_block, r = i % rows_per_block, n = tile * rows_per_block + r;
      if (m >= p.M || n >= p.N) continue;
      float v = sums[m * 128 + r];
      for (int s = 1; s < p.segments; s++) v = __fadd_rn(v, sums[m * 128 + s * rows_per_block + r]);
      f32_finish(p, head, m, n, v);
    }
    it = 0;
    tile += gridDim.x;
  }
}

// More rows: bound by the FMA units.  BM x 128 outputs a block of 128 threads, TM x 8 a thread as rows tm + i * (BM / TM)
// and columns tn + j * 16 (16-byte shared loads of neighbouring rows; no transposition, since a packed FMA takes two
// neighbouring k of either operand), two stages of 32 k by cp.async.  With 64 rows a thread holds 128 registers of the
// segment's sums, so an SM has two blocks of four warps; the sums over the segments, touched once in 256 k, lie in shared
// memory.  A packed FMA's operands come at one byte of shared memory a FMA, as much as an SM delivers: 44 TFLOP/s of 74.
// (Sums over the segments in registers, spilt, and three stages: 2 % slower; lanes of a warp as 4 x 8 in plain order: 2 %.)
// gridDim.y > 1: the segments are cut over gridDim.y blocks, every segment's sum goes to `parts` and
// linear_f32_parts_kernel adds them.
template <int BM, int TM, bool VEC>
__global__ void __launch_bounds__(128, 2)
linear_f32_tile_kernel(const F32Product p, const int m_tiles) {
  constexpr int BN = 128, TN = 8, STAGES = F32_TILE_STAGES, STAGE_FLOATS = (BM + BN) * F32_PITCH, MT = BM / TM, NT = BN / TN;
  static_assert(MT * NT == 128, "one thread per TM x TN outputs");
  extern __shared__ __align__(16) float smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, head = blockIdx.z;
  const int m0 = (blockIdx.x % m_tiles) * BM, n0 = (blockIdx.x / m_tiles) * BN;
  // a warp: 4 x 8 threads
  const int tm = (warp % (MT / 4)) * 4 + ((lane >> 4) << 1 | (lane & 1)), tn = (warp / (MT / 4)) * 8 + ((lane >> 1) & 7);
  const float* x = p.x + (size_t)head * p.x_step;
  const float* w = p.w + (size_t)head * p.w_step;
  const int per = (p.segments + gridDim.y - 1) / gridDim.y;
  const int s0 = blockIdx.y * per, s1 = min(p.segments, s0 + per);
  const int per_segment = p.segment / F32_BK;
  const int k_first = s0 * p.segment, k_end = min(p.K, s1 * p.segment);
  const int iters = (k_end - k_first + F32_BK - 1) / F32_BK;

  auto fetch = [&](int it) {
    float* st = smem + (it % STAGES) * STAGE_FLOATS;
    const int k = k_first + it * F32_BK + (tid & 7) * 4;
#pragma unroll
    for (int r = 0; r < (BM + BN) / 16; r++) {
      const int row = r * 16 + (tid >> 3);
      if (row < BM) {
        const int m = m0 + row;
        copy4<VEC>(st + row * F32_PITCH + (tid & 7) * 4, x + (size_t)(m < p.M ? m : 0) * p.ldx, k, p.K, m < p.M);
      } else {
        const int n = n0 + row - BM;
        copy4<VEC>(st + row * F32_PITCH + (tid & 7) * 4, w + (size_t)(n < p.N ? n : 0) * p.K, k, p.K, n < p.N);
      }
    }
  };

  f32x2 acc[TM][TN];
  float* total = smem + STAGES * STAGE_FLOATS + tid;      // sums over the segments: [TM * TN][128]
#pragma unroll
  for (int i = 0; i < TM; i++)
#pragma unroll
    for (int j = 0; j < TN; j++) acc[i][j] = 0;
#pragma unroll
  for (int it = 0; it < STAGES - 1; it++) {
    if (it < iters) fetch(it);
    copies_commit();
  }
  int s = s0, left = per_segment;                // stages left of segment s
  for (int it = 0; it < iters; it++) {
    copies_wait<STAGES - 2>();
    __syncthreads();
    if (it + STAGES - 1 < iters) fetch(it + STAGES - 1);
    copies_commit();
    const float* xs = smem + (it % STAGES) * STAGE_FLOATS + tm * F32_PITCH;
    const float* ws = smem + (it % STAGES) * STAGE_FLOATS + (BM + tn) * F32_PITCH;
#pragma unroll
    for (int c = 0; c < F32_BK / 4; c++) {
      ulonglong2 a[TM];
#pragma unroll
      for (int i = 0; i < TM; i++) a[i] = *reinterpret_cast<const ulonglong2*>(xs + i * MT * F32_PITCH + c * 4);
#pragma unroll
      for (int j = 0; j < TN; j++) {
        const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(ws + j * NT * F32_PITCH + c * 4);
#pragma unroll
        for (int i = 0; i < TM; i++) fma2(acc[i][j], a[i].x, b.x);
#pragma unroll
        for (int i = 0; i < TM; i++) fma2(acc[i][j], a[i].y, b.y);
      }
    }
    if (--left == 0 || it + 1 == iters) {        // the segment is complete
      if (gridDim.y > 1) {
        float* to = p.parts + ((size_t)head * p.segments + s) * p.M * p.N;
#pragma unroll
        for (int i = 0; i < TM; i++)
#pragma unroll
          for (int j = 0; j < TN; j++) {
            const int m = m0 + tm + i * MT, n = n0 + tn + j * NT;
            if (m < p.M && n < p.N) to[(size_t)m * p.N + n] = even_plus_odd(acc[i][j]);
            acc[i][j] = 0;
          }
      } else {
#pragma unroll
        for (int i = 0; i < TM; i++)
#pragma unroll
          for (int j = 0; j < TN; j++) {
            const float v = even_plus_odd(acc[i][j]);
            float& t = total[(i * TN + j) * 128];
            t = s == 0 ? v : __fadd_rn(t, v);
            acc[i][j] = 0;
          }
      }
      s++;
      left = per_segment;
    }
  }
  if (gridDim.y > 1) return;
#pragma unroll
  for (int i = 0; i < TM; i++)
#pragma unroll
    for (int j = 0; j < TN; j++) {
      const int m = m0 + tm + i * MT, n = n0 + tn + j * NT;
      if (m < p.M && n < p.N) f32_finish(p, head, m, n, total[(i * TN + j) * 128]);
    }
}

__global__ void __launch_bounds__(256) linear_f32_parts_kernel(const F32Product p) {
  const size_t size = (size_t)p.M * p.N, i = (size_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= size) return;
  const float* from = p.parts + (size_t)blockIdx.z * p.segments * size + i;
  float part[F32_MAX_SEGMENTS];
#pragma unroll
  for (int s = 0; s < F32_MAX_SEGMENTS; s++)
    if (s < p.segments) part[s] = from[(size_t)s * size];
  float v = part[0];
#pragma unroll
  for (int s = 1; s < F32_MAX_SEGMENTS; s++)
    if (s < p.segments) v = __fadd_rn(v, part[s]);
  f32_finish(p, blockIdx.z, (int)(i / p.N), (int)(i % p.N), v);
}

// How many blocks the segments of a tile are cut over: what makes the busiest SM's share smallest, counting two blocks
// to an SM of 148, plus what writing and reading the segments' sums costs.  In units of one segment of a 64 x 128 tile
// (k a segment: 64 * 128 * k FMA at half an SM's rate); the sums pass L2 at a few TB/s, an SM's share of which is about
// 6 floats a cycle both ways, against 64 FMA a cycle and block.
static int f32_cuts(int tiles, int segments, int segment, long long outputs, long long scratch_floats) {
  int best = 1;
  double best_cost = 0;
  for (int cuts = 1; cuts <= segments; cuts *= 2) {
    const int per = (segments + cuts - 1) / cuts, used = (segments + per - 1) / per;
    const long long blocks = (long long)tiles * used;
    double cost = (double)((blocks + 295) / 296) * per;
    if (used > 1) {
      if (outputs * segments > scratch_floats) break;
      cost += (outputs * segments / 148.0 / 6.0 + 4000.0) / (64.0 * 128.0 * segment / 64.0);
    }
    if (cuts == 1 || cost < best_cost) { best = used; best_cost = cost; }
  }
  return best;
}

#define F32_SCRATCH_FLOATS (16LL << 20)

static int f32_tile_rows(int M) { return M <= 32 ? 32 : 64; }
static int f32_tile_cuts(int M, int N, int K, int heads) {
  const int segment = f32_segment(K), segments = (K + segment - 1) / segment, bm = f32_tile_rows(M);
  const long long tiles = (long long)((M + bm - 1) / bm) * ((N + 127) / 128) * heads;
  return tiles > (1 << 20) ? 1 : f32_cuts((int)tiles, segments, segment, (long long)M * N * heads, F32_SCRATCH_FLOATS);
}

template <int MR, bool VEC, int STAGES>
static int launch_f32_few_stages(const F32Product& p, int heads, int rows_per_block, int tiles, cudaStream_t stream) {
  const int smem = (MR * 128 + 4 * STAGES * (32 + 2 * MR) * F32_PITCH) * 4;
  const cudaError_t e = cudaFuncSetAttribute(linear_f32_few_kernel<MR, VEC, STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  const int places = 148 * (STAGES == 4 ? 2 : 1);
  return launch_pdl(linear_f32_few_kernel<MR, VEC, STAGES>, dim3(tiles < places ? tiles : places, 1, heads), 128, smem, stream, p,
                    rows_per_block);
}

template <int MR, bool VEC>
static int launch_f32_few(const F32Product& p, int heads, cudaStream_t stream) {
  int lanes = 1;
  while (lanes < p.segments) lanes *= 2;
  const int rows_per_block = 128 / lanes, tiles = (p.N + rows_per_block - 1) / rows_per_block;
  return (long long)tiles * heads <= 148 ? launch_f32_few_stages<MR, VEC, 8>(p, heads, rows_per_block, tiles, stream)
                                         : launch_f32_few_stages<MR, VEC, 4>(p, heads, rows_per_block, tiles, stream);
}

template <int BM, int TM, bool VEC>
static int launch_f32_tile(const F32Product& p, int heads, int cuts, cudaStream_t stream) {
  const int smem = (F32_TILE_STAGES * (BM + 128) * F32_PITCH + BM * 128) * 4;
  const cudaError_t e = cudaFuncSetAttribute(linear_f32_tile_kernel<BM, TM, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  const int m_tiles = (p.M + BM - 1) / BM;
  const long long blocks = (long long)m_tiles * ((p.N + 127) / 128);
  if (blocks > 0x7fffffffLL) return STRATUM_ERR_LIMIT;
  linear_f32_tile_kernel<BM, TM, VEC><<<dim3((unsigned)blocks, cuts, heads), 128, smem, stream>>>(p, m_tiles);
  if (cuts > 1)
    linear_f32_parts_kernel<<<dim3((unsigned)(((long long)p.M * p.N + 255) / 256), 1, heads), 256, 0, stream>>>(p);
  return launch_status();
}

template <bool VEC>
static int launch_f32(F32Product p, int heads, cudaStream_t stream) {
  p.segment = f32_segment(p.K);
  p.segments = (p.K + p.segment - 1) / p.segment;
  if (p.M <= F32_FEW_ROWS) {
    if (p.M == 1) return launch_f32_few<1, VEC>(p, heads, stream);
    if (p.M == 2) return launch_f32_few<2, VEC>(p, heads, stream);
    if (p.M == 3) return launch_f32_few<3, VEC>(p, heads, stream);
    if (p.M == 4) return launch_f32_few<4, VEC>(p, heads, stream);
    if (p.M <= 6) return launch_f32_few<6, VEC>(p, heads, stream);
    return launch_f32_few<8, VEC>(p, heads, stream);
  }
  const int cuts = p.parts ? f32_tile_cuts(p.M, p.N, p.K, heads) : 1;
  return f32_tile_rows(p.M) == 32 ? launch_f32_tile<32, 4, VEC>(p, heads, cuts, stream)
                                  : launch_f32_tile<64, 8, VEC>(p, heads, cuts, stream);
}

static int launch_linear_f32(const void* x, const void* w, const float* bias, void* out, int epilogue, int M, int N,
                             int K, int ldx, int ldo, float* scratch, cudaStream_t stream, int heads = 1, int x_step = 0,
                             long long w_step = 0, int o_step = 0, int act = 0) {
  if (epilogue < 0 || epilogue > 2) return STRATUM_ERR_SHAPE;
  const F32Product p = {(const float*)x, (const float*)w, bias, (float*)out, scratch, M, N, K, ldx, ldo, x_step, o_step,
                        act, epilogue, 0, 0, w_step};
  const bool vec = K % 4 == 0 && ldx % 4 == 0 && x_step % 4 == 0 && ((uintptr_t)x | (uintptr_t)w) % 16 == 0;
  return vec ? launch_f32<true>(p, heads, stream) : launch_f32<false>(p, heads, stream);
}

// float32 numbers of scratch with which a float32 product cuts its tiles' segments over more blocks (0: it does not)
STRATUM_EXPORT long long stratum_linear_simple_scratch(int heads, int M, int N, int K) {
  if (M <= F32_FEW_ROWS || N <= 0 || K <= 0 || heads <= 0 || f32_tile_cuts(M, N, K, heads) == 1) return 0;
  const int segment = f32_segment(K);
  return (long long)heads * ((K + segment - 1) / segment) * M * N;
}

// x: [M][ldx] T (first K columns used); w: [N][K] T; bias: float32 [N] or null; out: [M][ldo].
// act (epilogue 0 only): an activation applied to what is stored, see common.cuh.
// scratch: as many float32 numbers as stratum_linear_simple_scratch says, or null (then no tile is cut).
STRATUM_EXPORT int stratum_linear_simple(const void* x, const void* w, const float* bias, void* out, int dtype,
                                         int epilogue, int M, int N, int K, int ldx, int ldo, int act,
                                         float* scratch, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || ldx < K || ldo < N) return STRATUM_ERR_SHAPE;
  if (act != 0 && epilogue != 0) return STRATUM_ERR_SHAPE;
  if ((M + LS_BM - 1) / LS_BM > 65535) return STRATUM_ERR_LIMIT;
  if (dtype == STRATUM_DT_F32)
    return launch_linear_f32(x, w, bias, out, epilogue, M, N, K, ldx, ldo, scratch, stream, 1, 0, 0, 0, act);
  if (dtype == STRATUM_DT_BF16)
    return launch_linear_simple(x, w, bias, out, epilogue, M, N, K, ldx, ldo, stream, 1, 0, 0, 0, act);
  return STRATUM_ERR_DTYPE;
}

// The same product once per head: head j multiplies columns [j * x_step, j * x_step + K) of x by the matrix
// w[j] ([heads][N][K]) into columns [j * o_step, j * o_step + N) of out.  No bias.
STRATUM_EXPORT int stratum_linear_heads(const void* x, const void* w, void* out, int dtype, int epilogue, int heads,
                                        int M, int N, int K, int ldx, int ldo, int x_step, int o_step,
                                        float* scratch, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || heads <= 0) return 0;
  if (K <= 0 || x_step < 0 || o_step < 0 || (long long)(heads - 1) * x_step + K > ldx ||
      (long long)(heads - 1) * o_step + N > ldo)
    return STRATUM_ERR_SHAPE;
  if ((M + LS_BM - 1) / LS_BM > 65535 || heads > 65535) return STRATUM_ERR_LIMIT;
  const long long w_step = (long long)N * K;
  if (dtype == STRATUM_DT_F32)
    return launch_linear_f32(x, w, nullptr, out, epilogue, M, N, K, ldx, ldo, scratch, stream, heads, x_step, w_step,
                             o_step);
  if (dtype == STRATUM_DT_BF16)
    return launch_linear_simple(x, w, nullptr, out, epilogue, M, N, K, ldx, ldo, stream, heads, x_step, w_step,
                                      o_step);
  return STRATUM_ERR_DTYPE;
}
