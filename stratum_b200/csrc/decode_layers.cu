// A decode step's layers, and the output head, as one resident kernel: every layer of a dense decoder (RMSNorm, grouped-query
// attention with neighbouring rotated pairs over the paged cache, RMSNorm, SwiGLU) for up to 16 rows of one new token each.
//
//   x += Wo attend(rope(Wqkv n_a(x)));  x += Wd (silu(Wg n_b(x)) * (Wu n_b(x)));  logits = Wh n_f(x)
// (stratum/native/stratum_arch_llama.inc.c:392-555; a step of one token per sequence: :1070-1218).
//
// What bounds it.  A step of so few rows reads every weight once, so the HBM rate is its floor; launched as ten kernels a
// layer it stood at 0.41 (1 row, Llama-3.2-1B shape) to 0.75 (8 rows, 8B shape) of it, because between two kernels the
// memory system runs empty.  Here one block per SM stays for the whole step.  A layer is five phases with a grid-wide
// meeting between them (the launch is cooperative, so all blocks are resident; every wait is bounded), and what a block
// streams, weights and cached keys and values alike, comes through one ring that a warp of its own fills with bulk copies in
// the order of use, whatever phase the other warps are in: while they wait for a meeting, the ring (165 KB an SM, 24 MB in
// all, 4 us of the HBM rate) fills with what the phases after will need.  Measured for the layers and the head (graph
// replays): 1B shape, 1 row behind 201 keys 616 us (one kernel after the other: 905), 8B shape, 8 rows behind 3,700 keys
// 104 us a layer (116).
//
// Split.  A block takes an equal share of the rows of every matrix, to a pair of rows, with all of k, so nothing has to be
// added across blocks; its eight warps cut every 1,024 values of k, and their partial sums meet in shared memory in the order
// of the warps.  A product's order of sums follows from k alone: its rows give the same bits in any batch.  Weights are the A
// operand of mma.sync.m16n8k16 (16 rows a tile), rows of x the B operand, straight from L2 into registers, k visited in an order of its
// own that both share (a lane takes the 8 contiguous values 8t..8t+7 of 32, see gemm_skinny.cu).  tcgen05 would add its trips
// through tensor memory to every phase, and mma.sync has three times the rate at which the weights arrive.
//
// Norms.  Whoever writes new rows r of the stream also writes bf16(r * gain) and, per block, the sum of r^2 over its columns;
// the product behind the norm multiplies its sums by 1 / sqrt(sum / size + eps).  The stream itself stays in the registers of
// the threads that add to it, in float32.
//
// Attention.  The pages of all (sequence, kv head) pairs form one list, cut evenly over the blocks.  Pairs of few pages are not
// cut, so a row of up to 512 visible keys gives the same bits in any batch of the kernel's; where a longer one is cut follows
// from the batch.  Four warps take 16 keys of a page each, two pages at a time; scores and values as in attention_mma.cu (keys
// along M).
// A pair seen by several blocks is merged by whichever of them comes last, in the order of its keys.  The new token's key and
// value, which another block may have written a phase ago, do not come through the ring: one warp takes them from L2.
#include "common.cuh"
#include "mma_common.cuh"
#include "tc_common.cuh"

#define STRATUM_ERR_RESIDENT (-6)     // the blocks cannot all be resident: nothing was launched

#define DL_WARPS 8                    // that compute; one more fills the ring (of a group of four: registers are dealt by fours)
#define DL_COMPUTE (DL_WARPS * 32)
#define DL_THREADS (DL_COMPUTE + 128)
#define DL_STAGES 5
#define DL_CHUNK 1024                 // values of k a step: 128 a warp
#define DL_PITCH (DL_CHUNK * 2 + 64)  // bytes from one weight row of a stage to the next: rows g, g+1 on different banks
#define DL_STAGE (16 * DL_PITCH)
#define DL_MAX_LAYERS 96
#define DL_MAX_ROWS 16
#define DL_MAX_BLOCKS 160
#define DL_PAGE 64
#define DL_MAX_PAGES 1024             // pages a block attends to
#define DL_WHOLE 8                    // up to this many pages a pair is not cut
#define DL_STRIDE 20                  // floats from one row of x to the next among the partial sums: no bank conflicts
#define DL_SPIN_LIMIT (1u << 21)      // polls of half a microsecond: a second.  (As a launch parameter: 0.6 % of a step of 8 rows)

struct DlLayer {
  const bf16 *w_qkv, *w_o, *w_gu, *w_down;
  const float *gain_ff, *gain_next;   // the norm in front of the feed-forward; the one behind it (next layer's, or the last)
  bf16 *k, *v;                        // [pages][n_kv][64][D]
};

struct DlParams {
  const float* x;                     // [M][H] embedded tokens
  const float* gain_first;
  const bf16* w_head; float* logits;  // [vocab][H]; [M][vocab]  (vocab 0: a step that wants no logits)
  bf16 *xb, *qb, *ob, *ab;            // [M][H], [M][n_q D], [M][n_q D], [M][F]
  float *ss;                          // [2][blocks][16]
  float *part_o, *part_ml;            // [2 blocks][8][D], [2 blocks][8][2]
  unsigned *counters;                 // [1 + M n_kv], zero before the launch
  const float2* rope;                 // [M][n_pairs]
  const int *pos, *seq, *block_table;
  int* status;
  int bt_stride, n_layers, M, H, F, n_q, n_kv, D, n_pairs, window, vocab;
  unsigned absent;                    // arrivals a meeting waits for beyond the blocks that are there: 0, but where a test lets one run out
  float eps, scale;
  DlLayer layer[DL_MAX_LAYERS];
};

enum { PH_QKV = 0, PH_O, PH_GU, PH_DOWN, PH_HEAD, PH_COUNT };

struct DlShare {                      // a block's share of a matrix
  int row0, rows, tiles, K, chunks;
};

struct DlSmem {
  uint8_t ring[DL_STAGES][DL_STAGE];            // 16 weight rows x 1,024 k; or pages: their keys, then their values
  float part[2][DL_WARPS * 32 * DL_STRIDE];     // [warp][tile][row of x][weight row]; also the attention's meeting place
  float ml[DL_WARPS][8][2];
  float ssw[DL_WARPS][4];
  float inv[DL_MAX_ROWS];
  uint64_t full[DL_STAGES], empty[DL_STAGES];
  int pre[DL_MAX_ROWS + 1];           // pages in front of each sequence (of one kv head)
  int first[DL_MAX_ROWS];             // a sequence's first page
  int live[DL_MAX_ROWS];
  int page0, pages;                   // this block's share of the list
  int place[DL_MAX_PAGES];            // where a page of the share lies in the cache, in pages of one kv head
  DlShare share[PH_COUNT];
  int abort_flag, last;
};

__device__ __forceinline__ void dl_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }      // the warps that compute

__device__ __forceinline__ void dl_bulk(uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

// ------------------------------------------------------------------------------------------ the list of pages
__device__ __forceinline__ int dl_page_share(const DlParams& P, const DlSmem& S) {
  return max(1, (S.pre[P.M] * P.n_kv + (int)gridDim.x - 1) / (int)gridDim.x);
}
// Where block c's share begins: an even cut, moved to the nearer end of a pair of few pages that it would fall into.
__device__ __forceinline__ int dl_cut(const DlParams& P, const DlSmem& S, int c) {
  const int all = S.pre[P.M] * P.n_kv;
  const long long even = (long long)c * dl_page_share(P, S);
  if (even >= all) return all;
  const int at = (int)even;
  int b = 0;
  while (S.pre[b + 1] * P.n_kv <= at) b++;
  const int n = S.pre[b + 1] - S.pre[b], r = (at - S.pre[b] * P.n_kv) % n;
  return n > DL_WHOLE ? at : 2 * r < n ? at - r : at - r + n;
}

// ------------------------------------------------------------------------------------------ the warp that fills the ring
template <int CH>
struct DlFeeder {
  const DlParams& P;
  DlSmem& S;
  const int lane;
  uint32_t stage, phase;              // the parity a free stage shows

  __device__ __forceinline__ bool free_stage() {
    const bool ok = __all_sync(0xffffffffu, mbar_wait(&S.empty[stage], phase, &S.abort_flag));
    if (!ok && lane == 0) { if (!*(volatile int*)&S.abort_flag) atomicCAS(P.status, 0, 431); S.abort_flag = 1; }
    return ok;
  }
  __device__ __forceinline__ void next() {
    if (++stage == DL_STAGES) { stage = 0; phase ^= 1; }
  }
  __device__ __forceinline__ bool tile(const DlShare& s, const bf16* w, int t, int c) {
    if (!free_stage()) return false;
    const int n = min(16, s.rows - 16 * t);
    const uint32_t bytes = 2 * min(DL_CHUNK, s.K - c * DL_CHUNK);
    if (lane == 0) mbar_expect_tx(&S.full[stage], n * bytes);
    __syncwarp();
    if (lane < n)
      dl_bulk(smem_u32(S.ring[stage]) + lane * DL_PITCH, w + (size_t)(s.row0 + 16 * t + lane) * s.K + c * DL_CHUNK, bytes, &S.full[stage]);
    next();
    return true;
  }
  __device__ __forceinline__ bool matrix(int ph, const bf16* w) {
    const DlShare s = S.share[ph];
    if (ph == PH_DOWN) {              // (its rows of x come chunk by chunk: all tiles of one, then the next)
      for (int c = 0; c < s.chunks; c++)
        for (int t = 0; t < s.tiles; t++)
          if (!tile(s, w, t, c)) return false;
    } else {
      for (int t = 0; t < s.tiles; t++)
        for (int c = 0; c < s.chunks; c++)
          if (!tile(s, w, t, c)) return false;
    }
    return true;
  }
  __device__ __forceinline__ bool pages(const DlLayer& L) {
    constexpr int PER = CH == 4 ? 1 : 2, BYTES = DL_PAGE * 32 * CH * 2;      // pages a stage; bytes of a page's keys
    for (int i = 0; i < S.pages; i += PER) {
      if (!free_stage()) return false;
      const int n = min(PER, S.pages - i);
      if (lane == 0) mbar_expect_tx(&S.full[stage], 2 * n * BYTES);
      __syncwarp();
      if (lane < 2 * n) {             // keys by even lanes, values by odd ones
        const size_t at = (size_t)S.place[i + (lane >> 1)] * (DL_PAGE * 32 * CH);
        dl_bulk(smem_u32(S.ring[stage]) + lane * BYTES, ((lane & 1) ? L.v : L.k) + at, BYTES, &S.full[stage]);
      }
      next();
    }
    return true;
  }
  __device__ __forceinline__ void run() {
    bool ok = true;
    for (int l = 0; l < P.n_layers && ok; l++) {
      const DlLayer& L = P.layer[l];
      ok = matrix(PH_QKV, L.w_qkv) && pages(L) && matrix(PH_O, L.w_o) && matrix(PH_GU, L.w_gu) && matrix(PH_DOWN, L.w_down);
    }
    if (ok) ok = matrix(PH_HEAD, P.w_head);
    // the block stays until everything that was asked for has landed: until all of it has been taken, or, where the warps that
    // compute gave up (the last copies may then be on their way still), for a while
    for (int s = 0; s < DL_STAGES && ok; s++) {
      ok = free_stage();
      next();
    }
    if (!ok)
      for (int i = 0; i < 2000; i++) __nanosleep(1000);
  }
};

// ------------------------------------------------------------------------------------------ grid-wide meetings
__device__ __forceinline__ void dl_arrive(const DlParams& P) {
  dl_sync();
  if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(P.counters) : "memory");
}
// False: a wait ran out, here or somewhere in the block before; every thread that computes gets the same answer.
__device__ __forceinline__ bool dl_meet(const DlParams& P, DlSmem& S, unsigned target, int code) {
  if (threadIdx.x == 0) {
    bool ok = false;
    for (unsigned i = 0; i < DL_SPIN_LIMIT; i++) {
      unsigned v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(P.counters) : "memory");
      if ((int)(v - target) >= 0) { ok = true; break; }
      if ((i & 1023u) == 1023u && *(volatile int*)&S.abort_flag) break;
    }
    if (!ok) { atomicCAS(P.status, 0, code); S.abort_flag = 1; }
    S.last = *(volatile int*)&S.abort_flag;      // (one reading for all: another warp may raise the flag meanwhile)
  }
  dl_sync();
  return S.last == 0;
}

// ------------------------------------------------------------------------------------------ products
template <int MT>
struct DlProduct {
  const DlParams& P;
  DlSmem& S;
  const int warp, lane;
  uint32_t stage, phase;
  int buf;                            // which half of the partial sums comes next

  // The ring's next stage, once it is filled.  (A wait that runs out leaves the flag for the next meeting; until then the
  // warp goes on with what it has.)
  __device__ __forceinline__ uint32_t ready() {
    if (!__all_sync(0xffffffffu, mbar_wait(&S.full[stage], phase, &S.abort_flag)) && lane == 0) {
      atomicCAS(P.status, 0, 432);
      S.abort_flag = 1;
    }
    return smem_u32(S.ring[stage]);
  }
  __device__ __forceinline__ void done() {
    __syncwarp();
    if (lane == 0) mbar_arrive(&S.empty[stage]);
    if (++stage == DL_STAGES) { stage = 0; phase ^= 1; }
  }
  // rows g and g+8 of N blocks of 32 values from `at` (this lane's first piece), as an A operand takes them
  template <int N>
  __device__ __forceinline__ void fragments(uint32_t at, uint32_t pitch, uint4 (&a0)[N], uint4 (&a1)[N]) {
#pragma unroll
    for (int u = 0; u < N; u++) {
      const uint32_t p = at + u * 64, q = p + 8 * pitch;
      asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(a0[u].x), "=r"(a0[u].y), "=r"(a0[u].z), "=r"(a0[u].w) : "r"(p) : "memory");
      asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(a1[u].x), "=r"(a1[u].y), "=r"(a1[u].z), "=r"(a1[u].w) : "r"(q) : "memory");
    }
  }
  // one step's products: 16 weight rows x this warp's 128 k of chunk c with the rows of x in b
  __device__ __forceinline__ void step(int K, int c, const uint4* b /* [4][MT] */, float (&acc)[MT][2][4]) {
    const uint32_t at = ready();
    if (c * DL_CHUNK + warp * 128 < K) {
      uint4 a0[4], a1[4];
      fragments<4>(at + (lane >> 2) * DL_PITCH + warp * 256 + (lane & 3) * 16, DL_PITCH, a0, a1);
#pragma unroll
      for (int u = 0; u < 4; u++) {
#pragma unroll
        for (int i = 0; i < MT; i++) {
          const uint4& x = b[u * MT + i];
          mma16816(acc[i][0], a0[u].x, a1[u].x, a0[u].y, a1[u].y, x.x, x.y);
          mma16816(acc[i][1], a0[u].z, a1[u].z, a0[u].w, a1[u].w, x.z, x.w);
        }
      }
    }
    done();
  }
  __device__ __forceinline__ void zero(float (&acc)[MT][2][4]) {
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
      for (int j = 0; j < 2; j++) acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.f;
  }
  // accumulator: [0],[1] -> (weight row g, rows of x 2t, 2t+1); [2],[3] -> weight row g+8
  __device__ __forceinline__ void leave(int tl, const float (&acc)[MT][2][4]) {
    const int g = lane >> 2, t = lane & 3;
    float* p = S.part[buf] + (warp * (4 / MT) + tl) * (8 * MT) * DL_STRIDE;
#pragma unroll
    for (int i = 0; i < MT; i++) {
      float* q = p + (8 * i + 2 * t) * DL_STRIDE + g;
      q[0] = acc[i][0][0] + acc[i][1][0];
      q[DL_STRIDE] = acc[i][0][1] + acc[i][1][1];
      q[8] = acc[i][0][2] + acc[i][1][2];
      q[DL_STRIDE + 8] = acc[i][0][3] + acc[i][1][3];
    }
  }
  // the sum over the warps, in their order, of the pair of weight rows 2p, 2p+1 of tile tl for row m of x
  __device__ __forceinline__ float2 gather(int tl, int m, int p) {
    float2 v = make_float2(0.f, 0.f);
#pragma unroll
    for (int w = 0; w < DL_WARPS; w++) {
      const float2 a = *reinterpret_cast<const float2*>(S.part[buf] + ((w * (4 / MT) + tl) * (8 * MT) + m) * DL_STRIDE + 2 * p);
      v.x += a.x;
      v.y += a.y;
    }
    return v;
  }
  // rows of x (operand B): this warp's 128 k of chunk c
  __device__ __forceinline__ void rows_of(const bf16* x, int K, int c, bool live_only, uint4* b /* [4][MT] */) {
    const int g = lane >> 2, t = lane & 3;
    const int k = c * DL_CHUNK + warp * 128;
#pragma unroll
    for (int i = 0; i < MT; i++) {
      const int m = 8 * i + g;
      const bool on = k < K && m < P.M && (!live_only || S.live[m]);
      const bf16* p = x + (size_t)(on ? m : 0) * K + (on ? k : 0) + t * 8;
#pragma unroll
      for (int u = 0; u < 4; u++)
        b[u * MT + i] = on ? ld_fresh(reinterpret_cast<const uint4*>(p + u * 32)) : make_uint4(0, 0, 0, 0);
    }
  }
  // 1 / rms of every row from the blocks' sums of squares: asked for with the rows of x, added up when the first products
  // are done (in front of them it cost 2 us a phase); known to all after the next meeting of the block's warps
  __device__ __forceinline__ void ask_factors(const float* ss, float (&f)[MT][DL_MAX_BLOCKS / 32]) {
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
      for (int c = 0; c < DL_MAX_BLOCKS / 32; c++)
        f[i][c] = lane + 32 * c < (int)gridDim.x ? ld_fresh(ss + (lane + 32 * c) * DL_MAX_ROWS + warp + 8 * i) : 0.f;
  }
  __device__ __forceinline__ void leave_factors(const float (&f)[MT][DL_MAX_BLOCKS / 32]) {
#pragma unroll
    for (int i = 0; i < MT; i++) {
      float v = 0.f;
#pragma unroll
      for (int c = 0; c < DL_MAX_BLOCKS / 32; c++) v += f[i][c];
      v = warp_sum(v);
      if (lane == 0) S.inv[warp + 8 * i] = 1.0f / sqrtf(v / (float)P.H + P.eps);
    }
  }
};

// Rows of the stream (their new values r0, r1 at columns n, n+1), rounded times the next norm's gain, and this block's sum of
// their squares, into `ss`.  Threads that hold nothing come with on = false.
template <int MT>
__device__ __forceinline__ void dl_hand_on(const DlParams& P, DlSmem& S, bool on, int m, int n, float r0, float r1, float2 gain, float* ss) {
  if (on) *reinterpret_cast<__nv_bfloat162*>(P.xb + (size_t)m * P.H + n) = __floats2bfloat162_rn(r0 * gain.x, r1 * gain.y);
  float q = on ? r0 * r0 + r1 * r1 : 0.f;
  q += __shfl_xor_sync(0xffffffffu, q, 1);
  q += __shfl_xor_sync(0xffffffffu, q, 2);
  q += __shfl_xor_sync(0xffffffffu, q, 4);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if ((lane & 7) == 0) S.ssw[warp][lane >> 3] = q;      // row of x 4 (warp % (2 MT)) + lane / 8
  dl_sync();
  if (threadIdx.x < 8 * MT) {
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < DL_WARPS; w += 2 * MT) v += S.ssw[w + (threadIdx.x >> 2)][threadIdx.x & 3];
    ss[blockIdx.x * DL_MAX_ROWS + threadIdx.x] = v;
  }
}

// ------------------------------------------------------------------------------------------ attention
template <int MT, int CH>
__device__ __forceinline__ void dl_attention(const DlParams& P, DlSmem& S, const DlLayer& L, DlProduct<MT>& W) {
  constexpr int HD = 32 * CH, PITCH = HD * 2, BYTES = DL_PAGE * PITCH;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int gs = P.n_q / P.n_kv;
  const int share = dl_page_share(P, S);
  const int p0 = S.page0, p1 = p0 + S.pages;
  const uint4 zero4 = make_uint4(0, 0, 0, 0);
  float* po = S.part[0];                                // [warp][8 heads][HD + 4]
  static_assert(DL_WARPS * 8 * (128 + 4) <= 2 * DL_WARPS * 32 * DL_STRIDE, "the warps' sums fit where the partial sums lie");
  uint32_t held = 0;                                    // the stage that holds page `at`
  int at = p0, b = 0;
  while (at < p1) {
    while (S.pre[b + 1] * P.n_kv <= at) b++;
    const int n = S.pre[b + 1] - S.pre[b];
    const int kvh = (at - S.pre[b] * P.n_kv) / n;
    const int s0 = S.pre[b] * P.n_kv + kvh * n, s1 = s0 + n, from = at, end = min(s1, p1);
    const int pos = P.pos[b];
    const int lo = (P.window > 0 && pos - P.window + 1 > 0) ? pos - P.window + 1 : 0;
    float o[2 * CH][4];
#pragma unroll
    for (int i = 0; i < 2 * CH; i++) { o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f; }
    float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
    uint4 qv[CH];
#pragma unroll
    for (int c = 0; c < CH; c++)
      qv[c] = g < gs ? ld_fresh(reinterpret_cast<const uint4*>(P.qb + ((size_t)b * P.n_q + kvh * gs + g) * HD + 32 * c + 8 * t)) : zero4;
    // the new key comes behind its pair's last page, as a block of 16 keys with one key; by a warp that has no part in that page
    const bool has_new = end == s1 && warp == ((n & 1) << 2);
    uint4 nk[CH], nv[CH];
    if (has_new) {
      const int page = P.block_table[(size_t)P.seq[b] * P.bt_stride + pos / DL_PAGE];
      const size_t off = (((size_t)page * P.n_kv + kvh) * DL_PAGE + pos % DL_PAGE) * HD + 8 * t;
#pragma unroll
      for (int c = 0; c < CH; c++) {
        nk[c] = g == 0 ? ld_fresh(reinterpret_cast<const uint4*>(L.k + off + 32 * c)) : zero4;
        nv[c] = g == 0 ? ld_fresh(reinterpret_cast<const uint4*>(L.v + off + 32 * c)) : zero4;
      }
    }
#pragma unroll 1
    for (; at <= end; at++) {
      const bool fresh = at == end;
      uint4 a0[CH], a1[CH];
      const int i = at - p0;
      bool mine;
      uint32_t keys = 0;
      if (!fresh) {
        if (CH == 4 || (i & 1) == 0) held = W.ready();
        mine = (warp >> 2) == ((at - s0) & 1);           // (by the pair's pages: the same sums in any batch)
        keys = held + (CH == 4 ? 0 : (i & 1) * 2 * BYTES) + (16 * (warp & 3) + g) * PITCH + t * 16;
      } else {
        mine = has_new;
      }
      const int key0 = (S.first[b] + at - s0) * DL_PAGE + 16 * (warp & 3);
      if (mine && (fresh || (key0 < pos && key0 + 15 >= lo))) {
        if (fresh) {
#pragma unroll
          for (int c = 0; c < CH; c++) { a0[c] = nk[c]; a1[c] = zero4; }
        } else {
          W.template fragments<CH>(keys, PITCH, a0, a1);
        }
        float s[4] = {0.f, 0.f, 0.f, 0.f};              // [0],[1] = (key g, heads 2t, 2t+1); [2],[3] = key g+8
        float z[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int c = 0; c < CH; c++) {
          mma16816(s, a0[c].x, a1[c].x, a0[c].y, a1[c].y, qv[c].x, qv[c].y);
          mma16816(z, a0[c].z, a1[c].z, a0[c].w, a1[c].w, qv[c].z, qv[c].w);
        }
        if (fresh) {
#pragma unroll
          for (int c = 0; c < CH; c++) a0[c] = nv[c];
        } else {
          W.template fragments<CH>(keys + BYTES, PITCH, a0, a1);
        }
        const bool ok0 = fresh ? g == 0 : key0 + g < pos && key0 + g >= lo;
        const bool ok1 = !fresh && key0 + g + 8 < pos && key0 + g + 8 >= lo;
        s[0] = ok0 ? (s[0] + z[0]) * P.scale : -INFINITY; s[1] = ok0 ? (s[1] + z[1]) * P.scale : -INFINITY;
        s[2] = ok1 ? (s[2] + z[2]) * P.scale : -INFINITY; s[3] = ok1 ? (s[3] + z[3]) * P.scale : -INFINITY;
        float bm[2] = {fmaxf(s[0], s[2]), fmaxf(s[1], s[3])}, corr[2], m_use[2];
#pragma unroll
        for (int e = 0; e < 2; e++) {
          bm[e] = fmaxf(bm[e], __shfl_xor_sync(0xffffffffu, bm[e], 4));
          bm[e] = fmaxf(bm[e], __shfl_xor_sync(0xffffffffu, bm[e], 8));
          bm[e] = fmaxf(bm[e], __shfl_xor_sync(0xffffffffu, bm[e], 16));
          const float m_new = fmaxf(m_run[e], bm[e]);
          m_use[e] = (m_new == -INFINITY) ? 0.f : m_new;
          corr[e] = __expf(m_run[e] - m_use[e]);
          m_run[e] = m_new;
        }
        const float e0 = __expf(s[0] - m_use[0]), e1 = __expf(s[1] - m_use[1]);
        const float e2 = __expf(s[2] - m_use[0]), e3 = __expf(s[3] - m_use[1]);
        l_run[0] = l_run[0] * corr[0] + e0 + e2;
        l_run[1] = l_run[1] * corr[1] + e1 + e3;
#pragma unroll
        for (int k = 0; k < 2 * CH; k++) {
          o[k][0] *= corr[0]; o[k][1] *= corr[1]; o[k][2] *= corr[0]; o[k][3] *= corr[1];
        }
        const uint32_t pb0 = transpose8x8(pack_bf16(e0, e1)), pb1 = transpose8x8(pack_bf16(e2, e3));
        // (places of keys the sequence does not hold have probability zero; what a page holds there is finite: zeros from
        // the start, or keys and values of this library)
#pragma unroll
        for (int c = 0; c < CH; c++) {
#pragma unroll
          for (int k = 0; k < 2; k++) {
            const uint32_t x0 = transpose8x8(reg_of(a0[c], 2 * k)), x1 = transpose8x8(reg_of(a0[c], 2 * k + 1));
            const uint32_t x2 = transpose8x8(reg_of(a1[c], 2 * k)), x3 = transpose8x8(reg_of(a1[c], 2 * k + 1));
            mma16816(o[2 * c + k], x0, x1, x2, x3, pb0, pb1);
          }
        }
      }
      if (!fresh && (CH == 4 || (i & 1) || at + 1 == p1)) W.done();
    }
    at = end;
    // the warps' sums meet: heads 2t+e, dims 32c + 8(g/2) + (g%2) + 2i of chunk c, register i
#pragma unroll
    for (int e = 0; e < 2; e++) {
      l_run[e] += __shfl_xor_sync(0xffffffffu, l_run[e], 4);
      l_run[e] += __shfl_xor_sync(0xffffffffu, l_run[e], 8);
      l_run[e] += __shfl_xor_sync(0xffffffffu, l_run[e], 16);
      if (g == 0) { S.ml[warp][2 * t + e][0] = m_run[e]; S.ml[warp][2 * t + e][1] = l_run[e]; }
      if (2 * t + e < gs) {
        float* q = po + (warp * 8 + 2 * t + e) * (HD + 4) + 8 * (g >> 1) + (g & 1);
#pragma unroll
        for (int c = 0; c < CH; c++)
#pragma unroll
          for (int i = 0; i < 4; i++) q[32 * c + 2 * i] = o[2 * c + (i >> 1)][2 * (i & 1) + e];
      }
    }
    dl_sync();
    const bool whole = from == s0 && end == s1;
    const int slot = 2 * blockIdx.x + (from == s0 ? 1 : 0);
    for (int i = threadIdx.x; i < gs * (HD / 2); i += DL_COMPUTE) {
      const int h = i / (HD / 2), d = 2 * (i % (HD / 2));
      float mx = -INFINITY;
#pragma unroll
      for (int w = 0; w < DL_WARPS; w++) mx = fmaxf(mx, S.ml[w][h][0]);
      const float mu = mx == -INFINITY ? 0.f : mx;
      float a0 = 0.f, a1 = 0.f, l = 0.f;
#pragma unroll
      for (int w = 0; w < DL_WARPS; w++) {               // (a warp without keys: factor exp(-inf) and sums of zero)
        const float f = __expf(S.ml[w][h][0] - mu);
        const float2 v = *reinterpret_cast<const float2*>(po + (w * 8 + h) * (HD + 4) + d);
        a0 += f * v.x; a1 += f * v.y; l += f * S.ml[w][h][1];
      }
      if (whole) {
        const float inv = 1.0f / l;
        *reinterpret_cast<__nv_bfloat162*>(P.ob + ((size_t)b * P.n_q + kvh * gs + h) * HD + d) = __floats2bfloat162_rn(a0 * inv, a1 * inv);
      } else {
        *reinterpret_cast<float2*>(P.part_o + ((size_t)slot * 8 + h) * HD + d) = make_float2(a0, a1);
        if (d == 0) *reinterpret_cast<float2*>(P.part_ml + (slot * 8 + h) * 2) = make_float2(mx, l);
      }
    }
    dl_sync();                                           // the meeting place is free again; the pieces are written
    if (!whole) {
      const int first = s0 / share, last = (s1 - 1) / share;           // the blocks that saw a part of this pair (see dl_cut)
      unsigned* counter = P.counters + 1 + b * P.n_kv + kvh;
      if (threadIdx.x == 0) {
        __threadfence();
        const bool is_last = atomicAdd(counter, 1u) == (unsigned)(last - first);
        if (is_last) *counter = 0;                       // (nobody else comes before the next layer)
        __threadfence();
        S.last = is_last;
      }
      dl_sync();
      if (S.last) {
        for (int i = threadIdx.x; i < gs * (HD / 2); i += DL_COMPUTE) {
          const int h = i / (HD / 2), d = 2 * (i % (HD / 2));
          float mx = -INFINITY, a0 = 0.f, a1 = 0.f, l = 0.f;
          for (int c0 = first; c0 <= last; c0 += 4) {    // four pieces' numbers under way at a time
            float2 ml[4], v[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
              const int c = min(c0 + k, last), sl = 2 * c + (c * share <= s0 ? 1 : 0);
              ml[k] = __ldcg(reinterpret_cast<const float2*>(P.part_ml + (sl * 8 + h) * 2));
              v[k] = __ldcg(reinterpret_cast<const float2*>(P.part_o + ((size_t)sl * 8 + h) * HD + d));
            }
#pragma unroll
            for (int k = 0; k < 4; k++) {
              if (c0 + k > last) break;
              const float m_new = fmaxf(mx, ml[k].x), mu = m_new == -INFINITY ? 0.f : m_new;
              const float f0 = __expf(mx - mu), f1 = __expf(ml[k].x - mu);
              a0 = a0 * f0 + f1 * v[k].x; a1 = a1 * f0 + f1 * v[k].y; l = l * f0 + f1 * ml[k].y;
              mx = m_new;
            }
          }
          const float inv = 1.0f / l;
          *reinterpret_cast<__nv_bfloat162*>(P.ob + ((size_t)b * P.n_q + kvh * gs + h) * HD + d) = __floats2bfloat162_rn(a0 * inv, a1 * inv);
        }
      }
      dl_sync();                                         // (S.last)
    }
  }
}

// ------------------------------------------------------------------------------------------ the kernel
template <int MT, int CH>
__global__ void __launch_bounds__(DL_THREADS, 1)
decode_layers_kernel(const __grid_constant__ DlParams P) {
  extern __shared__ __align__(128) uint8_t smem_raw[];
  DlSmem& S = *reinterpret_cast<DlSmem*>(smem_raw);
  constexpr int HD = 32 * CH;
  constexpr int TG = 4 / MT;                    // tiles whose partial sums meet at a time
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int G = gridDim.x;

  if (tid < PH_COUNT) {
    const int NQ = (P.n_q + 2 * P.n_kv) * HD;
    const int N = tid == PH_QKV ? NQ : tid == PH_O ? P.H : tid == PH_GU ? 2 * P.F : tid == PH_DOWN ? P.H : P.vocab;
    DlShare s;
    s.row0 = 2 * (int)((long long)blockIdx.x * (N / 2) / G);
    s.rows = 2 * (int)((long long)(blockIdx.x + 1) * (N / 2) / G) - s.row0;
    s.tiles = (s.rows + 15) / 16;
    s.K = tid == PH_O ? P.n_q * HD : tid == PH_DOWN ? P.F : P.H;
    s.chunks = (s.K + DL_CHUNK - 1) / DL_CHUNK;
    S.share[tid] = s;
  }
  if (tid == 32) {
    for (int s = 0; s < DL_STAGES; s++) { mbar_init(&S.full[s], 1); mbar_init(&S.empty[s], DL_WARPS); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    S.abort_flag = 0;
    int n = 0;
    S.pre[0] = 0;
    for (int b = 0; b < P.M; b++) {
      const int pos = P.pos[b], lo = (P.window > 0 && pos - P.window + 1 > 0) ? pos - P.window + 1 : 0;
      S.live[b] = P.seq[b] >= 0;
      S.first[b] = lo / DL_PAGE;
      n += S.live[b] ? max(pos - 1, lo) / DL_PAGE - lo / DL_PAGE + 1 : 0;    // pages of the keys in front of the new one
      S.pre[b + 1] = n;
    }
  }
  __syncthreads();
  {
    const int p0 = dl_cut(P, S, blockIdx.x), pages = min(DL_MAX_PAGES, dl_cut(P, S, blockIdx.x + 1) - p0);
    for (int i = tid; i < pages; i += DL_THREADS) {
      int b = 0;
      while (S.pre[b + 1] * P.n_kv <= p0 + i) b++;
      const int n = S.pre[b + 1] - S.pre[b], r = p0 + i - S.pre[b] * P.n_kv;
      S.place[i] = P.block_table[(size_t)P.seq[b] * P.bt_stride + S.first[b] + r % n] * P.n_kv + r / n;
    }
    if (tid == 0) { S.page0 = p0; S.pages = pages; }
  }
  __syncthreads();

  // 384 threads are launched with 168 registers each: 256 x 232 + 128 x 40 is the same
  if (warp >= DL_WARPS) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    if (warp == DL_WARPS) {
      DlFeeder<CH> feeder = {P, S, lane, 0, 1};
      feeder.run();
    }
    return;
  }
  asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
  DlProduct<MT> W = {P, S, warp, lane, 0, 0, 0};

  // where a thread stands among the sums that meet: pair ep of tile etl, row em of x
  const int ep = tid & 7, em = (tid >> 3) & (8 * MT - 1), etl = tid / (64 * MT);
  const bool m_ok = em < P.M;
  const int my_pos = m_ok ? P.pos[em] : 0, my_seq = m_ok ? P.seq[em] : -1;
  const int my_page = my_seq >= 0 ? P.block_table[(size_t)my_seq * P.bt_stride + my_pos / DL_PAGE] : 0;
  // the stream: every thread of the first two tiles of the block's share of H keeps its two values
  const int sn = S.share[PH_O].row0 + etl * 16 + 2 * ep;
  const bool s_on = m_ok && etl < S.share[PH_O].tiles && etl * 16 + 2 * ep < S.share[PH_O].rows;
  float r0 = 0.f, r1 = 0.f;
  float* ss_of[2] = {P.ss, P.ss + (size_t)G * DL_MAX_ROWS};      // in front of the attention's half; of the feed-forward's
  float2 gain = make_float2(0.f, 0.f);
  if (s_on) {
    const float2 v = __ldcg(reinterpret_cast<const float2*>(P.x + (size_t)em * P.H + sn));
    r0 = v.x; r1 = v.y;
    gain = *reinterpret_cast<const float2*>(P.gain_first + sn);
  }
  dl_hand_on<MT>(P, S, s_on, em, sn, r0, r1, gain, ss_of[0]);
  unsigned target = P.absent;

  // products whose rows of x fit into registers: all of this warp's k, one tile after the other
  auto wide = [&](int ph, const bf16* x, const float* ss, auto before, auto store) -> bool {
    const DlShare s = S.share[ph];
    before(0);
    target += G;
    if (!dl_meet(P, S, target, 401 + ph)) return false;
    uint4 b[16 * MT];
#pragma unroll
    for (int c = 0; c < 4; c++) W.rows_of(x, s.K, c, ph == PH_O, b + c * 4 * MT);
    float f[MT][DL_MAX_BLOCKS / 32];
    if (ss) W.ask_factors(ss, f);
#pragma unroll 1
    for (int t0 = 0; t0 < s.tiles; t0 += TG) {
      if (t0) before(t0);
#pragma unroll 1
      for (int tl = 0; tl < TG && t0 + tl < s.tiles; tl++) {
        float acc[MT][2][4];
        W.zero(acc);
#pragma unroll
        for (int c = 0; c < 4; c++)
          if (c < s.chunks) W.step(s.K, c, b + c * 4 * MT, acc);
        W.leave(tl, acc);
      }
      if (ss && t0 == 0) W.leave_factors(f);
      dl_sync();
      const int n = (t0 + etl) * 16 + 2 * ep;           // within the share
      const bool on = m_ok && t0 + etl < s.tiles && n < s.rows;
      float2 v = make_float2(0.f, 0.f);
      if (on) v = W.gather(etl, em, ep);
      store(on, s.row0 + n, v);
      W.buf ^= 1;
    }
    return true;
  };

  bool ok = true;
  dl_arrive(P);
#pragma unroll 1
  for (int l = 0; l < P.n_layers && ok; l++) {
    const DlLayer& L = P.layer[l];
    // ---------------------------------------------------------------- queries, keys, values
    float2 turn = make_float2(1.f, 0.f);
    ok = wide(PH_QKV, P.xb, ss_of[0],
              [&](int t0) {
                const int n = S.share[PH_QKV].row0 + (t0 + etl) * 16 + 2 * ep;
                const int d = (n % HD) >> 1;
                turn = make_float2(1.f, 0.f);
                if (m_ok && n < (P.n_q + P.n_kv) * HD && d < P.n_pairs) turn = P.rope[em * P.n_pairs + d];
              },
              [&](bool on, int n, float2 v) {
                if (!on) return;
                const float inv = S.inv[em];
                v.x *= inv; v.y *= inv;
                const __nv_bfloat162 y = __floats2bfloat162_rn(v.x * turn.x - v.y * turn.y, v.x * turn.y + v.y * turn.x);
                const int head = n / HD, d = n % HD;
                if (head < P.n_q) {
                  *reinterpret_cast<__nv_bfloat162*>(P.qb + (size_t)em * P.n_q * HD + n) = y;
                } else if (my_seq >= 0) {
                  const int h = head - P.n_q;
                  bf16* c = h < P.n_kv ? L.k : L.v;
                  const int kvh = h < P.n_kv ? h : h - P.n_kv;
                  *reinterpret_cast<__nv_bfloat162*>(c + (((size_t)my_page * P.n_kv + kvh) * DL_PAGE + my_pos % DL_PAGE) * HD + d) = y;
                }
              });
    if (!ok) break;
    dl_arrive(P);
    // ---------------------------------------------------------------- attention
    target += G;
    if (!(ok = dl_meet(P, S, target, 411))) break;
    dl_attention<MT, CH>(P, S, L, W);
    dl_arrive(P);
    // ---------------------------------------------------------------- output projection
    ok = wide(PH_O, P.ob, nullptr,
              [&](int) { if (s_on) gain = *reinterpret_cast<const float2*>(L.gain_ff + sn); },
              [&](bool on, int n, float2 v) {
                r0 += v.x; r1 += v.y;
                dl_hand_on<MT>(P, S, on, em, n, r0, r1, gain, ss_of[1]);
              });
    if (!ok) break;
    dl_arrive(P);
    // ---------------------------------------------------------------- gate and up
    ok = wide(PH_GU, P.xb, ss_of[1], [&](int) {},
              [&](bool on, int n, float2 v) {
                if (!on) return;
                const float inv = S.inv[em];
                P.ab[(size_t)em * P.F + (n >> 1)] = __float2bfloat16_rn(gated_as<STRATUM_ACT_NONE, false>(v.x * inv, v.y * inv, 0.f));
              });
    if (!ok) break;
    dl_arrive(P);
    // ---------------------------------------------------------------- down: k is long, its rows of x come as they are needed
    {
      if (s_on) gain = *reinterpret_cast<const float2*>(L.gain_next + sn);
      const DlShare s = S.share[PH_DOWN];
      target += G;
      if (!(ok = dl_meet(P, S, target, 421))) break;
      uint4 b[4 * MT], nb[4 * MT];
      W.rows_of(P.ab, s.K, 0, false, b);
      float acc0[MT][2][4], acc1[MT][2][4];
      W.zero(acc0);
      W.zero(acc1);
#pragma unroll 1
      for (int c = 0; c < s.chunks; c++) {
        W.rows_of(P.ab, s.K, c + 1, false, nb);
        W.step(s.K, c, b, acc0);
        if (s.tiles > 1) W.step(s.K, c, b, acc1);
#pragma unroll
        for (int i = 0; i < 4 * MT; i++) b[i] = nb[i];
      }
      W.leave(0, acc0);
      if (s.tiles > 1) W.leave(1, acc1);
      dl_sync();
      if (s_on) {
        const float2 v = W.gather(etl, em, ep);
        r0 += v.x; r1 += v.y;
      }
      W.buf ^= 1;
      dl_hand_on<MT>(P, S, s_on, em, sn, r0, r1, gain, ss_of[0]);
    }
    dl_arrive(P);
  }
  // ------------------------------------------------------------------ the head (of no tiles where no logits are wanted; asking
  // whether there is one costs 1.5 % of a step of 8 rows)
  if (ok)
    wide(PH_HEAD, P.xb, ss_of[0], [&](int) {},
         [&](bool on, int n, float2 v) {
           if (!on) return;
           const float inv = S.inv[em];
           *reinterpret_cast<float2*>(P.logits + (size_t)em * P.vocab + n) = make_float2(v.x * inv, v.y * inv);
         });
}

template <int MT, int CH>
static int launch_decode_layers(const DlParams& P, int blocks, cudaStream_t stream) {
  auto kern = decode_layers_kernel<MT, CH>;
  const int smem = (int)sizeof(DlSmem);
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  // the blocks meet, so all of them must be resident: where the device or this context cannot hold them the caller runs
  // the step another way
  int dev = 0, cooperative = 0, sms = 0, per_sm = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return (int)e;
  if ((e = cudaDeviceGetAttribute(&cooperative, cudaDevAttrCooperativeLaunch, dev)) != cudaSuccess) return (int)e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return (int)e;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, DL_THREADS, smem)) != cudaSuccess) return (int)e;
  if (!cooperative || per_sm * sms < blocks) return STRATUM_ERR_RESIDENT;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(DL_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  e = cudaLaunchKernelEx(&cfg, kern, P);
  if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported) {
    cudaGetLastError();                          // (nothing ran; the error is this launch's alone)
    return STRATUM_ERR_RESIDENT;
  }
  return (int)e;
}

// Bytes of DlParams, for callers that mirror it.
STRATUM_EXPORT int stratum_decode_layers_params() { return (int)sizeof(DlParams); }

// `blocks`: one per SM; the sizes of ss, part_o and part_ml follow from it.
STRATUM_EXPORT int stratum_decode_layers(const DlParams* p, int blocks, cudaStream_t stream) {
  const DlParams& P = *p;
  if (P.M < 1) return 0;
  if (P.M > DL_MAX_ROWS || P.n_layers > DL_MAX_LAYERS || blocks > DL_MAX_BLOCKS) return STRATUM_ERR_LIMIT;
  if (P.n_layers < 1 || blocks < 1 || (P.D != 64 && P.D != 128)) return STRATUM_ERR_SHAPE;
  if (P.n_kv < 1 || P.n_q % P.n_kv != 0 || P.n_q / P.n_kv > 8 || P.n_pairs < 0 || 2 * P.n_pairs > P.D) return STRATUM_ERR_SHAPE;
  const int KO = P.n_q * P.D;
  // a warp's 128 of every 1,024 k; the rows of x of the products over H and over the heads lie in registers
  if (P.H % 128 || P.F % 128 || KO % 128 || P.H > 4 * DL_CHUNK || KO > 4 * DL_CHUNK) return STRATUM_ERR_SHAPE;
  // two rows of every matrix for each block, two tiles of 16 of the stream at most
  if (P.H < 2 * blocks || 2 * P.F < 2 * blocks || (P.H / 2 + blocks - 1) / blocks > 16) return STRATUM_ERR_SHAPE;
  if ((P.n_q + 2 * P.n_kv) * P.D < 2 * blocks || P.vocab < 0 || P.vocab % 2 || (P.vocab && P.vocab < 2 * blocks)) return STRATUM_ERR_SHAPE;
  // a block's list of pages (the table's width bounds the sequences' lengths)
  if (P.bt_stride < 1 || (long long)P.M * P.n_kv * P.bt_stride > (long long)(DL_MAX_PAGES - 2 * DL_WHOLE - 1) * blocks)
    return STRATUM_ERR_LIMIT;
  if (P.vocab && (!P.w_head || !P.logits)) return STRATUM_ERR_SHAPE;
  if (!P.x || !P.gain_first || !P.pos || !P.seq || !P.block_table || (P.n_pairs && !P.rope))
    return STRATUM_ERR_SHAPE;
  if (!P.status || !P.counters || !P.xb || !P.qb || !P.ob || !P.ab || !P.ss || !P.part_o || !P.part_ml) return STRATUM_ERR_SHAPE;
  if (((uintptr_t)P.x | (uintptr_t)P.gain_first | (uintptr_t)P.w_head | (uintptr_t)P.logits | (uintptr_t)P.xb | (uintptr_t)P.qb |
       (uintptr_t)P.ob | (uintptr_t)P.ab | (uintptr_t)P.part_o | (uintptr_t)P.part_ml | (uintptr_t)P.rope) & 15) return STRATUM_ERR_ALIGN;
  for (int i = 0; i < P.n_layers; i++) {
    const DlLayer& L = P.layer[i];
    if (!L.w_qkv || !L.w_o || !L.w_gu || !L.w_down || !L.gain_ff || !L.gain_next || !L.k || !L.v) return STRATUM_ERR_SHAPE;
    if (((uintptr_t)L.w_qkv | (uintptr_t)L.w_o | (uintptr_t)L.w_gu | (uintptr_t)L.w_down | (uintptr_t)L.gain_ff |
         (uintptr_t)L.gain_next | (uintptr_t)L.k | (uintptr_t)L.v) & 15) return STRATUM_ERR_ALIGN;
  }
  if (P.M <= 8) return P.D == 64 ? launch_decode_layers<1, 2>(P, blocks, stream) : launch_decode_layers<1, 4>(P, blocks, stream);
  return P.D == 64 ? launch_decode_layers<2, 2>(P, blocks, stream) : launch_decode_layers<2, 4>(P, blocks, stream);
}
