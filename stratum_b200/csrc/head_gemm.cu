// One small matrix product per head, in one launch, in bfloat16 on tensor cores:
//   out[m][j * o_step + n] = sum_k x[m][j * x_step + k] * w[j][n][k]        (head j; w [heads][N][K])
// which is how a mixer carries per-head vectors from one space into another (queries into a latent space, mixed
// latents into value heads).  The matrices are small (tens to hundreds of rows and columns), so a launch per head
// would cost more than the work; here the heads are the grid's third dimension.
//
// More than 16 rows: a warp owns 32 rows of x (HG_TILES x 16) and 64 columns of one head: mma.sync.m16n8k16 with the rows of x as the A operand
// and 8 weight rows per B operand, both straight from global memory (lane t of a row takes the 8 contiguous values
// 8t..8t+7 of every 32 of k, for x and for w alike, so the products pair up as in the definition).  Up to 32 rows the
// four warps of a CTA take four column tiles and the kernel streams the weights once; with more (prompts) they take four
// row tiles and share the weight rows through L1.  float32 accumulation over k in order.
#include "common.cuh"
#include "mma_common.cuh"

#define HG_WARPS 4
#define HG_COLS 64
#define HG_TILES 2

__global__ void __launch_bounds__(HG_WARPS * 32)
head_gemm_kernel(const bf16* x, const bf16* __restrict__ w, bf16* out, int M, int N, int K, int ldx, int ldo,
                 int x_step, int o_step, int warps_split_columns) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int head = blockIdx.z;
  pdl_trigger();
  int row0, n0;
  if (warps_split_columns) {
    row0 = blockIdx.x * 16 * HG_TILES;
    n0 = (blockIdx.y * HG_WARPS + warp) * HG_COLS;
  } else {
    row0 = (blockIdx.x * HG_WARPS + warp) * 16 * HG_TILES;
    n0 = blockIdx.y * HG_COLS;
  }
  if (row0 >= M || n0 >= N) return;
  const bf16* xh = x + (size_t)head * x_step;
  const bf16* wh = w + (size_t)head * N * K;
  float acc[HG_TILES][8][4];
#pragma unroll
  for (int a = 0; a < HG_TILES; a++)
#pragma unroll
    for (int j = 0; j < 8; j++) { acc[a][j][0] = acc[a][j][1] = acc[a][j][2] = acc[a][j][3] = 0.f; }
  const uint4 zero4 = make_uint4(0, 0, 0, 0);
  pdl_wait();                                   // x comes from the kernel before this one
#pragma unroll 2
  for (int k0 = 0; k0 < K; k0 += 32) {
    const int k = k0 + 8 * t;
    const bool k_ok = k < K;
    uint4 xa[HG_TILES], xc[HG_TILES];
#pragma unroll
    for (int a = 0; a < HG_TILES; a++) {
      const int r = row0 + 16 * a + g;
      xa[a] = (k_ok && r < M) ? ld_fresh((const uint4*)(xh + (size_t)r * ldx + k)) : zero4;
      xc[a] = (k_ok && r + 8 < M) ? ld_fresh((const uint4*)(xh + (size_t)(r + 8) * ldx + k)) : zero4;
    }
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const int n = n0 + 8 * j + g;
      const uint4 wb = (k_ok && n < N) ? __ldg((const uint4*)(wh + (size_t)n * K + k)) : zero4;
#pragma unroll
      for (int a = 0; a < HG_TILES; a++) {
        mma16816(acc[a][j], xa[a].x, xc[a].x, xa[a].y, xc[a].y, wb.x, wb.y);
        mma16816(acc[a][j], xa[a].z, xc[a].z, xa[a].w, xc[a].w, wb.z, wb.w);
      }
    }
  }
  bf16* oh = out + (size_t)head * o_step;
#pragma unroll
  for (int a = 0; a < HG_TILES; a++) {
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const int n = n0 + 8 * j + 2 * t;
      if (n >= N) continue;                     // N % 8 == 0: a pair of columns is inside or outside together
      const int r = row0 + 16 * a + g;
      if (r < M) *reinterpret_cast<uint32_t*>(oh + (size_t)r * ldo + n) = pack_bf16(acc[a][j][0], acc[a][j][1]);
      if (r + 8 < M) *reinterpret_cast<uint32_t*>(oh + (size_t)(r + 8) * ldo + n) = pack_bf16(acc[a][j][2], acc[a][j][3]);
    }
  }
}

// Up to 16 rows of x (decode steps): a warp takes eight columns of one head and asks for all of its weights (STEPS blocks
// of 32 of k) before it waits for the kernel in front of it, so that a launch costs about one round trip to memory and the
// weights come in while that kernel still runs.  The sums are those of the kernel above, k in order.
// 32 heads of 128 x 512 and 512 x 128, six rows: 1.7 and 4.9 us in a step against 22 (64 columns a warp: 256 and 64 warps, sixteen
// dependent loads each).
template <int STEPS>
__global__ void __launch_bounds__(HG_WARPS * 32)
head_gemm_few_kernel(const bf16* x, const bf16* __restrict__ w, bf16* out, int M, int N, int K, int ldx, int ldo,
                     int x_step, int o_step) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, head = blockIdx.y;
  const int n0 = (blockIdx.x * HG_WARPS + warp) * 8;
  pdl_trigger();
  const uint4 zero4 = make_uint4(0, 0, 0, 0);
  const bf16* wr = w + ((size_t)head * N + n0 + g) * K;         // N % 8 == 0: the eight columns are there together
  const bf16* xr = x + (size_t)head * x_step + (size_t)g * ldx;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  for (int k0 = 0; k0 < K; k0 += 32 * STEPS) {
    uint4 wb[STEPS];
#pragma unroll
    for (int i = 0; i < STEPS; i++) {
      const int k = k0 + 32 * i + 8 * t;
      wb[i] = n0 < N && k < K ? __ldg((const uint4*)(wr + k)) : zero4;
    }
    if (k0 == 0) pdl_wait();                    // x comes from the kernel before this one
    if (n0 >= N) return;
#pragma unroll
    for (int i0 = 0; i0 < STEPS; i0 += 4) {
      uint4 xa[4], xc[4];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int k = k0 + 32 * (i0 + i) + 8 * t;
        xa[i] = k < K && g < M ? ld_fresh((const uint4*)(xr + k)) : zero4;
        xc[i] = k < K && g + 8 < M ? ld_fresh((const uint4*)(xr + (size_t)8 * ldx + k)) : zero4;
      }
#pragma unroll
      for (int i = 0; i < 4; i++) {
        mma16816(acc, xa[i].x, xc[i].x, xa[i].y, xc[i].y, wb[i0 + i].x, wb[i0 + i].y);
        mma16816(acc, xa[i].z, xc[i].z, xa[i].w, xc[i].w, wb[i0 + i].z, wb[i0 + i].w);
      }
    }
  }
  bf16* oh = out + (size_t)head * o_step + n0 + 2 * t;
  if (g < M) *reinterpret_cast<uint32_t*>(oh + (size_t)g * ldo) = pack_bf16(acc[0], acc[1]);
  if (g + 8 < M) *reinterpret_cast<uint32_t*>(oh + (size_t)(g + 8) * ldo) = pack_bf16(acc[2], acc[3]);
}

// x bf16 [M][ldx], w bf16 [heads][N][K], out bf16 [M][ldo].  Needs K % 8 == 0, N % 8 == 0, x_step % 8 == 0,
// ldx % 8 == 0, o_step and ldo even, x and w 16-byte aligned, out 4-byte aligned.
STRATUM_EXPORT int stratum_head_gemm(const void* x, const void* w, void* out, int heads, int M, int N, int K, int ldx,
                                     int ldo, int x_step, int o_step, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || heads <= 0) return 0;
  if (K <= 0 || K % 8 != 0 || N % 8 != 0 || x_step % 8 != 0 || ldx % 8 != 0 || o_step % 2 != 0 || ldo % 2 != 0)
    return STRATUM_ERR_SHAPE;
  if ((long long)(heads - 1) * x_step + K > ldx || (long long)(heads - 1) * o_step + N > ldo) return STRATUM_ERR_SHAPE;
  if ((((uintptr_t)x | (uintptr_t)w) & 15) != 0 || ((uintptr_t)out & 3) != 0) return STRATUM_ERR_ALIGN;
  if (heads > 65535) return STRATUM_ERR_LIMIT;
  const int col_tiles = (N + HG_COLS - 1) / HG_COLS;
  if (M <= 16) {
    const dim3 grid((N / 8 + HG_WARPS - 1) / HG_WARPS, heads);
    if (K <= 128)
      return launch_pdl(head_gemm_few_kernel<4>, grid, HG_WARPS * 32, 0, stream, (const bf16*)x, (const bf16*)w, (bf16*)out,
                        M, N, K, ldx, ldo, x_step, o_step);
    return launch_pdl(head_gemm_few_kernel<16>, grid, HG_WARPS * 32, 0, stream, (const bf16*)x, (const bf16*)w, (bf16*)out, M,
                      N, K, ldx, ldo, x_step, o_step);
  }
  if (M <= 32) {
    dim3 grid(1, (col_tiles + HG_WARPS - 1) / HG_WARPS, heads);
    return launch_pdl(head_gemm_kernel, grid, HG_WARPS * 32, 0, stream, (const bf16*)x, (const bf16*)w, (bf16*)out,
                      M, N, K, ldx, ldo, x_step, o_step, 1);
  }
  const long long row_groups = ((long long)M + 32 * HG_WARPS - 1) / (32 * HG_WARPS);
  if (row_groups > 0x7fffffffLL || col_tiles > 65535) return STRATUM_ERR_LIMIT;
  dim3 grid((unsigned)row_groups, col_tiles, heads);
  return launch_pdl(head_gemm_kernel, grid, HG_WARPS * 32, 0, stream, (const bf16*)x, (const bf16*)w, (bf16*)out, M,
                    N, K, ldx, ldo, x_step, o_step, 0);
}
