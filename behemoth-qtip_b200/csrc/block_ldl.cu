// Block LDL of the rotated, damped Hessian on the GPU, in fp64: H = (Lb + I) D (Lb + I)^T with 16 x 16 diagonal blocks,
// delivered as the strictly block-lower factor Lb in fp32 -- what LDLQ consumes. The reference computes it on the host
// (src/qtip_core.cpp:321-487: cholesky_inplace + block_ldl_to_L, fp64, OpenMP); at n = 28,672 that is the longest stage
// of a Hessian group once the Viterbi runs on a B200.
//
// Method (same algebra as the reference): symmetrise in fp64, A = (H + H^T) / 2; Cholesky A = C C^T (lower); for every
// 16-column block bj, Lb[:, bj] = C[:, bj] * inv(C[bj, bj]) below the diagonal block, zero on and above it.
// The Cholesky is right-looking with 128-column panels, two launches a panel:
//   1. chol_panel_kernel  rows below the diagonal block: x L11^T = a, 64 rows per CTA held in registers, sixteen columns
//                         at a time through the inverse of their diagonal block;
//   2. chol_update_kernel trailing update C -= P P^T on the lower triangle: 128 x 64 tiles on the fp64 tensor cores, the
//                         128-deep panels streamed through shared memory in 16-column slices. This is where the n^3 / 6
//                         multiply-adds are: bound by the fp64 pipes (64 lanes per SM and clock). The CTA of the first
//                         tile takes the next diagonal block whole and factors it in shared memory (chol_factor) while
//                         the other tiles are updated: the one serial stage of a panel is off the critical path as long
//                         as the update takes longer than one factorisation.
// The first diagonal block has a launch of its own (chol_first_kernel).
// A non-positive pivot or a non-finite result sets a status word in the workspace (qtip_block_ldl_status); the
// reference returns false in those cases.
#include "common.cuh"

namespace qb {

constexpr int kNb = 128;   // panel width
constexpr int kTile = 128; // trailing-update tile
constexpr int kKc = 16;    // panel columns per shared-memory slice

struct LdlHeader {
  int status;  // bit 0: a pivot was not positive; bit 1: a non-finite value in the factor
  int pad[63];
};

// A[i][j] = (H[i][j] + H[j][i]) / 2 in fp64, lower triangle (j <= i); the strict upper triangle is never read again.
__global__ void ldl_symmetrise_kernel(const float* __restrict__ H, double* __restrict__ A, long n) {
  __shared__ float t[32][33];
  const long bi = blockIdx.y, bj = blockIdx.x;
  if (bj > bi) return;
  const int tx = threadIdx.x, ty = threadIdx.y;  // 32 x 8
  for (int r = ty; r < 32; r += 8) {
    const long i = bj * 32 + r, j = bi * 32 + tx;  // the transposed block, read along its rows
    t[r][tx] = (i < n && j < n) ? H[i * n + j] : 0.f;
  }
  __syncthreads();
  for (int r = ty; r < 32; r += 8) {
    const long i = bi * 32 + r, j = bj * 32 + tx;
    if (i < n && j < n && j <= i) A[i * n + j] = 0.5 * (double(H[i * n + j]) + double(t[tx][r]));
  }
}

__device__ __forceinline__ void dmma_8x8x4(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// Cholesky of a kb x kb block (kb a multiple of 16, at most 128) in shared memory, packed lower triangle, by eight warps. Sixteen
// columns at a time: one warp factors the 16 x 16 diagonal block with a row per lane in registers and inverts it (a column
// per lane), then all warps take the rows below it through the inverse, a 16 x 16 block a warp on the fp64 tensor cores. What
// is right of them is updated by warps 1 to 7 while warp 0 updates, factors and inverts the next diagonal block. The
// inverses, which the panel kernel and the final block scaling need as well, go to `inv` (256 values a block, row-major,
// zeros above the diagonal).
// Bound by latency: the square roots of the pivots, one after another. 48 us a block of 128 where it was 127 (inverse 69,000, by
// divisions that each wait for the one before; factor 47,000; trailing updates 34,000 and the rows 19,000 in scalar
// multiply-adds behind the factor; the block's way in and out of shared memory, an element a thread at a time, the rest of
// 221,000 cycles). It is the floor of an update: 138 -> 70 us, which half of the panels of n = 12,288 and all of n = 4,096 met.
constexpr int kLd = kNb + 1;  // L11 in the panel kernel
constexpr int kInvLd = 17;
__device__ __forceinline__ int tri(int i) { return i * (i + 1) / 2; }  // first word of row i of a packed lower triangle

// c (2 x 2 fragments of 8 x 8) += x y^T over 16 columns; x(i, p) and y(j, p) read element p of row i / j of the two blocks.
template <typename X, typename Y>
__device__ __forceinline__ void chol_block_product(double (&c)[2][2][2], X x, Y y) {
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
#pragma unroll
  for (int p = 0; p < 16; p += 4) {
    const double a[2] = {x(g, p + q), x(g + 8, p + q)}, b[2] = {y(g, p + q), y(g + 8, p + q)};
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) dmma_8x8x4(c[i][j], a[i], b[j]);
  }
}
// Block (ra, rb) of 16 x 16 (rb <= ra): minus the product of the two row blocks' columns base .. base + 15. One warp.
__device__ __forceinline__ void chol_block_update(double* __restrict__ S, int ra, int rb, int base) {
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  double c[2][2][2] = {};
  chol_block_product(c, [&](int i, int p) { return S[tri(ra + i) + base + p]; },
                     [&](int j, int p) { return S[tri(rb + j) + base + p]; });
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = ra + 8 * i + g, col = rb + 8 * j + 2 * q + h;
        if (col <= r) S[tri(r) + col] -= c[i][j][h];
      }
}
// The 16 x 16 diagonal block at `base` and its inverse, by one warp.
__device__ __forceinline__ void chol_factor16(double* __restrict__ S, double* __restrict__ inv_s, int base,
                                              double* __restrict__ inv, int* status) {
  const int lane = threadIdx.x & 31, i = lane & 15;
  double a[16], own = 1.0;  // own: one over the diagonal element of the lane's row
#pragma unroll
  for (int c = 0; c < 16; ++c) a[c] = c <= i ? S[tri(base + i) + base + c] : 0.0;
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const double d = __shfl_sync(0xffffffffu, a[j], j);
    const bool ok = d > 0.0;
    if (!ok && lane == 0) atomicOr(status, 1);
    // a failed pivot is reported; the factor is then meaningless but finite
    const double dj = ok ? sqrt(d) : 1.0, rj = 1.0 / dj;
    if (i == j) own = rj;
    a[j] = i == j ? dj : a[j] * rj;
#pragma unroll
    for (int c = j + 1; c < 16; ++c) a[c] = fma(-a[j], __shfl_sync(0xffffffffu, a[j], c), a[c]);
  }
  double col[16];  // column i of the inverse
#pragma unroll
  for (int r = 0; r < 16; ++r) {
    double t = r == i ? 1.0 : 0.0;
#pragma unroll
    for (int q = 0; q < 16; ++q)
      if (q < r) t = fma(-__shfl_sync(0xffffffffu, a[q], r), col[q], t);
    col[r] = t * __shfl_sync(0xffffffffu, own, r);
  }
  if (lane < 16) {
#pragma unroll
    for (int c = 0; c < 16; ++c) {
      if (c <= i) S[tri(base + i) + base + c] = a[c];
      inv_s[c * kInvLd + i] = col[c];
      inv[(base / 16) * 256 + c * 16 + i] = col[c];
    }
  }
}
__device__ __forceinline__ void chol_factor(double* __restrict__ S, double* __restrict__ inv_s, int kb,
                                            double* __restrict__ inv, int* status) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  if (warp == 0) chol_factor16(S, inv_s, 0, inv, status);
  __syncthreads();
  for (int base = 0; base + 16 < kb; base += 16) {
    const int next = base + 16, blocks = (kb - next) / 16;
    if (warp < blocks) {  // rows below: x = a inv^T, in place (the warp has read its rows before it writes them)
      const int r0 = next + 16 * warp;
      double c[2][2][2] = {};
      chol_block_product(c, [&](int i, int p) { return S[tri(r0 + i) + base + p]; },
                         [&](int j, int p) { return inv_s[j * kInvLd + p]; });
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int h = 0; h < 2; ++h) S[tri(r0 + 8 * i + g) + base + 8 * j + 2 * q + h] = c[i][j][h];
    }
    __syncthreads();
    if (warp == 0) {
      chol_block_update(S, next, next, base);
      __syncwarp();
      chol_factor16(S, inv_s, next, inv, status);
    } else {
      int at = 0;  // the other blocks, dealt to warps 1 .. 7
      for (int ra = 1; ra < blocks; ++ra)
        for (int rb = 0; rb <= ra; ++rb, ++at)
          if (at % 7 == warp - 1) chol_block_update(S, next + 16 * ra, next + 16 * rb, base);
    }
    __syncthreads();
  }
}
// The diagonal block at (k, k): loaded, factored, stored by a CTA of 256 threads, a row a warp, four rows in flight.
__device__ __forceinline__ void chol_diagonal(double* __restrict__ A, long n, long k, double* __restrict__ sm,
                                              double* __restrict__ inv, int* status) {
  const int kb = int(min(long(kNb), n - k)), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i0 = warp; i0 < kb; i0 += 32) {
    double v[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int i = i0 + 8 * r, j = lane + 32 * c;
        v[r][c] = i < kb && j <= i ? A[(k + i) * n + k + j] : 0.0;
      }
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int i = i0 + 8 * r, j = lane + 32 * c;
        if (i < kb && j <= i) sm[tri(i) + j] = v[r][c];
      }
  }
  __syncthreads();
  chol_factor(sm, sm + tri(kNb), kb, inv, status);
  for (int i = warp; i < kb; i += 8)
    for (int j = lane; j <= i; j += 32) A[(k + i) * n + k + j] = sm[tri(i) + j];
}
__global__ __launch_bounds__(256) void chol_first_kernel(double* __restrict__ A, long n, double* __restrict__ inv,
                                                         int* status) {
  extern __shared__ double sm[];
  chol_diagonal(A, n, 0, sm, inv, status);
}

// Rows r0 + [64 b, 64 b + 64): x L11^T = a. Thread (ty, tx) holds rows ty + 16 a and columns tx + 16 j in registers. Sixteen
// columns at a time: x_b = s_b inv_b^T from shared memory, then every later column block takes x_b L11[j][b]^T off.
constexpr int kPanelRows = 64;
__global__ __launch_bounds__(256) void chol_panel_kernel(double* __restrict__ A, long n, long k,
                                                         const double* __restrict__ inv) {
  extern __shared__ double sm[];
  double* L11 = sm;                              // [kNb][kLd]
  double* inv_s = L11 + kNb * kLd;               // [kNb / 16][16][kInvLd]
  double* Y = inv_s + (kNb / 16) * 16 * kInvLd;  // [kPanelRows][kInvLd] right-hand side of the current block
  double* X = Y + kPanelRows * kInvLd;           // [kPanelRows][kInvLd] its solution
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const long r0 = k + kNb + long(blockIdx.x) * kPanelRows;
  const int rows = int(min(long(kPanelRows), n - r0));
  double acc[4][8];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[a][j] = ty + 16 * a < rows ? A[(r0 + ty + 16 * a) * n + k + tx + 16 * j] : 0.0;
  for (int i = ty; i < kNb; i += 16)
    for (int j = tx; j <= i; j += 16) L11[i * kLd + j] = A[(k + i) * n + k + j];
  for (int i = tid; i < kNb * 16; i += 256) inv_s[(i >> 4) * kInvLd + (i & 15)] = inv[i];
#pragma unroll
  for (int b = 0; b < 8; ++b) {
#pragma unroll
    for (int a = 0; a < 4; ++a) Y[(ty + 16 * a) * kInvLd + tx] = acc[a][b];
    __syncthreads();
    double x[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int p = 0; p < 16; ++p) {
      const double v = inv_s[(b * 16 + tx) * kInvLd + p];  // zero for p > tx
#pragma unroll
      for (int a = 0; a < 4; ++a) x[a] = fma(Y[(ty + 16 * a) * kInvLd + p], v, x[a]);
    }
#pragma unroll
    for (int a = 0; a < 4; ++a) acc[a][b] = x[a], X[(ty + 16 * a) * kInvLd + tx] = x[a];
    __syncthreads();
#pragma unroll
    for (int p = 0; p < 16; ++p) {
      double xr[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) xr[a] = X[(ty + 16 * a) * kInvLd + p];
#pragma unroll
      for (int j = b + 1; j < 8; ++j) {
        const double l = L11[(tx + 16 * j) * kLd + 16 * b + p];
#pragma unroll
        for (int a = 0; a < 4; ++a) acc[a][j] = fma(-xr[a], l, acc[a][j]);
      }
    }
  }
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (ty + 16 * a < rows) A[(r0 + ty + 16 * a) * n + k + tx + 16 * j] = acc[a][j];
}

// C[i][j] -= sum_p P[i][p] P[j][p] for a 128 x 64 tile of the lower triangle of the trailing matrix that starts at row /
// column r0; P = A[r0.., k .. k + 128). Eight warps as 4 x 2, each 32 x 32 outputs as 4 x 4 fp64 tensor-core fragments
// (m8n8k4). The two operand panels pass through a ring of 16-column slices (cp.async; row stride 20 doubles: the 4 x 4
// words that a half-warp reads for a fragment lie in 16 different bank pairs). Two CTAs share an SM, so that one reads and
// writes its part of C while the other multiplies. n = 12,288, all updates: 66 ms with scalar multiply-adds and 8 x 8
// outputs a thread, 29.9 ms with fragments and one 128 x 128 tile per SM, 27.2 ms so, 23.5 ms since the factorisation of the
// next diagonal block is shorter than most updates (the fp64 rate gives 16.6).
// Tile row ti has 2 ti + 2 tiles. The first CTA takes both tiles of the next diagonal block and factors it at once.
constexpr int kTileCols = 64, kSliceLd = kKc + 4, kSlices = kNb / kKc, kUpdThreads = 256, kUpdStages = 3;
constexpr int kStageDoubles = (kTile + kTileCols) * kSliceLd;
__device__ __forceinline__ void chol_update_tile(double* __restrict__ A, long n, long k, long i0, long j0, double* sm) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
  const int wi = (warp >> 1) * 32, wj = (warp & 1) * 32;
  // a slice is 128 + 64 rows of 16 doubles, 8 copies of 16 bytes a row; rows past n repeat the last one and are not stored
  auto stage = [&](int slice) {
    double* dst = sm + (slice % kUpdStages) * kStageDoubles;
#pragma unroll
    for (int c = 0; c < (kTile + kTileCols) * kKc / 2 / kUpdThreads; ++c) {
      const int idx = c * kUpdThreads + tid, row = idx >> 3, col = (idx & 7) * 2;
      const long src = min(row < kTile ? i0 + row : j0 + row - kTile, n - 1);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst + row * kSliceLd + col)),
                   "l"(A + src * n + k + slice * kKc + col));
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  double acc[4][4][2];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
#pragma unroll
  for (int s = 0; s < kUpdStages - 1; ++s) stage(s);
#pragma unroll 1
  for (int s = 0; s < kSlices; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kUpdStages - 2) : "memory");
    __syncthreads();  // slice s is there for all, and everyone has left the stage that is filled next
    if (s + kUpdStages - 1 < kSlices) stage(s + kUpdStages - 1);
    else asm volatile("cp.async.commit_group;" ::: "memory");
    const double* Pi = sm + (s % kUpdStages) * kStageDoubles + (wi + g) * kSliceLd + q;
    const double* Pj = sm + (s % kUpdStages) * kStageDoubles + (kTile + wj + g) * kSliceLd + q;
#pragma unroll
    for (int p = 0; p < kKc; p += 4) {
      double a[4], b[4];
#pragma unroll
      for (int x = 0; x < 4; ++x) a[x] = Pi[8 * x * kSliceLd + p], b[x] = Pj[8 * x * kSliceLd + p];
#pragma unroll
      for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y) dmma_8x8x4(acc[x][y], a[x], b[y]);
    }
  }
#pragma unroll
  for (int x = 0; x < 4; ++x) {
    const long i = i0 + wi + 8 * x + g;
    if (i >= n) continue;
    double2 c[4];
#pragma unroll
    for (int y = 0; y < 4; ++y) {
      const long j = j0 + wj + 8 * y + 2 * q;  // even: 16-byte aligned
      c[y] = j < n ? *reinterpret_cast<const double2*>(A + i * n + j) : make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int y = 0; y < 4; ++y) {
      const long j = j0 + wj + 8 * y + 2 * q;
      c[y].x -= acc[x][y][0], c[y].y -= acc[x][y][1];
      if (j < n) *reinterpret_cast<double2*>(A + i * n + j) = c[y];  // above the diagonal: never read
    }
  }
}
__global__ __launch_bounds__(kUpdThreads, 2) void chol_update_kernel(double* __restrict__ A, long n, long k, long r0,
                                                                     double* __restrict__ inv, int* status) {
  extern __shared__ __align__(16) double upd_sm[];
  // linear block index -> tile row ti, tile column cj of the ti (ti + 1) + cj tiles in row order
  const long t = blockIdx.x;
  long ti = long((sqrt(4.0 * double(t) + 1.0) - 1.0) * 0.5);
  while ((ti + 1) * (ti + 2) <= t) ++ti;
  while (ti * (ti + 1) > t) --ti;
  const long cj = t - ti * (ti + 1), j0 = r0 + cj * kTileCols;
  if (t == 1 || j0 >= n) return;  // the first CTA's second tile; columns past the edge
  chol_update_tile(A, n, k, r0 + ti * kTile, j0, upd_sm);
  if (t == 0) {
    __syncthreads();
    if (r0 + kTileCols < n) chol_update_tile(A, n, k, r0, r0 + kTileCols, upd_sm);
    __syncthreads();  // the block is in global memory, and the ring becomes its copy
    chol_diagonal(A, n, r0, upd_sm, inv, status);
  }
}

// L[r][16 bj + j] = sum_{p = j}^{15} C[r][16 bj + p] inv[bj][p][j] for bj < r / 16, zero on and above the diagonal
// block. One thread per row of a column block, the block's inverse in shared memory (broadcast reads); fp32 result,
// optionally the fp64 value beside it.
__global__ __launch_bounds__(128) void ldl_finish_kernel(const double* __restrict__ A, const double* __restrict__ inv,
                                                         long n, float* __restrict__ L, double* __restrict__ L64,
                                                         int* status) {
  __shared__ double iv[256];
  const long bj = blockIdx.y, r = long(blockIdx.x) * blockDim.x + threadIdx.x;
  for (int i = threadIdx.x; i < 256; i += blockDim.x) iv[i] = inv[bj * 256 + i];
  __syncthreads();
  if (r >= n) return;
  float4* out = reinterpret_cast<float4*>(L + r * n + bj * 16);
  double o[16];
  if (bj >= r / 16) {
#pragma unroll
    for (int j = 0; j < 16; ++j) o[j] = 0.0;
  } else {
    const double2* a = reinterpret_cast<const double2*>(A + r * n + bj * 16);
    double av[16];
#pragma unroll
    for (int p = 0; p < 8; ++p) {
      const double2 v = a[p];
      av[2 * p] = v.x, av[2 * p + 1] = v.y;
    }
    bool finite = true;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      double t = 0.0;
#pragma unroll
      for (int p = 0; p < 16; ++p)
        if (p >= j) t = fma(av[p], iv[p * 16 + j], t);
      o[j] = t;
      finite = finite && isfinite(t);
    }
    if (!finite) atomicOr(status, 2);
  }
#pragma unroll
  for (int q = 0; q < 4; ++q)
    out[q] = make_float4(float(o[4 * q]), float(o[4 * q + 1]), float(o[4 * q + 2]), float(o[4 * q + 3]));
  if (L64) {
#pragma unroll
    for (int j = 0; j < 16; ++j) L64[r * n + bj * 16 + j] = o[j];
  }
}

static size_t align256(size_t x) { return (x + 255) / 256 * 256; }
constexpr size_t kFactorSmem = size_t(kNb * (kNb + 1) / 2 + 16 * kInvLd) * 8;
constexpr size_t kUpdSmem = size_t(kUpdStages) * kStageDoubles * 8;
static_assert(kUpdSmem >= kFactorSmem, "the ring of the update is reused for the diagonal block");
constexpr size_t kPanelSmem = size_t(kNb * kLd + (kNb / 16) * 16 * kInvLd + 2 * kPanelRows * kInvLd) * 8;

int block_ldl_device_setup() {
  QB_CUDA(cudaFuncSetAttribute(chol_first_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kFactorSmem)));
  QB_CUDA(cudaFuncSetAttribute(chol_update_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kUpdSmem)));
  QB_CUDA(cudaFuncSetAttribute(chol_panel_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kPanelSmem)));
  return QTIP_OK;
}

}  // namespace qb

using namespace qb;

extern "C" size_t qtip_block_ldl_workspace_bytes(long n) {
  if (n <= 0) return 0;
  return sizeof(LdlHeader) + align256(size_t(n) * n * 8) + align256(size_t(n / 16) * 256 * 8);
}

extern "C" int qtip_block_ldl(const float* HR_d, long n, float* L_d, double* L64_d, void* workspace_d,
                              size_t workspace_bytes, void* stream) {
  QB_REQUIRE(HR_d && L_d && workspace_d, QTIP_E_ARG, "qtip_block_ldl: null pointer");
  QB_REQUIRE(n > 0 && n % 16 == 0, QTIP_E_GEOMETRY, "qtip_block_ldl: n = %ld must be a positive multiple of 16", n);
  QB_REQUIRE(workspace_bytes >= qtip_block_ldl_workspace_bytes(n), QTIP_E_WORKSPACE,
             "qtip_block_ldl: workspace of %zu bytes is too small (need %zu)", workspace_bytes,
             qtip_block_ldl_workspace_bytes(n));
  QB_REQUIRE(reinterpret_cast<uintptr_t>(L_d) % 16 == 0, QTIP_E_ARG, "qtip_block_ldl: L_d must be 16-byte aligned");
  if (!device_info()) return QTIP_E_DEVICE;
  cudaStream_t s = as_stream(stream);
  unsigned char* p = static_cast<unsigned char*>(workspace_d);
  int* status = reinterpret_cast<int*>(p);
  // 16-byte loads: a workspace that is only 8-byte aligned gives up the last 8 of the header's padding
  double* A = reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(p) + sizeof(LdlHeader)) & ~uintptr_t(15));
  double* inv = reinterpret_cast<double*>(reinterpret_cast<unsigned char*>(A) + align256(size_t(n) * n * 8));
  QB_CUDA(cudaMemsetAsync(status, 0, sizeof(LdlHeader), s));
  {
    const unsigned g = blocks_for(n, 32);
    ldl_symmetrise_kernel<<<dim3(g, g), dim3(32, 8), 0, s>>>(HR_d, A, n);
    QB_LAUNCHED();
  }
  chol_first_kernel<<<1, 256, kFactorSmem, s>>>(A, n, inv, status);
  QB_LAUNCHED();
  for (long k = 0; k + kNb < n; k += kNb) {
    const long r0 = k + kNb, nr = n - r0;
    chol_panel_kernel<<<blocks_for(nr, kPanelRows), 256, kPanelSmem, s>>>(A, n, k, inv + k / 16 * 256);
    QB_LAUNCHED();
    const long tiles = (nr + kTile - 1) / kTile;
    chol_update_kernel<<<unsigned(tiles * (tiles + 1)), kUpdThreads, kUpdSmem, s>>>(A, n, k, r0,
                                                                                         inv + r0 / 16 * 256, status);
    QB_LAUNCHED();
  }
  ldl_finish_kernel<<<dim3(blocks_for(n, 128), unsigned(n / 16)), 128, 0, s>>>(A, inv, n, L_d, L64_d, status);
  QB_LAUNCHED();
  return QTIP_OK;
}

extern "C" int qtip_block_ldl_status(const void* workspace_d, void* stream) {
  QB_REQUIRE(workspace_d, QTIP_E_ARG, "qtip_block_ldl_status: null workspace");
  int st = 0;
  QB_CUDA(cudaMemcpyAsync(&st, workspace_d, 4, cudaMemcpyDeviceToHost, as_stream(stream)));
  QB_CUDA(cudaStreamSynchronize(as_stream(stream)));
  QB_REQUIRE((st & 1) == 0, QTIP_E_NUMERIC, "block LDL: the matrix is not positive definite (a pivot was <= 0)");
  QB_REQUIRE((st & 2) == 0, QTIP_E_NUMERIC, "block LDL: non-finite values in the factor");
  return QTIP_OK;
}
