// Batched blocked eigensolver kernels for orders beyond the one-CTA shared-
// memory plan (n up to a few thousand).  A batch of B k-points is reduced
// together, one launch per column step:
//
//   blk_bloch_kernel    H(k) (full Hermitian, from the upper triangle), CTA per tile and four k
//   blk_column_kernel   zlatrd column step (lqm_blocked.cuh), CTA per k
//   blk_symv_kernel     y = A22 v from the lower triangle, 64 x 64 tiles x k,
//                       plus row slabs of the panel products t1, t2; ordered
//                       partials (summed by the next column step)
//   blk_finish_kernel   last w of a panel, CTA per k
//   (host)              rank-2nb trailing update, batched ZGEMM
//   ts_panel_reg_kernel, ts_w_kernel, ts_band_kernel, ts_chase_kernel, ts_q2g_kernel
//                       the two-stage reduction and its back-transformation
//   dc_large_kernel     divide and conquer per k (vectors in global memory,
//                       tiled merge updates), writes bands and Z (complex)
//   dc_root_kernel      the last merge's columns of Z, tiles over all k-points
//   blk_prep_kernel / blk_larft_kernel   compact WY factors per panel
//   (host)              U = (I - V T V^H) U per panel, batched ZGEMMs
//   blk_scale_f_kernel  Y = U diag(f), band energy; (host) rho_k = Y U^H
#pragma once
#include <cuda.h>

#include "lqm_blocked.cuh"
#include "lqm_kernels.cuh"
#include "lqm_twostage.cuh"

namespace lqm {

constexpr int kBlkNB = 32;      // panel width of the reduction (reflectors per panel)
constexpr int kBlkNBT = 64;     // panel width of the compact-WY back-transformation
constexpr int kBlkThreads = 256;
constexpr int kColThreads = 512;  // column step: latency-bound row passes, more rows in flight per k-point
constexpr int kSymvTB = 64;     // mat-vec tile (2 rows per lane of a 32-lane warp)
constexpr int kDcThreads = 512;
constexpr int kDcTileMin = 160; // merges with at least this many rows use the tiled update

struct BlkArgs {
  int n, nb;
  double2* A;    // B x (n x n)
  double2* W;    // B x (n x nb)
  double2* tau;  // B x n
  double* d;     // B x n
  double* e;     // B x n
  double2* t12;  // B x 2nb
  double2* part; // B x part_stride: mat-vec tile partials
  int64_t part_stride;
  double2* tpart;  // B x tpart_stride: panel-product slab partials
  int64_t tpart_stride;
};

// complex per k-point for the panel-product partials: slabs of 128 rows x 2nb
__host__ __device__ inline int64_t t12_part_stride(int n, int nb) {
  const int64_t nsl = (n - 1 + 127) / 128;
  return (nsl < 1 ? 1 : nsl) * 2 * nb;
}

// complex per k-point for the mat-vec partials: nblk^2 tiles of kSymvTB
__host__ __device__ inline int64_t symv_part_stride(int n) {
  const int64_t nbk = (n - 1 + kSymvTB - 1) / kSymvTB;
  return (nbk < 1 ? 1 : nbk * nbk) * kSymvTB;
}

// H(k) = sum_R H_R exp(i 2 pi k.R), from the upper triangle of the blocks: a CTA per 32 x 32
// tile of it and group of four k-points, so that an element of a block is read once for four
// k-points (the groups of a tile follow each other, so that the blocks come from HBM once);
// the mirrored tile is written through shared memory.  Bound by the writes of H(k).  With a
// CTA per k-point every one read all blocks: 6.5 ms at n = 1324 for 100 k-points.
// grid (tiles of the upper triangle x groups), R in slices of kBlochR.
constexpr int kBlochK = 4, kBlochR = 128;
__global__ void __launch_bounds__(kBlkThreads) blk_bloch_kernel(int n, int nR, int dim,
                                                                const double2* __restrict__ blocks,
                                                                const int64_t* __restrict__ keys, int64_t nk,
                                                                const double* __restrict__ ks, double2* A) {
  static_assert(kBlkThreads == 256, "eight warps, four columns each");
  __shared__ __align__(16) double2 ph[kBlochR][kBlochK];
  __shared__ __align__(16) double2 tl[2][32][33];  // [column][row] of the tile, by turns
  const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5;
  const int64_t ngrp = (nk + kBlochK - 1) / kBlochK;
  const int64_t k0 = (int64_t)(blockIdx.x % ngrp) * kBlochK;
  const int p = (int)(blockIdx.x / ngrp);
  int J = (int)((sqrt(8.0 * p + 1.0) - 1.0) * 0.5);  // p-th tile (I, J), I <= J, column by column
  while (J * (J + 1) / 2 > p) --J;
  while ((J + 1) * (J + 2) / 2 <= p) ++J;
  const int I = p - J * (J + 1) / 2;
  const int i = 32 * I + tx;
  const int64_t nn = (int64_t)n * n;
  double2 acc[4][kBlochK];
#pragma unroll
  for (int s = 0; s < 4; ++s)
#pragma unroll
    for (int q = 0; q < kBlochK; ++q) acc[s][q] = cmk(0.0, 0.0);
  for (int r0 = 0; r0 < nR; r0 += kBlochR) {
    const int nr = nR - r0 < kBlochR ? nR - r0 : kBlochR;
    __syncthreads();
    for (int e = tid; e < nr * kBlochK; e += kBlkThreads) {
      const int r = e / kBlochK, q = e % kBlochK;
      double dot = 0.0, s = 0.0, co = 0.0;
      if (k0 + q < nk) {
        for (int c = 0; c < dim; ++c) dot += ks[(k0 + q) * dim + c] * (double)keys[(int64_t)(r0 + r) * dim + c];
        lqm_sincospi(2.0 * dot, &s, &co);
      }
      ph[r][q] = cmk(co, s);
    }
    __syncthreads();
    for (int r = 0; r < nr; ++r) {
      double2 h[4];
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const int j = 32 * J + ty + 8 * s;
        h[s] = (i <= j && j < n) ? blocks[(int64_t)(r0 + r) * nn + i + (int64_t)j * n] : cmk(0.0, 0.0);
      }
#pragma unroll
      for (int q = 0; q < kBlochK; ++q) {
        const double2 f = ph[r][q];
#pragma unroll
        for (int s = 0; s < 4; ++s) acc[s][q] = cadd(acc[s][q], cmul(h[s], f));
      }
    }
  }
#pragma unroll
  for (int q = 0; q < kBlochK; ++q) {
    if (k0 + q >= nk) break;  // uniform
    double2* Ak = A + (k0 + q) * nn;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const int c = ty + 8 * s, j = 32 * J + c;
      if (i == j) acc[s][q].y = 0.0;
      if (i <= j && j < n) Ak[i + (int64_t)j * n] = acc[s][q];
      tl[q & 1][c][tx] = acc[s][q];
    }
    __syncthreads();
#pragma unroll
    for (int s = 0; s < 4; ++s) {  // rows 32 J + tx, column 32 I + c of the lower triangle
      const int c = ty + 8 * s, row = 32 * J + tx, col = 32 * I + c;
      if (row > col && row < n) Ak[row + (int64_t)col * n] = cconj(tl[q & 1][tx][c]);
    }
  }
}

__global__ void __launch_bounds__(kColThreads) blk_column_kernel(BlkArgs a, int j0, int i) {
  __shared__ double red[128];
  __shared__ __align__(16) double2 t12[2 * kBlkNB];
  const Team T = make_team();
  const int64_t b = blockIdx.x;
  const int n = a.n;
  blk_column(T, n, a.nb, j0, i, a.A + b * (int64_t)n * n, n, a.W + b * (int64_t)n * a.nb, n, a.tau + b * n,
             a.d + b * n, a.e + b * n, t12, red, a.part + b * a.part_stride, a.tpart + b * a.tpart_stride);
}

// Last column of a panel: finish its w from the partials.
__global__ void __launch_bounds__(kColThreads) blk_finish_kernel(BlkArgs a, int j0, int ip) {
  __shared__ double red[128];
  __shared__ __align__(16) double2 t12[2 * kBlkNB];
  const Team T = make_team();
  const int64_t b = blockIdx.x;
  const int n = a.n;
  blk_prev_w(T, n, a.nb, j0, ip, a.A + b * (int64_t)n * n, n, a.W + b * (int64_t)n * a.nb, n, a.tau + b * n, t12,
             red, a.part + b * a.part_stride, a.tpart + b * a.tpart_stride, nullptr);
}

// grid (nslabs, B): row slabs of the panel products of column j = j0 + i.
__global__ void __launch_bounds__(kBlkThreads) blk_t12_kernel(BlkArgs a, int j0, int i) {
  const Team T = make_team();
  const int64_t b = blockIdx.y;
  blk_t12_slab(T, a.n, a.nb, j0, i, blockIdx.x, a.A + b * (int64_t)a.n * a.n, a.n, a.W + b * (int64_t)a.n * a.nb, a.n,
               a.tpart + b * a.tpart_stride);
}

// ---- Hermitian mat-vec of one column, persistent and pipelined ----
// The same arithmetic and partial layout as blk_symv_tile (64 x 64 lower
// tiles, direct + transposed partials), but each CTA walks a list of tiles
// (all k-points of the batch) with a kSymvStages-deep cp.async pipeline, so
// that two tiles are in flight from HBM while a third is summed.
constexpr int kSymvStages = 3;
constexpr int kSymvThreads = 512;
constexpr int kSymvLd = kSymvTB + 1;
constexpr int kSymvStageC = kSymvTB * kSymvLd + 2 * kSymvTB;  // complex per stage: tile + v_R, v_C
constexpr int kSymvPipeSmem = (kSymvStages * kSymvStageC + 2 * (kSymvThreads / kSymvTB) * kSymvTB) * 16;
static_assert(kSymvPipeSmem <= 227 * 1024, "mat-vec pipeline exceeds shared memory");

__device__ __forceinline__ void cp_async16(void* sdst, const void* gsrc, bool valid) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(sdst);
  const int nbytes = valid ? 16 : 0;  // 0: the 16 bytes are zero-filled, nothing is read
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gsrc), "r"(nbytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_keep1() { asm volatile("cp.async.wait_group 1;\n" ::: "memory"); }

// tile t of the lower block triangle -> (R, C), R >= C, row-major
__device__ __forceinline__ void symv_tile_rc(int t, int* R, int* C) {
  int r = (int)((sqrt(8.0 * (double)t + 1.0) - 1.0) * 0.5);
  while ((r + 1) * (r + 2) / 2 <= t) ++r;
  while (r * (r + 1) / 2 > t) --r;
  *R = r;
  *C = t - r * (r + 1) / 2;
}

// Issue the copies of work item `it` (k-point it / ntiles, tile it % ntiles)
// into stage buffer `st`; rows/columns beyond m are zero-filled.
__device__ __forceinline__ void symv_issue(const BlkArgs& a, int j, int m, int ntiles, int64_t it, double2* st) {
  const int64_t b = it / ntiles;
  int R, C;
  symv_tile_rc((int)(it - b * ntiles), &R, &C);
  const double2* A = a.A + b * (int64_t)a.n * a.n;
  const double2* B = A + (j + 1) + (int64_t)(j + 1) * a.n;
  const double2* v = A + (j + 1) + (int64_t)j * a.n;
  const int x0 = R * kSymvTB, y0 = C * kSymvTB;
#pragma unroll
  for (int h = 0; h < (kSymvTB * kSymvTB) / kSymvThreads; ++h) {
    const int idx = threadIdx.x + h * kSymvThreads, rr = idx % kSymvTB, cc = idx / kSymvTB;
    const int x = x0 + rr, y = y0 + cc;
    const bool ok = x < m && y < m;
    cp_async16(st + rr + cc * kSymvLd, ok ? (const void*)(B + x + (int64_t)y * a.n) : (const void*)B, ok);
  }
  if (threadIdx.x < 2 * kSymvTB) {
    const int t = threadIdx.x;
    const int x = (t < kSymvTB) ? x0 + t : y0 + (t - kSymvTB);
    cp_async16(st + kSymvTB * kSymvLd + t, x < m ? (const void*)(v + x) : (const void*)v, x < m);
  }
}

// grid: persistent (about one CTA per SM), kSymvPipeSmem dynamic smem.
__global__ void __launch_bounds__(kSymvThreads, 1) blk_symv_pipe_kernel(BlkArgs a, int j, int64_t nitems) {
  extern __shared__ __align__(16) unsigned char smem[];
  double2* stg = (double2*)smem;
  double2* rd = stg + kSymvStages * kSymvStageC;           // [ng][TB] direct
  constexpr int ng = kSymvThreads / kSymvTB;
  double2* rt = rd + ng * kSymvTB;                         // [ng][TB] transposed
  const int m = a.n - j - 1;
  const int nbk = (m + kSymvTB - 1) / kSymvTB;
  const int ntiles = nbk * (nbk + 1) / 2;
  const int64_t first = blockIdx.x, step = gridDim.x;
  // prologue: stages 0 .. kSymvStages-2
#pragma unroll
  for (int s = 0; s < kSymvStages - 1; ++s) {
    const int64_t it = first + s * step;
    if (it < nitems) symv_issue(a, j, m, ntiles, it, stg + s * kSymvStageC);
    cp_async_commit();
  }
  int stage = 0;
  for (int64_t it = first; it < nitems; it += step) {
    cp_async_wait_keep1();  // the group of item `it` has landed (kSymvStages == 3)
    __syncthreads();
    {
      const int64_t nx = it + (kSymvStages - 1) * step;
      const int ns = (stage + kSymvStages - 1) % kSymvStages;
      if (nx < nitems) symv_issue(a, j, m, ntiles, nx, stg + ns * kSymvStageC);
      cp_async_commit();
    }
    const double2* ts = stg + stage * kSymvStageC;
    const double2* vR = ts + kSymvTB * kSymvLd;
    const double2* vC = vR + kSymvTB;
    const int64_t b = it / ntiles;
    int R, C;
    symv_tile_rc((int)(it - b * ntiles), &R, &C);
    const bool diag = (R == C);
    {
      // thread (q, g): direct product of row q and transposed product of column q
      // over u = g, g + ng, ... (two interleaved accumulators each)
      const int q = threadIdx.x % kSymvTB, g = threadIdx.x / kSymvTB;
      double2 ad0 = cmk(0.0, 0.0), ad1 = ad0, at0 = ad0, at1 = ad0;
      if (!diag) {
#pragma unroll
        for (int h = 0; h < kSymvTB / ng; h += 2) {
          const int u0 = g + h * ng, u1 = u0 + ng;
          ad0 = cadd(ad0, cmul(ts[q + u0 * kSymvLd], vC[u0]));
          at0 = cadd(at0, cmulc(ts[u0 + q * kSymvLd], vR[u0]));
          ad1 = cadd(ad1, cmul(ts[q + u1 * kSymvLd], vC[u1]));
          at1 = cadd(at1, cmulc(ts[u1 + q * kSymvLd], vR[u1]));
        }
      } else {
        // lower part only: direct uses columns u <= q (diagonal real), transposed rows u > q
#pragma unroll
        for (int h = 0; h < kSymvTB / ng; ++h) {
          const int u = g + h * ng;
          double2 x = ts[q + u * kSymvLd];
          if (u > q) x = cmk(0.0, 0.0);
          else if (u == q) x.y = 0.0;
          double2 y = ts[u + q * kSymvLd];
          if (u <= q) y = cmk(0.0, 0.0);
          if (h & 1) {
            ad1 = cadd(ad1, cmul(x, vC[u]));
            at1 = cadd(at1, cmulc(y, vR[u]));
          } else {
            ad0 = cadd(ad0, cmul(x, vC[u]));
            at0 = cadd(at0, cmulc(y, vR[u]));
          }
        }
      }
      rd[threadIdx.x] = cadd(ad0, ad1);
      rt[threadIdx.x] = cadd(at0, at1);
    }
    __syncthreads();
    if (threadIdx.x < kSymvTB) {
      const int x = threadIdx.x;
      double2 yd = cmk(0.0, 0.0), yt = cmk(0.0, 0.0);
#pragma unroll
      for (int g = 0; g < ng; ++g) {
        yd = cadd(yd, rd[g * kSymvTB + x]);
        yt = cadd(yt, rt[g * kSymvTB + x]);
      }
      double2* part = a.part + b * a.part_stride;
      if (diag) {
        part[((int64_t)R * nbk + C) * kSymvTB + x] = cadd(yd, yt);
      } else {
        part[((int64_t)R * nbk + C) * kSymvTB + x] = yd;
        part[((int64_t)C * nbk + R) * kSymvTB + x] = yt;
      }
    }
    stage = (stage + 1) % kSymvStages;
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// ---- Hermitian mat-vec of one column, tiles moved by TMA ----
// The same partial layout as blk_symv_pipe_kernel, with each 64 x 64 lower tile
// brought into shared memory by eight 3-D tensor copies (cp.async.bulk.tensor:
// box = 8 complex rows x 64 columns x 1 k-point, 128-byte swizzle) that complete
// on one mbarrier per stage, issued by one thread; rows and columns beyond the
// matrix read as zeros (out-of-bounds fill), so the tensor map covers the whole
// batch for every column.
// Each tile element is read from shared memory once and used for both products:
// warp w owns the 16 x 16 sub-block (rows 16 (w % 4) .., columns 16 (w / 4) ..);
// lane (a = lane % 8, b = lane / 8) holds rows a, a + 8 and columns b + 4 i
// (i < 4) of it (with the swizzle, the eight lanes of each load phase hit eight
// distinct 16-byte bank groups).  The direct partials (row sums over the lane's
// columns) are reduced over b and the transposed ones (column sums over its rows)
// over a, by reduce-scatter shuffles (each step halves what a lane keeps), then
// written to a double-buffered slot per warp; after the next tile's barrier the
// four column- (row-) blocks of each row (column) are added in order and written
// out.  So there is one block barrier per tile.  Every mbarrier wait is bounded;
// on expiry the kernel sets *err and stops (the host reports LQM_EDEVICE).
constexpr int kSymvTmaThreads = 512;
constexpr int kSymvTmaStages = 3;
constexpr int kSymvTileBytes = kSymvTB * kSymvTB * 16;  // 64 KB
constexpr int kSymvVecBytes = 2 * kSymvTB * 16;               // v over the tile's rows, then over its columns
constexpr int kSymvRedBytes = 2 * 2 * 4 * kSymvTB * 16;  // [buffer][direct, transposed][block][64] complex
constexpr int kSymvTmaSmem = kSymvTmaStages * (kSymvTileBytes + kSymvVecBytes) + kSymvRedBytes +
                             1024 /* alignment */ + 64 /* mbarriers */;
static_assert(kSymvTmaSmem <= 227 * 1024, "TMA mat-vec pipeline exceeds shared memory");
constexpr long long kSymvWaitLimit = 1LL << 22;  // mbarrier polls before giving up (well under a second)

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned bar, unsigned parity) {
  unsigned done;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}
// bounded wait: false when the limit ran out
__device__ __forceinline__ bool mbar_wait_bounded(unsigned bar, unsigned parity) {
  for (long long i = 0; i < kSymvWaitLimit; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}
__device__ __forceinline__ void tma_load_3d(unsigned dst, const CUtensorMap* map, int c0, int c1, int c2,
                                            unsigned bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
      "[%5];\n" ::"r"(dst),
      "l"((unsigned long long)map), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
      : "memory");
}

// byte offset of element (row r, column c) of a staged tile (eight swizzled boxes)
__device__ __forceinline__ int symv_sw(int r, int c) {
  return ((r >> 3) << 13) + (c << 7) + ((((r & 7) ^ (c & 7))) << 4);
}

// The tile of work item `it` (eight boxes) and the two 64-element segments of the
// reflector v = A(j+1:, j) it multiplies (rows of the tile's row block and of its
// column block; one box each from the vector map), all on the stage's mbarrier.
__device__ __forceinline__ void symv_tma_issue(const CUtensorMap* map, const CUtensorMap* vmap, int j, int ntiles,
                                               int64_t it, unsigned dst, unsigned vdst, unsigned bar) {
  const int64_t b = it / ntiles;
  int R, C;
  symv_tile_rc((int)(it - b * ntiles), &R, &C);
  mbar_arrive_expect_tx(bar, (unsigned)(kSymvTileBytes + kSymvVecBytes));
  const int row0 = j + 1 + R * kSymvTB, col0 = j + 1 + C * kSymvTB;
#pragma unroll
  for (int bx = 0; bx < kSymvTB / 8; ++bx)
    tma_load_3d(dst + (unsigned)(bx << 13), map, 2 * (row0 + 8 * bx), col0, (int)b, bar);
  tma_load_3d(vdst, vmap, 2 * row0, j, (int)b, bar);
  tma_load_3d(vdst + kSymvTB * 16, vmap, 2 * col0, j, (int)b, bar);
}

// Finish of one tile from its warp partials (red: [direct, transposed][block][64 rows]
// complex, as doubles): thread t < 256 adds the four blocks of output o = t / 2,
// component t % 2, in block order; outputs 0..63 are the direct rows, 64..127 the
// transposed columns (on a diagonal tile both go to the same row, summed).
__device__ __forceinline__ void symv_tma_finish(const double* red, double2* part, int nbk, int R, int C) {
  const int t = threadIdx.x;
  if (t >= 2 * 2 * kSymvTB) return;
  const int o = t >> 1, comp = t & 1;
  const bool diag = (R == C);
  if (diag && o >= kSymvTB) return;
  const int kind = o >= kSymvTB ? 1 : 0, x = o & (kSymvTB - 1);
  const double* src = red + kind * (4 * kSymvTB * 2) + x * 2 + comp;
  double v = src[0];
#pragma unroll
  for (int q = 1; q < 4; ++q) v += src[q * kSymvTB * 2];
  if (diag) {
    const double* s2 = red + 4 * kSymvTB * 2 + x * 2 + comp;
    double w = s2[0];
#pragma unroll
    for (int q = 1; q < 4; ++q) w += s2[q * kSymvTB * 2];
    v += w;
  }
  double* dst = (double*)(part + ((int64_t)(kind ? C : R) * nbk + (kind ? R : C)) * kSymvTB + x);
  dst[comp] = v;
}

__global__ void __launch_bounds__(kSymvTmaThreads, 1)
    blk_symv_tma_kernel(const __grid_constant__ CUtensorMap map, const __grid_constant__ CUtensorMap vmap, BlkArgs a,
                        int j, int64_t nitems, int* err) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const unsigned raw = smem_u32(smem_raw);
  const unsigned base = (raw + 1023u) & ~1023u;                // 1024-byte aligned tiles (128-byte swizzle)
  unsigned char* tiles = smem_raw + (base - raw);
  const unsigned vbase = base + kSymvTmaStages * kSymvTileBytes;  // v segments of each stage
  const unsigned char* vsm = tiles + kSymvTmaStages * kSymvTileBytes;
  double* redsm = (double*)(tiles + kSymvTmaStages * (kSymvTileBytes + kSymvVecBytes));  // 2 buffers
  const unsigned bars = vbase + kSymvTmaStages * kSymvVecBytes + kSymvRedBytes;  // one mbarrier per stage
  const int m = a.n - j - 1;
  const int nbk = (m + kSymvTB - 1) / kSymvTB;
  const int ntiles = nbk * (nbk + 1) / 2;
  const int64_t first = blockIdx.x, step = gridDim.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int la = lane & 7, lb = lane >> 3;
  const int rw = (warp & 3) * 16, cw = (warp >> 2) * 16;  // the warp's sub-block
  if (*(volatile int*)err != 0) return;  // an earlier launch gave up: the pass is void, end at once
  if (threadIdx.x == 0) {
    for (int s = 0; s < kSymvTmaStages; ++s) mbar_init(bars + 8 * s, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int s = 0; s < kSymvTmaStages - 1; ++s) {
      const int64_t it = first + s * step;
      if (it < nitems)
        symv_tma_issue(&map, &vmap, j, ntiles, it, base + s * kSymvTileBytes, vbase + s * kSymvVecBytes, bars + 8 * s);
    }
  }
  int stage = 0;
  unsigned parity = 0;
  int64_t pk = -1;               // k-point of the previous tile (finished after this tile's barrier), or -1
  int pR = 0, pC = 0;
  int rb = 0;                    // reduction buffer of this tile
  for (int64_t it = first; it < nitems; it += step) {
    const int64_t b = it / ntiles;
    int R, C;
    symv_tile_rc((int)(it - b * ntiles), &R, &C);
    // the stage's copies have landed, and every thread is past the previous tile (so
    // its stage may be refilled and its partials read); the outcome of the bounded
    // wait is the block's
    const int ok = __syncthreads_and(mbar_wait_bounded(bars + 8 * stage, parity) ? 1 : 0);
    if (!ok) {
      if (threadIdx.x == 0) {
        atomicExch(err, 1);
        // leave no copy in flight: the stage of this item and, if issued, the next one
        mbar_wait_bounded(bars + 8 * stage, parity);
        if (it + step < nitems) {
          const int s1 = (stage + 1) % kSymvTmaStages;
          mbar_wait_bounded(bars + 8 * s1, s1 == 0 ? parity ^ 1u : parity);
        }
      }
      return;
    }
    if (threadIdx.x == 0) {
      const int64_t nx = it + (kSymvTmaStages - 1) * step;
      const int ns = (stage + kSymvTmaStages - 1) % kSymvTmaStages;
      if (nx < nitems)
        symv_tma_issue(&map, &vmap, j, ntiles, nx, base + ns * kSymvTileBytes, vbase + ns * kSymvVecBytes,
                       bars + 8 * ns);
    }
    if (pk >= 0) symv_tma_finish(redsm + (rb ^ 1) * (2 * 4 * kSymvTB * 2), a.part + pk * a.part_stride, nbk, pR, pC);
    const unsigned char* ts = tiles + stage * kSymvTileBytes;
    const double2* vR = (const double2*)(vsm + stage * kSymvVecBytes);  // zeros past the matrix edge
    const double2* vC = vR + kSymvTB;
    const bool diag = (R == C);
    const int r0 = rw + la, r1 = r0 + 8;
    const double2 vr0 = vR[r0], vr1 = vR[r1];
    double2 yd0 = cmk(0.0, 0.0), yd1 = yd0, yt[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int u = cw + lb + 4 * i;
      const double2 vc = vC[u];
      double2 e0 = *(const double2*)(ts + symv_sw(r0, u));
      double2 e1 = *(const double2*)(ts + symv_sw(r1, u));
      double2 f0 = e0, f1 = e1;  // the transposed product's copies
      if (diag) {  // lower part only: direct uses u <= row (diagonal real), transposed u < row
        if (u > r0) e0 = cmk(0.0, 0.0); else if (u == r0) e0.y = 0.0;
        if (u > r1) e1 = cmk(0.0, 0.0); else if (u == r1) e1.y = 0.0;
        if (u >= r0) f0 = cmk(0.0, 0.0);
        if (u >= r1) f1 = cmk(0.0, 0.0);
      }
      yd0 = cadd(yd0, cmul(e0, vc));
      yd1 = cadd(yd1, cmul(e1, vc));
      yt[i] = cadd(cmulc(f0, vr0), cmulc(f1, vr1));
    }
    constexpr unsigned FULL = 0xffffffffu;
    // direct: reduce over lb (lane bits 3, 4); the lane keeps row r0 + 8 (lb & 1), component lb >> 1
    double dk;
    {
      const bool h = lb & 1;
      double k0 = h ? yd1.x : yd0.x, k1 = h ? yd1.y : yd0.y;
      const double s0 = h ? yd0.x : yd1.x, s1 = h ? yd0.y : yd1.y;
      k0 += __shfl_xor_sync(FULL, s0, 8);
      k1 += __shfl_xor_sync(FULL, s1, 8);
      const bool h2 = lb & 2;
      dk = h2 ? k1 : k0;
      dk += __shfl_xor_sync(FULL, h2 ? k0 : k1, 16);
    }
    // transposed: reduce over la (lane bits 0..2); the lane keeps column
    // cw + lb + 4 (2 (la & 1) + ((la >> 1) & 1)), component (la >> 2) & 1
    double tk;
    {
      const bool g0 = la & 1;
      double q0 = g0 ? yt[2].x : yt[0].x, q1 = g0 ? yt[2].y : yt[0].y;
      double q2 = g0 ? yt[3].x : yt[1].x, q3 = g0 ? yt[3].y : yt[1].y;
      const double s0 = g0 ? yt[0].x : yt[2].x, s1 = g0 ? yt[0].y : yt[2].y;
      const double s2 = g0 ? yt[1].x : yt[3].x, s3 = g0 ? yt[1].y : yt[3].y;
      q0 += __shfl_xor_sync(FULL, s0, 1);
      q1 += __shfl_xor_sync(FULL, s1, 1);
      q2 += __shfl_xor_sync(FULL, s2, 1);
      q3 += __shfl_xor_sync(FULL, s3, 1);
      const bool g1 = la & 2;
      double p0 = g1 ? q2 : q0, p1 = g1 ? q3 : q1;
      const double u0 = g1 ? q0 : q2, u1 = g1 ? q1 : q3;
      p0 += __shfl_xor_sync(FULL, u0, 2);
      p1 += __shfl_xor_sync(FULL, u1, 2);
      const bool g2 = la & 4;
      tk = g2 ? p1 : p0;
      tk += __shfl_xor_sync(FULL, g2 ? p0 : p1, 4);
    }
    {
      double* red = redsm + rb * (2 * 4 * kSymvTB * 2);
      const int xr = r0 + 8 * (lb & 1), cd = lb >> 1;
      red[((warp >> 2) * kSymvTB + xr) * 2 + cd] = dk;
      const int xc = cw + lb + 4 * (2 * (la & 1) + ((la >> 1) & 1)), ct = (la >> 2) & 1;
      red[((4 + (warp & 3)) * kSymvTB + xc) * 2 + ct] = tk;
    }
    pk = b; pR = R; pC = C;
    rb ^= 1;
    stage = (stage + 1) % kSymvTmaStages;
    if (stage == 0) parity ^= 1u;
  }
  __syncthreads();
  if (pk >= 0) symv_tma_finish(redsm + (rb ^ 1) * (2 * 4 * kSymvTB * 2), a.part + pk * a.part_stride, nbk, pR, pC);
}

// off: the row offset of the reflectors (1 one-stage, the half-bandwidth two-stage)
__global__ void __launch_bounds__(kBlkThreads) blk_prep_kernel(int n, double2* A, int off) {
  const Team T = make_team();
  blk_prep_reflectors(T, n, A + (int64_t)blockIdx.x * n * n, n, off);
}

// grid (P, B); Tm: B x P x (nb x nb); dynamic smem: G (nb x nb double2); Gg: the
// Gram matrices V_p^H V_p laid out as Tm, or null (formed in the kernel)
// off: the row offset of the reflectors; their count is n - off
__global__ void __launch_bounds__(kBlkThreads) blk_larft_kernel(int n, int nb, int P, const double2* A,
                                                                const double2* tau, double2* Tm,
                                                                const double2* Gg, int off) {
  extern __shared__ __align__(16) unsigned char smem[];
  const Team T = make_team();
  const int p = blockIdx.x;
  const int64_t b = blockIdx.y;
  const int j0 = p * nb;
  int nbr = n - off - j0;
  if (nbr > nb) nbr = nb;
  double2* Tp = Tm + (b * P + p) * (int64_t)nb * nb;
  if (nbr <= 0) {
    for (int q = T.tid; q < nb * nb; q += T.nt) Tp[q] = cmk(0.0, 0.0);
    return;
  }
  blk_larft(T, n, nb, j0, nbr, A + b * (int64_t)n * n, n, tau + b * n, Tp, (double2*)smem,
            Gg ? Gg + (b * P + p) * (int64_t)nb * nb : nullptr, off);
}

struct DCLargeArgs {
  int n;
  int64_t nk;
  DCPlan plan;
  const double* d;   // nk x n (hetrd diagonal)
  const double* e;   // nk x n (subdiagonal, n-1 used)
  double* bands;     // nk x n
  double2* U;        // nk x (n x n): Z as complex, or null (eigenvalues only)
  double* slots;     // gridDim.x slots
  int64_t slot_doubles;
  unsigned long long* phase_cycles;  // [16] as eigh_kernel's (d&c total and merge steps), or null
  double* Qk;        // nk x (n x n): the vectors before the last merge, left to dc_root_kernel with
  double* rec;       // nk x dc_root_rec_doubles(n); or null (U is written here)
};

// doubles of one k-point's record of its last merge (DCRootRec)
__host__ __device__ inline int64_t dc_root_rec_doubles(int n) { return 5 * (int64_t)n + (2 * (int64_t)n + 4 + 1) / 2; }
__host__ __device__ inline DCRootRec dc_root_rec(double* p, int n) {
  DCRootRec r;
  r.zh = p; r.dl = p + n; r.lorg = p + 2 * (int64_t)n; r.tq = p + 3 * (int64_t)n; r.sc = p + 4 * (int64_t)n;
  r.cidx = (int*)(p + 5 * (int64_t)n); r.src = r.cidx + n; r.hdr = r.src + n;
  return r;
}

__host__ __device__ inline int64_t dc_large_slot_doubles(int n, bool vec) {
  const int64_t nn = (int64_t)n * n;
  const int64_t vecs = 13 * (int64_t)n + 8 + (10 * (int64_t)n + 1) / 2 + 1 + 2 * (int64_t)(kDcThreads / 32) * n + 2;
  return (vec ? 3 * nn : 4 * (int64_t)n + 4) + vecs;
}

// dynamic shared memory: the merge GEMM's cp.async ring and the column indices of one merge
__host__ __device__ inline int dc_tile_smem(int n) { return kDcTileRing * 8 + ((n + 3) / 4) * 16; }

// NT = 512 (one CTA per SM) for orders with tiled merges; below kDcTileMin the
// merges are small and latency-bound, and NT = 128 with four CTAs per SM keeps
// four k-points in flight per SM.
template <int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) dc_large_kernel(DCLargeArgs a) {
  __shared__ double red[128];
  extern __shared__ __align__(16) double tile[];
  const Team T = make_team();
  const int n = a.n;
  const bool vec = a.U != nullptr;
  const int64_t nn = (int64_t)n * n;
  double* slot = a.slots + (int64_t)blockIdx.x * a.slot_doubles;
  double* Q = slot;
  double* Qt = vec ? Q + nn : nullptr;
  double* Ub = vec ? Q + 2 * nn : nullptr;
  double* db = slot + (vec ? 3 * nn : 4 * (int64_t)n + 4);
  EighVec S;
  S.d = db; S.e = db + n; S.D = db + 2 * n; S.z = db + 3 * n; S.dl = db + 4 * n; S.zl = db + 5 * n;
  S.troot = db + 6 * n; S.zhat = db + 7 * n; S.vals = db + 8 * n; S.dval = db + 9 * n; S.rc = db + 10 * n;
  S.rs = db + 11 * n; S.nrho = db + 12 * n;
  S.red = red;
  int* ib = (int*)(db + 13 * (int64_t)n + 8);
  S.perm = ib; S.colnd = ib + n; S.org = ib + 2 * n; S.dcol = ib + 3 * n; S.newpos = ib + 4 * n;
  S.ri = ib + 5 * n; S.rj = ib + 6 * n; S.nk = ib + 7 * n; S.nrot = ib + 8 * n; S.ndef = ib + 9 * n;
  double* pb = db + 13 * (int64_t)n + 8 + (10 * (int64_t)n + 1) / 2 + 1;
  S.pbuf = (double2*)(((uintptr_t)pb + 15) & ~(uintptr_t)15);
  S.tau = S.v = S.w = S.vn = S.pn = S.bc = nullptr;
  S.tile = tile;
  DCRootRec rec;
  const bool prof = a.phase_cycles != nullptr;
  unsigned long long dsub[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  unsigned long long dtot = 0;
  for (int64_t k = blockIdx.x; k < a.nk; k += gridDim.x) {
    for (int i = T.tid; i < n; i += T.nt) {
      S.d[i] = a.d[k * n + i];
      S.e[i] = (i < n - 1) ? a.e[k * n + i] : 0.0;
    }
    team_sync();
    const long long t0 = prof ? clock64() : 0;
    if (a.Qk) {
      Q = a.Qk + k * nn;
      rec = dc_root_rec(a.rec + k * dc_root_rec_doubles(n), n);
    }
    dc_solve(T, n, a.plan, S, Q, Qt, prof ? dsub : nullptr, vec, Ub, kDcTileMin, a.Qk ? &rec : nullptr);
    if (prof) dtot += (unsigned long long)(clock64() - t0);
    for (int i = T.tid; i < n; i += T.nt) a.bands[k * n + i] = S.D[i];
    if (vec && !a.Qk) {
      double2* Uk = a.U + k * nn;
      for (int c = T.wid; c < n; c += T.nw)
        for (int r = T.lane; r < n; r += T.nl) Uk[r + (int64_t)c * n] = cmk(Q[r + (int64_t)c * n], 0.0);
    }
    team_sync();
  }
  if (prof && T.tid == 0) {
    atomicAdd(&a.phase_cycles[PH_DC], dtot);
    for (int i = 0; i < 8; ++i) atomicAdd(&a.phase_cycles[PH_DCSUB + i], dsub[i]);
  }
}

// The last merge of every k-point: columns c0 .. c0 + K - 1 of its eigenvectors, as complex
// numbers, from the vectors before it (Q) and its record.  The work of dc_tile_gemm (same order
// of the poles, each child's rows over its own and the shared ones), but over all SMs however few the k-points are,
// only for the wanted columns, and with the secular vectors formed as the B tile is
// staged.  grid (ceil(K / 64), row tiles of both children, nk): 128 x 64 tiles, eight warps of
// 32 x 32, a ring of three 16-deep stages.  Three quarters of all merge products are this one.
// Bound by the FP64 tensor path.  With it (and the halved sums below it) the density matrix
// took 331 ms against 363 at n = 1324 on 144 k-points and 919 against 1232 at n = 2884 on 36,
// where one block per k-point left three quarters of the SMs idle.
constexpr int kDcRootThreads = 256;
constexpr int kDcRootPA = 132, kDcRootPB = 68;  // pitches == 4 mod 16: conflict-free fragment reads
constexpr int kDcRootStage = 16 * (kDcRootPA + kDcRootPB);
constexpr int kDcRootSmem = 3 * kDcRootStage * 8;
__host__ __device__ inline int dc_root_row_tiles(int n, int mid) { return (mid + 127) / 128 + (n - mid + 127) / 128; }
__global__ void __launch_bounds__(kDcRootThreads, 2) dc_root_kernel(int n, int mid, int c0, int K, const double* Qk,
                                                                    const double* recs, double2* U) {
  extern __shared__ __align__(16) double rtile[];
  constexpr int BK = 16, PA = kDcRootPA, PB = kDcRootPB;
  const int64_t b = blockIdx.z;
  const DCRootRec rec = dc_root_rec((double*)recs + b * dc_root_rec_doubles(n), n);
  const double* Q = Qk + b * (int64_t)n * n;
  double2* Uk = U + b * (int64_t)n * n;
  const int k = rec.hdr[0], nu = rec.hdr[1], nm = rec.hdr[2];
  const int tu = (mid + 127) / 128, rt = blockIdx.y;
  const int r0 = rt < tu ? rt * 128 : mid + (rt - tu) * 128;
  const int rend = rt < tu ? mid : n;
  const int pb = rt < tu ? 0 : nu, pe = rt < tu ? nm : k;
  const int cb = c0 + blockIdx.x * 64, cend = c0 + K;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int wr = (warp & 3) * 32, wc = (warp >> 2) * 32;
  // B: thread's column of the tile (fixed) and rows tid / 64 + 4 h of a stage
  const int bc = cb + (tid & 63);
  const bool bok = bc < cend && rec.src[bc] < 0;
  const double lorg = bok ? rec.lorg[bc] : 0.0, tq = bok ? rec.tq[bc] : 0.0, sc = bok ? rec.sc[bc] : 0.0;
  auto stage_a = [&](int p0, int st) {
    double* As = rtile + st * kDcRootStage;
#pragma unroll
    for (int h = 0; h < 8; ++h) {
      const int pp = (tid >> 7) + 2 * h, x = tid & 127, p = p0 + pp, r = r0 + x;
      const bool ok = p < pe && r < rend;
      lqm_cp_async8(As + pp * PA + x, ok ? (const void*)(Q + r + (int64_t)rec.cidx[p] * n) : (const void*)Q, ok);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  auto stage_b = [&](int p0, int st) {
    double* Bs = rtile + st * kDcRootStage + 16 * PA;
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const int pp = (tid >> 6) + 4 * h, p = p0 + pp;
      double u = 0.0;
      if (bok && p < pe) u = lqm_div_normal(rec.zh[p], (rec.dl[p] - lorg) - tq) * sc;
      Bs[pp * PB + (tid & 63)] = u;
    }
  };
  double acc[4][4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  const int nst = (pe - pb + BK - 1) / BK;
  stage_a(pb, 0);
  stage_a(pb + BK, 1);
  stage_b(pb, 0);
  for (int it = 0; it < nst; ++it) {
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    __syncthreads();  // stage it is in place; stages it + 1 (B) and it + 2 (A) are free to be filled
    stage_a(pb + (it + 2) * BK, (it + 2) % 3);
    if (it + 1 < nst) stage_b(pb + (it + 1) * BK, (it + 1) % 3);
    const double* As = rtile + (it % 3) * kDcRootStage;
    const double* Bs = As + 16 * PA;
#pragma unroll
    for (int kk = 0; kk < BK; kk += 4) {
      double av[4], bv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) av[i] = As[(kk + t) * PA + wr + 8 * i + g];
#pragma unroll
      for (int j = 0; j < 4; ++j) bv[j] = Bs[(kk + t) * PB + wc + 8 * j + g];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) dmma_884(acc[i][j][0], acc[i][j][1], av[i], bv[j]);
    }
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int c = cb + wc + 8 * j + 2 * t + h;
      if (c >= cend) continue;
      const int src = rec.src[c];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = r0 + wr + 8 * i + g;
        if (r < rend) Uk[r + (int64_t)c * n] = cmk(src < 0 ? acc[i][j][h] : Q[r + (int64_t)src * n], 0.0);
      }
    }
}

// Y[k] = U[k] diag(f(eps - mu)) and eband_k = w_k sum_j f_j eps_j; CTA per k.
__global__ void __launch_bounds__(kBlkThreads) blk_scale_f_kernel(int n, int64_t nk, const double2* U,
                                                                  const double* bands, double mu_val,
                                                                  const double* mu_ptr, double T_,
                                                                  const double* w, double2* Y,
                                                                  double* eband_k) {
  __shared__ double red[128];
  extern __shared__ __align__(16) unsigned char smem[];
  double* f = (double*)smem;
  const Team T = make_team();
  const int64_t k = blockIdx.x;
  const double mu = mu_ptr ? *mu_ptr : mu_val;
  const int64_t nn = (int64_t)n * n;
  double eb = 0.0;
  for (int j = T.tid; j < n; j += T.nt) {
    const double ej = bands[k * n + j];
    const double fj = fermi(ej - mu, T_);
    f[j] = fj;
    eb += ej * fj;
  }
  eb = team_sum(T, eb, red);
  if (T.tid == 0 && eband_k) eband_k[k] = w[k] * eb;
  for (int c = T.wid; c < n; c += T.nw) {
    const double fc = f[c];
    for (int r = T.lane; r < n; r += T.nl) Y[k * nn + r + (int64_t)c * n] = cscale(fc, U[k * nn + r + (int64_t)c * n]);
  }
}

// Occupation span of each k-point's states (eigenvalues ascending, so the exactly
// filled states, f == 1, form a prefix and the exactly empty ones, f == 0, a suffix):
// span[0] = max over k of the states that are not exactly filled, span[1] = max over k
// of the states that are not exactly empty (integer maxima: order-independent).
__global__ void __launch_bounds__(kBlkThreads) blk_occ_span_kernel(int n, const double* bands, double mu,
                                                                   double T_, int* span) {
  __shared__ int cnt[2];
  const int64_t k = blockIdx.x;
  if (threadIdx.x < 2) cnt[threadIdx.x] = 0;
  __syncthreads();
  int notfull = 0, notempty = 0;
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    const double fj = fermi(bands[k * n + j] - mu, T_);
    notfull += fj != 1.0;
    notempty += fj != 0.0;
  }
  atomicAdd(&cnt[0], notfull);
  atomicAdd(&cnt[1], notempty);
  __syncthreads();
  if (threadIdx.x == 0) {
    atomicMax(&span[0], cnt[0]);
    atomicMax(&span[1], cnt[1]);
  }
}

// rho_k from the K columns [c0, c0 + K) of U that carry it: Y[:, c] = U[:, c0 + c] f
// (direct: the first K states hold every nonzero f) or U[:, c0 + c] (1 - f)
// (complement: the last K states hold every f < 1, rho_k = I - Y U_K^H); the band
// energy sum_j w f_j eps_j over all states as blk_scale_f_kernel computes it.
__global__ void __launch_bounds__(kBlkThreads) blk_scale_f_cols_kernel(int n, const double2* U, const double* bands,
                                                                       double mu, double T_, const double* w,
                                                                       double2* Y, double* eband_k, int c0, int K,
                                                                       int complement) {
  __shared__ double red[128];
  extern __shared__ __align__(16) unsigned char smem[];
  double* f = (double*)smem;
  const Team T = make_team();
  const int64_t k = blockIdx.x;
  const int64_t nn = (int64_t)n * n;
  double eb = 0.0;
  for (int j = T.tid; j < n; j += T.nt) {
    const double ej = bands[k * n + j];
    const double fj = fermi(ej - mu, T_);
    f[j] = fj;
    eb += ej * fj;
  }
  eb = team_sum(T, eb, red);
  if (T.tid == 0 && eband_k) eband_k[k] = w[k] * eb;
  for (int c = T.wid; c < K; c += T.nw) {
    const double fc = complement ? 1.0 - f[c0 + c] : f[c0 + c];
    const double2* Uc = U + k * nn + (int64_t)(c0 + c) * n;
    double2* Yc = Y + k * nn + (int64_t)c * n;
    for (int r = T.lane; r < n; r += T.nl) Yc[r] = cscale(fc, Uc[r]);
  }
}

// rho_k is Hermitian and only its lower column blocks are formed: the strictly upper
// part of each 32 x 32 tile pair (I < J) is the conjugate transpose of tile (J, I),
// moved through shared memory so both the reads and the writes are coalesced.
// grid (tiles above the diagonal (J > I) of the 32-tile grid, nk).
__global__ void __launch_bounds__(256) blk_herm_mirror_kernel(int n, double2* R) {
  __shared__ double2 t[32][33];
  const int nt = (n + 31) / 32;
  int p = blockIdx.x, I = 0;  // p-th pair (I, J), J > I, row-major over I
  while (p >= nt - 1 - I) { p -= nt - 1 - I; ++I; }
  const int J = I + 1 + p;
  double2* Rk = R + (int64_t)blockIdx.y * n * n;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
  // read tile (J, I) of the lower part: rows 32J + tx, columns 32I + c
  for (int c = ty; c < 32; c += 8) {
    const int r = 32 * J + tx, col = 32 * I + c;
    if (r < n && col < n) t[c][tx] = Rk[r + (int64_t)col * n];
  }
  __syncthreads();
  // write tile (I, J): rows 32I + tx, columns 32J + c, value conj(R[32J + c, 32I + tx])
  for (int c = ty; c < 32; c += 8) {
    const int r = 32 * I + tx, col = 32 * J + c;
    if (r < n && col < n) Rk[r + (int64_t)col * n] = cconj(t[tx][c]);
  }
}

// rho_k = I - (Y U_K^H): the identity added to the diagonal (complement form).
__global__ void __launch_bounds__(kBlkThreads) blk_add_identity_kernel(int n, double2* R) {
  const int64_t nn = (int64_t)n * n;
  double2* Rk = R + blockIdx.x * nn;
  for (int i = threadIdx.x; i < n; i += blockDim.x) Rk[i + (int64_t)i * n].x += 1.0;
}


// ---- Two-stage reduction (lqm_twostage.cuh) ----
constexpr int kTsB = 16;              // half-bandwidth of the stage-1 band
constexpr int kTsPanelThreads = 512;  // panel QR: latency-bound row passes, CTA per k-point
constexpr int kTsWaitPolls = 1 << 26; // bound of one inter-warp wait of the chase (shared-memory polls, ~1 s)

// complex per k-point of the stage-2 reflector store (sweeps 0..n-2, tmax slots of kTsB each)
__host__ __device__ inline int64_t ts_v2_stride(int n) {
  return (int64_t)(n > 1 ? n - 1 : 1) * ts_tmax(n, kTsB) * kTsB;
}
__host__ __device__ inline int64_t ts_tau2_stride(int n) { return (int64_t)(n > 1 ? n - 1 : 1) * ts_tmax(n, kTsB); }

// grid (B): panel j0 of every k-point.  Vb: B x (n x kTsB), Tm: B x (kTsB x kTsB).
__global__ void __launch_bounds__(kTsPanelThreads) ts_panel_kernel(int n, int j0, double2* A, double2* tau,
                                                                   double2* Vb, double2* Tm) {
  __shared__ __align__(16) double2 sm[(kTsPanelThreads / 32 + 2) * kTsB + kTsB * kTsB];
  const Team T = make_team();
  const int64_t b = blockIdx.x;
  ts_panel_qr<kTsB>(T, n, j0, A + b * (int64_t)n * n, n, tau + b * n, Vb + b * (int64_t)n * kTsB, n,
                    Tm + b * kTsB * kTsB, sm);
}

// ---- cluster helpers (all blocks of a cluster work on one k-point) ----
__device__ __forceinline__ void cluster_barrier() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// store 16 bytes at the shared-memory address of block `rank` that corresponds to p
__device__ __forceinline__ void cluster_st16(void* p, int rank, double2 v) {
  unsigned ra;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(ra) : "r"(smem_u32(p)), "r"(rank));
  asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};\n" ::"r"(ra), "d"(v.x), "d"(v.y) : "memory");
}

// Sums of 16 values over the warp: every lane gets the total of value lane % 16
// (an exchange tree: 16 shuffles instead of 80).
__device__ __forceinline__ double warp_sum16(double (&v)[16], int lane) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1)
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const bool up = lane & o;
      const double keep = up ? v[i + o] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, up ? v[i] : v[i + o], o);
    }
  return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 16);
}

// The panel factorisation of ts_panel_qr with the panel in registers: thread = one row of
// the panel (16 complex), a cluster of cs = ceil(m / 512) blocks per k-point, each with its
// share of the rows (blockDim.x of them).
// A column takes one reduction: the sums of conj(x_r) a_l(r) over the rows below the
// head, for all 16 columns l at once, hold the column's norm, the products with
// the columns to the right (scaled afterwards, the head row added) and with the finished
// reflectors to the left, which are the Gram matrix that T is formed from.  One block
// barrier per column (and one cluster barrier where cs > 1), against five barriers and three
// passes over global memory in ts_panel_qr.  The registers rotate by a column per step, so
// that the loop is not unrolled: unrolled, its 16 different steps are fetched from L2 once
// each and take 91 us at m = 348.  Bound by that chain of 16 steps: 31 us per panel of the
// n = 364 reduction (32 k-points, average) and 100 of the n = 1324 one (144), against 97 and 165
// in ts_panel_qr's form.
constexpr int kTsPanelMaxCluster = 8;  // the portable cluster size; longer panels take ts_panel_kernel
__global__ void __launch_bounds__(kTsPanelThreads, 1) ts_panel_reg_kernel(int n, int j0, int cs, double2* A,
                                                                          double2* tau, double2* Vb, double2* Tm) {
  constexpr int B = kTsB, NW = kTsPanelThreads / 32;
  static_assert(B == 16, "half a warp holds the sums of the 16 columns");
  __shared__ __align__(16) double2 part[2][NW][B];               // warp sums
  __shared__ __align__(16) double2 head[2][B];                   // the head row before its column
  __shared__ __align__(16) double2 tot[2][kTsPanelMaxCluster][B];  // block sums of the cluster
  __shared__ __align__(16) double2 wv[NW][B];                    // per warp: conj(tau) w_l
  __shared__ __align__(16) double2 G[B][B];                      // G[q][l] = v_q^H v_l, q < l
  __shared__ double2 taus[B];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  const int rank = blockIdx.x % cs;  // grid (cs nk), clusters of cs consecutive blocks
  const int64_t b = blockIdx.x / cs;
  const int m = n - j0 - B, nr = m < B ? m : B;
  const int r = rank * (int)blockDim.x + tid;  // this thread's row, counted from j0 + B
  const bool valid = r < m;
  double2* Ar = A + b * (int64_t)n * n + (int64_t)j0 * n + (j0 + B) + r;  // + l n: column l
  double2* Vr = Vb + b * (int64_t)n * B + r;
  double2 a[B];  // slot l: column (c + l) % 16 at step c (the finished ones hold their reflectors)
#pragma unroll
  for (int l = 0; l < B; ++l) a[l] = valid ? Ar[(int64_t)l * n] : cmk(0.0, 0.0);
  for (int e = tid; e < B * B; e += blockDim.x) ((double2*)G)[e] = cmk(0.0, 0.0);
  if (tid < B) taus[tid] = cmk(0.0, 0.0);
  if (cs > 1) cluster_barrier();  // every block of the cluster runs before its shared memory is written
#pragma unroll 1
  for (int c = 0; c < nr; ++c) {
    const int par = c & 1;
    const double2 x = (r > c) ? a[0] : cmk(0.0, 0.0);
    double t[B];
#pragma unroll
    for (int l = 0; l < B; ++l) t[l] = x.x * a[l].x + x.y * a[l].y;
    const double sr = warp_sum16(t, lane);
#pragma unroll
    for (int l = 0; l < B; ++l) t[l] = x.x * a[l].y - x.y * a[l].x;
    const double si = warp_sum16(t, lane);
    if (lane < B) part[par][warp][lane] = cmk(sr, si);
    if (r == c) {
#pragma unroll
      for (int l = 0; l < B; ++l) head[par][l] = a[l];
    }
    __syncthreads();
    // lane l (and l + 16): the block's sum of slot l, every second warp in each half
    const int l0 = lane & 15;
    double2 v = cmk(0.0, 0.0);
    if (cs == 1 || warp == 0) {
#pragma unroll
      for (int q = 0; q < NW; q += 2)
        if (q + (lane >> 4) < nw) v = cadd(v, part[par][q + (lane >> 4)][l0]);
      v.x += __shfl_xor_sync(0xffffffffu, v.x, 16);
      v.y += __shfl_xor_sync(0xffffffffu, v.y, 16);
    }
    if (cs > 1) {
      if (warp == 0 && lane < B) {
        for (int q = 0; q < cs; ++q) cluster_st16(&tot[par][rank][lane], q, v);
        if (rank == 0)
          for (int q = 1; q < cs; ++q) cluster_st16(&head[par][lane], q, head[par][lane]);
      }
      cluster_barrier();
      v = cmk(0.0, 0.0);
      for (int q = 0; q < cs; ++q) v = cadd(v, tot[par][q][l0]);
    }
    const double s = __shfl_sync(0xffffffffu, v.x, 0);
    double2 tj, scal;
    double beta;
    zlarfg_scalars(head[par][0], s, &tj, &beta, &scal);
    const double2 w = cadd(head[par][l0], cmulc(scal, v));  // v_c^H a_l
    const bool right = l0 > 0 && c + l0 < B;                // a column still to be reduced
    if (lane < B) wv[warp][lane] = right ? cmul(cconj(tj), w) : cmk(0.0, 0.0);
    if (rank == 0 && warp == 0 && lane < B && c + lane >= B) G[c + lane - B][c] = cconj(w);
    if (rank == 0 && tid == 0) { taus[c] = tj; tau[b * n + j0 + c] = tj; }
    __syncwarp();
    // column c: R above the head, beta in it, the reflector below; the explicit reflector
    const double2 vc = (r == c) ? cmk(1.0, 0.0) : cmul(scal, x);
    if (valid) {
      Ar[(int64_t)c * n] = (r < c) ? a[0] : (r == c) ? cmk(beta, 0.0) : vc;
      Vr[(int64_t)c * n] = vc;
    }
#pragma unroll
    for (int l = 0; l + 1 < B; ++l) a[l] = csub(a[l + 1], cmul(vc, wv[warp][l + 1]));
    a[B - 1] = vc;
  }
  if (valid)
#pragma unroll
    for (int l = 0; l < B; ++l)
      if (nr + l < B) Ar[(int64_t)(nr + l) * n] = a[l];
  // T = (diag(1 / tau) + striu(G))^-1 (zlarft forward), column `lane` by back-substitution:
  // t_s = -tau_s sum_{i > s} G(s, i) t_i; a zero tau gives a zero row
  if (rank == 0 && warp == 0) {
    __syncwarp();
    double2 acc[B];
#pragma unroll
    for (int i = 0; i < B; ++i) acc[i] = cmk(0.0, 0.0);
#pragma unroll
    for (int s2 = B - 1; s2 >= 0; --s2) {
      const double2 ts = taus[s2];
      const double2 tv = (s2 == lane)  ? ts
                         : (s2 < lane) ? cmul(cmk(-ts.x, -ts.y), acc[s2])
                                       : cmk(0.0, 0.0);
#pragma unroll
      for (int i = 0; i < s2; ++i) acc[i] = cadd(acc[i], cmul(G[i][s2], tv));
      if (lane < B) Tm[b * B * B + s2 + lane * B] = tv;
    }
  }
}

// W = X - V Z / 2 of the trailing update A22 -= V W^H + W V^H, from V, T and Y = A22 V:
// X = Y T, Z = T^H V^H X.  With G = V^H Y this is W = Y T - V (T^H G T / 2), one pass over V
// and Y for G and one for W, tensor steps (DMMA) straight from global memory in both; a
// cluster of cs blocks per k-point, each with a slice of `rows` rows (a multiple of 16).
// As five to seven GEMM launches this took 84 us per panel of the n = 364 reduction (32
// k-points), now 10; 32 us at n = 1324 (144 k-points).  Bound by latency and, for many
// k-points, by reading V and Y.
constexpr int kTsWThreads = 256;
constexpr int kTsWMaxCluster = 8;
constexpr int kTsWSmem = (kTsWThreads / 32 + kTsWMaxCluster + 4) * kTsB * kTsB * 16;
__global__ void __launch_bounds__(kTsWThreads, 2) ts_w_kernel(int n, int m, int nr, int cs, int rows,
                                                              const double2* V, const double2* Y, const double2* Tm,
                                                              double2* Wo) {
  constexpr int B = kTsB, NW = kTsWThreads / 32, BB = B * B;
  static_assert(BB == kTsWThreads, "a thread per entry of the 16 x 16 products");
  extern __shared__ __align__(16) unsigned char tsw_smem[];
  double2* part = (double2*)tsw_smem;        // NW x BB warp sums of G
  double2* tot = part + NW * BB;             // cs x BB block sums
  double2* Gm = tot + kTsWMaxCluster * BB;   // G, then S = G T
  double2* Sm = Gm + BB;
  double2* Cf = Sm + BB;                     // 32 x 16: T over -Z (row-major)
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int rank = blockIdx.x % cs;
  const int64_t b = blockIdx.x / cs;
  const double2* Vk = V + b * (int64_t)n * B;
  const double2* Yk = Y + b * (int64_t)n * B;
  double2* Wk = Wo + b * (int64_t)n * B;
  const int rbeg = rank * rows, rend = (rbeg + rows < m) ? rbeg + rows : m;
  Cf[tid] = Tm[b * BB + (tid / B) + (tid % B) * B];  // Cf[k][l] = T(k, l)
  if (cs > 1) cluster_barrier();  // every block of the cluster runs before its shared memory is written
  // G(q, l) = sum_r conj(V(r, q)) Y(r, l)
  double re[2][2][2], im[2][2][2];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) re[i][j][0] = re[i][j][1] = im[i][j][0] = im[i][j][1] = 0.0;
  for (int r0 = rbeg + 16 * warp; r0 < rend; r0 += 16 * NW) {
    double2 av[4][2], bv[4][2];
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      const int r = r0 + 4 * kk + t;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const bool ok = r < rend && 8 * i + g < nr;
        av[kk][i] = ok ? Vk[r + (int64_t)(8 * i + g) * n] : cmk(0.0, 0.0);
        bv[kk][i] = ok ? Yk[r + (int64_t)(8 * i + g) * n] : cmk(0.0, 0.0);
      }
    }
#pragma unroll
    for (int kk = 0; kk < 4; ++kk)
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          dmma_884(re[i][j][0], re[i][j][1], av[kk][i].x, bv[kk][j].x);
          dmma_884(re[i][j][0], re[i][j][1], av[kk][i].y, bv[kk][j].y);
          dmma_884(im[i][j][0], im[i][j][1], av[kk][i].x, bv[kk][j].y);
          dmma_884(im[i][j][0], im[i][j][1], -av[kk][i].y, bv[kk][j].x);
        }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        part[warp * BB + (8 * i + g) * B + 8 * j + 2 * t + h] = cmk(re[i][j][h], im[i][j][h]);
  __syncthreads();
  double2 sum = part[tid];
#pragma unroll
  for (int w = 1; w < NW; ++w) sum = cadd(sum, part[w * BB + tid]);
  if (cs > 1) {
    for (int q = 0; q < cs; ++q) cluster_st16(tot + rank * BB + tid, q, sum);
    cluster_barrier();
    sum = tot[tid];
    for (int q = 1; q < cs; ++q) sum = cadd(sum, tot[q * BB + tid]);
  }
  Gm[tid] = sum;
  __syncthreads();
  const int q = tid / B, l = tid % B;
  double2 acc = cmk(0.0, 0.0);
#pragma unroll
  for (int k = 0; k < B; ++k) acc = cadd(acc, cmul(Gm[q * B + k], Cf[k * B + l]));
  Sm[tid] = acc;
  __syncthreads();
  acc = cmk(0.0, 0.0);
#pragma unroll
  for (int k = 0; k < B; ++k) acc = cadd(acc, cmulc(Cf[k * B + q], Sm[k * B + l]));
  Cf[BB + tid] = cmk(-0.5 * acc.x, -0.5 * acc.y);
  __syncthreads();
  // W = [Y V] Cf: the coefficients stay in registers as B fragments
  double2 bf[8][2];
#pragma unroll
  for (int k = 0; k < 8; ++k)
#pragma unroll
    for (int j = 0; j < 2; ++j) bf[k][j] = Cf[(4 * k + t) * B + 8 * j + g];
  for (int r0 = rbeg + 8 * warp; r0 < rend; r0 += 8 * NW) {
    const int r = r0 + g;
    double2 av[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int cc = 4 * (k & 3) + t;
      const double2* src = (k < 4) ? Yk : Vk;
      av[k] = (r < rend && cc < nr) ? src[r + (int64_t)cc * n] : cmk(0.0, 0.0);
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      double wr[2] = {0.0, 0.0}, wi[2] = {0.0, 0.0};
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        dmma_884(wr[0], wr[1], av[k].x, bf[k][j].x);
        dmma_884(wr[0], wr[1], -av[k].y, bf[k][j].y);
        dmma_884(wi[0], wi[1], av[k].x, bf[k][j].y);
        dmma_884(wi[0], wi[1], av[k].y, bf[k][j].x);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int cc = 8 * j + 2 * t + h;
        if (r < rend && cc < nr) Wk[r + (int64_t)cc * n] = cmk(wr[h], wi[h]);
      }
    }
  }
}

// grid (B): the band (2 kTsB x n per k-point) out of the stage-1 result.
__global__ void __launch_bounds__(kBlkThreads) ts_band_kernel(int n, const double2* A, double2* Bd) {
  const Team T = make_team();
  const int64_t b = blockIdx.x;
  ts_band_extract<kTsB>(T, n, A + b * (int64_t)n * n, n, Bd + b * 2 * kTsB * (int64_t)n);
}

// Bulge chase of one k-point (the tasks of ts_chase_sweep): grid (B), kTsPairs pairs of
// warps; pair p takes the sweeps s = p, p + kTsPairs, ...  Before task t of sweep s the pair
// waits until sweep s - 1 has finished its tasks 0 .. t + 2 (those whose rows and columns
// overlap task t's), read from a per-pair progress word in shared memory.
// A pair is a two-stage pipeline over the tasks of its sweep.  The maker takes task t's
// column x, forms the reflector v and applies it to the block E below (E <- E H), which
// holds the next task's x, and so runs along the only chain within a sweep; the applier,
// one task behind at most, applies v to the rest F of the block that the task started
// from and two-sided to the diagonal block D, writes both back and publishes the task.
// They meet on the pair's named barrier once per task.  E passes through three buffers in
// shared memory (row by lane pair in the maker, column by lane pair in the applier); D and
// E live in registers while they are changed; rows past the matrix's end are zeros.
// The band stays in global memory (L1/L2): the applier's stores are fenced at block scope
// before it publishes, and a waiting warp fences after it reads the progress word.  Every
// wait is bounded (wait_polls polls): on expiry the kernel records an error in *err, every
// pair stops at its next task, and d / e are written as zeros.  V2 / tau2 (or null): the
// reflectors for the back-transformation.  Outputs: d (n) and e (n - 1) of the real
// tridiagonal.  Bound by the latency of a task: 3 n of them follow each other at least.  One warp
// per sweep that did a whole task by itself (1560 instructions) took 44 ms at n = 1324 for up
// to 148 k-points; with pairs whole calls went from 12.2 to 9.0 ms (bands, n = 364, 32 k-points) and from 155 to 135 ms
// (n = 1324, 100).  Eight pairs of 128 registers a thread; ten of 96 spill.
constexpr int kTsPairs = 8;
constexpr int kTsLw = kTsB + 1;  // block pitch (odd: row and column walks conflict-free)
constexpr int kTsBlk = kTsB * kTsLw;
constexpr int kTsPairWin = 4 * kTsBlk + 3 * kTsB + 4;  // three E buffers, D | v (2), w | tau, beta (2 each)
constexpr int kTsChaseSmem = kTsPairs * kTsPairWin * 16;
static_assert(kTsChaseSmem <= 225 * 1024, "chase windows exceed shared memory");
static_assert(kTsB == 16, "a lane pair per row or column, eight elements each");

__device__ __forceinline__ double ts_warp_sum(double v) {  // every lane gets the sum (two tensor steps)
  double a0 = 0.0, a1 = 0.0, b0 = 0.0, b1 = 0.0;
  dmma_884(a0, a1, 1.0, v);
  dmma_884(b0, b1, 1.0, a0 + a1);
  return b0;
}
__device__ __forceinline__ double2 ts_pair_add(double2 v) {  // + the value of lane ^ 16
  v.x += __shfl_xor_sync(0xffffffffu, v.x, 16);
  v.y += __shfl_xor_sync(0xffffffffu, v.y, 16);
  return v;
}

__global__ void __launch_bounds__(kTsPairs * 64, 1) ts_chase_kernel(int n, double2* Bd, double2* V2, double2* tau2,
                                                                    double* d, double* e, int* err,
                                                                    long long wait_polls) {
  extern __shared__ __align__(16) double2 tswin[];
  __shared__ long long prog[kTsPairs];
  __shared__ int stop;
  // the meeting at which the maker gives up, or -1: a number, as the applier may still be on its
  // way from the last meeting when the maker writes it, and has to come to this one too
  __shared__ int halt[kTsPairs];
  constexpr int B = kTsB, LW = kTsLw, ldb = 2 * B;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, pair = w >> 1;
  const bool maker = (w & 1) == 0;
  const int r = lane & 15, hh = lane >> 4;
  const int64_t b = blockIdx.x;
  double2* Bk = Bd + b * ldb * (int64_t)n;
  double2* buf = tswin + pair * kTsPairWin;  // block i at buf + i kTsBlk, (row, column) at row + LW column
  double2* Dm = buf + 3 * kTsBlk;            // the part of D above the diagonal, by rows of its mirror
  double2* vb = Dm + kTsBlk;                 // v of even and odd tasks
  double2* wv = vb + 2 * B;
  double2* sc = wv + B;                      // tau, (beta, 0) of even and odd tasks
  const int tmax = ts_tmax(n, B);
  const long long unit = tmax + 1;  // progress: s * unit + tasks done
  if (threadIdx.x < kTsPairs) { prog[threadIdx.x] = -1; halt[threadIdx.x] = -1; }
  if (threadIdx.x == 0) stop = (err && *(volatile int*)err) ? 1 : 0;
  __syncthreads();
  volatile long long* vprog = prog;
  volatile int* vstop = &stop;
  const int pp = (pair + kTsPairs - 1) % kTsPairs;  // the pair of sweep s - 1
  auto meet = [&] { asm volatile("bar.sync %0, 64;\n" ::"r"(1 + pair) : "memory"); };
  const bool go = *vstop == 0;
  int it = 0;  // tasks of this pair so far: the buffers' turn (the maker's next sweep overlaps the applier's last task)
  for (int s = pair; go && s <= n - 2; s += kTsPairs) {
    const int nt = ts_tasks(n, B, s), ntp = s > 0 ? ts_tasks(n, B, s - 1) : 0;
    double2* vo = V2 ? V2 + b * ts_v2_stride(n) + (int64_t)s * tmax * B : nullptr;
    double2* to = tau2 ? tau2 + b * ts_tau2_stride(n) + (int64_t)s * tmax : nullptr;
    bool ok = true;
    if (maker) {
      for (int t = 0; t < nt; ++t, ++it) {
        // R0: first row of the task; rows R0 .. R0 + 15 (zeros past n), E below them
        const int R0 = s + 1 + t * B, R1 = R0 + B;
        if (s > 0) {
          const long long need = (long long)(s - 1) * unit + (t + 3 < ntp ? t + 3 : ntp);
          if (lane == 0) {
            long long polls = 0;
            while (vprog[pp] < need) {
              if (*vstop) { ok = false; break; }
              if (++polls > wait_polls) {
                *vstop = 1;
                if (err) atomicExch(err, 2);
                ok = false;
                break;
              }
            }
          }
          ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
          __threadfence_block();
        }
        if (!ok) break;
        double2 E[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int q = 8 * hh + k;
          E[k] = (R1 + r < n) ? Bk[(B + r - q) + (int64_t)(R0 + q) * ldb] : cmk(0.0, 0.0);
        }
        double2* X = buf + (it % 3) * kTsBlk;  // x: its first column
        double2 x = cmk(0.0, 0.0);
        if (t == 0) x = (R0 + r < n) ? Bk[(1 + r) + (int64_t)s * ldb] : cmk(0.0, 0.0);
        else x = X[r];
        const double nrm = ts_warp_sum((hh == 0 && r > 0) ? x.x * x.x + x.y * x.y : 0.0);
        const double2 alpha = shfl_c(x, 0);
        double2 tj, scal;
        double beta;
        zlarfg_scalars(alpha, nrm, &tj, &beta, &scal);
        const double2 vr = r == 0 ? cmk(1.0, 0.0) : cmul(scal, x);
        double2* v = vb + (it & 1) * B;
        if (hh == 0) {
          v[r] = vr;
          if (vo) vo[(int64_t)t * B + r] = vr;
        }
        if (lane == 0) {
          sc[2 * (it & 1)] = tj;
          sc[2 * (it & 1) + 1] = cmk(beta, 0.0);
          if (to) to[t] = tj;
        }
        __syncwarp();
        // E <- E H: z = E v, E -= tau z v^H
        double2 vq[8], e0 = cmk(0.0, 0.0), e1 = e0;
#pragma unroll
        for (int k = 0; k < 8; ++k) vq[k] = v[8 * hh + k];
#pragma unroll
        for (int k = 0; k < 8; k += 2) {
          e0 = cfma(e0, E[k], vq[k]);
          e1 = cfma(e1, E[k + 1], vq[k + 1]);
        }
        const double2 z = cmul(tj, ts_pair_add(cadd(e0, e1)));
        double2* EN = buf + ((it + 1) % 3) * kTsBlk;
#pragma unroll
        for (int k = 0; k < 8; ++k) EN[r + LW * (8 * hh + k)] = cfms(E[k], z, cconj(vq[k]));
        meet();  // v, E and the reflector's scalars are the applier's; it is done with task t - 1
      }
      if (!ok) {
        if (lane == 0) ((volatile int*)halt)[pair] = it;
        meet();
        break;
      }
    } else {
      for (int t = 0; t < nt; ++t, ++it) {
        meet();
        if (((volatile int*)halt)[pair] == it) { ok = false; break; }
        const int R0 = s + 1 + t * B, c = t == 0 ? s : R0 - B;
        double2 D[8];  // D(r, 8 hh + k), the lower triangle
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int q = 8 * hh + k;
          D[k] = (q <= r && R0 + r < n) ? Bk[(r - q) + (int64_t)(R0 + q) * ldb] : cmk(0.0, 0.0);
        }
        const double2* v = vb + (it & 1) * B;
        const double2 tj = sc[2 * (it & 1)], beta = sc[2 * (it & 1) + 1];
        double2* X = buf + (it % 3) * kTsBlk;
        // F <- H^H F, column r (1 .. 15), rows 8 hh ..; the first column becomes beta e1
        if (t > 0) {
          double2 f[8], vf[8], a0 = cmk(0.0, 0.0), a1 = a0;
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            f[k] = X[8 * hh + k + LW * r];
            vf[k] = v[8 * hh + k];
          }
#pragma unroll
          for (int k = 0; k < 8; k += 2) {
            a0 = cfma_conj(a0, vf[k], f[k]);
            a1 = cfma_conj(a1, vf[k + 1], f[k + 1]);
          }
          const double2 fl = cmul(cconj(tj), ts_pair_add(cadd(a0, a1)));
#pragma unroll
          for (int k = 0; k < 8; ++k)
            X[8 * hh + k + LW * r] = r > 0 ? cfms(f[k], vf[k], fl) : (hh == 0 && k == 0) ? beta : cmk(0.0, 0.0);
          __syncwarp();
#pragma unroll
          for (int k = 0; k < 8; ++k) {  // back to the band, by columns: two at a time
            const int l = 2 * k + hh;
            if (R0 + r < n) Bk[(B + r - l) + (int64_t)(c + l) * ldb] = X[r + LW * l];
          }
        } else if (hh == 0 && R0 + r < n) {
          Bk[(1 + r) + (int64_t)s * ldb] = r == 0 ? beta : cmk(0.0, 0.0);
        }
        // D <- H^H D H: y = D v, gamma = v^H y, w = tau y - 1/2 |tau|^2 gamma v,
        // D -= w v^H + v w^H
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int q = 8 * hh + k;
          if (q < r) Dm[q + LW * r] = cconj(D[k]);
        }
        __syncwarp();
        double2 vq[8], a0 = cmk(0.0, 0.0), a1 = a0;
#pragma unroll
        for (int k = 0; k < 8; ++k) vq[k] = v[8 * hh + k];
#pragma unroll
        for (int k = 0; k < 8; k += 2) {
          const int q = 8 * hh + k;
          a0 = cfma(a0, q <= r ? D[k] : Dm[r + LW * q], vq[k]);
          a1 = cfma(a1, q + 1 <= r ? D[k + 1] : Dm[r + LW * (q + 1)], vq[k + 1]);
        }
        const double2 y = ts_pair_add(cadd(a0, a1)), vr = v[r];
        const double g = ts_warp_sum(hh == 0 ? cmulc(vr, y).x : 0.0);
        const double h = -0.5 * (tj.x * tj.x + tj.y * tj.y) * g;
        const double2 wr = cadd(cmul(tj, y), cscale(h, vr));
        if (hh == 0) wv[r] = wr;
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int q = 8 * hh + k;
          double2 x = cfms(cfms(D[k], wr, cconj(vq[k])), vr, cconj(wv[q]));
          if (q == r) x.y = 0.0;
          if (q <= r && R0 + r < n) Bk[(r - q) + (int64_t)(R0 + q) * ldb] = x;
        }
        __threadfence_block();
        __syncwarp();
        if (lane == 0) vprog[pair] = (long long)s * unit + t + 1;
      }
      if (!ok) break;
    }
  }
  __syncthreads();
  const bool fin = *vstop == 0;  // after a failed wait: zeros, so the solver that follows stays bounded
  __threadfence_block();
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    d[b * n + i] = fin ? Bk[(int64_t)i * ldb].x : 0.0;
    e[b * n + i] = (fin && i + 1 < n) ? Bk[1 + (int64_t)i * ldb].x : 0.0;
  }
}

// Q2 Z in the grouped order (ts_q2_apply_grouped_host): grid (ceil(K / kTsQ2gThreads), B),
// thread = one of the columns c0 .. c0+K-1 of U (n x n per k-point, in place).
// Each (group of 16 sweeps, task t) step applies 16 reflectors to a window of 31
// rows of the thread's column, held in registers (all indices compile-time); the
// window slides by 16 rows per step, so a group streams the column once.  The
// step's reflectors and taus (16 x 16 + 16 complex; zeros where a sweep has no
// task t) are copied into shared memory by cp.async one step ahead.
// Bound by the FP64 pipe (64 FMA per row and reflector pair) as long as the window's
// traffic stays off it: a column per lane makes every direct access 32 separate lines,
// as many LSU cycles per step as the arithmetic takes, and all warps at once behind the
// step's barrier.  So the 16 rows that enter and leave move through a 32-column
// exchange block per warp, 256 contiguous bytes of a column per half-warp, the entering
// rows by cp.async one step ahead.  144 k-points of n = 1324 (693 columns each): 86 ms,
// 16 TFLOP/s, against 115 ms with direct accesses (256 threads, rows prefetched into L1).
// Two blocks of 128 let one compute while the other waits at its barrier; 64 and 32 threads,
// four partial sums, or two reflectors at a time (with their Gram element) are not faster.
constexpr int kTsQ2gThreads = 128;
constexpr int kTsQ2gCtas = 2;
constexpr int kTsQ2gStep = kTsB * kTsB + kTsB;  // complex per staged step
constexpr int kTsQ2gPitch = kTsB + 1;           // complex per column of the exchange block (conflict-free)
constexpr int kTsQ2gSmem = (3 * kTsQ2gStep + kTsQ2gThreads * kTsQ2gPitch) * 16;
__global__ void __launch_bounds__(kTsQ2gThreads, kTsQ2gCtas) ts_q2g_kernel(int n, int c0, int K, const double2* V2,
                                                                           const double2* tau2, double2* U) {
  constexpr int B = kTsB, W = 2 * kTsB - 1, P = kTsQ2gPitch;
  static_assert(B == 16, "a half-warp moves one column's rows");
  extern __shared__ __align__(16) unsigned char q2g_smem[];
  double2* sv = (double2*)q2g_smem;  // three steps of reflectors
  const int lane = threadIdx.x & 31;
  double2* xb = sv + 3 * kTsQ2gStep + (threadIdx.x >> 5) * 32 * P;  // the warp's exchange block, [column][row]
  const int64_t b = blockIdx.y;
  const int cw = blockIdx.x * kTsQ2gThreads + (threadIdx.x & ~31);  // the warp's first column
  const int xc = lane >> 4, xr = lane & 15;                          // this lane's part of a moved column pair
  double2* Uw = U + b * (int64_t)n * n + (int64_t)(c0 + cw + xc) * n + xr;
  const double2* Vk = V2 + b * ts_v2_stride(n);
  const double2* tk = tau2 + b * ts_tau2_stride(n);
  const int tmax = ts_tmax(n, B);
  const int ns = n - 1;
  if (ns <= 0) return;
  const int g0 = (ns - 1) / B;  // highest group
  // step (g, t) -> shared buffer: reflector i of the step = sweep g B + i, task t
  auto stage = [&](int g, int t, double2* dst) {
    for (int e = threadIdx.x; e < kTsQ2gStep; e += kTsQ2gThreads) {
      const int i = (e < B * B) ? e / B : e - B * B;
      const int s = g * B + i;
      const bool ok = s < ns && t < ts_tasks(n, B, s);
      const double2* src = (e < B * B) ? Vk + ((int64_t)s * tmax + t) * B + (e - i * B) : tk + (int64_t)s * tmax + t;
      cp_async16(dst + e, ok ? (const void*)src : (const void*)Vk, ok);
    }
  };
  // rows r0 .. r0 + 15 of the warp's columns into / out of the exchange block (rows past
  // n and columns past K: zeros in, nothing out)
  auto rows_in = [&](int r0) {
#pragma unroll 4
    for (int q = 0; q < 16; ++q) {
      const bool ok = r0 + xr < n && cw + 2 * q + xc < K;
      cp_async16(xb + (2 * q + xc) * P + xr, ok ? (const void*)(Uw + r0 + (int64_t)(2 * q) * n) : (const void*)Vk, ok);
    }
  };
  auto rows_out = [&](int r0) {
#pragma unroll 4
    for (int q = 0; q < 16; ++q)
      if (r0 + xr < n && cw + 2 * q + xc < K) Uw[r0 + (int64_t)(2 * q) * n] = xb[(2 * q + xc) * P + xr];
  };
  double2* xl = xb + lane * P;  // this lane's column
  int buf = 0;
  stage(g0, 0, sv);
  cp_async_commit();
  for (int g = g0; g >= 0; --g) {
    const int s0 = g * B;
    const int nt = ts_tasks(n, B, s0);
    double2 z[W];
    const int w0 = s0 + 1;
    // the group's first window, in two passes of the exchange block
    rows_in(w0);
    cp_async_commit();
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncwarp();
#pragma unroll
    for (int j = 0; j < B; ++j) z[j] = xl[j];
    __syncwarp();
    rows_in(w0 + B);
    cp_async_commit();
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncwarp();
#pragma unroll
    for (int j = B; j < W; ++j) z[j] = xl[j - B];
    __syncwarp();
    if (nt > 1) rows_in(w0 + W);  // the first slide's rows
    cp_async_commit();
    for (int t = 0; t < nt; ++t) {
      // next step: (g, t + 1), or the next group's first.  In flight after this commit, in
      // order: this step's reflectors, the entering rows, the next step's reflectors.  The
      // buffer being filled was last read two steps ago, before the last barrier.
      const int nb = (buf == 2) ? 0 : buf + 1;
      if (t + 1 < nt) stage(g, t + 1, sv + nb * kTsQ2gStep);
      else if (g > 0) stage(g - 1, 0, sv + nb * kTsQ2gStep);
      cp_async_commit();
      asm volatile("cp.async.wait_group 2;\n" ::: "memory");
      __syncthreads();
      const double2* vs = sv + buf * kTsQ2gStep;
#pragma unroll
      for (int i = B - 1; i >= 0; --i) {
        const double2 tj = vs[B * B + i];
        double2 a[2] = {cmk(0.0, 0.0), cmk(0.0, 0.0)};
#pragma unroll
        for (int r = 0; r < B; ++r) a[r & 1] = cfma_conj(a[r & 1], vs[i * B + r], z[i + r]);
        const double2 f = cmul(tj, cadd(a[0], a[1]));
#pragma unroll
        for (int r = 0; r < B; ++r) z[i + r] = cfms(z[i + r], vs[i * B + r], f);
      }
      buf = nb;
      const int wt = w0 + t * B;  // first row of this step's window
      if (t + 1 < nt) {
        cp_async_wait_keep1();  // the entering rows
        __syncwarp();
        const double2 zl = z[B - 1];  // leaves too, but its place is taken by the first entering row
#pragma unroll
        for (int j = 0; j < B; ++j) {  // each lane swaps its own column: row wt + j out, row wt + W + j in
          const double2 in = xl[j];
          xl[j] = (j < B - 1) ? z[j] : zl;
          if (j < W - B) z[j] = z[j + B];
          z[W - B + j] = in;
        }
        __syncwarp();
        rows_out(wt);
        __syncwarp();
        if (t + 2 < nt) rows_in(wt + B + W);
        cp_async_commit();
      } else {
#pragma unroll
        for (int j = 0; j < B; ++j) xl[j] = z[j];
        __syncwarp();
        rows_out(wt);
        __syncwarp();
#pragma unroll
        for (int j = B; j < W; ++j) xl[j - B] = z[j];
        __syncwarp();
        if (xr < W - B) rows_out(wt + B);
        __syncwarp();  // the next group reads these rows from other lanes of this warp
      }
    }
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

}  // namespace lqm
