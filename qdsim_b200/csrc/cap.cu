// Products of the complex-symmetric open-system pencil (config with a complex
// absorbing potential): AX = (H + i Himag) X and MX = M X for a block of b
// complex vectors, in one pass over the CSR arrays.
//
// H, Himag and M share one CSR pattern (qd_assemble writes all three), so a
// row's column indices are read once for the three matrices.  Blocks are
// row-major complex (re, im interleaved), X[row * ldx + c], with a leading
// dimension so that column slices of a wider basis can be read and written in
// place.
//
// Replaces the complex SpMV of the shift-invert Arnoldi that scipy's eigs
// runs for the reference's complex eigenvalue path (a12:
// backend/src/schrodinger.cpp:699-818 solves the same pencil densely with
// ComplexEigenSolver; fused_gpu_kernels.cu:97-125 is its never-launched
// scalar complex CSR SpMV).
#include <cuda_runtime.h>
#include <algorithm>
#include <atomic>
#include <cstdint>
#include "common.h"

namespace {

template <typename T> struct Vec2;
template <> struct Vec2<float> { using type = float2; };
template <> struct Vec2<double> { using type = double2; };

constexpr int kLanes = 16;          // lanes per row: two rows per warp
constexpr int kRowsPerBlock = 16;   // 256 threads

// The order in which rows are taken: tiles of 16 rows, 4 x 4 of a lattice or 16
// of one line, marching along the line; a block takes `run` consecutive tiles,
// then skips the runs of the other blocks, so that the blocks move through the
// lattice together and find each other's lines in L2.
struct RowOrder {
  int width, lines;              // rows per line, lines
  int shift;                     // a tile is 1 << shift rows along the line
  int tiles_i, run;              // tiles per band, tiles per run
  int runs_i, runs;              // runs per band, runs
};

// One half-warp's rows, tile after tile.
struct RowWalk {
  int i0, j0, place, left, run;
  __device__ RowWalk(const RowOrder &o, int half) {
    run = blockIdx.x;
    place = half;
    start(o);
  }
  __device__ void start(const RowOrder &o) {   // the first tile of run `run`
    const int band = run / o.runs_i, first = (run - band * o.runs_i) * o.run;
    i0 = first << o.shift;
    j0 = band << (4 - o.shift);
    left = min(o.run, o.tiles_i - first);
  }
  // The row of the current tile (-1: none), then on to the next tile.  Places
  // 2q, 2q + 1 (the two rows of a warp) lie two apart along the line; the warps
  // trade places from tile to tile.
  __device__ int next(const RowOrder &o) {
    if (run >= o.runs) return -1;
    const int along = place & ((1 << o.shift) - 1);
    const int i = i0 + ((along & ~3) | (along >> 1 & 1) | (along & 1) << 1);
    const int j = j0 + (place >> o.shift);
    place = (place + 2) & 15;
    i0 += 1 << o.shift;
    if (--left == 0) {
      run += gridDim.x;
      start(o);
    }
    return i < o.width && j < o.lines ? j * o.width + i : -1;
  }
};

// Tiles of all runs of this block.
__device__ __forceinline__ int tiles_of(const RowOrder &o) {
  int sum = 0;
  for (int r = blockIdx.x; r < o.runs; r += gridDim.x)
    sum += min(o.run, o.tiles_i - r % o.runs_i * o.run);
  return sum;
}

// Two kernels, the same sums in the same order (equal bits).  Both take kLanes
// lanes per row; lane l owns columns l, l + 16, ... (C of them, so a 48-column
// block keeps every lane busy), so each half-warp's vector loads are 16
// consecutive complex values.
//
// cap_spmm_rows_kernel: a block per 16 rows; the row's CSR entries are loaded 16
// at a time, one per lane, and broadcast by shuffles.  Small registers and no
// set-up: where the vectors come from L2 and many rows in flight hide its latency
// it is the faster one (tiles_pay).
template <typename T, int C>
__global__ void __launch_bounds__(kRowsPerBlock * kLanes, 4)
cap_spmm_rows_kernel(int32_t n, int b, int ldx, int ldy, const int32_t *__restrict__ rowptr,
                     const int32_t *__restrict__ col, const T *__restrict__ H,
                     const T *__restrict__ G, const T *__restrict__ M,
                     const typename Vec2<T>::type *__restrict__ X, typename Vec2<T>::type *AX,
                     typename Vec2<T>::type *MX) {
  using V = typename Vec2<T>::type;
  const int row = blockIdx.x * kRowsPerBlock + (threadIdx.x / kLanes);
  const int lane = threadIdx.x % kLanes;
  // the two rows of a warp are independent: shuffles stay inside each half
  const unsigned mask = 0xffffu << (threadIdx.x & 16);
  const bool live = row < n;
  T ar[C], ai[C], mr[C], mi[C];
#pragma unroll
  for (int c = 0; c < C; ++c) ar[c] = ai[c] = mr[c] = mi[c] = T(0);
  const int p0 = live ? rowptr[row] : 0, p1 = live ? rowptr[row + 1] : 0;
  for (int base = p0; base < p1; base += kLanes) {
    const int p = base + lane;
    int cj = 0;
    T h = T(0), g = T(0), m = T(0);
    if (p < p1) {
      cj = col[p];
      h = H[p];
      g = G ? G[p] : T(0);
      m = M[p];
    }
    const int cnt = min(kLanes, p1 - base);
    for (int q = 0; q < cnt; ++q) {
      const int j = __shfl_sync(mask, cj, q, kLanes);
      const T hq = __shfl_sync(mask, h, q, kLanes);
      const T gq = __shfl_sync(mask, g, q, kLanes);
      const T mq = __shfl_sync(mask, m, q, kLanes);
      const V *xr = X + size_t(j) * ldx;
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const int cc = c * kLanes + lane;
        if (cc < b) {
          const V x = xr[cc];
          // (h + i g)(xr + i xi) = (h xr - g xi) + i (h xi + g xr)
          ar[c] = fma(hq, x.x, fma(-gq, x.y, ar[c]));
          ai[c] = fma(hq, x.y, fma(gq, x.x, ai[c]));
          mr[c] = fma(mq, x.x, mr[c]);
          mi[c] = fma(mq, x.y, mi[c]);
        }
      }
    }
  }
  if (!live) return;
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const int cc = c * kLanes + lane;
    if (cc < b) {
      V a, mm;
      a.x = ar[c];
      a.y = ai[c];
      mm.x = mr[c];
      mm.y = mi[c];
      AX[size_t(row) * ldy + cc] = a;
      MX[size_t(row) * ldy + cc] = mm;
    }
  }
}

// cap_spmm_kernel: rows in tiles of the lattice (RowOrder).  The row's CSR entries
// are copied to shared memory and read from there by all lanes (two or three reads
// per entry; by shuffles it takes seven).  A warp's two rows lie two apart: on a P2
// lattice neighbours have 19 and 9 entries, and half of the warp would wait.
//
// The latency of the gathers bounds it: a row reads 11 vector rows of 768 bytes
// (P2, b = 48, FP64).  Sixteen rows of one line share 45 % of them in L1; a
// 4 x 4 tile that marches along the line shares more.  The loads run ahead:
// while a warp works on a row, the next row's entries and the pointers of the
// one after it are on their way, and so are the vector rows of the next three
// entries, also across the end of a row.  The warps of a block trade places from
// tile to tile, so that none keeps the long rows.  FP64, b = 48, P2 400 x 200
// cells: 376 us by cap_spmm_rows_kernel, 253 us here (FP32: 203 and 174 us).
constexpr int kEntries = 24;        // entries staged at once (P1, P2: a whole row)
// Blocks per SM and vector rows in flight per half-warp.  FP64: with one column
// per lane a fourth block fits; with four columns two rows in flight do without
// spills (four of them spilled: P2 400 x 200, b = 49, 425 us, now 336).
template <typename T, int C> struct TileShape { static constexpr int BLOCKS = 3, AHEAD = 4; };
template <> struct TileShape<double, 1> { static constexpr int BLOCKS = 4, AHEAD = 4; };
template <> struct TileShape<double, 2> { static constexpr int BLOCKS = 2, AHEAD = 4; };
template <> struct TileShape<double, 3> { static constexpr int BLOCKS = 2, AHEAD = 4; };
template <> struct TileShape<double, 4> { static constexpr int BLOCKS = 2, AHEAD = 2; };
template <typename T> struct __align__(16) CsrEntry { T h, g, m; int j; };

template <int N> __device__ __forceinline__ void copy_async(void *smem, const void *gmem) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(s), "l"(gmem), "n"(N) : "memory");
}

template <typename T, int C>
__global__ void __launch_bounds__(kRowsPerBlock * kLanes, TileShape<T, C>::BLOCKS)
cap_spmm_kernel(RowOrder o, int b, int ldx, int ldy, const int32_t *__restrict__ rowptr,
                const int32_t *__restrict__ col, const T *__restrict__ H,
                const T *__restrict__ G, const T *__restrict__ M,
                const typename Vec2<T>::type *__restrict__ X, typename Vec2<T>::type *AX,
                typename Vec2<T>::type *MX) {
  using V = typename Vec2<T>::type;
  using Entry = CsrEntry<T>;
  constexpr int kAhead = TileShape<T, C>::AHEAD;
  __shared__ Entry s_e[2][kRowsPerBlock][kEntries];
  const int lane = threadIdx.x % kLanes, half = threadIdx.x / kLanes;
  // the two rows of a warp are independent: barriers stay inside each half
  const unsigned mask = 0xffffu << (threadIdx.x & 16);
  RowWalk walk(o, half);
  auto stage = [&](Entry *dst, int p, int p1) {   // up to kEntries of [p, p1)
#pragma unroll
    for (int u = 0; u < kEntries; u += kLanes) {
      const int i = u + lane;
      if (i < kEntries && p + i < p1) {
        copy_async<4>(&dst[i].j, col + p + i);
        copy_async<sizeof(T)>(&dst[i].h, H + p + i);
        copy_async<sizeof(T)>(&dst[i].m, M + p + i);
        if (G)
          copy_async<sizeof(T)>(&dst[i].g, G + p + i);
        else
          dst[i].g = T(0);
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  auto staged = [&]() {
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncwarp(mask);
  };
  int row = walk.next(o), nrow = walk.next(o);
  int p0 = 0, p1 = 0, n0 = 0, n1 = 0;         // this row's range and the next one's
  if (row >= 0) {
    p0 = rowptr[row];
    p1 = rowptr[row + 1];
  }
  if (nrow >= 0) {
    n0 = rowptr[nrow];
    n1 = rowptr[nrow + 1];
  }
  // this lane's columns; past the block's end the last column again (not
  // stored): skipping those loads by a predicate took 188 us where this takes
  // 175 (FP32, b = 48)
  int off[C];
#pragma unroll
  for (int c = 0; c < C; ++c) off[c] = min(c * kLanes + lane, b - 1);
  T ar[C], ai[C], mr[C], mi[C];
  V x[kAhead][C];                             // vector rows of the next entries
  const Entry *cur = s_e[0][half];
  auto load = [&](int q, V (&y)[C]) {
    const V *xr = X + int64_t(cur[q].j) * ldx;
#pragma unroll
    for (int c = 0; c < C; ++c) y[c] = xr[off[c]];
  };
  auto add = [&](int q, const V (&y)[C]) {
    const Entry e = cur[q];
#pragma unroll
    for (int c = 0; c < C; ++c) {
      // (h + i g)(xr + i xi) = (h xr - g xi) + i (h xi + g xr)
      ar[c] = fma(e.h, y[c].x, fma(-e.g, y[c].y, ar[c]));
      ai[c] = fma(e.h, y[c].y, fma(e.g, y[c].x, ai[c]));
      mr[c] = fma(e.m, y[c].x, mr[c]);
      mi[c] = fma(e.m, y[c].y, mi[c]);
    }
  };
  auto first = [&](int cnt) {
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
      if (u < cnt) load(u, x[u]);
  };
  stage(s_e[0][half], p0, p1);
  staged();
  first(min(kEntries, p1 - p0));
  int buf = 0;
  for (int left = tiles_of(o); left > 0; --left, buf ^= 1) {
    if (p1 - p0 <= kEntries) stage(s_e[buf ^ 1][half], n0, n1);
    const int frow = walk.next(o);
    int f0 = 0, f1 = 0;                       // the range after that
    if (frow >= 0) {
      f0 = rowptr[frow];
      f1 = rowptr[frow + 1];
    }
#pragma unroll
    for (int c = 0; c < C; ++c) ar[c] = ai[c] = mr[c] = mi[c] = T(0);
    for (int base = p0; base < p1; base += kEntries) {
      if (base > p0) {                        // a long row: the rest, not run ahead
        __syncwarp(mask);                     // the last entries have been read
        stage(s_e[buf][half], base, p1);
        staged();
        first(min(kEntries, p1 - base));
      }
      const int cnt = min(kEntries, p1 - base);
      for (int q = 0; q < cnt; q += kAhead) {
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
          if (q + u < cnt) {
            add(q + u, x[u]);
            if (q + u + kAhead < cnt) load(q + u + kAhead, x[u]);
          }
      }
    }
    if (p1 - p0 > kEntries) stage(s_e[buf ^ 1][half], n0, n1);
    staged();
    cur = s_e[buf ^ 1][half];
    first(min(kEntries, n1 - n0));
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const int cc = c * kLanes + lane;
      if (row >= 0 && cc < b) {
        V a, mm;
        a.x = ar[c];
        a.y = ai[c];
        mm.x = mr[c];
        mm.y = mi[c];
        AX[int64_t(row) * ldy + cc] = a;
        MX[int64_t(row) * ldy + cc] = mm;
      }
    }
    row = nrow;
    nrow = frow;
    p0 = n0;
    p1 = n1;
    n0 = f0;
    n1 = f1;
  }
}

// Whether the tiles are the faster form: by the type, the columns per lane, the
// rows and the nonzeros per row z (P1 7, P2 11, P3 17), timed on lattices of 361 to
// 319,000 rows with 1 to 64 columns against the rows kernel.  Gains and losses of
// the tiles where they are taken, and why not elsewhere:
//   FP64, 33 to 48 columns: 1.1 to 1.7 times faster everywhere; 49 to 64 columns:
//     1.0 to 1.5; up to 16 columns: 1.0 to 1.5 from some thousand rows on.
//   FP64, 17 to 32 columns: 1.04 to 1.12 on P2; P1 0.89 to 0.98, P3 0.90 to 0.98.
//   FP32: 1.05 to 1.19 where X passes 19 MB (the traffic that tiles save is then
//     what counts) and 1.0 to 1.06 on small P2 lattices up to 16 columns; 0.8 to
//     1.0 otherwise and on P3; 49 to 64 columns 0.7 to 1.0.
// z is not known (0) where the caller gives no pattern size: P2 is assumed.
// Without a lattice the tiles are 16 rows of one line, and only the widest FP64
// blocks gain (1.2 to 1.4 at 33 to 48 columns, P3 1.0).
bool tiles_pay(bool fp32, int32_t n, int b, double z, bool lattice) {
  if (z <= 0.0) z = 11.4;
  const int c = (b + kLanes - 1) / kLanes;
  if (fp32)
    return lattice && c <= 3 && z < 14.0 &&
           (int64_t(n) * b >= 2400000 || (c == 1 && z > 9.0 && n <= 32768));
  if (!lattice) return c == 3;
  return c == 1 ? n >= 2048 : c != 2 || (z > 9.0 && z < 14.0);
}

template <typename T, int C>
int launch_c(RowOrder o, int32_t n, bool tiles, int b, int ldx, int ldy, const int32_t *rowptr,
             const int32_t *col, const T *h, const T *g, const T *m, const typename Vec2<T>::type *x,
             typename Vec2<T>::type *ax, typename Vec2<T>::type *mx, cudaStream_t s) {
  constexpr int threads = kRowsPerBlock * kLanes;
  if constexpr (sizeof(T) == 8 || C <= 3) {
    if (tiles) {
      static std::atomic<int> per_sm{0};
      int res = per_sm.load(std::memory_order_relaxed);
      if (res == 0) {
        QD_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&res, cap_spmm_kernel<T, C>, threads, 0));
        if (res < 1) return QD_ERR_CUDA;
        per_sm.store(res, std::memory_order_relaxed);
      }
      // runs of 8 tiles (longer ones share no more, and leave the last wave
      // emptier: 276 us at 25), shorter where a block would have fewer than four
      const int bands = (o.lines - 1) / (16 >> o.shift) + 1;
      const int64_t count = int64_t(o.tiles_i) * bands, resident = int64_t(res) * 148;
      o.run = int(std::max<int64_t>(1, std::min<int64_t>(8, count / (4 * resident))));
      o.runs_i = (o.tiles_i - 1) / o.run + 1;
      o.runs = o.runs_i * bands;
      const unsigned blocks = unsigned(std::min<int64_t>(o.runs, resident));
      cap_spmm_kernel<T, C><<<blocks, threads, 0, s>>>(o, b, ldx, ldy, rowptr, col, h, g, m, x, ax, mx);
      QD_CHECK_LAUNCH();
      return QD_OK;
    }
  }
  const unsigned blocks = unsigned((int64_t(n) + kRowsPerBlock - 1) / kRowsPerBlock);
  cap_spmm_rows_kernel<T, C><<<blocks, threads, 0, s>>>(n, b, ldx, ldy, rowptr, col, h, g, m, x, ax, mx);
  QD_CHECK_LAUNCH();
  return QD_OK;
}

template <typename T>
int launch(int32_t n, int64_t nnz, int width, int b, int ldx, int ldy, const int32_t *rowptr,
           const int32_t *col, const void *H, const void *G, const void *M, const void *X, void *AX,
           void *MX, cudaStream_t s) {
  using V = typename Vec2<T>::type;
  const T *h = static_cast<const T *>(H), *g = static_cast<const T *>(G),
          *m = static_cast<const T *>(M);
  const V *x = static_cast<const V *>(X);
  V *ax = static_cast<V *>(AX), *mx = static_cast<V *>(MX);
  // 4 x 4 tiles on a lattice of at least four lines, else 16 rows in a line
  RowOrder o{};
  const bool lattice = width >= 4 && width < n && n % width == 0 && n / width >= 4;
  o.width = lattice ? width : n;
  o.lines = n / o.width;
  o.shift = lattice ? 2 : 4;
  o.tiles_i = ((o.width - 1) >> o.shift) + 1;
  const bool t = tiles_pay(sizeof(T) == 4, n, b, double(nnz) / n, lattice);
  switch ((b + kLanes - 1) / kLanes) {
    case 1: return launch_c<T, 1>(o, n, t, b, ldx, ldy, rowptr, col, h, g, m, x, ax, mx, s);
    case 2: return launch_c<T, 2>(o, n, t, b, ldx, ldy, rowptr, col, h, g, m, x, ax, mx, s);
    case 3: return launch_c<T, 3>(o, n, t, b, ldx, ldy, rowptr, col, h, g, m, x, ax, mx, s);
    default: return launch_c<T, 4>(o, n, t, b, ldx, ldy, rowptr, col, h, g, m, x, ax, mx, s);
  }
}

}  // namespace

extern "C" int qd_cap_spmm_pattern(int32_t n, int64_t nnz, int32_t width, int b, int vec_fp32,
                                   const int32_t *d_rowptr, const int32_t *d_col,
                                   const void *d_H, const void *d_Himag, const void *d_M,
                                   const void *d_X, int ldx, void *d_AX, void *d_MX, int ldy,
                                   void *stream) {
  if (n < 0 || nnz < 0 || b < 1 || b > 64 || ldx < b || ldy < b || !d_rowptr || !d_col || !d_H ||
      !d_M || !d_X || !d_AX || !d_MX)
    return QD_ERR_INVALID;
  if (n == 0) return QD_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (vec_fp32)
    return launch<float>(n, nnz, width, b, ldx, ldy, d_rowptr, d_col, d_H, d_Himag, d_M, d_X, d_AX,
                         d_MX, s);
  return launch<double>(n, nnz, width, b, ldx, ldy, d_rowptr, d_col, d_H, d_Himag, d_M, d_X, d_AX,
                        d_MX, s);
}

extern "C" int qd_cap_spmm_lattice(int32_t n, int32_t width, int b, int vec_fp32,
                                   const int32_t *d_rowptr, const int32_t *d_col,
                                   const void *d_H, const void *d_Himag, const void *d_M,
                                   const void *d_X, int ldx, void *d_AX, void *d_MX, int ldy,
                                   void *stream) {
  return qd_cap_spmm_pattern(n, 0, width, b, vec_fp32, d_rowptr, d_col, d_H, d_Himag, d_M, d_X, ldx,
                             d_AX, d_MX, ldy, stream);
}

extern "C" int qd_cap_spmm(int32_t n, int b, int vec_fp32, const int32_t *d_rowptr,
                           const int32_t *d_col, const void *d_H, const void *d_Himag,
                           const void *d_M, const void *d_X, int ldx, void *d_AX, void *d_MX,
                           int ldy, void *stream) {
  return qd_cap_spmm_pattern(n, 0, 0, b, vec_fp32, d_rowptr, d_col, d_H, d_Himag, d_M, d_X, ldx,
                             d_AX, d_MX, ldy, stream);
}
