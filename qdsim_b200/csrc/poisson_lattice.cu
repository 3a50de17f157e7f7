// Poisson step on a structured rectangle: conjugate gradients, FP64, with a
// fast separable solver as the preconditioner.
//
// Replaces PoissonSolver::solve (backend/src/poisson.cpp:320-334,
// SimplicialLDLT) and the spsolve / cg calls of CythonPoissonSolver.solve
// (qdsim_cython/solvers/poisson_solver.pyx:238-247) on lattices; other
// matrices go to the Jacobi form in pcg.cu.
//
// The P1 stiffness of right triangles couples lattice neighbours only, with
// one conductance per lattice edge.  Averaging the conductances of each column
// of x-edges (gx[i]) and of y-edges (gy[i]) over y gives
//     Kt = Gx (x) My + diag(gy) (x) Ky,
// Gx the tridiagonal Dirichlet matrix of gx, Ky / My the Neumann second
// difference and its lumped mass.  Ky V = My V diag(2 - 2 cos(pi k / ny)) with
// V the cosine matrix (V^T My V = I), so Kt^-1 is a cosine transform along y,
// one tridiagonal solve along x per mode, and the transform back.  Kt differs
// from K only by the variation of eps along y: the condition number of
// Kt^-1 K is at most the largest over the smallest ratio of an edge's
// conductance to its column's mean (1 for layered devices), whatever the
// mesh.  Jacobi needs a count of iterations proportional to the mesh width:
// 300 x 100 cells with 64 right-hand sides took ~1000 iterations and 65.5 ms
// where this form takes 1.2 ms, and 100 x 50 cells with one right-hand side
// 31.5 ms against 0.24 ms (residual 1e-12, whole call, layered eps).
//
// Vectors are row-major [node][rhs], node = j (nx + 1) + i, i.e. [j][q] with
// q = i nrhs + c: both transforms are products with unit stride along q.  One
// iteration is five launches:
//   spmv    p = z + beta p_prev fused into A p; p.Ap -> alpha
//   axpy    x += alpha p, r -= alpha Ap; r.r -> converged flag
//   cosine  s = V^T r, folded (even modes from r_j + r_{ny-j}, odd ones from
//           the difference: half the products), on the FP64 matrix
//           instructions
//   sweep   the tridiagonal solves, eliminated from both ends to the middle
//   cosine  z = V s, unfolded; r.z -> beta
// Every reduction is summed in a fixed order by the block that finishes last.
#include <cuda_runtime.h>
#include <algorithm>
#include <cmath>
#include <vector>
#include "common.h"

namespace {

constexpr int kMaxRhs = 256;
constexpr int kT = 256;            // threads of every kernel but the sweep
constexpr int kMaxNx = 8000;       // one line of one column fits in shared memory
constexpr int kMaxNy = 16384;      // 2.1 GB of cosine matrices
constexpr int kNT = 64;            // lattice columns q per transform tile
constexpr int kMT = 64;            // modes (rows) per transform tile
constexpr int kKC = 16;            // contraction depth per stage
constexpr int kAP = kKC + 4, kBP = kNT + 4;   // pitches: fragments without bank conflicts
constexpr int kSweepT = 128;
// shared memory of a sweep block with cw columns: a line's factors and values
__host__ __device__ constexpr size_t sweep_bytes(int nx, int cw) {
  return size_t(nx + 1) * (sizeof(double2) + 8 * size_t(cw));
}
constexpr size_t kSweepWide = size_t(100) << 10;              // most for cw > 1
constexpr size_t kSweepMax = sweep_bytes(kMaxNx, 1);          // most of all: one column
static_assert(kSweepMax >= kSweepWide && kSweepMax <= (size_t(227) << 10), "fits an SM");

struct Dims {
  int nx, ny, nrhs, n;    // n = (nx + 1)(ny + 1)
  int Q;                  // (nx + 1) nrhs
  int H, Ho, Hp;          // even modes, odd modes, H rounded up to kMT
};

__host__ Dims dims_of(int nx, int ny, int nrhs) {
  Dims d;
  d.nx = nx;
  d.ny = ny;
  d.nrhs = nrhs;
  d.n = (nx + 1) * (ny + 1);
  d.Q = (nx + 1) * nrhs;
  d.H = ny / 2 + 1;
  d.Ho = (ny + 1) / 2;
  d.Hp = (d.H + kMT - 1) / kMT * kMT;
  return d;
}

// Plan of one lattice (doubles): four Hp x Hp cosine matrices, zero-padded
// (Ve^T, Vo^T for the forward transform, Ve, Vo for the way back), then per
// mode (nx + 1) pairs (1 / pivot, multiplier) of the tridiagonal factors.
__host__ __device__ inline size_t plan_mats(int Hp) { return size_t(4) * Hp * Hp; }

// ---------------------------------------------------------------------------
// Plan
// ---------------------------------------------------------------------------
__global__ void plan_cos_kernel(Dims d, double *plan) {
  const int64_t per = int64_t(d.Hp) * d.Hp;
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < 4 * per;
       e += int64_t(gridDim.x) * blockDim.x) {
    const int which = int(e / per), r = int((e % per) / d.Hp), c = int(e % d.Hp);
    // forward (0, 1): row = mode m, column = j; back (2, 3): row = j, column = m
    const int m = which < 2 ? r : c, j = which < 2 ? c : r;
    const int odd = which & 1, k = 2 * m + odd;
    double v = 0.0;
    if (j < d.H && m < (odd ? d.Ho : d.H)) {
      const double w = (k == 0 || k == d.ny) ? 1.0 / d.ny : 2.0 / d.ny;
      v = sqrt(w) * cospi(double((int64_t(j) * k) % (2 * int64_t(d.ny))) / d.ny);
    }
    plan[e] = v;
  }
}

// Tridiagonal factors of mode k (one thread each): pivots eliminated from both
// ends to the middle column; tri[k][i] = (1 / pivot_i, multiplier_i) with
// multiplier g / pivot along the edge towards the middle.
__global__ void plan_tri_kernel(Dims d, const double *gx, const double *gy, double2 *tri) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k > d.ny) return;
  const double mu = 2.0 - 2.0 * cospi(double(k) / d.ny);
  double2 *t = tri + size_t(k) * (d.nx + 1);
  const int mid = (d.nx + 1) / 2;
  t[0] = t[d.nx] = make_double2(0.0, 0.0);
  double carry = 0.0;                        // g^2 / pivot of the previous column
  for (int i = 1; i < mid; ++i) {
    const double di = 1.0 / (gx[i - 1] + gx[i] + gy[i] * mu - carry);
    t[i] = make_double2(di, gx[i] * di);
    carry = gx[i] * gx[i] * di;
  }
  const double left = carry;
  carry = 0.0;
  for (int i = d.nx - 1; i > mid; --i) {
    const double di = 1.0 / (gx[i - 1] + gx[i] + gy[i] * mu - carry);
    t[i] = make_double2(di, gx[i - 1] * di);
    carry = gx[i - 1] * gx[i - 1] * di;
  }
  if (mid > 0 && mid < d.nx)
    t[mid] = make_double2(1.0 / (gx[mid - 1] + gx[mid] + gy[mid] * mu - left - carry), 0.0);
}

// ---------------------------------------------------------------------------
// Reductions
// ---------------------------------------------------------------------------

// step scalars per right-hand side; `done` and the iteration count follow them
struct Scal {
  double rz, ref, alpha, beta, rr;
};

__device__ inline bool last_block(unsigned *counter, unsigned total) {
  __shared__ unsigned s_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(counter, 1u) == total - 1;
  }
  __syncthreads();
  if (s_last) __threadfence();
  return s_last;
}

// Sum over the rows r < rows of red[r * nrhs + j], a fixed tree; the result in
// red[j].  Every thread of the block calls it.
__device__ inline void tree_cols(double *red, int rows, int nrhs) {
  __syncthreads();
  while (rows > 1) {
    const int h = (rows + 1) / 2;
    for (int e = threadIdx.x; e < (rows - h) * nrhs; e += blockDim.x) red[e] += red[e + h * nrhs];
    __syncthreads();
    rows = h;
  }
}

// Column sums of per-thread values (thread t holds column t % nrhs, t below
// the largest multiple of nrhs) into part[blockIdx.x][j].
__device__ inline void block_cols(double v, double *red, int nrhs, double *part) {
  const int rows = blockDim.x / nrhs;
  __syncthreads();
  red[threadIdx.x] = v;
  tree_cols(red, rows, nrhs);
  for (int j = threadIdx.x; j < nrhs; j += blockDim.x)
    part[size_t(blockIdx.x) * nrhs + j] = red[j];
}

// In the last block: red[j] = sum over m < count of part[m * nrhs + j].
__device__ inline void gather_cols(const double *part, int count, int nrhs, double *red) {
  const int rows = blockDim.x / nrhs;          // lanes per column
  const int j = threadIdx.x % nrhs, l = threadIdx.x / nrhs;
  double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
  if (l < rows) {
    int m = l;
    for (; m + 3 * rows < count; m += 4 * rows) {
      a0 += __ldcg(part + size_t(m) * nrhs + j);
      a1 += __ldcg(part + size_t(m + rows) * nrhs + j);
      a2 += __ldcg(part + size_t(m + 2 * rows) * nrhs + j);
      a3 += __ldcg(part + size_t(m + 3 * rows) * nrhs + j);
    }
    for (; m < count; m += rows) a0 += __ldcg(part + size_t(m) * nrhs + j);
  }
  __syncthreads();
  if (l < rows) red[l * nrhs + j] = (a0 + a1) + (a2 + a3);
  tree_cols(red, rows, nrhs);
}

// ---------------------------------------------------------------------------
// Kernels of the iteration
// ---------------------------------------------------------------------------

struct Ends {   // Dirichlet values per right-hand side (x = 0 and x = Lx)
  double vp[kMaxRhs], vn[kMaxRhs];
};

struct Ctl {
  Scal *sc;
  int *done;         // [0] every column converged, [1] iterations
  unsigned *counter;
  double *part;
  double tol;
};

// X = the Dirichlet values on x = 0, Lx and X0 (or 0) elsewhere;
// r = alpha M rho - K X on the free nodes; the reference residual takes only
// the Dirichlet part of X
__global__ void __launch_bounds__(kT)
lat_init_kernel(Dims d, const int32_t *__restrict__ rowptr, const int32_t *__restrict__ col,
                const double *__restrict__ K, const double *__restrict__ M,
                const double *__restrict__ rho, double alpha, const __grid_constant__ Ends ends,
                const double *X0, double *X, double *R, double *P, Ctl ctl) {
  __shared__ double red[kT];
  const int rpb = blockDim.x / d.nrhs;
  const int j = threadIdx.x % d.nrhs;
  const double vp = ends.vp[j], vn = ends.vn[j];
  const int w = d.nx + 1;
  double rr = 0.0, r0 = 0.0;
  for (int row = blockIdx.x * rpb + threadIdx.x / d.nrhs; row < d.n; row += gridDim.x * rpb) {
    const size_t idx = size_t(row) * d.nrhs + j;
    const int i = row % w;
    const bool fixed = i == 0 || i == d.nx;
    double r = 0.0, rd = 0.0;
    if (!fixed) {
      double b = 0.0, ax = 0.0, ad = 0.0;
      for (int p = rowptr[row]; p < rowptr[row + 1]; ++p) {
        const int cj = col[p], ci = cj % w;
        const double a = K[p];
        const size_t at = size_t(cj) * d.nrhs + j;
        b = fma(M[p], rho[at], b);
        if (ci == 0 || ci == d.nx)
          ad = fma(a, ci == 0 ? vp : vn, ad);
        else if (X0)
          ax = fma(a, X0[at], ax);
      }
      rd = alpha * b - ad;
      r = rd - ax;
    }
    X[idx] = fixed ? (i == 0 ? vp : vn) : (X0 ? X0[idx] : 0.0);
    R[idx] = r;
    P[idx] = 0.0;
    rr += r * r;
    r0 += rd * rd;
  }
  block_cols(rr, red, d.nrhs, ctl.part);
  block_cols(r0, red, d.nrhs, ctl.part + size_t(gridDim.x) * d.nrhs);
  if (!last_block(ctl.counter, gridDim.x)) return;
  __shared__ int s_open;
  if (threadIdx.x == 0) s_open = 0;
  gather_cols(ctl.part, gridDim.x, d.nrhs, red);
  double s_rr = threadIdx.x < d.nrhs ? red[threadIdx.x] : 0.0;
  gather_cols(ctl.part + size_t(gridDim.x) * d.nrhs, gridDim.x, d.nrhs, red);
  if (threadIdx.x < d.nrhs) {
    const double ref = red[threadIdx.x] > 0.0 ? red[threadIdx.x] : s_rr;
    ctl.sc[threadIdx.x] = Scal{0.0, ref, 0.0, 0.0, s_rr};
    if (!(s_rr <= ctl.tol * ctl.tol * ref)) atomicOr(&s_open, 1);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    ctl.done[0] = !s_open;
    ctl.done[1] = 0;
    *ctl.counter = 0u;
  }
}

__global__ void __launch_bounds__(kT)
lat_spmv_kernel(Dims d, const int32_t *__restrict__ rowptr, const int32_t *__restrict__ col,
                const double *__restrict__ K, const double *__restrict__ Z,
                const double *__restrict__ Pprev, double *__restrict__ P, double *__restrict__ AP,
                Ctl ctl) {
  __shared__ double red[kT];
  if (*ctl.done) return;
  const int rpb = blockDim.x / d.nrhs;
  const int j = threadIdx.x % d.nrhs;
  const int w = d.nx + 1;
  const double beta = ctl.sc[j].beta;
  double pap = 0.0;
  for (int row = blockIdx.x * rpb + threadIdx.x / d.nrhs; row < d.n; row += gridDim.x * rpb) {
    const size_t idx = size_t(row) * d.nrhs + j;
    const int i = row % w;
    double ap = 0.0;
    if (i != 0 && i != d.nx) {
      const int p1 = rowptr[row + 1];
#pragma unroll 8
      for (int p = rowptr[row]; p < p1; ++p) {
        const size_t q = size_t(col[p]) * d.nrhs + j;
        ap = fma(K[p], fma(beta, Pprev[q], Z[q]), ap);
      }
    }
    const double pi = fma(beta, Pprev[idx], Z[idx]);
    P[idx] = pi;
    AP[idx] = ap;
    pap = fma(pi, ap, pap);
  }
  block_cols(pap, red, d.nrhs, ctl.part);
  if (!last_block(ctl.counter, gridDim.x)) return;
  gather_cols(ctl.part, gridDim.x, d.nrhs, red);
  if (threadIdx.x < d.nrhs) {
    Scal &s = ctl.sc[threadIdx.x];
    const double pa = red[threadIdx.x];
    s.alpha = (pa > 0.0 && s.rr > ctl.tol * ctl.tol * s.ref) ? s.rz / pa : 0.0;
  }
  if (threadIdx.x == 0) *ctl.counter = 0u;
}

__global__ void __launch_bounds__(kT)
lat_axpy_kernel(Dims d, double *__restrict__ X, double *__restrict__ R,
                const double *__restrict__ P, const double *__restrict__ AP, Ctl ctl) {
  __shared__ double red[kT];
  if (*ctl.done) return;
  const int rpb = blockDim.x / d.nrhs;
  const int j = threadIdx.x % d.nrhs;
  const double alpha = ctl.sc[j].alpha;
  double rr = 0.0;
  for (int row = blockIdx.x * rpb + threadIdx.x / d.nrhs; row < d.n; row += gridDim.x * rpb) {
    const size_t idx = size_t(row) * d.nrhs + j;
    X[idx] = fma(alpha, P[idx], X[idx]);
    const double r = fma(-alpha, AP[idx], R[idx]);
    R[idx] = r;
    rr = fma(r, r, rr);
  }
  block_cols(rr, red, d.nrhs, ctl.part);
  if (!last_block(ctl.counter, gridDim.x)) return;
  __shared__ int s_open;
  if (threadIdx.x == 0) s_open = 0;
  gather_cols(ctl.part, gridDim.x, d.nrhs, red);
  if (threadIdx.x < d.nrhs) {
    Scal &s = ctl.sc[threadIdx.x];
    s.rr = red[threadIdx.x];
    if (!(s.rr <= ctl.tol * ctl.tol * s.ref)) atomicOr(&s_open, 1);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    ctl.done[0] = !s_open;
    ctl.done[1] += 1;
    *ctl.counter = 0u;
  }
}

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// One stage of operands: both parities of the matrix (kMT x kKC) and of the
// data (kKC x kNT).
struct Stage {
  double a[2][kMT * kAP];
  double b[2][kKC * kBP];
};

// Cosine transform of a tile of kNT lattice columns.  FWD: out rows are modes
// 2m + parity, in rows j folded.  Back: out rows j and ny - j unfolded from
// modes; also r.z per column q into dotq[blockIdx.y][q], summed by the last
// block.  Eight warps, each 8 columns x 64 rows x both parities (16 fragment
// pairs of the FP64 matrix instruction); the data tile is read from memory
// once for both parities, the next stage is loaded while the current one
// multiplies.
template <bool FWD>
__global__ void __launch_bounds__(kT, 2)
lat_cos_kernel(Dims d, const double *__restrict__ plan, const double *__restrict__ in,
               double *__restrict__ out, const double *__restrict__ R, double *dotq, Ctl ctl) {
  extern __shared__ __align__(16) unsigned char sm_raw[];
  Stage *st = reinterpret_cast<Stage *>(sm_raw);
  if (*ctl.done) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int q0 = blockIdx.x * kNT, m0 = blockIdx.y * kMT;
  const size_t per = size_t(d.Hp) * d.Hp;
  const double *Ae = plan + (FWD ? 0 : 2) * per, *Ao = Ae + per;
  const int depth = d.H;                       // H >= Ho
  const int nst = (depth + kKC - 1) / kKC;
  // loads of a thread: 4 + 4 matrix entries, 4 + 4 data entries
  const int ar = tid >> 2, ac = (tid & 3) * 4;          // row, first of 4 columns
  const int bq = tid & 63, br = tid >> 6;               // column, first row (step 4)
  const bool qin = q0 + bq < d.Q;
  double la[2][4], lb[2][4];
  auto load = [&](int s) {
    const size_t ao = size_t(m0 + ar) * d.Hp + s * kKC + ac;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      la[0][u] = Ae[ao + u];
      la[1][u] = Ao[ao + u];
      const int h = s * kKC + br + 4 * u;
      double x0 = 0.0, x1 = 0.0;
      if (qin) {
        if (FWD) {
          if (h < d.H) {
            const double up = in[size_t(h) * d.Q + q0 + bq];
            const double dn = d.ny - h != h ? in[size_t(d.ny - h) * d.Q + q0 + bq] : 0.0;
            x0 = up + dn;
            x1 = d.ny - h != h ? up - dn : 0.0;
          }
        } else {
          if (h < d.H) x0 = in[size_t(2 * h) * d.Q + q0 + bq];
          if (h < d.Ho) x1 = in[size_t(2 * h + 1) * d.Q + q0 + bq];
        }
      }
      lb[0][u] = x0;
      lb[1][u] = x1;
    }
  };
  auto store = [&](int s) {
    Stage &g = st[s & 1];
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        g.a[p][ar * kAP + ac + u] = la[p][u];
        g.b[p][(br + 4 * u) * kBP + bq] = lb[p][u];
      }
  };
  double c[2][8][2];
#pragma unroll
  for (int p = 0; p < 2; ++p)
#pragma unroll
    for (int t = 0; t < 8; ++t) c[p][t][0] = c[p][t][1] = 0.0;
  // row tiles of 8 in use (the matrices are zero-padded)
  const int mt = min(8, (d.H - m0 + 7) / 8);
  load(0);
  store(0);
  __syncthreads();
  for (int s = 0; s < nst; ++s) {
    if (s + 1 < nst) load(s + 1);
    const Stage &g = st[s & 1];
    const int fr = lane >> 2, fk = lane & 3;
#pragma unroll
    for (int k4 = 0; k4 < kKC; k4 += 4) {
      const double be = g.b[0][(k4 + fk) * kBP + warp * 8 + fr];
      const double bo = g.b[1][(k4 + fk) * kBP + warp * 8 + fr];
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        if (t < mt) {
          dmma(c[0][t], g.a[0][(t * 8 + fr) * kAP + k4 + fk], be);
          dmma(c[1][t], g.a[1][(t * 8 + fr) * kAP + k4 + fk], bo);
        }
      }
    }
    if (s + 1 < nst) store(s + 1);   // the other buffer: last read a barrier ago
    __syncthreads();
  }
  const int row0 = m0 + (lane >> 2), qc = q0 + warp * 8 + 2 * (lane & 3);
  double dt[2] = {0.0, 0.0};
#pragma unroll
  for (int t = 0; t < 8; ++t) {
    const int h = row0 + 8 * t;
#pragma unroll
    for (int v = 0; v < 2; ++v) {
      if (t >= mt || h >= d.H || qc + v >= d.Q) continue;
      if (FWD) {
        out[size_t(2 * h) * d.Q + qc + v] = c[0][t][v];
        if (h < d.Ho) out[size_t(2 * h + 1) * d.Q + qc + v] = c[1][t][v];
      } else {
        const size_t up = size_t(h) * d.Q + qc + v;
        const double z = c[0][t][v] + c[1][t][v];
        out[up] = z;
        dt[v] = fma(R[up], z, dt[v]);
        if (d.ny - h != h) {
          const size_t dn = size_t(d.ny - h) * d.Q + qc + v;
          const double y = c[0][t][v] - c[1][t][v];
          out[dn] = y;
          dt[v] = fma(R[dn], y, dt[v]);
        }
      }
    }
  }
  if (FWD) return;
#pragma unroll
  for (int v = 0; v < 2; ++v) {
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) dt[v] += __shfl_xor_sync(0xffffffffu, dt[v], o);
    if (lane < 4 && qc + v < d.Q) dotq[size_t(blockIdx.y) * d.Q + qc + v] = dt[v];
  }
  if (!last_block(ctl.counter, gridDim.x * gridDim.y)) return;
  double *red = reinterpret_cast<double *>(sm_raw);
  // dotq is [gridDim.y][nx + 1][nrhs]
  gather_cols(dotq, int(gridDim.y) * (d.nx + 1), d.nrhs, red);
  if (tid < d.nrhs) {
    Scal &s = ctl.sc[tid];
    s.beta = s.rz > 0.0 ? red[tid] / s.rz : 0.0;
    s.rz = red[tid];
  }
  if (tid == 0) *ctl.counter = 0u;
}

// Tridiagonal solves along x: block (mode k, columns c0 .. c0 + cw).  The line
// is staged in shared memory; two warps eliminate from both ends to the middle
// and substitute back, so the serial chain is half the line.
__global__ void __launch_bounds__(kSweepT)
lat_sweep_kernel(Dims d, int cw, const double2 *__restrict__ tri, double *__restrict__ S, Ctl ctl) {
  extern __shared__ __align__(16) unsigned char sm_raw[];
  if (*ctl.done) return;
  double2 *t = reinterpret_cast<double2 *>(sm_raw);               // [nx + 1]
  double *y = reinterpret_cast<double *>(t + d.nx + 1);           // [nx + 1][cw]
  const int k = blockIdx.x, c0 = blockIdx.y * cw, tid = threadIdx.x;
  const int nc = min(cw, d.nrhs - c0);
  double *line = S + size_t(k) * d.Q + c0;
  for (int i = tid; i <= d.nx; i += kSweepT) t[i] = tri[size_t(k) * (d.nx + 1) + i];
  for (int e = tid; e < (d.nx + 1) * cw; e += kSweepT) {
    const int i = e / cw, c = e - i * cw;
    y[e] = c < nc ? line[size_t(i) * d.nrhs + c] : 0.0;
  }
  __syncthreads();
  const int mid = (d.nx + 1) / 2, side = tid >> 5, c = tid & 31;
  if (side < 2 && c < cw) {
    const int step = side ? -1 : 1;
    int i = side ? d.nx - 1 : 1;
    const int count = side ? d.nx - 1 - mid : mid - 1;   // columns before the middle
    double a = 0.0, m = 0.0;
#pragma unroll 8
    for (int u = 0; u < count; ++u, i += step) {
      a = fma(m, a, y[i * cw + c]);
      y[i * cw + c] = a;
      m = t[i].y;
    }
    // this side's contribution to the middle column, in its own end row
    y[(side ? d.nx : 0) * cw + c] = m * a;
  }
  __syncthreads();
  double x = 0.0;
  if (side < 2 && c < cw) x = (y[mid * cw + c] + y[c] + y[d.nx * cw + c]) * t[mid].x;
  __syncthreads();
  if (side < 2 && c < cw) {
    if (side == 0) y[mid * cw + c] = x;
    const int step = side ? 1 : -1;
    int i = mid + step;
    const int count = side ? d.nx - 1 - mid : mid - 1;
#pragma unroll 8
    for (int u = 0; u < count; ++u, i += step) {
      x = fma(t[i].y, x, y[i * cw + c] * t[i].x);
      y[i * cw + c] = x;
    }
    y[(side ? d.nx : 0) * cw + c] = 0.0;
  }
  __syncthreads();
  for (int e = tid; e < (d.nx + 1) * cw; e += kSweepT) {
    const int i = e / cw, c1 = e - i * cw;
    if (c1 < nc) line[size_t(i) * d.nrhs + c1] = y[e];
  }
}

// ---------------------------------------------------------------------------
// Host
// ---------------------------------------------------------------------------
struct Layout {
  double *R, *S, *Z, *P[2], *AP, *part, *dotq;
  Scal *sc;        // [nrhs], then done[2]
  unsigned *counter;
};

constexpr int kBlocks = 4 * 148;   // elementwise kernels: at most four blocks per SM

int elem_threads(const Dims &d) { return kT / d.nrhs * d.nrhs; }
int elem_blocks(const Dims &d) {
  const int rpb = kT / d.nrhs;
  return std::max(1, std::min((d.n + rpb - 1) / rpb, kBlocks));
}

void carve(qd::Arena &ar, const Dims &d, Layout &L) {
  const size_t nv = size_t(d.n) * d.nrhs;
  L.R = ar.take<double>(nv);
  L.S = ar.take<double>(nv);
  L.Z = ar.take<double>(nv);
  L.P[0] = ar.take<double>(nv);
  L.P[1] = ar.take<double>(nv);
  L.AP = ar.take<double>(nv);
  L.part = ar.take<double>(size_t(2) * kBlocks * d.nrhs);
  L.dotq = ar.take<double>(size_t(d.Hp / kMT) * d.Q);
  L.sc = reinterpret_cast<Scal *>(ar.take<double>(size_t(d.nrhs) * (sizeof(Scal) / 8) + 1));
  L.counter = ar.take<unsigned>(4);
}

bool valid_lattice(int nx, int ny, int nrhs) {
  return nx >= 1 && nx <= kMaxNx && ny >= 1 && ny <= kMaxNy && nrhs >= 1 && nrhs <= kMaxRhs &&
         (int64_t(nx) + 1) * (int64_t(ny) + 1) <= INT32_MAX &&
         (int64_t(nx) + 1) * nrhs <= INT32_MAX;
}

}  // namespace

extern "C" int qd_poisson_lattice_plan_size(int nx, int ny, size_t *bytes) {
  if (!bytes || !valid_lattice(nx, ny, 1)) return QD_ERR_INVALID;
  const Dims d = dims_of(nx, ny, 1);
  *bytes = (plan_mats(d.Hp) + size_t(2) * (ny + 1) * (nx + 1)) * sizeof(double);
  return QD_OK;
}

extern "C" int qd_poisson_lattice_plan(int nx, int ny, const double *d_gx, const double *d_gy,
                                       void *d_plan, size_t plan_bytes, void *stream) {
  if (!valid_lattice(nx, ny, 1) || !d_gx || !d_gy || !d_plan) return QD_ERR_INVALID;
  const Dims d = dims_of(nx, ny, 1);
  size_t need = 0;
  qd_poisson_lattice_plan_size(nx, ny, &need);
  if (plan_bytes < need || reinterpret_cast<uintptr_t>(d_plan) % 16) return QD_ERR_WORKSPACE;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  double *plan = static_cast<double *>(d_plan);
  plan_cos_kernel<<<296, 256, 0, s>>>(d, plan);
  QD_CHECK_LAUNCH();
  plan_tri_kernel<<<(ny + 1 + 63) / 64, 64, 0, s>>>(
      d, d_gx, d_gy, reinterpret_cast<double2 *>(plan + plan_mats(d.Hp)));
  QD_CHECK_LAUNCH();
  return QD_OK;
}

extern "C" int qd_poisson_lattice_workspace_size(int nx, int ny, int nrhs, size_t *bytes) {
  if (!bytes || !valid_lattice(nx, ny, nrhs)) return QD_ERR_INVALID;
  qd::Arena ar(nullptr, 0);
  Layout L;
  carve(ar, dims_of(nx, ny, nrhs), L);
  *bytes = ar.used;
  return QD_OK;
}

extern "C" int qd_poisson_lattice_solve(int nx, int ny, int nrhs, const int32_t *d_rowptr,
                                        const int32_t *d_col, const double *d_K,
                                        const double *d_M, const double *d_rho, double alpha,
                                        const double *h_left, const double *h_right,
                                        const double *d_X0, double *d_X, const void *d_plan,
                                        double tol, int max_iter, int32_t *h_iters,
                                        double *h_relres, void *d_work, size_t work_bytes,
                                        void *stream) {
  if (!valid_lattice(nx, ny, nrhs) || !d_rowptr || !d_col || !d_K || !d_M || !d_rho || !h_left ||
      !h_right || !d_X || d_X == d_X0 || !d_plan || !d_work || !(tol > 0.0) || max_iter < 1)
    return QD_ERR_INVALID;
  if (reinterpret_cast<uintptr_t>(d_plan) % 16) return QD_ERR_INVALID;
  const Dims d = dims_of(nx, ny, nrhs);
  {
    qd::Arena need(nullptr, 0);
    Layout t;
    carve(need, d, t);
    if (need.used > work_bytes) return QD_ERR_WORKSPACE;
  }
  if (reinterpret_cast<uintptr_t>(d_work) % 256) return QD_ERR_WORKSPACE;
  qd::Arena ar(d_work, work_bytes);
  Layout L;
  carve(ar, d, L);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  Ends ends;
  for (int j = 0; j < kMaxRhs; ++j) {
    ends.vp[j] = j < nrhs ? h_left[j] : 0.0;
    ends.vn[j] = j < nrhs ? h_right[j] : 0.0;
  }
  Ctl ctl;
  ctl.sc = L.sc;
  ctl.done = reinterpret_cast<int *>(L.sc + nrhs);
  ctl.counter = L.counter;
  ctl.part = L.part;
  ctl.tol = tol;
  const double *plan = static_cast<const double *>(d_plan);
  const double2 *tri = reinterpret_cast<const double2 *>(plan + plan_mats(d.Hp));
  const int T = elem_threads(d), G = elem_blocks(d);
  const dim3 cgrid((d.Q + kNT - 1) / kNT, d.Hp / kMT);
  const int cbytes = 2 * int(sizeof(Stage));
  int cw = std::min(32, nrhs);
  while (cw > 1 && sweep_bytes(nx, cw) > kSweepWide) cw = (cw + 1) / 2;
  const dim3 sgrid(ny + 1, (nrhs + cw - 1) / cw);
  QD_CUDA_TRY(cudaFuncSetAttribute(lat_cos_kernel<true>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, cbytes));
  QD_CUDA_TRY(cudaFuncSetAttribute(lat_cos_kernel<false>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, cbytes));
  // a constant, as for every kernel: the limit belongs to the process, and a
  // smaller one set for a small lattice would fail another thread's launch
  QD_CUDA_TRY(cudaFuncSetAttribute(lat_sweep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   int(kSweepMax)));
  qd::prof_begin(qd::PK_PCG, s);
  QD_CUDA_TRY(cudaMemsetAsync(L.counter, 0, 4 * sizeof(unsigned), s));
  lat_init_kernel<<<G, T, 0, s>>>(d, d_rowptr, d_col, d_K, d_M, d_rho, alpha, ends, d_X0, d_X, L.R,
                                  L.P[0], ctl);
  QD_CHECK_LAUNCH();
  auto precond = [&]() -> int {
    lat_cos_kernel<true><<<cgrid, kT, cbytes, s>>>(d, plan, L.R, L.S, nullptr, nullptr, ctl);
    QD_CHECK_LAUNCH();
    lat_sweep_kernel<<<sgrid, kSweepT, sweep_bytes(nx, cw), s>>>(d, cw, tri, L.S, ctl);
    QD_CHECK_LAUNCH();
    lat_cos_kernel<false><<<cgrid, kT, cbytes, s>>>(d, plan, L.S, L.Z, L.R, L.dotq, ctl);
    QD_CHECK_LAUNCH();
    return QD_OK;
  };
  int st = precond();
  if (st != QD_OK) return st;
  // scalars and flags come back in one copy; the host looks after every kCheck
  // iterations (the launches left over return at once)
  constexpr int kCheck = 4;
  std::vector<double> back(size_t(nrhs) * (sizeof(Scal) / 8) + 1);
  int flags[2] = {0, 0};
  for (int it = 0; it < max_iter && !flags[0];) {
    const int upto = std::min(max_iter, it + kCheck);
    for (; it < upto; ++it) {
      lat_spmv_kernel<<<G, T, 0, s>>>(d, d_rowptr, d_col, d_K, L.Z, L.P[it & 1], L.P[(it + 1) & 1],
                                      L.AP, ctl);
      QD_CHECK_LAUNCH();
      lat_axpy_kernel<<<G, T, 0, s>>>(d, d_X, L.R, L.P[(it + 1) & 1], L.AP, ctl);
      QD_CHECK_LAUNCH();
      if ((st = precond()) != QD_OK) return st;
    }
    QD_CUDA_TRY(cudaMemcpyAsync(back.data(), L.sc, back.size() * sizeof(double),
                                cudaMemcpyDeviceToHost, s));
    QD_CUDA_TRY(cudaStreamSynchronize(s));
    std::copy_n(reinterpret_cast<const int *>(back.data() + back.size() - 1), 2, flags);
    bool finite = true;   // NaN inputs never converge: no more iterations for them
    for (int j = 0; j < nrhs; ++j)
      finite = finite && std::isfinite(reinterpret_cast<const Scal *>(back.data())[j].rr);
    if (!finite) break;
  }
  qd::prof_end(qd::PK_PCG, s);
  const Scal *sc = reinterpret_cast<const Scal *>(back.data());
  double worst = 0.0;
  for (int j = 0; j < nrhs; ++j)
    worst = std::max(worst, sc[j].ref > 0.0 ? std::sqrt(sc[j].rr / sc[j].ref) : 0.0);
  if (h_iters) *h_iters = flags[1];
  if (h_relres) *h_relres = worst;
  return flags[0] ? QD_OK : QD_ERR_NOT_CONVERGED;
}
