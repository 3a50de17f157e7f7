// Adjoint (Hellmann-Feynman) gradients of L = Re sum_s w_s E_s.
//
// For the Hermitian pencil (H, M) with M-normalised real eigenvectors and for
// the complex-symmetric open-system pencil (H + i Himag, M) with bilinearly
// normalised complex eigenvectors (x^T M x = 1, no conjugation, so that the
// left eigenvector is x itself), M depends on neither V nor c and
//   dE_s/dp = x_s^T (dH/dp) x_s.
// Per element e with local nodes i, j and U_ij = Re sum_s w_s x_si x_sj
// (complex weights w_s = dL/dRe E_s - i dL/dIm E_s):
//   dL/dV_g = sum_{(e, l): node g} A_e sum_ij T_lij U_ij
//   dL/dc_e = A_e sum_ij (g00 Sxx + g01 Sxy + g11 Syy)_ij U_ij
// with the assembly kernel's reference tables (T_lij = int phi_l phi_i phi_j
// on the reference triangle).
//
// Two launches.  The element pass takes a thread per element: the products
// U_ij of the K (K + 1) / 2 pairs i <= j (U, T and the stiffness tables are
// symmetric in i, j) build up in registers state by state, then go through the
// tables, which are constant operands of the arithmetic, into dL/dc_e and the
// element's K nodal contributions (caller scratch, [K][num_elems]).  The node
// pass sums each node's contributions over its incident elements in adjacency
// order, so every result is reproducible without atomics, and each element is
// evaluated once.  T_lij is the integral of three basis functions, symmetric in
// all of l, i, j: each of its values is read once and serves up to three sums
// (the constant cache holds 2 KB of the 8.8 KB table, so the walk over it is
// what the element pass waits for).  Latency bounds both passes at these sizes
// (a P3 mesh of 22,500 elements is 700 warps).  Before, a group of 8 to 32 lanes shared an element
// through shared memory and summed its K + 1 results by shuffles: 54 us where
// this takes 15 us cold (P3, 22,500 elements, 4 states; a whole gradient call
// 76 us before, 18 us now, with the weights passed in the launch).
// No reference counterpart (the reference has no derivatives); checked against
// central finite differences and the FP64 oracle gradient.
#include <cuda_runtime.h>
#include <algorithm>
#include "common.h"
#include "devtables.cuh"

namespace {

constexpr int kMaxStates = 16;
constexpr int kThreads = 64;      // small blocks: the element pass has few warps per SM

// Weights by value (host weights) or in device memory.
struct Weights {
  const double *d;                 // [ns], or (re, im) per state; nullptr: v
  double v[2 * kMaxStates];
};

// Place of (i, j), i <= j, among the pairs in row order.
__host__ __device__ constexpr int pair_at(int k, int i, int j) {
  return i * k - i * (i - 1) / 2 + (j - i);
}

// Pass 1, one thread per element: dL/dc_e and gl[l][e] = A_e sum_ij T_lij U_ij.
template <int K, bool CPLX>
__global__ void __launch_bounds__(kThreads)
adjoint_elem_kernel(int64_t ne, int ns, const double2 *__restrict__ nodes,
                    const int32_t *__restrict__ elems, const int32_t *__restrict__ dofmap,
                    const double *__restrict__ psi, const __grid_constant__ Weights w,
                    double *__restrict__ dLdc, double *__restrict__ gl) {
  constexpr int KK = K * K, NP = K * (K + 1) / 2, B0 = TabBase<K>::v;
  const int64_t e = int64_t(blockIdx.x) * kThreads + threadIdx.x;
  if (e >= ne) return;
  int dof[K];
  double2 p0, p1, p2;
  {
    int g[K];
#pragma unroll
    for (int i = 0; i < K; ++i) g[i] = elems[e * K + i];
    p0 = nodes[g[0]];
    p1 = nodes[g[1]];
    p2 = nodes[g[2]];
#pragma unroll
    for (int i = 0; i < K; ++i) dof[i] = dofmap[g[i]];
  }
  double U[NP];                    // twice U_ij for i < j
#pragma unroll
  for (int q = 0; q < NP; ++q) U[q] = 0.0;
  for (int s = 0; s < ns; ++s) {
    double re[K], im[CPLX ? K : 1];
#pragma unroll
    for (int i = 0; i < K; ++i) {
      re[i] = 0.0;
      if constexpr (CPLX) im[i] = 0.0;
      if (dof[i] >= 0) {
        if constexpr (CPLX) {
          const double2 z = reinterpret_cast<const double2 *>(psi)[size_t(dof[i]) * ns + s];
          re[i] = z.x;
          im[i] = z.y;
        } else {
          re[i] = psi[size_t(dof[i]) * ns + s];
        }
      }
    }
    if constexpr (CPLX) {
      const double wr = w.d ? w.d[2 * s] : w.v[2 * s], wi = w.d ? w.d[2 * s + 1] : w.v[2 * s + 1];
#pragma unroll
      for (int i = 0, q = 0; i < K; ++i) {
        // Re (w x_i) x_j, with (a + i b) = w x_i
        const double a = wr * re[i] - wi * im[i], b = wr * im[i] + wi * re[i];
#pragma unroll
        for (int j = i; j < K; ++j, ++q)
          U[q] = fma(j == i ? a : 2.0 * a, re[j], fma(j == i ? -b : -2.0 * b, im[j], U[q]));
      }
    } else {
      const double ws = w.d ? w.d[s] : w.v[s];
#pragma unroll
      for (int i = 0, q = 0; i < K; ++i) {
        const double a = ws * re[i], a2 = 2.0 * a;
#pragma unroll
        for (int j = i; j < K; ++j, ++q) U[q] = fma(j == i ? a : a2, re[j], U[q]);
      }
    }
  }
  const double ja = p1.x - p0.x, jb = p2.x - p0.x, jc = p1.y - p0.y, jd = p2.y - p0.y;
  const double det = ja * jd - jb * jc;
  const double A = 0.5 * fabs(det);
  const double inv2 = 1.0 / (det * det);
  const double g00 = (jd * jd + jb * jb) * inv2;
  const double g01 = -(jd * jc + jb * ja) * inv2;
  const double g11 = (jc * jc + ja * ja) * inv2;
  double sx = 0.0, sm = 0.0, sy = 0.0;
#pragma unroll
  for (int i = 0, q = 0; i < K; ++i)
#pragma unroll
    for (int j = i; j < K; ++j, ++q) {
      sx = fma(c_tab[B0 + KK + i * K + j], U[q], sx);
      sm = fma(c_tab[B0 + 2 * KK + i * K + j], U[q], sm);
      sy = fma(c_tab[B0 + 3 * KK + i * K + j], U[q], sy);
    }
  dLdc[e] = A * (g00 * sx + g01 * sm + g11 * sy);
  double v[K];
#pragma unroll
  for (int l = 0; l < K; ++l) v[l] = 0.0;
#pragma unroll
  for (int a = 0; a < K; ++a)
#pragma unroll
    for (int b = a; b < K; ++b)
#pragma unroll
      for (int c = b; c < K; ++c) {
        const double t = c_tab[B0 + 4 * KK + a * KK + b * K + c];
        v[a] = fma(t, U[pair_at(K, b, c)], v[a]);
        if (b != a) v[b] = fma(t, U[pair_at(K, a, c)], v[b]);
        if (c != b) v[c] = fma(t, U[pair_at(K, a, b)], v[c]);
      }
#pragma unroll
  for (int l = 0; l < K; ++l) gl[size_t(l) * ne + e] = A * v[l];
}

// Pass 2, one thread per node: dL/dV_g = sum over the node's incident
// (element, local index) pairs, in adjacency order, of gl[l][e].
template <int K>
__global__ void adjoint_node_kernel(int64_t nn, int64_t ne, const int32_t *__restrict__ nadjptr,
                                    const int32_t *__restrict__ nadj,
                                    const double *__restrict__ gl, double *__restrict__ dLdV) {
  for (int64_t g = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; g < nn;
       g += int64_t(gridDim.x) * blockDim.x) {
    double acc = 0.0;
    for (int t = nadjptr[g]; t < nadjptr[g + 1]; ++t) {
      const int packed = nadj[t];
      acc += gl[size_t(packed & 15) * ne + (packed >> 4)];
    }
    dLdV[g] = acc;
  }
}

template <int K>
int launch_adjoint(int64_t nn, int64_t ne, int ns, bool cplx, const double *nodes,
                   const int32_t *elems, const int32_t *dofmap, const double *psi,
                   const Weights &w, const int32_t *nadjptr, const int32_t *nadj, double *dLdV,
                   double *dLdc, double *gl, cudaStream_t s) {
  const double2 *nd = reinterpret_cast<const double2 *>(nodes);
  const unsigned eblocks = unsigned((ne + kThreads - 1) / kThreads);
  qd::prof_begin(qd::PK_ADJOINT, s);
  if (cplx)
    adjoint_elem_kernel<K, true><<<eblocks, kThreads, 0, s>>>(ne, ns, nd, elems, dofmap, psi, w,
                                                             dLdc, gl);
  else
    adjoint_elem_kernel<K, false><<<eblocks, kThreads, 0, s>>>(ne, ns, nd, elems, dofmap, psi,
                                                              w, dLdc, gl);
  QD_CHECK_LAUNCH();
  const int nblocks = int(std::min<int64_t>((nn + 255) / 256, 148 * 16));
  adjoint_node_kernel<K><<<nblocks, 256, 0, s>>>(nn, ne, nadjptr, nadj, gl, dLdV);
  QD_CHECK_LAUNCH();
  qd::prof_end(qd::PK_ADJOINT, s);
  return QD_OK;
}

int adjoint_any(int order, int64_t num_nodes, int64_t num_elems, int n_states, int is_complex,
                const double *d_nodes, const int32_t *d_elems, const int32_t *d_dofmap,
                const double *d_psi, const Weights &w, const int32_t *d_nadjptr,
                const int32_t *d_nadj, double *d_dLdV, double *d_dLdc, double *d_work,
                void *stream) {
  if (num_elems >= (int64_t(1) << 27) || num_nodes >= (int64_t(1) << 31)) return QD_ERR_LIMIT;
  if (!d_nodes || !d_elems || !d_dofmap || !d_psi || !d_nadjptr || !d_nadj || !d_dLdV || !d_dLdc ||
      !d_work)
    return QD_ERR_INVALID;
  if (is_complex && (reinterpret_cast<uintptr_t>(d_psi) & 15)) return QD_ERR_INVALID;
  int st = ensure_tables();
  if (st != QD_OK) return st;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const bool c = is_complex != 0;
  switch (order) {
    case 1: return launch_adjoint<3>(num_nodes, num_elems, n_states, c, d_nodes, d_elems, d_dofmap, d_psi, w, d_nadjptr, d_nadj, d_dLdV, d_dLdc, d_work, s);
    case 2: return launch_adjoint<6>(num_nodes, num_elems, n_states, c, d_nodes, d_elems, d_dofmap, d_psi, w, d_nadjptr, d_nadj, d_dLdV, d_dLdc, d_work, s);
    default: return launch_adjoint<10>(num_nodes, num_elems, n_states, c, d_nodes, d_elems, d_dofmap, d_psi, w, d_nadjptr, d_nadj, d_dLdV, d_dLdc, d_work, s);
  }
}
}  // namespace

extern "C" int qd_adjoint(int order, int64_t num_nodes, int64_t num_elems, int n_states,
                          int is_complex, const double *d_nodes, const int32_t *d_elems,
                          const int32_t *d_dofmap, const double *d_psi, const double *d_w,
                          const int32_t *d_nadjptr, const int32_t *d_nadj, double *d_dLdV,
                          double *d_dLdc, double *d_work, void *stream) {
  if (order < 1 || order > 3 || num_nodes <= 0 || num_elems <= 0) return QD_ERR_INVALID;
  if (n_states < 1 || n_states > kMaxStates) return QD_ERR_LIMIT;
  if (!d_w) return QD_ERR_INVALID;
  Weights w{};
  w.d = d_w;
  return adjoint_any(order, num_nodes, num_elems, n_states, is_complex, d_nodes, d_elems, d_dofmap,
                     d_psi, w, d_nadjptr, d_nadj, d_dLdV, d_dLdc, d_work, stream);
}

extern "C" int qd_adjoint_host_weights(int order, int64_t num_nodes, int64_t num_elems,
                                       int n_states, int is_complex, const double *d_nodes,
                                       const int32_t *d_elems, const int32_t *d_dofmap,
                                       const double *d_psi, const double *h_w,
                                       const int32_t *d_nadjptr, const int32_t *d_nadj,
                                       double *d_dLdV, double *d_dLdc, double *d_work,
                                       void *stream) {
  if (order < 1 || order > 3 || num_nodes <= 0 || num_elems <= 0) return QD_ERR_INVALID;
  if (n_states < 1 || n_states > kMaxStates) return QD_ERR_LIMIT;
  if (!h_w) return QD_ERR_INVALID;
  Weights w{};
  for (int i = 0; i < (is_complex ? 2 : 1) * n_states; ++i) w.v[i] = h_w[i];
  return adjoint_any(order, num_nodes, num_elems, n_states, is_complex, d_nodes, d_elems, d_dofmap,
                     d_psi, w, d_nadjptr, d_nadj, d_dLdV, d_dLdc, d_work, stream);
}
