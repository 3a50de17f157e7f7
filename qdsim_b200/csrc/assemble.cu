// Finite-element assembly into a precomputed CSR pattern.
//
// Replaces FEMSolver::assemble_element_matrix (backend/src/fem.cpp:736-990),
// the per-element / batched GPU element kernels (backend/src/gpu_kernels.cu:
// 46-336, 442-745) and the host triplet scatter of
// GPUAccelerator::assemble_matrices (backend/src/gpu_accelerator.cpp:439-642).
//
// A block takes a range of CSR rows: a thread per incident (element, local
// node) pair computes that row of the element matrices into shared memory,
// then a thread per CSR slot sums the slot's contributions in the fixed
// (element id, local column) order given by the host plan.  No atomics, so the
// result is bitwise reproducible; every slot is written exactly once and the
// block's slots are contiguous, so stores are coalesced.
//
// Element formulas (per element, A = area, Ginv = J^-1 J^-T):
//   FEM:        H_ab = c A (g00 Sxx + g01 Sxy + g11 Syy)_ab + A sum_l V_l T_lab
//               M_ab = A Mr_ab,  Himag_ab = -A sum_l W_l T_lab
//   REF_CYTHON: schrodinger_solver.pyx:201-251 -- correct P1 stiffness, element
//               V lumped as V A/3 on the diagonal, added a second time at local
//               nodes 1 and 2 (:224-236); consistent mass.
//   REF_FIXED:  fixed_open_system_solver.pyx:225-255 -- c A/3 on the diagonal and
//               c A/6 off it (no gradients), V A/3 on the diagonal; consistent mass.
//   REF_CPP:    SchrodingerSolver::assemble_matrices_cpu (backend/src/schrodinger.cpp:
//               92-230) -- correct P1 stiffness; the potential and the mass by the
//               one-point centroid rule, every entry V A/9 and A/9.
#include <cuda_runtime.h>
#include <algorithm>
#include <atomic>
#include "common.h"
#include "devtables.cuh"

namespace qd {
std::atomic<uint64_t> g_launches{0};
}

namespace {

// Most and least rows per block, threads per block and element-matrix entries staged
// at once, by nodes per element.  A structured P1 / P2 / P3 mesh has at most 18 / 24 / 33
// entries per row on average over a lattice line, so one pass of a block takes
// all of its rows; rows of higher valence (refined meshes, up to 16 elements)
// take more passes.
template <int K> struct AsmShape;
template <> struct AsmShape<3> { static constexpr int ROWS = 128, LEAST = 16, THREADS = 256, CAP = 2304; };
template <> struct AsmShape<6> { static constexpr int ROWS = 96, LEAST = 16, THREADS = 256, CAP = 2304; };
template <> struct AsmShape<10> { static constexpr int ROWS = 64, LEAST = 8, THREADS = 128, CAP = 2240; };

// Shared memory of a block, bytes.  Tables: M, Sxx, Sxy, Syy as [a][b] and the
// potential weights as [a][b][l], rows padded so that lanes with different a
// hit different banks; a pair's entries are an odd number of 16-byte words
// apart, for the same reason.
template <int K, bool HAS_W>
struct AsmLayout {
  using SH = AsmShape<K>;
  static constexpr int CAP = SH::CAP, CE = CAP / K;          // entries, pairs
  static constexpr int KP = K % 2 ? K : K + 1;               // pitch of a pair's entries
  static constexpr int TP = K * K + (K % 2 ? 0 : 2), NT = 4 * K * K;
  static constexpr int HEAVY = 2 * SH::ROWS, BYTES = CAP + 16;
  static constexpr size_t hm = 0, w = hm + size_t(CE) * KP * 16,
                          tab = w + (HAS_W ? size_t(CE) * KP * 8 : 0),
                          slot = tab + size_t(NT + K * TP + 1) / 2 * 16, pair = slot + (CAP + 8) * 4,
                          con = pair + CE * 4, cnt = con + BYTES, heavy = cnt + BYTES,
                          bytes = heavy + HEAVY * 2;
};

__device__ __forceinline__ void cp_async4(void *dst, const void *src) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
}

// Asynchronous copy of bytes [0, count) of src to shared memory such that byte
// i lands at dst + (src & 3) + i (dst 4-byte aligned): whole words where they
// lie inside the range, single bytes at its ends.
__device__ __forceinline__ void stage_bytes(uint8_t *dst, const uint8_t *src, int count, int tid,
                                            int nt) {
  const int off = int(reinterpret_cast<uintptr_t>(src) & 3);
  const uint8_t *base = src - off;                 // word aligned
  const int words = (off + count + 3) / 4;
  for (int i = tid; i < words; i += nt) {
    const int lo = i * 4, hi = lo + 4;
    if (lo >= off && hi <= off + count) {
      cp_async4(dst + lo, base + lo);
    } else {
      for (int k = max(lo, off); k < min(hi, off + count); ++k) dst[k] = base[k];
    }
  }
}

// One block takes ROWS consecutive rows, whose incident (element, local node a)
// pairs, slots and contributions are each one contiguous range of the plan,
// copied to shared memory at once.
//  (1) A thread per pair: the element's nodes, coefficient and nodal V in
//      registers, then the K entries of row a of its H and M (and W term) to
//      shared memory.
//  (2) A thread per row writes where each of its slots' contributions begin,
//      four counts at a time.
//  (3) A thread per slot sums its contributions in the plan's order and writes
//      H and M, contiguous across the block.  Two nodes share at most two
//      elements, so only the diagonal slots have more than two contributions:
//      those are listed in (2) and summed last, and no warp waits on them.
// Instruction issue and the L1 pipe (gathers, staged entries) bound it.
// Before, one row was staged per 8 to 32 lanes, most of which waited on the
// chain adjacency -> element -> nodes of a few pairs: 64 P2 dots (2.4M rows)
// took 1351 us and the P2 400 x 200-cell mesh with W 361 us; now 488 and 142 us.
// Sorting the pairs by a (tables as constant operands) and prefetching the next
// chunk's plan cost as many instructions as they saved (550 us); a thread per
// row, its slots in shared memory, leaves ten warps on an SM (729 us).
// HAS_W: a CAP amplitude is given (Himag is assembled); without it the W terms
// are compiled out.  FEM: the weak form with nodal V; without it the
// reference-compatible P1 modes.
template <int K, bool HAS_W, bool FEM>
__global__ void __launch_bounds__(AsmShape<K>::THREADS)
assemble_rows_kernel(int mode, int32_t n, int rows, int pairs8, const double2 *__restrict__ nodes,
                     const int32_t *__restrict__ elems, const double *__restrict__ cvec,
                     const double *__restrict__ V, const double *__restrict__ W,
                     const int32_t *__restrict__ rowptr, const int32_t *__restrict__ adjptr,
                     const int32_t *__restrict__ adj, const int32_t *__restrict__ cptr,
                     const uint8_t *__restrict__ contrib, const uint8_t *__restrict__ slotcnt,
                     double *__restrict__ H, double *__restrict__ M, double *__restrict__ Him,
                     int32_t *__restrict__ status, const double *__restrict__ tables) {
  using LY = AsmLayout<K, HAS_W>;
  constexpr int ROWS = AsmShape<K>::ROWS, TH = AsmShape<K>::THREADS, CAP = LY::CAP, KP = LY::KP;
  constexpr int KK = K * K, B0 = TabBase<K>::v;
  extern __shared__ __align__(16) unsigned char asm_sm[];
  double2 *s_hm = reinterpret_cast<double2 *>(asm_sm + LY::hm);      // [pair][KP] (H, M)
  double *s_w = reinterpret_cast<double *>(asm_sm + LY::w);
  double *s_tab = reinterpret_cast<double *>(asm_sm + LY::tab);
  uint32_t *s_slot = reinterpret_cast<uint32_t *>(asm_sm + LY::slot);
  int32_t *s_pair = reinterpret_cast<int32_t *>(asm_sm + LY::pair);
  uint16_t *s_heavy = reinterpret_cast<uint16_t *>(asm_sm + LY::heavy);
  __shared__ int32_t s_adj[ROWS + 1], s_rp[ROWS + 1], s_cp[ROWS + 1];
  __shared__ int s_nheavy;
  const int tid = threadIdx.x;
  for (int i = tid; i < 4 * KK + K * KK; i += TH) {
    if (i < 4 * KK) {
      s_tab[i] = tables[B0 + i];
    } else {
      const int l = (i - 4 * KK) / KK, ab = (i - 4 * KK) % KK;
      s_tab[LY::NT + ab / K * LY::TP + ab % K * K + l] = tables[B0 + i];
    }
  }
  const int64_t step = int64_t(gridDim.x) * rows;
  for (int64_t r0 = int64_t(blockIdx.x) * rows; r0 < n; r0 += step) {
    const int nrows = int(min(int64_t(rows), n - r0));
    for (int i = tid; i <= nrows; i += TH) {
      s_adj[i] = adjptr[r0 + i];
      s_rp[i] = rowptr[r0 + i];
      s_cp[i] = cptr[r0 + i];
    }
    __syncthreads();
    int ra = 0;
    while (ra < nrows) {
      // rows [ra, rb): the most whose pairs fit (a row has at most 16 of them,
      // 16 K <= CAP, and no more contributions than K per pair); the same search
      // in every thread
      const int a0 = s_adj[ra];
      int rb = nrows;
      if ((s_adj[nrows] - a0) * K > CAP) {
        rb = ra + 1;
        while (rb < nrows && (s_adj[rb + 1] - a0) * K <= CAP) ++rb;
      }
      const int na = s_adj[rb] - a0, rp0 = s_rp[ra], ns = s_rp[rb] - rp0, c0 = s_cp[ra],
                nc = s_cp[rb] - c0;
      stage_bytes(asm_sm + LY::cnt, slotcnt + rp0, ns, tid, TH);
      stage_bytes(asm_sm + LY::con, contrib + c0, nc, tid, TH);
      for (int p = tid; p < na; p += TH) cp_async4(s_pair + p, adj + a0 + p);
      asm volatile("cp.async.commit_group;\n" ::: "memory");
      const uint8_t *con = asm_sm + LY::con + (reinterpret_cast<uintptr_t>(contrib + c0) & 3);
      const uint8_t *sc = asm_sm + LY::cnt + (reinterpret_cast<uintptr_t>(slotcnt + rp0) & 3);
      if (tid == 0) s_nheavy = 0;
      // (1); P3 and few pairs: `parts` threads share a pair's entries
      const int parts = K < 10 || 2 * na > TH ? 1 : (5 * na > TH ? 2 : 5);
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
      if (parts > 1) __syncthreads();   // else a thread reads the pairs that it copied itself
      for (int item = tid; item < na * parts; item += TH) {
        const int p = K < 10 ? item : item / parts, part = K < 10 ? 0 : item - p * parts;
        const int packed = s_pair[p], e = packed >> 4, a = packed & 15;
        int g[K];
        const int32_t *ep = elems + size_t(e) * K;
        if (K % 2 == 0 && pairs8) {   // rows of K ints on 8-byte boundaries
#pragma unroll
          for (int l = 0; l < K / 2; ++l) {
            const int2 q = reinterpret_cast<const int2 *>(ep)[l];
            g[2 * l] = q.x;
            g[2 * l + 1] = q.y;
          }
        } else {
#pragma unroll
          for (int l = 0; l < K; ++l) g[l] = ep[l];
        }
        const double ce = cvec[e];
        const double2 p0 = nodes[g[0]], p1 = nodes[g[1]], p2 = nodes[g[2]];
        double v[K], w[HAS_W ? K : 1];
        bool bad = false;
        if constexpr (FEM) {
#pragma unroll
          for (int l = 0; l < K; ++l) {
            v[l] = V[g[l]];
            if constexpr (HAS_W) w[l] = W[g[l]];
            bad |= !isfinite(v[l]);
          }
        } else {
          v[0] = V[e];
          bad = !isfinite(v[0]);
        }
        const double ja = p1.x - p0.x, jb = p2.x - p0.x, jc = p1.y - p0.y, jd = p2.y - p0.y;
        const double det = ja * jd - jb * jc;
        const double A = 0.5 * fabs(det);
        const double inv2 = 1.0 / (det * det);
        const double g00 = (jd * jd + jb * jb) * inv2;
        const double g01 = -(jd * jc + jb * ja) * inv2;
        const double g11 = (jc * jc + ja * ja) * inv2;
        const double cA = ce * A;
        if (bad) atomicOr(status, 2);
        if (!(det != 0.0) || !isfinite(det) || !isfinite(ce)) atomicOr(status, 1);
        const double *Mr = s_tab + a * K, *T = s_tab + LY::NT + a * LY::TP;
#pragma unroll(K <= 6 ? K : 2)
        for (int b = part; b < K; b += parts) {
          const double st = g00 * Mr[KK + b] + g01 * Mr[2 * KK + b] + g11 * Mr[3 * KK + b];
          double hk, mk = A * Mr[b];
          if constexpr (FEM) {
            double vs = 0.0, ws = 0.0;
            if constexpr (K % 2 == 0) {
              const double2 *t2 = reinterpret_cast<const double2 *>(T + b * K);
#pragma unroll
              for (int l = 0; l < K / 2; ++l) {
                const double2 tl = t2[l];
                vs += v[2 * l] * tl.x;
                vs += v[2 * l + 1] * tl.y;
                if constexpr (HAS_W) {
                  ws += w[2 * l] * tl.x;
                  ws += w[2 * l + 1] * tl.y;
                }
              }
            } else {
#pragma unroll
              for (int l = 0; l < K; ++l) {
                vs += v[l] * T[b * K + l];
                if constexpr (HAS_W) ws += w[l] * T[b * K + l];
              }
            }
            hk = cA * st;
            hk += A * vs;
            if constexpr (HAS_W) s_w[p * KP + b] = A * ws;
          } else if (mode == QD_ASM_REF_CYTHON) {
            hk = cA * st;
            if (a == b) hk += (a == 0 ? 1.0 : 2.0) * (v[0] * A / 3.0);
          } else if (mode == QD_ASM_REF_FIXED) {
            hk = (cA / 3.0) * (a == b ? 1.0 : 0.5);
            if (a == b) hk += v[0] * A / 3.0;
          } else {
            hk = cA * st + v[0] * A / 9.0;
            mk = A / 9.0;
          }
          s_hm[p * KP + b] = make_double2(hk, mk);
        }
      }
      __syncthreads();   // entries and byte lists of every thread
      // (2) slot: first contribution | its row's first pair << 16
      for (int r = ra + tid; r < rb; r += TH) {
        const uint32_t base = uint32_t(s_adj[r] - a0) << 16;
        const int q0 = s_rp[r] - rp0, len = s_rp[r + 1] - s_rp[r];
        const uint8_t *first = sc + q0;
        const int sh = int(reinterpret_cast<uintptr_t>(first) & 3) * 8;
        const uint32_t *wd = reinterpret_cast<const uint32_t *>(first - sh / 8);
        uint32_t lo = wd[0], at = uint32_t(s_cp[r] - c0);
        for (int q = 0; q < len; q += 4) {
          const uint32_t hi = wd[q / 4 + 1], four = __funnelshift_r(lo, hi, sh);
          lo = hi;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            if (q + u < len) {
              const uint32_t c = four >> (8 * u) & 255u;
              s_slot[q0 + q + u] = base | at;
              if (c > 2) {
                const int i = atomicAdd(&s_nheavy, 1);
                if (i < LY::HEAVY) s_heavy[i] = uint16_t(q0 + q + u);
              }
              at += c;
            }
          }
        }
      }
      if (tid == 0) s_slot[ns] = uint32_t(nc);
      __syncthreads();
      // (3)
      const bool listed = s_nheavy <= LY::HEAVY;   // else every slot is summed in turn
      auto place = [&](uint32_t base, int id) { return int(base) * KP + id + (KP == K ? 0 : id / K); };
      for (int q = tid; q < ns; q += TH) {
        const uint32_t sl = s_slot[q], base = sl >> 16;
        const int u = int(sl & 0xffffu), cnt = int(s_slot[q + 1] & 0xffffu) - u;
        if (cnt > 2 && listed) continue;
        double h = 0.0, mm = 0.0, wi = 0.0;
        if (cnt > 0) {
          const int x0 = place(base, con[u]), x1 = cnt > 1 ? place(base, con[u + 1]) : x0;
          const double2 y0 = s_hm[x0], y1 = s_hm[x1];
          h = 0.0 + y0.x;
          mm = 0.0 + y0.y;
          if constexpr (HAS_W) wi = 0.0 - s_w[x0];
          if (cnt > 1) {
            h += y1.x;
            mm += y1.y;
            if constexpr (HAS_W) wi -= s_w[x1];
          }
          for (int x = 2; x < cnt; ++x) {
            const int xx = place(base, con[u + x]);
            h += s_hm[xx].x;
            mm += s_hm[xx].y;
            if constexpr (HAS_W) wi -= s_w[xx];
          }
        }
        H[rp0 + q] = h;
        M[rp0 + q] = mm;
        if (Him) Him[rp0 + q] = wi;
      }
      const int nheavy = listed ? s_nheavy : 0;
      for (int i = tid; i < nheavy; i += TH) {
        const int q = s_heavy[i];
        const uint32_t sl = s_slot[q], base = sl >> 16;
        const int end = int(s_slot[q + 1] & 0xffffu);
        double h = 0.0, mm = 0.0, wi = 0.0;
        for (int u = int(sl & 0xffffu); u < end; ++u) {
          const int x = place(base, con[u]);
          const double2 y = s_hm[x];
          h += y.x;
          mm += y.y;
          if constexpr (HAS_W) wi -= s_w[x];
        }
        H[rp0 + q] = h;
        M[rp0 + q] = mm;
        if (Him) Him[rp0 + q] = wi;
      }
      __syncthreads();
      ra = rb;
    }
  }
}

template <int K, bool HAS_W, bool FEM>
int launch_rows(int mode, int32_t n, const double *nodes, const int32_t *elems, const double *c,
                const double *V, const double *W, const int32_t *rowptr, const int32_t *adjptr,
                const int32_t *adj, const int32_t *cptr, const uint8_t *contrib,
                const uint8_t *slotcnt, double *H, double *M, double *Him, int32_t *status,
                const double *tables, cudaStream_t s) {
  constexpr size_t smem = AsmLayout<K, HAS_W>::bytes;
  QD_CUDA_TRY(cudaFuncSetAttribute(assemble_rows_kernel<K, HAS_W, FEM>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
  // a block builds its tables once: as many blocks as are resident, and on small
  // meshes no more rows per block than it takes to give each of them some (at the
  // most rows per block P1 100 x 50 cells took 8.5 us and P3 16 x 8 cells 16.4, the row
  // per 8 to 32 lanes before 6.8 and 11.3; with fewer rows, and for P3 threads that
  // share a pair, 6.2 and 10.2)
  static std::atomic<int> per_sm{0};
  int res = per_sm.load(std::memory_order_relaxed);
  if (res == 0) {
    QD_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &res, assemble_rows_kernel<K, HAS_W, FEM>, AsmShape<K>::THREADS, smem));
    if (res < 1) return QD_ERR_CUDA;
    per_sm.store(res, std::memory_order_relaxed);
  }
  const int64_t resident = int64_t(res) * 148;
  const int rows = int(std::clamp<int64_t>((n + resident - 1) / resident, AsmShape<K>::LEAST,
                                           AsmShape<K>::ROWS));
  const int64_t chunks = (int64_t(n) + rows - 1) / rows;
  const int blocks = int(std::min<int64_t>(chunks, resident));
  qd::prof_begin(qd::PK_ASSEMBLE, s);
  assemble_rows_kernel<K, HAS_W, FEM><<<blocks, AsmShape<K>::THREADS, smem, s>>>(
      mode, n, rows, reinterpret_cast<uintptr_t>(elems) % 8 == 0, reinterpret_cast<const double2 *>(nodes),
      elems, c, V, W, rowptr, adjptr, adj, cptr, contrib, slotcnt, H, M, Him, status, tables);
  qd::prof_end(qd::PK_ASSEMBLE, s);
  QD_CHECK_LAUNCH();
  return QD_OK;
}

template <int K>
int launch_assemble(int mode, int32_t n, const double *nodes, const int32_t *elems,
                    const double *c, const double *V, const double *W, const int32_t *rowptr,
                    const int32_t *adjptr, const int32_t *adj, const int32_t *cptr,
                    const uint8_t *contrib, const uint8_t *slotcnt, double *H, double *M,
                    double *Him, int32_t *status, const double *tables, cudaStream_t s) {
  if (n == 0) return QD_OK;
  if constexpr (K == 3) {   // the reference-compatible modes are P1
    if (mode != QD_ASM_FEM)
      return launch_rows<K, false, false>(mode, n, nodes, elems, c, V, W, rowptr, adjptr, adj, cptr,
                                          contrib, slotcnt, H, M, Him, status, tables, s);
  }
  if (W)
    return launch_rows<K, true, true>(mode, n, nodes, elems, c, V, W, rowptr, adjptr, adj, cptr,
                                      contrib, slotcnt, H, M, Him, status, tables, s);
  return launch_rows<K, false, true>(mode, n, nodes, elems, c, V, W, rowptr, adjptr, adj, cptr,
                                     contrib, slotcnt, H, M, Him, status, tables, s);
}

}  // namespace

extern "C" int qd_assemble(int order, int mode, int64_t num_nodes, int64_t num_elems,
                           int32_t n_dofs, const double *d_nodes, const int32_t *d_elems,
                           const double *d_c, const double *d_V, const double *d_W,
                           const int32_t *d_rowptr, const int32_t *d_adjptr,
                           const int32_t *d_adj, const int32_t *d_cptr,
                           const uint8_t *d_contrib, const uint8_t *d_slotcnt, double *d_H,
                           double *d_M, double *d_Himag, int32_t *d_status, void *stream) {
  if (order < 1 || order > 3) return QD_ERR_INVALID;
  if (mode != QD_ASM_FEM && mode != QD_ASM_REF_CYTHON && mode != QD_ASM_REF_FIXED &&
      mode != QD_ASM_REF_CPP)
    return QD_ERR_INVALID;
  if (mode != QD_ASM_FEM && order != 1) return QD_ERR_INVALID;
  if (num_nodes <= 0 || num_elems <= 0 || n_dofs < 0) return QD_ERR_INVALID;
  if (!d_nodes || !d_elems || !d_c || !d_V || !d_rowptr || !d_adjptr || !d_adj || !d_cptr ||
      !d_contrib || !d_slotcnt || !d_H || !d_M || !d_status)
    return QD_ERR_INVALID;
  if (reinterpret_cast<uintptr_t>(d_nodes) % 16 != 0) return QD_ERR_INVALID;
  const double *tables = nullptr;
  int st = ensure_tables(&tables);
  if (st != QD_OK) return st;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  switch (order) {
    case 1:
      return launch_assemble<3>(mode, n_dofs, d_nodes, d_elems, d_c, d_V, d_W, d_rowptr,
                                d_adjptr, d_adj, d_cptr, d_contrib, d_slotcnt, d_H, d_M,
                                d_Himag, d_status, tables, s);
    case 2:
      return launch_assemble<6>(mode, n_dofs, d_nodes, d_elems, d_c, d_V, d_W, d_rowptr,
                                d_adjptr, d_adj, d_cptr, d_contrib, d_slotcnt, d_H, d_M,
                                d_Himag, d_status, tables, s);
    default:
      return launch_assemble<10>(mode, n_dofs, d_nodes, d_elems, d_c, d_V, d_W, d_rowptr,
                                 d_adjptr, d_adj, d_cptr, d_contrib, d_slotcnt, d_H, d_M,
                                 d_Himag, d_status, tables, s);
  }
}

extern "C" const char *qd_version(void) { return "qdsim_b200 0.1.0 (sm_100a)"; }

extern "C" uint64_t qd_kernel_launch_count(void) {
  return qd::g_launches.load(std::memory_order_relaxed);
}

extern "C" const char *qd_status_string(int status) {
  switch (status) {
    case QD_OK: return "ok";
    case QD_ERR_INVALID: return "invalid argument";
    case QD_ERR_CUDA: return "CUDA runtime error";
    case QD_ERR_NOT_CONVERGED: return "not converged";
    case QD_ERR_BREAKDOWN: return "breakdown (Gram matrix not positive definite)";
    case QD_ERR_WORKSPACE: return "workspace too small";
    case QD_ERR_DEGENERATE: return "degenerate element or non-finite coefficient";
    case QD_ERR_LIMIT: return "size exceeds a compiled-in limit";
    case QD_ERR_TIMEOUT: return "device-side wait exceeded its time bound";
    default: return "unknown status";
  }
}
